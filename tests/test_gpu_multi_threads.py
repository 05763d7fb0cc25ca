"""The uneven batch beside other callers of its plans: a second thread on the same
stream, and two batch objects over the same plans in another order."""
import threading

import pytest

pytestmark = pytest.mark.gpu
K = [0.0, 3.0, 4.0]


def _plans(sc, sizes, batch):
    plans = [sc.prepare_shearing_filters_cuda([2, 3], [16, 16], H, W, batch=batch) for H, W in sizes]
    for p in plans:
        p.set_scalars([0.1] * p.nbands)
    return plans


def test_threads_share_the_plans(built_lib, cuda):
    import torch
    import shearcuda_gb300 as sc
    sizes = ((192, 256), (256, 256), (256, 384))
    plans = _plans(sc, sizes, 2)
    g = torch.Generator(device='cuda').manual_seed(3)
    sets = [[100 + 20 * torch.randn(s, device='cuda', generator=g) for s in sizes] for _ in range(2)]
    multis = [sc.MultiBatch(plans), sc.MultiBatch(plans[::-1])]  # the same plans, in another order
    sig = [[5.0, 15.0, 25.0], [40.0, 50.0, 60.0]]
    refs = [[sc.nsst_denoise(x, p, s, K, mode=sc.THRESH_SOFT) for x, p, s in zip(xs, plans, ss)] for xs, ss in zip(sets, sig)]
    single = [sc.nsst_denoise(sets[0][k], p, 80.0, K, mode=sc.THRESH_SOFT) for k, p in enumerate(plans)]
    torch.cuda.synchronize()
    errors = []

    def batch(m, again):
        try:
            xs, ss, rs = sets[m], sig[m], refs[m]
            if m:
                xs, ss, rs = xs[::-1], ss[::-1], rs[::-1]
            bufs = [[torch.empty_like(x) for x in xs] for _ in range(2)]
            for i in range(60):
                outs = bufs[0 if again else i % 2]  # replayed, or launched directly every time
                multis[m].denoise(xs, ss, K, mode=sc.THRESH_SOFT, outs=outs)
                for o, r in zip(outs, rs):
                    assert torch.equal(o, r)
        except Exception as e:  # noqa: BLE001 - reported by the test's own thread
            errors.append(e)

    def alone():
        try:
            for i in range(150):
                k = i % len(plans)
                assert torch.equal(sc.nsst_denoise(sets[0][k], plans[k], 80.0, K, mode=sc.THRESH_SOFT), single[k])
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    for again in (False, True):
        jobs = [threading.Thread(target=batch, args=(0, again)), threading.Thread(target=batch, args=(1, again)),
                threading.Thread(target=alone)]
        for t in jobs:
            t.start()
        for t in jobs:
            t.join(120)
            assert not t.is_alive()
        assert not errors, errors[0]
