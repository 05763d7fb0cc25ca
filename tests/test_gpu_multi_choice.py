"""The uneven batch after another choice of its plans' directional kernels, between
two calls with the same buffers."""
import pytest

pytestmark = pytest.mark.gpu
K = [0.0, 3.0, 4.0]


def _plans(sc, sizes, batch):
    plans = [sc.prepare_shearing_filters_cuda([2, 3], [16, 16], H, W, batch=batch) for H, W in sizes]
    for p in plans:
        p.set_scalars([0.1] * p.nbands)
    return plans


def test_another_choice_is_not_replayed_away(built_lib, cuda):
    import torch
    import shearcuda_gb300 as sc
    sizes = ((192, 256), (256, 384))
    plans = _plans(sc, sizes, 1)
    multi = sc.MultiBatch(plans)
    g = torch.Generator(device='cuda').manual_seed(3)
    xs = [100 + 20 * torch.randn(s, device='cuda', generator=g) for s in sizes]
    outs = [torch.empty_like(x) for x in xs]
    for _ in range(4):  # direct, captured, replayed
        multi.denoise(xs, [20.0, 20.0], K, mode=sc.THRESH_SOFT, outs=outs)
    c0 = sc.launch_count()
    multi.denoise(xs, [20.0, 20.0], K, mode=sc.THRESH_SOFT, outs=outs)
    assert sc.launch_count() == c0  # a replay
    for name in ('split/level/rows8/synthesis', 'split/level-tma/rows8/synthesis-regs'):
        plans[1].select_directional(1, plans[1].directional_candidates().index(name))
        refs = [sc.nsst_denoise(x, p, 20.0, K, mode=sc.THRESH_SOFT) for x, p in zip(xs, plans)]
        for call in range(3):
            c0 = sc.launch_count()
            multi.denoise(xs, [20.0, 20.0], K, mode=sc.THRESH_SOFT, outs=outs)
            launched = sc.launch_count() - c0
            for o, r in zip(outs, refs):
                assert torch.equal(o, r)
            assert call > 0 or launched > 0  # the old choice's kernels are not replayed
