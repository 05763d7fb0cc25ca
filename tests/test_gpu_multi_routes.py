"""The uneven batch's three routes (launched directly, captured, replayed) and
calls from two streams give the outputs of the single-image path."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('counts', [(1, 1), (3, 5)])
def test_direct_captured_and_replayed_calls_agree(built_lib, cuda, counts):
    import torch
    import shearcuda_gb300 as sc
    sizes = ((192, 256), (256, 384))
    plans = [sc.prepare_shearing_filters_cuda([2, 3], [16, 16], H, W, batch=n) for (H, W), n in zip(sizes, counts)]
    for p in plans:
        p.set_scalars([0.1] * p.nbands)
    multi = sc.MultiBatch(plans)
    g = torch.Generator(device='cuda').manual_seed(4)
    K = [0.0, 3.0, 4.0]

    def images():
        return [100 + 20 * torch.randn(s, device='cuda', generator=g) for s, n in zip(sizes, counts) for _ in range(n)]
    sets = [images() for _ in range(3)]
    sigmas = [10.0 + i for i in range(len(sets[0]))]
    which = [p for p, n in zip(plans, counts) for _ in range(n)]
    refs = [[sc.nsst_denoise(x, p, s, K, mode=sc.THRESH_SOFT) for x, p, s in zip(xs, which, sigmas)] for xs in sets]
    outs = [[torch.empty_like(x) for x in xs] for xs in sets]
    side = torch.cuda.Stream()
    # 0 1 2: new pointers; 0 0 0: direct, captured, replayed; then alternating streams
    for k, stream in [(0, None), (1, None), (2, None), (0, None), (0, None), (0, None), (1, side), (1, None), (2, side),
                      (2, side), (2, None)]:
        for o in outs[k]:
            o.zero_()
        if stream is not None:
            stream.wait_stream(torch.cuda.current_stream())
        multi.denoise(sets[k], sigmas, K, mode=sc.THRESH_SOFT, outs=outs[k], stream=stream)
        if stream is not None:
            torch.cuda.current_stream().wait_stream(stream)
        for o, r in zip(outs[k], refs[k]):
            assert torch.equal(o, r)
    # a bad item is refused before anything runs, and the next call is sound
    with pytest.raises(sc.NsstError):
        multi.denoise(sets[0], [-1.0] + sigmas[1:], K, outs=outs[0])
    multi.denoise(sets[0], sigmas, K, mode=sc.THRESH_SOFT, outs=outs[0])
    for o, r in zip(outs[0], refs[0]):
        assert torch.equal(o, r)
