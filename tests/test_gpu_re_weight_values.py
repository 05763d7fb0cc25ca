"""re_weight_band where a transform of the whole image would show: a pixel that
is not finite stays within the filters' support, the output may overlap the
input, and a result much smaller than the image keeps its precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def sc(built_lib, cuda):
    import shearcuda_gb300 as sc
    return sc


@pytest.mark.parametrize('lpfilt,levels', [('maxflat', 1), ('maxflat', 2), ('9-7', 3), ('pyrexc', 2)])
@pytest.mark.parametrize('value', [float('nan'), float('inf')])
def test_a_pixel_that_is_not_finite_stays_local(sc, lpfilt, levels, value):
    import torch
    H, W, r, c = 384, 512, 200, 131
    plan = sc.prepare_shearing_filters_cuda([3, 3, 4], [32, 32, 16], H, W, lpfilt)
    x = 100 + 20 * torch.randn((H, W), device='cuda', generator=torch.Generator(device='cuda').manual_seed(levels))
    w = [0.5, 1.5, 2.0, 0.25][:levels + 1]
    ref = sc.re_weight_band(x, w, plan)
    x[r, c] = value
    y = sc.re_weight_band(x, w, plan)
    # an analysis and a synthesis filter of at most 19 taps per level, dilated by 2^level
    reach = 2 * sum((1 << l) * 9 for l in range(levels))
    far = torch.ones((H, W), dtype=torch.bool, device='cuda')
    far[max(r - reach, 0):r + reach + 1, max(c - reach, 0):c + reach + 1] = False
    assert not torch.isfinite(y[r, c])
    assert torch.equal(y[far], ref[far])


@pytest.mark.parametrize('rows', [0, 8, -8, 300])
def test_the_output_may_overlap_the_image(sc, rows):
    import torch
    H, W = 384, 512
    plan = sc.prepare_shearing_filters_cuda([3, 3], [32, 32], H, W)
    buf = torch.empty((2 * H + 16, W), device='cuda')
    g = torch.Generator(device='cuda').manual_seed(1)
    x0 = 100 + 20 * torch.randn((H, W), device='cuda', generator=g)
    ref = sc.re_weight_band(x0, [0.5, 1.5, 2.0], plan)
    x, out = buf[8:8 + H], buf[8 + rows:8 + rows + H]
    for _ in range(5):
        x.copy_(x0)
        assert torch.equal(sc.re_weight_band(x, [0.5, 1.5, 2.0], plan, out=out), ref)


@pytest.mark.parametrize('w', [[1, 0, 0, 0, 0], [100, 1, 1, 1, 1], [0, 1], [0.1, 0.1, 1.5, 1.5]])
def test_precision_of_small_results(sc, w):
    # 2 x 4 chained FP32 convolutions: a few float roundings of each plane's own size
    import torch
    from oracle import nsst2d
    H, W = 256, 384
    plan = sc.prepare_shearing_filters_cuda([3, 3, 4, 4], [32, 32, 16, 16], H, W)
    x = np.random.default_rng(5).standard_normal((H, W)).astype(np.float32)
    got = sc.re_weight_band(torch.tensor(x, device='cuda'), w, plan).cpu().numpy().astype(np.float64)
    ref = nsst2d.re_weight_band(x.astype(np.float64), w)
    assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref)
