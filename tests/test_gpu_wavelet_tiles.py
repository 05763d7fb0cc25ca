"""The one-kernel wavelet levels over filter lengths, widths, level counts and
batch sizes (row groups of 8, 4 and 2, partial groups, taps that wrap more than
once, the untabled length) and with the output over the input."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
# the other wavelet tests' bound: FP32 FMA chains of at most 2 x 32 taps a level
TOL = 2e-6


@pytest.fixture(scope='module')
def sc(built_lib, cuda):
    import shearcuda_gb300 as sc
    return sc


def _maxrel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize('fam,par,n,H,W,L', [
    ('Symmlet', 4, 1, 256, 256, 4), ('Symmlet', 10, 3, 192, 128, 5), ('Daubechies', 4, 40, 64, 96, 3),
    ('Haar', 0, 2, 2, 8, 1), ('Daubechies', 20, 1, 32, 16, 4), ('Vaidyanathan', 0, 2, 48, 64, 2),
    ('Coiflet', 2, 1, 36, 2052, 2), ('Beylkin', 0, 1, 16, 8192, 1), ('Symmlet', 8, 24, 128, 512, 2)])
def test_levels_match_oracle(sc, fam, par, n, H, W, L):
    import torch
    from oracle import rwt
    h = sc.MakeONFilter(fam, par)
    g = np.random.default_rng(H * W + L)
    x = g.standard_normal((n, H, W)).astype(np.float32)
    xt = torch.tensor(x, device='cuda')
    yl, yh = sc.mrdwt_cuda(xt, h, L)
    keep = yh.clone()
    rec = sc.mirdwt_cuda(yl, yh, h, L)
    assert torch.equal(yh, keep)
    for i in (0, n - 1):
        ol, oh = rwt.mrdwt(x[i].astype(np.float64), h, L)
        assert _maxrel(yl[i].cpu().numpy(), ol) <= TOL
        for k in range(3 * L):
            assert np.abs(yh[i, k].cpu().numpy() - oh[k]).max() <= TOL * max(np.abs(ol).max(), np.abs(oh[k]).max()), k
        assert _maxrel(rec[i].cpu().numpy(), rwt.mirdwt(ol, oh, h, L)) <= 2 * TOL
    # x may be yl in both directions
    a = xt.clone()
    yl2, yh2 = sc.mrdwt_cuda(a, h, L, yl=a)
    assert torch.equal(yl2, yl) and torch.equal(yh2, yh)
    b = yl.clone()
    assert torch.equal(sc.mirdwt_cuda(b, yh, h, L, x=b), rec)


@pytest.mark.parametrize('H,W', [(2, 2), (32, 34), (62, 128), (256, 96)])
def test_tv_tiles(sc, H, W):
    import torch
    from oracle import rwt
    x = (40 * np.random.default_rng(H + W).standard_normal((3, H, W))).astype(np.float32)
    y = sc.tv_correction_cuda(torch.tensor(x, device='cuda'), 3.0).cpu().numpy()
    for i in range(3):
        assert _maxrel(y[i], rwt.tv_correction(x[i].astype(np.float64), 3.0)) <= TOL
