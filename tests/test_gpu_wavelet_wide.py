"""Wavelet levels of long and of few rows, which CTAs share by columns: widths
around the parts' sizes, taps that reach around the row's end and across a whole
part, and the same bits whatever the rows are split into."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
# the other wavelet tests' bound: FP32 FMA chains of at most 2 x 32 taps a level
TOL = 2e-6


def _close(a, b, tol):
    return float(np.abs(a - b).max()) <= tol * float(np.abs(b).max())


@pytest.mark.parametrize('fam,par', [('Haar', 0), ('Symmlet', 4), ('Symmlet', 10), ('Battle', 1), ('Coiflet', 5)])
@pytest.mark.parametrize('H,W,L', [(8, 8192, 1), (32, 8192, 5), (64, 4096, 6), (4, 2052, 2), (16, 2064, 4), (24, 3000, 3),
                                   (6, 262, 1), (8, 512, 3), (16, 1040, 4), (2, 1026, 1), (36, 2048, 2)])
def test_wide_rows(built_lib, cuda, fam, par, H, W, L):
    import torch
    import shearcuda_gb300 as sc
    from oracle import rwt
    h = sc.MakeONFilter(fam, par)
    x = np.random.default_rng(H * W + L).standard_normal((H, W)).astype(np.float32)
    yl, yh = sc.mrdwt_cuda(torch.tensor(x, device='cuda'), h, L)
    rec = sc.mirdwt_cuda(yl, yh, h, L)
    ol, oh = rwt.mrdwt(x.astype(np.float64), h, L)
    top = max(np.abs(ol).max(), np.abs(oh).max())
    assert _close(yl.cpu().numpy(), ol, TOL)
    for k in range(3 * L):
        assert np.abs(yh[k].cpu().numpy() - oh[k]).max() <= TOL * top, k
    assert _close(rec.cpu().numpy(), rwt.mirdwt(ol, oh, h, L), 2 * TOL)


@pytest.mark.parametrize('H,W,n', [(64, 512, 24), (32, 1024, 40), (128, 2048, 12), (16, 4096, 70)])
def test_an_image_of_a_batch_has_the_bits_of_one_alone(built_lib, cuda, H, W, n):
    import torch
    import shearcuda_gb300 as sc
    for h in (sc.MakeONFilter('Symmlet', 6), sc.MakeONFilter('Coiflet', 4)):
        x = torch.randn((n, H, W), device='cuda', generator=torch.Generator(device='cuda').manual_seed(W))
        yl, yh = sc.mrdwt_cuda(x, h, 3)
        rec = sc.mirdwt_cuda(yl, yh, h, 3)
        for i in (0, n - 1):
            a, b = sc.mrdwt_cuda(x[i], h, 3)
            assert torch.equal(a, yl[i]) and torch.equal(b, yh[i])
            assert torch.equal(sc.mirdwt_cuda(a, b, h, 3), rec[i])
