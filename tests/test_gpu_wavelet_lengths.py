"""Every filter length up to the longest, tabled or not, odd ones too, against
the oracle: row groups of 8, 4 and 2, a partial group, fewer rows per phase than
the group or the filter has."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
# the other wavelet tests' bound: FP32 FMA chains of at most 2 x 32 taps a level
TOL = 2e-6


def _close(a, b, tol):
    return float(np.abs(a - b).max()) <= tol * float(np.abs(b).max())


@pytest.mark.parametrize('lh', list(range(1, 33)))
@pytest.mark.parametrize('n,H,W,L', [(40, 72, 64, 2), (12, 104, 96, 1), (1, 20, 36, 2)])
def test_length(built_lib, cuda, lh, n, H, W, L):
    import torch
    import shearcuda_gb300 as sc
    from oracle import rwt
    g = np.random.default_rng(100 * lh + n)
    h = g.standard_normal(lh)
    h /= np.abs(h).sum()
    x = g.standard_normal((n, H, W)).astype(np.float32)
    yl, yh = sc.mrdwt_cuda(torch.tensor(x, device='cuda'), h, L)
    rec = sc.mirdwt_cuda(yl, yh, h, L)
    for i in (0, n - 1):
        ol, oh = rwt.mrdwt(x[i].astype(np.float64), h, L)
        assert _close(yl[i].cpu().numpy(), ol, TOL)
        for k in range(3 * L):
            assert _close(yh[i, k].cpu().numpy(), oh[k], TOL), k
        assert _close(rec[i].cpu().numpy(), rwt.mirdwt(ol, oh, h, L), 2 * TOL)
