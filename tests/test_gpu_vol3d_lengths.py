"""The volume FFT passes over the grids' transform lengths: bands against the
oracle's convolution, the band sum without a threshold against its input, and
the backward's dot product, for sides that differ per axis (partial line
groups, odd radices, a chunked level)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-5  # the other volume tests' bound on one FP32 transform chain

# (shape, num_dirs, grid, batch): every side's grid and level lengths differ within a case where they can
CASES = [
    ((40, 44, 36), (2, 2), 'fast', 2),          # 48 -> 32
    ((90, 48, 130), (2, 2), 'fast', 1),         # 96, 48, 144 -> 64, 32, 96
    ((120, 131, 195), (2, 2, 4), 'marshal', 1),  # 132, 132, 204 -> 88, 44 and 136, 68
    ((185, 125, 90), (3, 2, 2), 'marshal', 2),  # 192, 132, 96 and an odd number of bands
    ((70, 80, 96), (8, 4, 4), 'fast', 2),       # more band pairs than one pass over the work buffer takes
]


@pytest.fixture(scope='module')
def s3(built_lib, cuda):
    import shearcuda_gb300 as sc
    return sc


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize('shape,num_dirs,grid,batch', CASES)
def test_bands_band_sum_and_adjoint(s3, shape, num_dirs, grid, batch):
    import torch
    from oracle import nsst3d
    p = s3.VolumePlan(*shape, num_dirs=num_dirs, batch=batch, grid=grid)
    g = torch.Generator(device='cuda').manual_seed(7)
    x = 100 + 30 * torch.randn((batch,) + shape, device='cuda', generator=g)
    flat, subs = s3.do_pyr_dec(x, p)
    assert _rel(s3.do_pyr_rec(flat, p), x) < TOL
    F = nsst3d.band_list(nsst3d.meyer_filters_3d(list(num_dirs)))
    first = 0
    for level, nd in enumerate(num_dirs):
        nb = 3 * nd * nd
        got = s3.sh_dec(flat, level, p)
        for k in sorted({0, nb // 2, nb - 1}):
            ref = nsst3d.convnfft_same_level(subs[level][-1].double().cpu().numpy(), [F[first + k][4]])[0]
            assert _rel(got[-1, k], torch.tensor(ref, device='cuda')) < TOL, (level, k)
        first += nb
        del got
    # T = 0 keeps every coefficient, and the filters sum to the identity
    rec = p.split(s3.sh_dec_th_rec_cuda(flat, p, 30.0, [0] * len(num_dirs), scalars=np.ones(p.nbands)))
    for level in range(len(num_dirs) + 1):
        assert _rel(rec[level], subs[level]) < TOL, level
    # the thresholded denoise is linear at fixed masks: <gy, J x> = <J^T gy, x>
    p.set_scalars(np.full(p.nbands, 0.3))
    p.enable_grad()
    out = s3.denoise3(x, p, 30.0, [3.0] * len(num_dirs))
    gy = out + 10 * torch.randn(out.shape, device='cuda', generator=g)
    gx = s3.denoise3_backward(gy, p)
    lhs, rhs = float((gy.double() * out.double()).sum()), float((gx.double() * x.double()).sum())
    assert abs(lhs - rhs) <= 1e-6 * float(gy.double().norm() * out.double().norm())
