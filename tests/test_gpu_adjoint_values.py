"""The operator adjoints where a transform of the whole image would show: their
precision, pixels that are not finite, and outputs over the inputs."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
# the convolutions' and the directional transforms' own rounding: at most 3.1e-7 over sizes of 192 x 256 to
# 1024 x 1024, all filter sets and two to four levels
TOL = 3.4e-7


@pytest.fixture(scope='module')
def sc(built_lib, cuda):
    import shearcuda_gb300 as sc
    return sc


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize('lpfilt', ['maxflat', '9-7', 'pyr', 'pyrexc'])
def test_precision(sc, lpfilt):
    import torch
    from oracle import nsst2d
    H, W, dcomp, dsize = 192, 256, [2, 3], [16, 16]
    plan = sc.prepare_shearing_filters_cuda(dcomp, dsize, H, W, lpfilt)
    S = nsst2d.shear_spectra(H, W, dcomp, dsize)
    g = np.random.default_rng(3)
    c = g.standard_normal((plan.nbands, H, W)).astype(np.float32)
    x = g.standard_normal((H, W)).astype(np.float32)
    bands = np.split(c[1:].astype(np.float64), [len(S[0])])
    y = [c[0].astype(np.float64)] + [np.real(np.fft.ifft2((np.conj(s) * np.fft.fft2(b)).sum(0))) for s, b in zip(S, bands)]
    got = sc.shear_trans_adjoint(torch.tensor(c, device='cuda'), plan).cpu().numpy()
    assert _rel(got, nsst2d.atrousdec_adjoint(y, lpfilt)) <= TOL
    y = nsst2d.atrousrec_adjoint(x.astype(np.float64), len(dcomp), lpfilt)
    ref = np.concatenate([y[0][None]] + [np.real(np.fft.ifft2(s * np.fft.fft2(b))) for s, b in zip(S, y[1:])])
    got = sc.inverse_shear_adjoint(torch.tensor(x, device='cuda'), plan).cpu().numpy()
    assert _rel(got, ref) <= TOL


@pytest.mark.parametrize('lpfilt,levels', [('maxflat', 1), ('maxflat', 3), ('9-7', 2), ('pyrexc', 4)])
@pytest.mark.parametrize('value', [float('nan'), float('inf')])
def test_a_value_that_is_not_finite_stays_local_in_the_lowpass(sc, lpfilt, levels, value):
    import torch
    H, W, r, q = 384, 512, 200, 131
    plan = sc.prepare_shearing_filters_cuda([2, 3, 3, 3][:levels], [16] * levels, H, W, lpfilt)
    g = torch.Generator(device='cuda').manual_seed(levels)
    x = 100 + 20 * torch.randn((H, W), device='cuda', generator=g)
    c = torch.randn((plan.nbands, H, W), device='cuda', generator=g)
    low, a = sc.inverse_shear_adjoint(x, plan)[0], sc.shear_trans_adjoint(c, plan)
    x[r, q] = value
    c[0, r, q] = value
    reach = 9 * ((1 << levels) - 1)  # filters of at most 19 taps, dilated by 2^level
    far = torch.ones((H, W), dtype=torch.bool, device='cuda')
    far[max(r - reach, 0):r + reach + 1, max(q - reach, 0):q + reach + 1] = False
    assert torch.equal(sc.inverse_shear_adjoint(x, plan)[0][far], low[far])
    assert torch.equal(sc.shear_trans_adjoint(c, plan)[far], a[far])


@pytest.mark.parametrize('levels', [1, 2, 4])
@pytest.mark.parametrize('plane', [0, 1])
def test_the_output_over_the_input(sc, levels, plane):
    import torch
    from shearcuda_gb300._lib import lib
    H, W = 256, 384
    plan = sc.prepare_shearing_filters_cuda([2, 3, 3, 3][:levels], [16] * levels, H, W, '9-7')
    g = torch.Generator(device='cuda').manual_seed(levels)
    c = torch.randn((plan.nbands, H, W), device='cuda', generator=g)
    x = torch.randn((H, W), device='cuda', generator=g)
    a, b = sc.shear_trans_adjoint(c, plan), sc.inverse_shear_adjoint(x, plan)
    buf = c.clone()
    image, stream = ctypes.c_void_p(buf[plane].data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib().nsst_shear_trans_adjoint(plan.handle, ctypes.c_void_p(buf.data_ptr()), image, stream) == 0
    assert torch.equal(buf[plane], a)
    buf[plane].copy_(x)
    assert lib().nsst_inverse_shear_adjoint(plan.handle, image, ctypes.c_void_p(buf.data_ptr()), stream) == 0
    assert torch.equal(buf, b)
