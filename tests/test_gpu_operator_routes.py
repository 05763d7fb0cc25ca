"""The single-image adjoints on the spectral pyramid against the direct one."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def sc(built_lib, cuda):
    import shearcuda_gb300 as sc
    return sc


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize('H,W,lpfilt,batch', [(192, 256, 'maxflat', 1), (256, 192, '9-7', 1), (384, 512, 'pyr', 3),
                                              (768, 384, 'pyrexc', 1), (1024, 768, 'maxflat', 1)])
def test_adjoints_on_the_spectral_pyramid_match_the_direct_one(sc, H, W, lpfilt, batch):
    # the same operators up to FP32 rounding: 1e-5, the bound between the two pyramids elsewhere
    import torch
    dcomp, dsize = [3, 3, 4, 4], [32, 32, 16, 16]
    plans = [sc.prepare_shearing_filters_cuda(dcomp, dsize, H, W, lpfilt=lpfilt, pyramid=m, batch=batch)
             for m in (sc.PYRAMID_AUTO, sc.PYRAMID_DIRECT)]
    g = torch.Generator(device='cuda').manual_seed(H + W)
    x = 100 + 20 * torch.randn((H, W), device='cuda', generator=g)
    c = torch.randn((plans[0].nbands, H, W), device='cuda', generator=g)
    a, d = (sc.shear_trans_adjoint(c, p) for p in plans)
    assert _rel(a, d) <= 1e-5
    ca, cd = (sc.inverse_shear_adjoint(x, p) for p in plans)
    assert _rel(ca, cd) <= 1e-5
    # an image that is not 16-byte aligned takes the direct pyramid
    buf = torch.empty(H * W + 1, device='cuda')
    xm = buf[1:].view(H, W)
    xm.copy_(x)
    assert torch.equal(sc.inverse_shear_adjoint(xm, plans[0]), cd)
    # <A x, c> = <x, A^T c>
    Ax = sc.shear_trans_cuda(x, lpfilt, plans[0])
    lhs, rhs = float((Ax.double() * c.double()).sum()), float((x.double() * a.double()).sum())
    assert abs(lhs - rhs) <= 1e-6 * float(Ax.double().norm() * c.double().norm())


@pytest.mark.parametrize('H,W,lpfilt', [(192, 256, 'maxflat'), (384, 192, '9-7'), (512, 384, 'pyr'),
                                        (256, 1024, 'pyrexc')])
@pytest.mark.parametrize('levels', [1, 2, 4])
def test_band_weights_on_the_spectral_pyramid_match_the_direct_one(sc, H, W, lpfilt, levels):
    import torch
    plans = [sc.prepare_shearing_filters_cuda([3, 3, 4, 4], [32, 32, 16, 16], H, W, lpfilt=lpfilt, pyramid=m)
             for m in (sc.PYRAMID_AUTO, sc.PYRAMID_DIRECT)]
    g = torch.Generator(device='cuda').manual_seed(H + levels)
    x = 100 + 20 * torch.randn((H, W), device='cuda', generator=g)
    w = [0.1, 1.5, 0.0, 2.0, -1.0][:levels + 1]
    a, d = (sc.re_weight_band(x, w, p) for p in plans)
    assert _rel(a, d) <= 1e-5
    # in place, and from an image that is not 16-byte aligned (the direct pyramid)
    y = x.clone()
    assert torch.equal(sc.re_weight_band(y, w, plans[0], out=y), a)
    buf = torch.empty(H * W + 1, device='cuda')
    xm = buf[1:].view(H, W)
    xm.copy_(x)
    assert torch.equal(sc.re_weight_band(xm, w, plans[0], out=torch.empty_like(x)), d)
