"""The threshold kernel's two forms (16-byte groups, single values) against the
rule itself, exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def sc(built_lib, cuda):
    import shearcuda_gb300 as sc
    return sc


@pytest.mark.parametrize('H,W', [(128, 128), (192, 384), (256, 256)])
@pytest.mark.parametrize('aligned', [True, False])
@pytest.mark.parametrize('soft', [False, True])
def test_threshold_values(sc, H, W, aligned, soft):
    import torch
    plan = sc.prepare_shearing_filters_cuda([2, 3], [16, 16], H, W)
    g = torch.Generator(device='cuda').manual_seed(3)
    buf = 10 * torch.randn(plan.nbands * H * W + 1, device='cuda', generator=g)
    c = (buf[:-1] if aligned else buf[1:]).view(plan.nbands, H, W)
    c[1, 0, :6] = torch.tensor([float('nan'), float('inf'), -float('inf'), 0.0, -0.0, 3.0], device='cuda')
    scal = np.linspace(0.5, 2.0, plan.nbands)
    t = torch.tensor((3.0 * scal).astype(np.float32), device='cuda')[:, None, None]
    if soft:
        m = c.abs() - t
        ref = torch.where(m > 0, torch.copysign(m, c), torch.zeros_like(c))
    else:
        ref = torch.where(c.abs() > t, c, torch.zeros_like(c))
    first, last = buf[0].clone(), buf[-1].clone()
    sc.thresh_cuda(c, 1.0, [3.0] * 3, scal, plan, sc.THRESH_SOFT if soft else sc.THRESH_HARD)
    assert torch.equal(c, ref)
    assert torch.equal(buf[-1] if aligned else buf[0], last if aligned else first)  # nothing beyond the planes
