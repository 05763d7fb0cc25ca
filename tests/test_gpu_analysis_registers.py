"""The level analysis with the spectrum's columns in registers against the
cp.async kernels, at every column length that takes it and at the narrowest and
a wide row; one image alone and as part of a batch gives the same bits."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('H,W,n', [(256, 128, 3), (256, 512, 2), (512, 128, 3), (512, 768, 2), (1024, 128, 2),
                                   (1024, 1024, 1), (2048, 128, 2), (2048, 512, 1)])
def test_analysis_registers(built_lib, cuda, H, W, n):
    import torch
    import shearcuda_gb300 as sc
    plan = sc.prepare_shearing_filters_cuda([2, 3], [16, 16], H, W, batch=n)
    plan.set_scalars([0.1] * plan.nbands)
    names = plan.directional_candidates()
    g = torch.Generator(device='cuda').manual_seed(H + W + n)
    xs = [100 + 20 * torch.randn((H, W), device='cuda', generator=g) for _ in range(n)]
    K = [0.5, 3.0, 4.0]
    got = {}
    for name in ('split/level/rows8/synthesis', 'split/level-tma/rows8/synthesis-regs'):
        plan.select_directional(n, names.index(name))
        got[name] = sc.nsst_denoise_batch(xs, plan, 20.0, K, mode=sc.THRESH_SOFT)
        plan.check_device()
    # soft thresholds do not amplify a rounding: the two agree to a few float roundings of the image
    for a, b in zip(*got.values()):
        assert float((a.double() - b.double()).norm()) <= 1e-6 * float(b.double().norm())
    plan.select_directional(n, -1)
    outs = sc.nsst_denoise_batch(xs, plan, 20.0, K, mode=sc.THRESH_SOFT)
    assert torch.equal(sc.nsst_denoise(xs[-1], plan, 20.0, K, mode=sc.THRESH_SOFT), outs[-1])
