"""The differentiable path on the TMA column kernels against the cp.async ones:
outputs and gradients, saved and recomputed, over row pitches of 512 bytes to 4 KB."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('H,W,n', [(128, 128, 3), (192, 192, 2), (256, 256, 5), (384, 768, 1), (512, 384, 2),
                                   (768, 1024, 1)])
def test_gradients_agree(built_lib, cuda, H, W, n):
    import torch
    import shearcuda_gb300 as sc
    dcomp, dsize = [2, 3], [16, 16]
    got = []
    for route in ('split/level/rows8/synthesis', None):
        plan = sc.prepare_shearing_filters_cuda(dcomp, dsize, H, W, batch=n)
        if route is not None:
            plan.select_directional(n, plan.directional_candidates().index(route))
        g = torch.Generator(device='cuda').manual_seed(H + W + n)
        x = (100 + 20 * torch.randn((n, H, W), device='cuda', generator=g)).requires_grad_(True)
        net = sc.NsstDenoiser(plan, [0.1] * plan.nbands, 20.0, [0.5, 3.0, 4.0])
        gy = torch.randn((n, H, W), device='cuda', generator=g)
        out = net(x)
        out.backward(gy)
        saved = x.grad.clone(), net.tau.grad.clone()
        x.grad = net.tau.grad = None
        out = net(x)
        with torch.no_grad():
            net(x.detach() * 0.5)  # the plan's saved coefficients are another forward's: the backward recomputes
        out.backward(gy)
        assert torch.equal(x.grad, saved[0]) and torch.equal(net.tau.grad, saved[1])
        got.append((out.detach(),) + saved)
        plan.check_device()
    # the two stagings run the same arithmetic; the fused column passes round alike
    for a, b in zip(*got):
        assert float((a.double() - b.double()).norm()) <= 1e-6 * float(b.double().norm())
