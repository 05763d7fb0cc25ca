"""The differentiable path on the TMA level analysis, in the plan's arena and in
the gradient workspace, against the cp.async kernels: fused column pass (256 and
512 rows), the register form with it, and the lengths that keep the plane;
saved and recomputed, in a plan that holds more items than the call has."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('H,W,n,batch', [(256, 128, 2, 2), (256, 256, 1, 3), (512, 256, 2, 3), (384, 512, 2, 2),
                                         (768, 384, 1, 2), (192, 256, 3, 4), (1024, 256, 1, 1)])
def test_gradients_agree(built_lib, cuda, H, W, n, batch):
    import torch
    import shearcuda_gb300 as sc
    got = []
    for route in ('split/level/rows8/synthesis', 'split/level-tma/rows8/synthesis-regs'):
        plan = sc.prepare_shearing_filters_cuda([2, 3], [16, 16], H, W, batch=batch)
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
