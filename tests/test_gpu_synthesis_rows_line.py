"""The synthesis rows on both sides of the line between the cluster and the serial
form (10.5 row tiles per SM, 1596 on 152): a batch just below it, one just above it
and an image alone give the same bits, for every row length and level count that
the cluster form takes."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('H,W,levels,tile', [(128, 192, 1, 8), (192, 256, 2, 8), (256, 384, 3, 8), (128, 128, 2, 8),
                                             (384, 512, 4, 8), (256, 1024, 4, 8), (256, 2048, 4, 4), (192, 768, 2, 8)])
def test_both_forms_give_the_same_bits(built_lib, cuda, H, W, levels, tile):
    import torch
    import shearcuda_gb300 as sc
    line = 21 * torch.cuda.get_device_properties(0).multi_processor_count // 2 // (H // tile)  # most images below it
    plan = sc.prepare_shearing_filters_cuda([2, 2, 3, 3][:levels], [16] * levels, H, W, batch=line + 1)
    plan.set_scalars([0.1] * plan.nbands)
    g = torch.Generator(device='cuda').manual_seed(H + W)
    xs = [100 + 20 * torch.randn((H, W), device='cuda', generator=g) for _ in range(line + 1)]
    K = [0.0] + [3.0] * levels
    for n in (line, line + 1):
        outs = sc.nsst_denoise_batch(xs[:n], plan, 20.0, K, mode=sc.THRESH_SOFT)
        for i in (0, n // 2, n - 1):
            assert torch.equal(sc.nsst_denoise(xs[i], plan, 20.0, K, mode=sc.THRESH_SOFT), outs[i])
        del outs
