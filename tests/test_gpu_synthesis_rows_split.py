"""The synthesis rows as clusters (few row tiles) give the bits of the serial
form (many): one image alone and as part of a batch whose tiles do not fit the
cluster form's range, for row lengths and level counts around its limits."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('H,W,levels,n', [(128, 192, 1, 80), (192, 256, 2, 64), (256, 384, 3, 40), (256, 128, 2, 64),
                                          (384, 512, 4, 32), (256, 1024, 4, 40), (256, 2048, 4, 20), (384, 256, 5, 32)])
def test_one_image_equals_the_batch(built_lib, cuda, H, W, levels, n):
    import torch
    import shearcuda_gb300 as sc
    dcomp, dsize = [2, 2, 3, 3, 3][:levels], [16] * levels
    # the fifth level's 16-fold dilated 19-tap filter needs 305 rows and columns: the 9-tap set reaches 256
    plan = sc.prepare_shearing_filters_cuda(dcomp, dsize, H, W, lpfilt='9-7' if levels == 5 else 'maxflat', batch=n)
    plan.set_scalars([0.1] * plan.nbands)
    g = torch.Generator(device='cuda').manual_seed(H + W)
    xs = [100 + 20 * torch.randn((H, W), device='cuda', generator=g) for _ in range(n)]
    K = [0.0] + [3.0] * levels
    outs = sc.nsst_denoise_batch(xs, plan, 20.0, K, mode=sc.THRESH_SOFT)
    for i in (0, n // 2, n - 1):
        assert torch.equal(sc.nsst_denoise(xs[i], plan, 20.0, K, mode=sc.THRESH_SOFT), outs[i])
