"""mrdwt takes no scratch from the device, whatever the level count, and allows
its input to overlap the planes that it writes after the first level."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def sc(built_lib, cuda):
    import shearcuda_gb300 as sc
    return sc


def _pool_high(reset):
    """Most bytes in use in the device's stream-ordered pool since the last reset."""
    cu, pool, v = ctypes.CDLL('libcuda.so.1'), ctypes.c_void_p(), ctypes.c_uint64(0)
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    used_high = 8
    if reset:
        assert cu.cuMemPoolSetAttribute(pool, used_high, ctypes.byref(v)) == 0
    assert cu.cuMemPoolGetAttribute(pool, used_high, ctypes.byref(v)) == 0
    return v.value


@pytest.mark.parametrize('L', [1, 2, 3, 4])
@pytest.mark.parametrize('n', [1, 3])
def test_analysis_without_scratch(sc, n, L):
    import torch
    h = sc.MakeONFilter('Symmlet', 4)
    x = torch.randn((n, 64, 96), device='cuda', generator=torch.Generator(device='cuda').manual_seed(L))
    torch.cuda.synchronize()
    before = _pool_high(True)
    yl, yh = sc.mrdwt_cuda(x, h, L)
    torch.cuda.synchronize()
    assert _pool_high(False) == before
    # levels one by one give the same planes
    cur = x
    for l in range(1, L + 1):
        ref = sc.mrdwt_cuda(x, h, l)
        assert torch.equal(ref[1], yh[:, :3 * l])
        cur = ref[0]
    assert torch.equal(cur, yl)


@pytest.mark.parametrize('L', [1, 2, 3, 4])
def test_input_over_the_outputs(sc, L):
    import torch
    H, W = 64, 96
    h = sc.MakeONFilter('Daubechies', 6)
    x0 = torch.randn((H, W), device='cuda', generator=torch.Generator(device='cuda').manual_seed(L))
    yl, yh = sc.mrdwt_cuda(x0, h, L)
    buf = torch.empty((2 * H, W), device='cuda')
    for off in (0, 1, H // 2):  # over the lowpass plane, whole or in part
        x = buf[off:off + H]
        x.copy_(x0)
        a = sc.mrdwt_cuda(x, h, L, yl=buf[:H])
        assert torch.equal(a[0], yl) and torch.equal(a[1], yh)
    if L > 1:  # over the last level's planes, which are written after the input was read
        for k in range(3):
            out = torch.empty_like(yh)
            x = out[3 * (L - 1) + k]
            x.copy_(x0)
            a = sc.mrdwt_cuda(x, h, L, yh=out)
            assert torch.equal(a[0], yl) and torch.equal(a[1], yh)
