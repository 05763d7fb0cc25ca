"""A volume plan on a device without room for all band pairs in flight: one pair at
a time, in no more memory than plans took when that was the only form (1.232 GB
and 0.045 GB here), and the same bits."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape,num_dirs,batch,most', [((128, 128, 128), (2, 2, 4), 4, 1.232e9), ((48, 48, 48), (2, 2), 4, 0.0455e9)])
def test_one_pair_at_a_time(built_lib, cuda, shape, num_dirs, batch, most):
    import torch
    import shearcuda_gb300 as sc
    from shearcuda_gb300._lib import lib
    g = torch.Generator(device='cuda').manual_seed(1)
    x = 100 + 30 * torch.randn((batch,) + shape, device='cuda', generator=g)
    gy = torch.randn(x.shape, device='cuda', generator=g)
    got, bytes_ = [], []
    for fail in (0, 1):
        lib().nsst_debug_fail_next_alloc(fail)  # the plan's first allocation, as if it did not fit
        try:
            p = sc.VolumePlan(*shape, num_dirs=num_dirs, batch=batch)
        finally:
            lib().nsst_debug_fail_next_alloc(0)
        bytes_.append(p.device_bytes())
        p.set_scalars([0.3] * p.nbands)
        p.enable_grad()
        out = sc.denoise3(x, p, 30.0, [3.0] * len(num_dirs))
        flat, _ = sc.do_pyr_dec(x, p)
        got.append((out, sc.denoise3_backward(gy, p), sc.sh_dec(flat, 0, p)))
        del p
    assert bytes_[1] <= most and bytes_[1] < bytes_[0]
    for a, b in zip(*got):
        assert torch.equal(a, b)
