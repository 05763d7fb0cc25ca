"""Volumes whose padded grid is 216 (a side of 210 to 215): the grid's lengths
216, 144 and 72 with a convolution length above 228, along every axis."""
import pytest

import test_gpu_vol3d_lengths as lengths

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape,num_dirs,batch', [
    ((213, 45, 69), (2,), 1), ((45, 215, 69), (2,), 2), ((69, 45, 214), (2,), 1),   # one level: 216 -> 144
    ((210, 44, 66), (2, 2), 1), ((44, 215, 66), (2, 2), 1), ((66, 44, 211), (3, 2), 2)])  # two: 216 -> 144 -> 72
def test_bands_band_sum_and_adjoint(built_lib, cuda, shape, num_dirs, batch):
    import shearcuda_gb300 as sc
    p = sc.VolumePlan(*shape, num_dirs=num_dirs, batch=batch, grid='marshal')
    assert max(p.grid) == 216
    del p
    lengths.test_bands_band_sum_and_adjoint(sc, shape, num_dirs, 'marshal', batch)
