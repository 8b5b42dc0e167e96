"""Device grids off the boundaries that the kernels' accesses need are refused on the host,
before anything is launched."""
import pytest

from ct2_b200 import ics
from ct2_b200._lib import CT2GError
from ct2_b200.gravity import Gravity

pytestmark = pytest.mark.gpu

CT2G_EINVAL = 1


def test_misaligned_grids_are_refused(gpu):
    import torch
    N = 16
    g = Gravity(mesh=8, order=1, bwidth=1.0, hsoft=1e-3)
    g.upload_dict(ics.plummer_spheres(100, seed=1, nspheres=1, a=0.1))
    real = torch.zeros(N ** 3 + 8, dtype=torch.float32, device="cuda")
    spec = torch.zeros(N * N * (N // 2 + 1) + 8, dtype=torch.complex64, device="cuda")
    grid = torch.zeros(4 * N ** 3 + 8, dtype=torch.complex64, device="cuda")
    assert all(t.data_ptr() % 16 == 0 for t in (real, spec, grid))
    before = g.launch_count()
    for ro, so in ((4, 0), (8, 0), (12, 8), (2, 0), (0, 4), (0, 2), (16, 12)):
        for d in (1, -1):
            with pytest.raises(CT2GError) as e:
                g.fft3d_r2c_dev(real.data_ptr() + ro, spec.data_ptr() + so, N, 1, dir=d)
            assert e.value.status == CT2G_EINVAL, (ro, so, d)
    for o in (1, 2):
        with pytest.raises(CT2GError) as e:
            g.cic_deposit(N, grid.data_ptr() + o)
        assert e.value.status == CT2G_EINVAL, o
    assert g.launch_count() == before
    # and what the checks let through runs
    g.fft3d_r2c_dev(real.data_ptr() + 16, spec.data_ptr() + 8, N, 1)
    g.cic_deposit(N, grid.data_ptr() + 8)
    assert g.synchronize_status() == 0
    g.close()
