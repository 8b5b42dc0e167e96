"""A replayed step leaves the context in the state of an eager one: the particles have
moved, so that whatever was binned or computed before it no longer holds."""
import numpy as np
import pytest

from ct2_b200 import ics
from ct2_b200._lib import CT2GError
from ct2_b200.gravity import Batch, Gravity, kick_params

pytestmark = pytest.mark.gpu

CT2G_ESTATE = 4


@pytest.mark.parametrize("how", ["eager", "graph", "batch"])
def test_a_step_invalidates_an_earlier_binning(gpu, how):
    n, kp = 3000, kick_params(t0=1e-3)
    g = Gravity(mesh=32, order=2, bwidth=2.0, hsoft=1e-3, GM=1.0 / n)
    g.upload_dict(ics.plummer_spheres(n, seed=3, nspheres=2, a=0.05))
    b = Batch([g]) if how == "batch" else None

    def step():
        if b is not None:
            b.kick_drift(kp, 1e-3, 1.0)
        else:
            g.kick_drift(kp, 1e-3, 1.0, graph=how == "graph")

    step()
    g.particle_to_grid()
    g.compute_forces()
    step()  # the second one: a replay of the first's recording
    for call in (g.compute_forces, g.compute_multipoles, lambda: g.kick(kp)):
        with pytest.raises(CT2GError) as e:
            call()
        assert e.value.status == CT2G_ESTATE
    g.particle_to_grid()
    g.compute_forces()
    assert np.isfinite(g.forces()[0]).all()
    if b is not None:
        b.close()
    g.close()
