"""Contexts of several meshes side by side: each one's near field walks its own
mesh's neighbouring blocks, whatever contexts were created after it (the batch
form steps boxes of meshes 32 to 256 together)."""
import numpy as np
import pytest

from ct2_b200 import ics
from ct2_b200.gravity import Gravity

pytestmark = pytest.mark.gpu


def _forces(g, P):
    g.upload_dict(P)
    g.particle_to_grid()
    g.compute_forces()
    return g.forces()[0]


@pytest.mark.parametrize("other", [8, 16, 64])
def test_a_later_context_leaves_the_neighbour_walk_alone(gpu, other):
    n = 20000
    P = ics.plummer_spheres(n, seed=5, nspheres=6, a=0.02)
    kw = dict(mesh=32, order=2, bwidth=3.0, hsoft=1e-3, GM=1.0 / n)
    g = Gravity(**kw)
    alone = _forces(g, P)
    with Gravity(**{**kw, "mesh": other}) as h:
        _forces(h, P)
        beside = _forces(g, P)
    g.close()
    assert np.array_equal(alone, beside)
