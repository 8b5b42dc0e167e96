"""Stencil radii whose FP32 square rounds up to a whole number: the cells at that distance
belong to the mesh, for the sinks of every path of the near field."""
import numpy as np
import pytest

from ct2_b200 import ics
from ct2_b200.gravity import Gravity
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rms(f, ref):
    return np.sqrt(np.mean(np.sum((f - ref) ** 2, 1)) / np.mean(np.sum(ref ** 2, 1)))


@pytest.mark.parametrize("d2", [3, 12])
@pytest.mark.parametrize("dense_cell", [1, 48])
def test_radius_just_below_a_cell_distance(gpu, d2, dense_cell):
    bw = np.float32(np.sqrt(float(d2)))
    assert float(bw) ** 2 < d2 <= float(bw * bw)
    n, mbits, p, kernel = 6000, 5, 3, 0
    M, GM = 1 << mbits, 1.0 / n
    soft = float(np.float32(0.02 / M))
    P = ics.plummer_spheres(n, seed=d2, nspheres=6, a=2.0 / M)
    g = Gravity(mesh=M, order=p, bwidth=float(bw), hsoft=soft, GM=GM, kernel=kernel)
    r = O.method_forces(P["x"], P["y"], P["z"], mbits, p, kernel, soft, float(bw), GM)
    ref = r["ffar"] + r["fnear"]
    for path in (0, 1, 2):
        g.set_tuning(**{**g.tuning(), "dense_cell": dense_cell, "sparse_path": path})
        g.upload_dict(P)
        g.particle_to_grid()
        g.compute_forces()
        # FP32 sums against FP64, as in the plain parity tests; a shell of cells summed
        # twice is a percent
        assert _rms(g.forces()[0], ref) < 1e-5, path
    g.close()


def test_widening_to_such_a_radius(gpu):
    bw, bwx = np.float32(np.sqrt(3.0)), np.float32(np.sqrt(12.0))
    n, mbits, p = 6000, 5, 3
    M, GM = 1 << mbits, 1.0 / n
    soft = float(np.float32(0.02 / M))
    P = ics.plummer_spheres(n, seed=5, nspheres=6, a=2.0 / M)
    g = Gravity(mesh=M, order=p, bwidth=float(bw), hsoft=soft, GM=GM)
    r = O.method_forces(P["x"], P["y"], P["z"], mbits, p, 0, soft, float(bwx), GM)
    g.upload_dict(P)
    g.learned_enable(float(bwx))
    g.learned_select("all")
    g.particle_to_grid()
    g.compute_forces()
    # every cell widened: the method at the wider radius
    assert _rms(g.forces()[0], r["ffar"] + r["fnear"]) < 1e-5
    g.close()
