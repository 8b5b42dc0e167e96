"""The near field's potentials where its kernels change form, and its capped grids (tuning
near_chunks_per_warp, beside the mesh solve), whose blocks leave after a few chunks each and
must still cover every chunk."""
import numpy as np
import pytest

from ct2_b200 import ics
from ct2_b200.gravity import Gravity
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# few chunks (several warps each), heavy sparse chunks, dense cells of one and two sinks a
# lane, the sphere kernel inside and outside its radius
@pytest.mark.parametrize("n,mbits,bw,kernel,nsph,a,dense_cell", [
    (33, 3, 3.0, 1, 1, 0.05, 16),
    (6000, 3, 3.0, 0, 1, 0.03, 16),
    (20011, 5, 4.0, 0, 40, 0.02, 16),
    (20011, 5, 3.0, 1, 1, 0.02, 40),
    (12000, 4, 2.0, 1, 3, 0.03, 4096),
    (12000, 4, 2.0, 0, 3, 0.03, 4096),
])
def test_potentials_match_the_method(gpu, n, mbits, bw, kernel, nsph, a, dense_cell):
    M, p = 1 << mbits, 2
    soft, GM = float(np.float32(1.0 / (2 * M))), 1.0 / n
    P = ics.plummer_spheres(n, seed=n % 97, nspheres=nsph, a=a)
    g = Gravity(mesh=M, order=p, bwidth=bw, hsoft=soft, GM=GM, kernel=kernel)
    g.set_tuning(**{**g.tuning(), "dense_cell": dense_cell})
    g.upload_dict(P)
    g.particle_to_grid()
    g.compute_forces()
    _, pot = g.forces()
    ids = g.download()["id"]
    g.close()
    r = O.method_forces(P["x"], P["y"], P["z"], mbits, p, kernel, soft, bw, GM)
    assert np.array_equal(ids, r["perm"])
    # FP32 sums of up to n terms of one sign: sqrt(n) eps = 1e-5 of the sum at most
    rms = np.sqrt(np.mean(r["pot"] ** 2))
    assert np.sqrt(np.mean((pot - r["pot"]) ** 2)) <= 1e-5 * rms


@pytest.mark.parametrize("sparse_path", [1, 2])
@pytest.mark.parametrize("n,mesh,nsph,a,dense_cell", [(700, 16, 2, 0.05, 4096), (700, 16, 2, 0.05, 1),
                                                      (60000, 64, 12, 0.01, 16)])
def test_capped_grids_take_every_chunk(gpu, n, mesh, nsph, a, dense_cell, sparse_path):
    P = ics.plummer_spheres(n, seed=8, nspheres=nsph, a=a)
    g = Gravity(mesh=mesh, order=2, bwidth=3.0, hsoft=1.0 / (50 * mesh), GM=1.0 / n)
    out = []
    for overlap, cap in ((0, 0), (1, 1), (1, 4)):
        g.set_tuning(**{**g.tuning(), "overlap": overlap, "near_chunks_per_warp": cap,
                        "sparse_path": sparse_path, "dense_cell": dense_cell})
        g.upload_dict(P)
        g.particle_to_grid()
        g.compute_forces()
        out.append((*g.forces(), g.interaction_count()))
    g.close()
    assert out[0][2] > 0
    for f, pot, inter in out[1:]:
        assert inter == out[0][2]
        assert np.array_equal(f, out[0][0]) and np.array_equal(pot, out[0][1])
