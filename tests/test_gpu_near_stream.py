"""The streamed near field against the FP64 restatement of the method, at the
sizes where it changes form: few chunks (shared by several warps), chunks
whose neighbourhood is heavy (shared by a block), partial batches, both
kernels, and the smallest meshes."""
import numpy as np
import pytest

from ct2_b200 import ics
from ct2_b200.gravity import Gravity
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,mbits,bw,kernel,nsph,a", [
    (1, 4, 2.0, 0, 1, 0.02),
    (33, 3, 3.0, 1, 1, 0.05),
    (700, 3, 2.5, 0, 2, 0.05),
    (6000, 3, 3.0, 0, 1, 0.03),
    (1728, 4, 4.0, 1, 3, 0.03),
    (20011, 5, 4.0, 0, 40, 0.02),
    (20011, 5, 3.0, 1, 1, 0.02),
    (30001, 4, 2.0, 0, 1, 0.01),
    (30001, 6, 4.0, 1, 1, 0.01),
])
def test_streamed_near_field_matches_the_method(gpu, n, mbits, bw, kernel, nsph, a):
    M, p = 1 << mbits, 2
    soft, GM = 1.0 / (25 * M), 1.0 / n
    P = ics.plummer_spheres(n, seed=n % 97, nspheres=nsph, a=a)
    g = Gravity(mesh=M, order=p, bwidth=bw, hsoft=soft, GM=GM, kernel=kernel)
    g.upload_dict(P)
    g.particle_to_grid()
    g.compute_forces()
    f, _ = g.forces()
    ids = g.download()["id"]
    g.close()
    r = O.method_forces(P["x"], P["y"], P["z"], mbits, p, kernel, soft, bw, GM)
    ref = r["ffar"] + r["fnear"]
    assert np.array_equal(ids, r["perm"])
    # FP32 sums of up to n terms in windows of a few thousand: sqrt(3e4) eps
    # = 1e-5 of the terms' size at most
    scale = np.sqrt(np.mean(np.sum(ref ** 2, 1)))
    err = np.sqrt(np.mean(np.sum((f - ref) ** 2, 1)))
    assert err <= 1e-5 * max(scale, 1e-30) + 1e-6
