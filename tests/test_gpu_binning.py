"""Binning at the edges of its sort and cell passes against a stable sort by
Morton key: one item, the edges of a radix tile, the change of tile size (65536
items) and of the passes' form (128 tiles of 4096), digits of 6 to 9 bits, and
tiles of the cell pass with more particles than mark their cells one by one."""
import numpy as np
import pytest

from ct2_b200 import ics
from ct2_b200.gravity import Gravity
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,mbits,nsph,a", [
    (1, 3, 1, 0.1), (1023, 4, 2, 0.1), (1024, 5, 2, 0.1), (1025, 3, 2, 0.1), (65536, 6, 1, 0.01),
    (65537, 6, 1, 0.01), (65537, 7, 20, 0.02), (524288, 6, 100, 0.02), (524289, 5, 100, 0.02),
])
def test_binning_matches_a_stable_sort(gpu, n, mbits, nsph, a):
    P = ics.plummer_spheres(n, seed=n % 89, nspheres=nsph, a=a)
    g = Gravity(mesh=1 << mbits, order=1, bwidth=1.0, hsoft=1e-3, GM=1.0 / n)
    g.upload_dict(P)
    for _ in range(2):  # a second binning keeps the order
        g.particle_to_grid()
        d = g.download()
        b, e = g.cells()
    perm, cs = O.bin_stable(P["x"], P["y"], P["z"], mbits)
    assert np.array_equal(d["id"], perm)
    assert np.array_equal(d["x"], P["x"][perm])
    M = 1 << mbits
    i, j, k = np.meshgrid(*[np.arange(M)] * 3, indexing="ij")
    key = O.morton(i.ravel(), j.ravel(), k.ravel()).astype(np.int64)
    cs = np.asarray(cs)
    assert np.array_equal(b, cs[key]) and np.array_equal(e, cs[key + 1])
    g.close()
