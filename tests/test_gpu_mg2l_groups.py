"""The Green's contraction dealt to thread groups (all groups' sums, one barrier, all
groups' stores) at every number of groups and at rows fewer than a warp, the Green's values from
shared memory or straight from the table, against the three-kernel form."""
import numpy as np
import pytest

from ct2_b200 import ics
from ct2_b200.gravity import Gravity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh,p,x_tma,direct", [(8, 6, 2, 0), (16, 4, 2, 1), (32, 6, 2, 1), (64, 5, 0, 1),
                                                 (64, 6, 1, 0), (128, 5, 2, 0), (128, 6, 0, 1),
                                                 (128, 6, 1, 1), (128, 6, 2, 0)])
def test_grouped_contraction_matches_the_three_kernels(gpu, mesh, p, x_tma, direct):
    n = 5000
    P = ics.plummer_spheres(n, seed=mesh + p, nspheres=3, a=0.05)
    g = Gravity(mesh=mesh, order=p, bwidth=1.0, hsoft=1.0 / (25 * mesh), GM=1.0 / n)
    L = {}
    for split in (0, 1):
        g.set_tuning(**{**g.tuning(), "split_mg2l": split, "x_tma": x_tma,
                        "mg2l_greens_direct": direct})
        g.upload_dict(P)
        g.particle_to_grid()
        g.compute_multipoles()
        g.compute_expansions()
        L[split] = g.expansions()
    g.close()
    # the same FP32 transforms and sums in another order: a few rounding
    # steps of the largest value of each component
    for a, b in zip(L[0], L[1]):
        assert np.abs(a - b).max() <= 2e-6 * np.abs(b).max()
