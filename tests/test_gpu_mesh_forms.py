"""The fused x pass + Green's multiply at the meshes and orders where its
contraction is split over thread groups, against the three-kernel form; and the
P2M of a crowded cell inside the z pass, against the moment grid."""
import numpy as np
import pytest

from ct2_b200 import ics
from ct2_b200.gravity import Gravity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh,p,x_tma", [(8, 1, 2), (16, 2, 2), (16, 3, 0), (32, 5, 2), (64, 3, 1),
                                          (64, 5, 2), (64, 6, 2), (128, 2, 2), (128, 4, 0)])
def test_split_contraction_matches_the_three_kernels(gpu, mesh, p, x_tma):
    n = 5000
    P = ics.plummer_spheres(n, seed=mesh + p, nspheres=3, a=0.05)
    g = Gravity(mesh=mesh, order=p, bwidth=1.0, hsoft=1.0 / (25 * mesh), GM=1.0 / n)
    L = {}
    for split in (0, 1):
        g.set_tuning(**{**g.tuning(), "split_mg2l": split, "x_tma": x_tma})
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


@pytest.mark.parametrize("n", [255, 256, 257, 3001])
def test_crowded_cell_moments(gpu, n):
    """n particles of one cell (summed by a warp up to 256, by the block beyond)
    beside 50 spread ones: the moments formed inside the z pass give the forces of
    the moment grid's (both FP64 sums stored FP32: one FP32 rounding apart)."""
    mesh, p = 16, 4
    rng = np.random.default_rng(n)
    pos = np.concatenate([5.5 / mesh + rng.uniform(-0.4, 0.4, (n, 3)) / mesh,
                          rng.uniform(0, 1, (50, 3))])
    P = ics._pack(pos, len(pos))
    f = []
    for grid in (True, False):
        g = Gravity(mesh=mesh, order=p, bwidth=1.0, hsoft=1e-3, GM=1.0 / n)
        g.upload_dict(P)
        g.particle_to_grid()
        if grid:
            g.compute_multipoles()
        g.compute_forces()
        f.append(g.forces()[0])
        g.close()
    scale = np.sqrt(np.mean(np.sum(f[0] ** 2, 1)))
    assert np.abs(f[0] - f[1]).max() <= 1e-5 * scale


@pytest.mark.parametrize("mesh,p", [(8, 1), (8, 6), (16, 2), (16, 5), (32, 3), (32, 6), (64, 1), (64, 4),
                                    (64, 5), (64, 6), (128, 2), (128, 4), (128, 5), (128, 6)])
def test_line_moments(gpu, mesh, p):
    """Cells of 1 .. 6 particles (a thread each, the components dealt to the line's
    thread groups), 7 .. 40 (a warp) and 300 (the block) along two lines, against the
    moment grid's: as above, one FP32 rounding of the moments apart."""
    rng = np.random.default_rng(mesh + p)
    pos = []
    for z, n in zip((0, 1, 3, 4, mesh // 2, mesh - 2, mesh - 1), (1, 6, 7, 40, 300, 2, 33)):
        for line in ((2, 3), (mesh - 1, 0)):
            c = (np.array([line[0], line[1], z]) + 0.5) / mesh
            pos.append(c + rng.uniform(-0.45, 0.45, (n, 3)) / mesh)
    pos = np.concatenate(pos)
    P = ics._pack(pos, len(pos))
    f = []
    for grid in (True, False):
        g = Gravity(mesh=mesh, order=p, bwidth=1.0, hsoft=0.5 / mesh, GM=1.0 / len(pos))
        g.upload_dict(P)
        g.particle_to_grid()
        if grid:
            g.compute_multipoles()
        g.compute_forces()
        f.append(g.forces()[0])
        g.close()
    scale = np.sqrt(np.mean(np.sum(f[0] ** 2, 1)))
    assert np.abs(f[0] - f[1]).max() <= 1e-5 * scale
