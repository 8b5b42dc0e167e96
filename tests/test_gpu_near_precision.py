"""The precision of the near field's sparse sinks: close pairs inside one cell, a
softening length or so apart, whose separation is exact in FP32 when it is formed
from the particles' offsets from their own cell's centre."""
import numpy as np
import pytest

from ct2_b200 import ics
from ct2_b200.gravity import Gravity
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def close_pairs(pairs, mbits, cells, hsoft, seed):
    """Pairs 0.5 to 2 softening lengths apart, both of a pair in one cell of the
    first `cells` along each axis; coordinates are multiples of 2^-30 (four units of
    the fixed-point store), so that the offsets from the cell centres are FP32 numbers."""
    rng = np.random.default_rng(seed)
    unit, M = 1 << 30, 1 << mbits
    cell = rng.integers(0, cells, (pairs, 3))
    w = unit // M                      # steps a cell
    a = rng.integers(w // 8, w - w // 8, (pairs, 3))
    d = rng.normal(size=(pairs, 3))
    d *= (rng.uniform(0.5, 2.0, pairs) * hsoft * unit / np.linalg.norm(d, axis=1))[:, None]
    b = a + np.rint(d).astype(np.int64)
    assert b.min() >= 0 and b.max() < w
    P = ics._pack(np.zeros((2 * pairs, 3)), 2 * pairs)
    pos = 4 * np.concatenate([cell * w + a, cell * w + b])
    P["x"], P["y"], P["z"] = (np.ascontiguousarray(c, dtype=np.uint32) for c in pos.T)
    return P


# 600 pairs all over the box: a warp per chunk; 700 pairs within 10 cells of a corner: more
# sources in a chunk's neighbourhood than one warp takes
@pytest.mark.parametrize("kernel,pairs,cells", [(1, 600, 32), (1, 700, 10)])
def test_sparse_pairs_keep_their_separation(gpu, kernel, pairs, cells):
    mbits, p, bw = 5, 2, 3.0
    M, n = 1 << mbits, 2 * pairs
    hsoft = float(np.float32(1.0 / (25 * M)))
    P = close_pairs(pairs, mbits, cells, hsoft, seed=pairs)
    g = Gravity(mesh=M, order=p, bwidth=bw, hsoft=hsoft, GM=1.0 / n, kernel=kernel)
    out = {}
    for path in (1, 2):
        g.set_tuning(**{**g.tuning(), "sparse_path": path})
        g.upload_dict(P)
        g.particle_to_grid()
        b, e = g.cells()
        assert (e - b).max() < g.tuning()["dense_cell"]  # every sink is a sparse one
        g.compute_forces()
        out[path] = g.forces()
    ids = g.download()["id"]
    g.close()
    r = O.method_forces(P["x"], P["y"], P["z"], mbits, p, kernel, hsoft, bw, 1.0 / n)
    ref = r["ffar"] + r["fnear"]
    assert np.array_equal(ids, r["perm"])
    scale = np.sqrt(np.mean(np.sum(ref ** 2, 1)))
    # a pair's force dominates (1/hsoft^2 against 1/(a few cells)^2) and its separation is
    # exact: what is left are some six FP32 roundings of r^2, 1/r^3 and the products, the
    # sums, and those of a far field of up to a twentieth of the force: ten roundings at
    # most.  (Separations formed in the frame of a 4-cell block are off by up to 16
    # units of 2^-32 where the pair is 2^27 / 25 apart: 3.5e-6.)
    bound = 10 * 2.0 ** -24
    for path in (1, 2):
        err = np.sqrt(np.mean(np.sum((out[path][0] - ref) ** 2, 1)))
        assert err <= bound * scale, (path, err / scale)
    # the far field is the same in both forms, so the potentials differ by the near field's
    # roundings alone
    p1, p2 = (out[k][1].astype(np.float64) for k in (1, 2))
    assert np.sqrt(np.mean((p1 - p2) ** 2)) <= bound * np.sqrt(np.mean(p1 ** 2))
