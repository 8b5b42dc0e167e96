"""The FP32 device transforms on grids off the 16-byte boundary (they take the
plain column passes, the aligned ones TMA tiles), the CIC deposit onto such a
grid, and the FP64 host transforms of several grids, against FP64."""
import numpy as np
import pytest

from ct2_b200 import ics
from ct2_b200.gravity import Gravity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,batch,shift", [(16, 3, 0), (64, 2, 0), (64, 2, 1), (128, 1, 1), (256, 1, 0)])
def test_r2c_round_trip_off_alignment(gpu, N, batch, shift):
    import torch
    rng = np.random.default_rng(N + shift)
    x = rng.normal(size=(batch, N, N, N)).astype(np.float32)
    g = Gravity(mesh=8, order=1, bwidth=1.0, hsoft=1e-3)
    real = torch.from_numpy(x).cuda()
    nk = batch * N * N * (N // 2 + 1)
    buf = torch.zeros(nk + 1, dtype=torch.complex64, device="cuda")
    spec = buf[shift:shift + nk]  # shift 1: 8 bytes past the allocation's boundary
    g.fft3d_r2c_dev(real.data_ptr(), spec.data_ptr(), N, batch, dir=1)
    X = spec.cpu().numpy().reshape(batch, N, N, N // 2 + 1)
    ref = np.fft.rfftn(x.astype(np.float64), axes=(1, 2, 3))
    # FP32 transforms of 3 log2 N steps: a few eps of the rms
    assert np.sqrt(np.mean(np.abs(X - ref) ** 2)) <= 1e-6 * np.sqrt(np.mean(np.abs(ref) ** 2))
    back = torch.empty_like(real)
    g.fft3d_r2c_dev(back.data_ptr(), spec.data_ptr(), N, batch, dir=-1)
    b = back.cpu().numpy() / float(N) ** 3
    assert np.sqrt(np.mean((b - x) ** 2)) <= 1e-6
    g.close()


@pytest.mark.parametrize("shift", [0, 1])
def test_cic_deposit_off_alignment(gpu, shift):
    import torch
    N, n = 32, 3000
    P = ics.plummer_spheres(n, seed=4, nspheres=2, a=0.1)
    g = Gravity(mesh=8, order=1, bwidth=1.0, hsoft=1e-3)
    g.upload_dict(P)
    buf = torch.full((4 * N ** 3 + 1,), 7.0, dtype=torch.complex64, device="cuda")
    grid = buf[shift:shift + 4 * N ** 3]
    g.cic_deposit(N, grid.data_ptr())
    got = grid.cpu().numpy().reshape(4, N, N, N)
    g.close()
    ref = np.zeros((4, N ** 3))
    u = [P[k].astype(np.float64) * (N * 2.0 ** -32) - 0.5 for k in ("x", "y", "z")]
    m = [np.floor(v) for v in u]
    for c in range(8):
        b = [(c >> (2 - d)) & 1 for d in range(3)]
        o = [u[d] - m[d] - b[d] for d in range(3)]
        w = (1 - np.abs(o[0])) * (1 - np.abs(o[1])) * (1 - np.abs(o[2]))
        i = [(m[d].astype(np.int64) + b[d]) % N for d in range(3)]
        q = (i[0] * N + i[1]) * N + i[2]
        for k in range(4):
            np.add.at(ref[k], q, w if k == 0 else w * o[k - 1])
    # FP32 sums of up to a few hundred weights of at most 1
    assert np.abs(got.real.reshape(4, -1) - ref).max() <= 1e-5 * ref[0].max()
    assert np.all(got.imag == 0)


@pytest.mark.parametrize("N,batch", [(4, 5), (32, 3)])
def test_fp64_host_transforms_of_a_batch(gpu, N, batch):
    rng = np.random.default_rng(N)
    x = rng.normal(size=(batch, N, N, N))
    g = Gravity(mesh=8, order=1, bwidth=1.0, hsoft=1e-3)
    y = g.fft_r2c_3d(x)
    X = np.fft.rfftn(x, axes=(1, 2, 3)).reshape(batch, -1)
    ref = np.concatenate([X.real, X.imag], 1)
    assert np.abs(y - ref).max() <= 1e-13 * np.abs(ref).max()
    assert np.abs(g.fft_c2r_3d(y, N) / N ** 3 - x).max() <= 1e-13 * np.abs(x).max()
    g.close()
