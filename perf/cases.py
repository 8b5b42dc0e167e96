"""The work this library is measured on.

Every case goes through the public entry points: the host-state step
(particles in host memory in, the stepped particles out), the rung-hierarchical
kick_step, the forces alone, many boxes in one context, the learned
correction, the training gradient, and the 3D FFTs (FP32 on device buffers,
the CIC deposit with its complex batch, the reference's FP64 host interface).
Sizes and options are those of the configurations, the tests and the
benchmark, with ragged particle counts beside the round ones.

Positions come back from the library as 32-bit fixed point; the programs here
take them in box units, as floats in [-1/2, 1/2).
"""
import math

import numpy as np
import torch

from ct2_b200 import _lib, ics
from ct2_b200.gravity import Gravity, kick_params

ETA = 0.15
# a base step below every particle's own acceleration limit: rung 0 throughout
T0 = 2e-5


def listed():
    return [
        # the smallest call: 12^3 lattice particles on a 16^3 mesh, all latency
        dict(name="step_lattice_12", kind="step", ic="lattice", n=12 ** 3, mesh=16, order=3,
             bwidth=2.0, kernel="plummer", nbox=1, graph=True),
        # the reference's step driver at the CPU-parity configuration: upload,
        # kick_step, download
        dict(name="kick_step_lattice_32", kind="kick_step", ic="lattice", n=32 ** 3, mesh=64,
             order=4, bwidth=3.0, kernel="plummer", nbox=1, graph=False),
        # an ordinary small clustered box, a ragged count, plain stream launches
        dict(name="step_spheres_50k", kind="step", ic="spheres", n=50021, mesh=64, order=5,
             bwidth=4.0, kernel="plummer", nbox=1, graph=False),
        # many small independent boxes in one context
        dict(name="step_boxes_12x64", kind="step", ic="spheres", n=12 * 30011, mesh=64, order=5,
             bwidth=4.0, kernel="plummer", nbox=12, graph=True),
        # the headline configuration: 128^3 particles, 256^3 mesh
        dict(name="step_spheres_128", kind="step", ic="spheres", n=128 ** 3, mesh=256, order=4,
             bwidth=4.0, kernel="plummer", nbox=1, graph=True),
        # strongly clustered halos: the near field is most of the step
        dict(name="step_halos_2p5M", kind="step", ic="halos", n=2500009, mesh=256, order=4,
             bwidth=4.0, kernel="plummer", nbox=1, graph=True),
        # forces and potential with the reference's softening kernel
        dict(name="forces_sphere_300k", kind="forces", ic="halos", n=300007, mesh=128, order=4,
             bwidth=3.0, kernel="sphere", nbox=1, graph=False),
        # the learned correction: forces with network-selected cells widened
        dict(name="learned_spheres_64", kind="learned", ic="spheres", n=64 ** 3, mesh=128, order=4,
             bwidth=3.0, kernel="plummer", nbox=1, graph=False),
        # training the network: loss and gradient of one set of samples
        dict(name="mlp_gradients_20k", kind="gradients", n=20011),
        # a particle-mesh solve on device buffers: r2c, k-space kernel, c2r
        dict(name="poisson_256x3", kind="poisson", N=256, batch=3),
        # density and first moments on four 512^3 grids and their spectra
        dict(name="cic_c2c_512", kind="cic", ic="spheres", n=128 ** 3, N=512),
        # the reference's FP64 transforms on host arrays, both directions
        dict(name="fft64_128", kind="fft64", N=128, batch=1),
    ]


def _mesh_for(n, lo=16, hi=256):
    return int(min(max(2 ** round(math.log2(2.0 * n ** (1.0 / 3.0))), lo), hi))


def draw(rng):
    """One more case: sizes spread over their logarithm, odd counts among them."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "boxes", "forces", "kick_step", "learned",
                       "gradients", "poisson", "cic", "fft64"])
    if kind == "gradients":
        return dict(kind=kind, n=size(1000, 80000))
    if kind == "poisson":
        N = rng.choice([32, 64, 128, 256])
        return dict(kind=kind, N=N, batch=rng.randint(1, {256: 3, 128: 9}.get(N, 20)))
    if kind == "fft64":
        N = rng.choice([16, 32, 64, 128])
        return dict(kind=kind, N=N, batch=1 if N == 128 else rng.randint(1, 6))
    if kind == "cic":
        return dict(kind=kind, ic="spheres", n=size(20000, 2000000), N=rng.choice([128, 256, 512]))
    if kind == "boxes":
        nbox, per = rng.randint(2, 12), size(3000, 35000)
        return dict(kind="step", ic="spheres", n=nbox * per, mesh=_mesh_for(per, 32, 64),
                    order=rng.choice([4, 5]), bwidth=4.0, kernel="plummer", nbox=nbox, graph=True)
    ic = rng.choice(["spheres", "spheres", "halos", "lattice"])
    n = size(2000, 400000) if kind in ("forces", "kick_step", "learned") else size(1500, 2000000)
    if kind == "learned":
        ic = "spheres"
    if ic == "lattice":
        n = max(8, round(n ** (1.0 / 3.0))) ** 3
    mesh = _mesh_for(n)
    order = rng.choice([3, 4, 5] if mesh <= 64 else [3, 4])
    bwidth = 3.0 if kind == "learned" else rng.choice([3.0, 4.0])
    if mesh == 16 and (kind == "learned" or bwidth > 3):
        mesh = 32
    kernel = rng.choice(["plummer", "sphere"]) if kind == "forces" else "plummer"
    return dict(kind=kind, ic=ic, n=n, mesh=mesh, order=order, bwidth=bwidth, kernel=kernel, nbox=1,
                graph=kind == "step" and rng.random() < 0.7)


# ---- inputs -------------------------------------------------------------------

def _box(ic, n, seed):
    if ic == "lattice":
        return ics.lattice(round(n ** (1.0 / 3.0)), seed=seed)
    if ic == "halos":
        return ics.nfw_halos(n, seed=seed, nhalos=max(4, round(2000 * n / 2 ** 24)))
    return ics.plummer_spheres(n, seed=seed, nspheres=max(1, round(512 * n / 2 ** 21)))


def _counts(case):
    """Particles of each box: ragged around the mean, fixed by the case."""
    nb = case.get("nbox", 1)
    if nb == 1:
        return [case["n"]]
    per = case["n"] // nb
    c = [per + (37 * (b % 5) - 74) * per // 200 for b in range(nb)]
    c[-1] += case["n"] - sum(c)
    return c


def _particles(case, seed):
    parts = [_box(case["ic"], c, 1000 * seed + b) for b, c in enumerate(_counts(case))]
    return {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}


def _soft(case):
    return 1.0 / (25 * case["mesh"])


def _context(case, P):
    counts = _counts(case)
    kernel = _lib.SOFT_SPHERE if case["kernel"] == "sphere" else _lib.SOFT_PLUMMER
    g = Gravity(mesh=case["mesh"], order=case["order"], bwidth=case["bwidth"], hsoft=_soft(case),
                eta=ETA, GM=1.0 / counts[0], kernel=kernel, max_particles=case["n"],
                nbox=case["nbox"])
    g.upload_dict(P)
    if case["nbox"] > 1:
        g.set_boxes(counts, [1.0 / c for c in counts])
    return g


def _pinned(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=True)


def _mlp_params(rng):
    """He-scaled weights of the 24 -> 64 -> 64 -> 1 network, in the library's order."""
    return np.concatenate([rng.normal(0, math.sqrt(2 / 24), 64 * 24), rng.normal(0, 0.1, 64),
                           rng.normal(0, math.sqrt(2 / 64), 64 * 64), rng.normal(0, 0.1, 64),
                           rng.normal(0, math.sqrt(1 / 64), 64), [0.0]]).astype(np.float32)


def _samples(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    p = _mlp_params(rng)
    fmean, fstd = rng.normal(0, 2, 24), rng.uniform(0.5, 3, 24)
    X = (rng.normal(size=(case["n"], 24)) * fstd + fmean).astype(np.float32)
    T = rng.normal(-4.0, 0.7, case["n"]).astype(np.float32)  # log10 residuals
    return p, fmean.astype(np.float32), fstd.astype(np.float32), X, T


def _laplace(N):
    """-1/k^2 of the half spectrum (zero at k = 0), FP32 on the GPU."""
    k = torch.fft.fftfreq(N, 1.0 / N, dtype=torch.float64)
    k2 = (k[:, None, None] ** 2 + k[None, :, None] ** 2
          + torch.arange(N // 2 + 1, dtype=torch.float64)[None, None, :] ** 2)
    k2[0, 0, 0] = math.inf
    return (-1.0 / k2).float().cuda()


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "gradients":
        p, fmean, fstd, X, T = _samples(case, seed)
        s["g"] = Gravity(mesh=8, order=2, bwidth=1.0, hsoft=1e-3)
        s["g"].learned_enable(2.0)
        s["g"].mlp_set(p, fmean, fstd)
        s.update(X=X, T=T)
    elif kind == "poisson":
        N, b = case["N"], case["batch"]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        s["g"] = Gravity(mesh=8, order=1, bwidth=1.0, hsoft=1e-3)
        s["rho"] = torch.randn(b, N, N, N, device="cuda", generator=gen)
        s["k"] = _laplace(N)
        s["spec"] = torch.empty(b, N, N, N // 2 + 1, dtype=torch.complex64, device="cuda")
        s["phik"] = torch.empty_like(s["spec"])
        s["phi"] = torch.empty_like(s["rho"])
    elif kind == "cic":
        s["g"] = Gravity(mesh=8, order=1, bwidth=1.0, hsoft=1e-3, max_particles=case["n"])
        s["g"].upload_dict(_box(case["ic"], case["n"], seed))
        N = case["N"]
        s["grid"] = torch.empty(4, N, N, N, dtype=torch.complex64, device="cuda")
    elif kind == "fft64":
        rng = np.random.Generator(np.random.PCG64(seed))
        N = case["N"]
        s["g"] = Gravity(mesh=8, order=1, bwidth=1.0, hsoft=1e-3)
        s["x"] = rng.normal(size=(case["batch"], N, N, N))
    else:
        P = _particles(case, seed)
        g = s["g"] = _context(case, P)
        n = case["n"]
        s["kp"] = kick_params(ascending=True, descending=True, top=True, first=False, rung=0,
                              t0=T0, eta=ETA, max_dt=1.0, scale=1.0)
        s["P"] = P
        if kind == "step":
            s["in"] = {}
            for k, v in P.items():
                t = _pinned(n, torch.int8 if v.dtype == np.int8 else torch.int32)
                s["in"][k] = t.numpy().view(v.dtype)
                s["in"][k][:] = v
            raw = {k: _pinned(n, torch.int32) for k in ("x", "y", "z", "id")}
            vel = {k: _pinned(n, torch.float32) for k in ("vx", "vy", "vz")}
            rung = _pinned(n, torch.int8)
            s["raw"] = raw
            s["out"] = {**{k: t.numpy().view(np.uint32) for k, t in raw.items()},
                        **{k: t.numpy() for k, t in vel.items()}, "rung": rung.numpy()}
            s["pos"] = {k: torch.empty(n) for k in ("x", "y", "z")}
            s["res"] = {**s["pos"], **vel, "rung": rung, "id": raw["id"]}
        elif kind in ("forces", "learned"):
            s["f"] = [_pinned(n, torch.float32) for _ in range(4)]
            if kind == "learned":
                rng = np.random.Generator(np.random.PCG64(seed))
                p = _mlp_params(rng)
                g.learned_enable(case["bwidth"] + 1.0)
                g.mlp_set(p, np.zeros(24), np.ones(24))
                g.learned_select("mlp", 1e30)
                g.particle_to_grid()
                g.compute_forces()
                X = g.learned_cells()["X"].astype(np.float64)
                two = lambda v: np.array([float("%.1e" % q) for q in v])  # noqa: E731
                g.mlp_set(p, two(X.mean(0)), np.maximum(two(X.std(0)), 1e-3))
                g.learned_select("mlp", 0.0)
    return s


def run(s):
    case, g = s["case"], s["g"]
    kind = case["kind"]
    if kind == "step":
        mr = g.kick_drift_host(s["kp"], T0, s["in"], s["out"], 1.0, graph=case["graph"])
        for k in ("x", "y", "z"):
            torch.mul(s["raw"][k], 2.0 ** -32, out=s["pos"][k])
        return {**s["res"], "max_rung": mr}
    if kind == "kick_step":
        g.upload_dict(s["P"])
        mr, minrung = g.kick_step(0, 0, 1.0, 1.0, 1.0, T0, 0)
        d = g.download()
        for k in ("x", "y", "z"):
            d[k] = d[k].view(np.int32) * np.float32(2.0 ** -32)
        d["id"] = d["id"].view(np.int32)
        return {**d, "max_rung": mr, "minrung": minrung}
    if kind in ("forces", "learned"):
        g.particle_to_grid()
        g.compute_forces()
        rc = _lib.load().ct2g_download_forces(g.handle, *[t.data_ptr() for t in s["f"]])
        if rc != 0:
            raise _lib.CT2GError(rc, "download_forces")
        return dict(zip(("fx", "fy", "fz", "pot"), s["f"]))
    if kind == "gradients":
        grad, loss = g.mlp_gradients(s["X"], s["T"])
        return {"grad": grad, "loss": np.float32(loss)}
    if kind == "poisson":
        N, b = case["N"], case["batch"]
        g.fft3d_r2c_dev(s["rho"].data_ptr(), s["spec"].data_ptr(), N, b, dir=1)
        torch.mul(s["spec"], s["k"], out=s["phik"])
        g.fft3d_r2c_dev(s["phi"].data_ptr(), s["phik"].data_ptr(), N, b, dir=-1)
        return {"spec": s["spec"], "phi": s["phi"]}
    if kind == "cic":
        g.cic_deposit(case["N"], s["grid"].data_ptr())
        g.fft3d_c2c_dev(s["grid"].data_ptr(), case["N"], 4, dir=1)
        return s["grid"]
    y = g.fft_r2c_3d(s["x"])
    return {"spec": y, "back": g.fft_c2r_3d(y, case["N"])}


# ---- what a pass cannot do without ----------------------------------------------

def _interactions(case):
    """Direct-sum pairs: every particle with those of its stencil's cells."""
    M, bw = case["mesh"], case["bwidth"] + (0.5 if case["kind"] == "learned" else 0.0)
    r = int(bw)
    o = np.arange(-r, r + 1)
    near = (o[:, None, None] ** 2 + o[None, :, None] ** 2 + o[None, None, :] ** 2) <= bw * bw
    if case["ic"] == "lattice":
        return case["n"] * (case["n"] / M ** 3) * float(near.sum())
    total = 0.0
    sh = 32 - int(math.log2(M))
    ker = np.zeros((M, M, M), np.float32)
    ker[np.ix_(o % M, o % M, o % M)] = near
    kf = torch.fft.rfftn(torch.from_numpy(ker))
    for b, c in enumerate(_counts(case)):
        P = _box(case["ic"], c, b)
        cell = ((P["x"] >> sh).astype(np.int64) * M + (P["y"] >> sh)) * M + (P["z"] >> sh)
        cnt = torch.from_numpy(np.bincount(cell, minlength=M ** 3).astype(np.float32)).view(M, M, M)
        conv = torch.fft.irfftn(torch.fft.rfftn(cnt) * kf, s=(M, M, M))
        total += float((cnt.double() * conv.double()).sum())
    return total


def work(case):
    kind = case["kind"]
    if kind == "gradients":
        # forward, input and weight gradients of 24*64 + 64*64 + 64 weights
        return dict(bytes=4.0 * 25 * case["n"] + 8.0 * 5825, flops=6.0 * 5696 * case["n"])
    if kind in ("poisson", "fft64", "cic"):
        N = case["N"]
        b = case.get("batch", 4)
        lg = 5.0 * N ** 3 * math.log2(N ** 3)
        if kind == "cic":
            return dict(bytes=12.0 * case["n"] + 32.0 * N ** 3, flops=4 * lg + 100.0 * case["n"])
        word = 8 if kind == "fft64" else 4
        # real field in, half spectrum out and real field out (and the kernel in)
        io = word * (2.0 * N ** 3 * b + N * N * (N / 2 + 1) * (2 * b + (kind == "poisson")))
        return dict(bytes=io, flops=lg * b)
    n, M, p = case["n"], case["mesh"], case["order"]
    nc = (p + 1) * (p + 2) * (p + 3) / 6
    cells = case["nbox"] * float(M) ** 3
    fft = 2 * 2.5 * cells * math.log2(float(M) ** 3) * nc
    pairs = math.comb(p + 6, 6)  # (a, b) with |a| + |b| <= p
    flops = 20.0 * _interactions(case) + fft + 4.0 * pairs * cells / 2 + 8.0 * nc * n
    return dict(bytes=(25.0 + 29.0) * n if kind in ("step", "kick_step") else (12.0 + 16.0) * n,
                flops=flops)


# ---- the values in 64 bits ----------------------------------------------------

def _spread3(v):
    out = np.zeros(v.shape, np.uint64)
    for b in range(10):
        out |= ((v.astype(np.uint64) >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b)
    return out


def _cell_order(case, P, lo, hi):
    sh = np.uint32(32 - int(math.log2(case["mesh"])))
    key = ((_spread3(P["x"][lo:hi] >> sh) << np.uint64(2))
           | (_spread3(P["y"][lo:hi] >> sh) << np.uint64(1)) | _spread3(P["z"][lo:hi] >> sh))
    return lo + np.argsort(key, kind="stable")


def _ewald(q, GM, soft, sphere, alpha=10.5, rc=0.5, kmax=20):
    """FP64 periodic accelerations and potentials of equal masses (torch, GPU):
    softened minimum-image pairs, the Ewald correction of the images."""
    q = torch.from_numpy(q).cuda()
    n = len(q)
    f, pot = torch.empty(n, 3, dtype=torch.float64, device="cuda"), torch.empty(
        n, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 25) // n)
    spi = math.sqrt(math.pi)
    for i in range(0, n, step):
        d = q[i:i + step, None, :] - q[None, :, :]
        d -= torch.round(d)
        r2 = (d * d).sum(-1)
        same = r2 == 0
        r = torch.sqrt(r2).masked_fill_(same, 1.0)
        ri = 1 / r
        ec = torch.where(r2 < rc * rc, torch.special.erfc(alpha * r), torch.zeros_like(r))
        ex = torch.where(r2 < rc * rc, 2 * alpha * r / spi * torch.exp(-alpha ** 2 * r2),
                         torch.zeros_like(r))
        if sphere:
            inner = r2 < soft * soft
            g = torch.where(inner, torch.full_like(r, soft ** -3), ri ** 3)
            pk = torch.where(inner, 1.5 / soft - 0.5 * r2 / soft ** 3, ri)
        else:
            s = torch.rsqrt(r2 + soft * soft)
            g, pk = s ** 3, s
        g = (g + (ec + ex - 1) * ri ** 3).masked_fill_(same, 0.0)
        pk = torch.where(same, torch.full_like(r, (1.5 if sphere else 1.0) / soft
                                               - 2 * alpha / spi), pk + (ec - 1) * ri)
        f[i:i + step] = -(d * g[..., None]).sum(1)
        pot[i:i + step] = pk.sum(1)
    k = torch.arange(-kmax, kmax + 1, dtype=torch.float64, device="cuda")
    kv = torch.stack(torch.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
    k2 = (kv * kv).sum(1)
    on = (k2 > 0) & (k2 <= kmax * kmax)
    kv, k2 = kv[on], k2[on]
    w = torch.exp(-math.pi ** 2 * k2 / alpha ** 2) / (math.pi * k2)
    step = max(1, (1 << 25) // n)
    for i in range(0, len(kv), step):
        ph = 2 * math.pi * (q @ kv[i:i + step].T)
        c, s = torch.cos(ph), torch.sin(ph)
        sc, ss = c.sum(0), s.sum(0)
        pot += (c * sc + s * ss) @ w[i:i + step]
        f += ((s * sc - c * ss) * (-2 * math.pi * w[i:i + step])) @ kv[i:i + step]
    pot -= math.pi / alpha ** 2 * n
    return (GM * f).cpu().numpy(), (-GM * pot).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradients":
        p, fmean, fstd, X, T = _samples(case, seed)
        w = torch.from_numpy(p).bfloat16().double().requires_grad_()  # BF16 weights
        x = (torch.from_numpy(X).double() - torch.from_numpy(fmean).double()) \
            / torch.from_numpy(fstd).double()
        o = np.cumsum([64 * 24, 64, 64 * 64, 64, 64])
        h = torch.relu(x @ w[:o[0]].view(64, 24).T + w[o[0]:o[1]])
        h = torch.relu(h @ w[o[1]:o[2]].view(64, 64).T + w[o[2]:o[3]])
        y = h @ w[o[3]:o[4]] + w[o[4]]
        loss = ((y - torch.from_numpy(T).double()) ** 2).mean()
        loss.backward()
        return {"grad": w.grad.numpy(), "loss": loss.item()}
    if kind == "poisson":
        N, b = case["N"], case["batch"]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        rho = torch.randn(b, N, N, N, device="cuda", generator=gen).double()
        spec = torch.fft.rfftn(rho, dim=(1, 2, 3))
        phi = torch.fft.irfftn(spec * _laplace(N).double(), s=(N, N, N), dim=(1, 2, 3))
        return {"spec": spec, "phi": phi * float(N) ** 3}
    if kind == "cic":
        N = case["N"]
        P = _box(case["ic"], case["n"], seed)
        grid = torch.zeros(4, N ** 3, dtype=torch.float64, device="cuda")
        u = [torch.from_numpy(P[k].astype(np.float64)).cuda() * (N * 2.0 ** -32) - 0.5
             for k in ("x", "y", "z")]
        m = [torch.floor(v) for v in u]
        for corner in range(8):
            b = [(corner >> (2 - d)) & 1 for d in range(3)]
            off = [u[d] - m[d] - b[d] for d in range(3)]
            w = (1 - off[0].abs()) * (1 - off[1].abs()) * (1 - off[2].abs())
            i = [(m[d].long() + b[d]) % N for d in range(3)]
            q = (i[0] * N + i[1]) * N + i[2]
            for c in range(4):
                grid[c].index_add_(0, q, w if c == 0 else w * off[c - 1])
        return torch.fft.fftn(grid.view(4, N, N, N).to(torch.complex128), dim=(1, 2, 3))
    if kind == "fft64":
        rng = np.random.Generator(np.random.PCG64(seed))
        N = case["N"]
        x = rng.normal(size=(case["batch"], N, N, N))
        X = np.fft.rfftn(x, axes=(1, 2, 3))
        spec = np.concatenate([X.real.reshape(len(x), -1), X.imag.reshape(len(x), -1)], 1)
        return {"spec": spec, "back": x * float(N) ** 3}
    counts = _counts(case)
    # selected cells have no closed form; a lattice's net forces are small
    # residues of cancelling pulls, so the expansion's truncation is most of
    # their error; larger sums take too long
    if kind == "learned" or case["ic"] == "lattice" or sum(c * c for c in counts) > 2e10:
        return None
    P = _particles(case, seed)
    pos = np.stack([P[k].view(np.int32) * 2.0 ** -32 for k in ("x", "y", "z")], 1)
    order, F, pot, lo = [], [], [], 0
    for c in counts:
        o = _cell_order(case, P, lo, lo + c)
        f, p = _ewald(pos[o], 1.0 / c, _soft(case), case["kernel"] == "sphere")
        order.append(o)
        F.append(f)
        pot.append(p)
        lo += c
    order, F, pot = np.concatenate(order), np.concatenate(F), np.concatenate(pot)
    if kind == "forces":
        return {"fx": F[:, 0], "fy": F[:, 1], "fz": F[:, 2], "pot": pot}
    v = T0 * F
    x = pos[order] + T0 * v
    x -= np.floor(x + 0.5)
    out = {k: x[:, d] for d, k in enumerate("xyz")}
    out.update({"v" + k: v[:, d] for d, k in enumerate("xyz")})
    out.update({k: None for k in ("rung", "id", "max_rung")})
    if kind == "kick_step":
        out["minrung"] = None
    return out
