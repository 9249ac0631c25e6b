"""Workloads whose speed this project measures, through its public entry points.

A case is one call sequence of a user's program, in the ranges of the tests and the benchmark:

  solve     conductivity -> head -> face velocities on one grid, with the solver handle kept: set_K,
            solve to ||b - A h|| / ||b|| <= 1e-10 and the compact velocity (the reference's solve_head
            followed by compute_velocity_from_head)
  ensemble  the same for several realisations on grids of their own, as one BatchSolver
  velocity  padded face velocities of a head and their divergence, curl and helicity
  kfield    a log-normal conductivity field by the randomization method (1000 modes)
  predict   the learned initial guess of a conductivity field
  train     loss and gradients of the learned guess over a minibatch
"""
from __future__ import annotations

import math

import numpy as np
import torch

import macroflow3d_b200 as M

PREC = {"fp64": M.PREC_FP64, "fp32": M.PREC_FP32, "bf16": M.PREC_BF16}
# channels in, channels out, resolution level of the learned guess's convolutions
LAYERS = [(16, 16, 0), (16, 16, 0), (16, 32, 1), (32, 32, 1), (32, 64, 2), (64, 64, 2),
          (64, 64, 3), (64, 64, 3), (128, 64, 2), (96, 32, 1), (48, 16, 0), (16, 16, 0)]


def _solve(name, nx, ny, nz, prec, sigma2, lam, lam_z=None, bc="darcy"):
    c = {"kind": "solve", "nx": nx, "ny": ny, "nz": nz, "prec": prec, "sigma2": sigma2, "lam": lam,
         "lam_z": lam if lam_z is None else lam_z, "bc": bc}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one small plain FP64 solve, bound by launches and latency: the smallest problem of the benchmark
        _solve("solve_64_fp64", 64, 64, 64, "fp64", 1.0, 4.0),
        # a site model whose axes are no powers of two: short coarse rows, a ragged coarsest level
        _solve("solve_100x76x52_mixed", 100, 76, 52, "fp32", 2.0, 6.0),
        # a slab periodic in y and z (no wall effects), plain FP64
        _solve("solve_160x96x128_periodic", 160, 96, 128, "fp64", 1.0, 6.0, bc="periodic_yz"),
        # the BF16-coefficient preconditioner on an ordinary grid
        _solve("solve_192x160x128_bf16", 192, 160, 128, "bf16", 2.0, 8.0),
        # the headline workload, mixed precision and plain FP64
        _solve("solve_256_mixed", 256, 256, 256, "fp32", 4.0, 8.0),
        _solve("solve_256_fp64", 256, 256, 256, "fp64", 4.0, 8.0),
        # the largest single solve: 134 M cells, anisotropic field
        _solve("solve_512_mixed", 512, 512, 512, "fp32", 1.0, 16.0, lam_z=4.0),
        # Monte Carlo: realisations of uneven grids (edges 64, 96, 128 or 160), mixed precision
        {"name": "ensemble_16_mixed", "kind": "ensemble", "count": 16, "prec": "fp32", "sigma2": 2.0, "lam": 6.0,
         "edges": "64,96,128,160", "pick": 1},
        # post-processing of one head: padded velocities for a particle tracker and their diagnostics
        {"name": "velocity_201x150x99", "kind": "velocity", "nx": 201, "ny": 150, "nz": 99, "bc": "darcy"},
        # the input field of one realisation
        {"name": "kfield_128", "kind": "kfield", "nx": 128, "ny": 128, "nz": 128, "sigma2": 2.0, "lam": 6.0,
         "lam_z": 6.0, "modes": 1000},
        # inference and one training minibatch at the size the network is trained at
        {"name": "predict_128", "kind": "predict", "nx": 128, "ny": 128, "nz": 128, "sigma2": 2.5, "lam": 8.0},
        {"name": "train_128_x4", "kind": "train", "nx": 128, "ny": 128, "nz": 128, "sigma2": 2.5, "lam": 8.0,
         "count": 4},
    ]


def draw(rng):
    kind = rng.choice(["solve"] * 5 + ["ensemble", "velocity", "kfield", "predict", "train"])
    sigma2, lam = round(rng.uniform(0.5, 4.0), 2), round(rng.uniform(3.0, 12.0), 2)
    if kind == "solve":
        prec = rng.choice(["fp64", "fp32", "fp32", "bf16"])
        bc = rng.choice(["darcy", "darcy", "periodic_yz"])
        while True:  # axes a * 2^p of 32 .. 384 cells whose coarsest level has 4 .. 20 cells an axis
            p = rng.randint(2, 5)
            n = [rng.randint(4, 20) << p for _ in range(3)]
            if min(n) >= 32 and max(n) <= 384 and n[0] * n[1] * n[2] <= 300 ** 3:
                break
        return _solve(None, n[0], n[1], n[2], prec, sigma2, lam, round(lam * rng.choice([0.25, 0.5, 1.0]), 2), bc)
    if kind == "ensemble":
        return {"kind": "ensemble", "count": rng.randint(2, 16), "prec": rng.choice(["fp64", "fp32", "fp32"]),
                "sigma2": sigma2, "lam": lam, "edges": rng.choice(["64,96,128,160", "48,64,80,112", "32,40,64,96"]),
                "pick": rng.randint(2, 10 ** 6)}
    if kind == "velocity":
        n = [int(math.exp(rng.uniform(math.log(24), math.log(300)))) for _ in range(3)]
        return {"kind": "velocity", "nx": n[0], "ny": n[1], "nz": n[2], "bc": rng.choice(["darcy", "periodic_yz"])}
    if kind == "kfield":
        n = [int(math.exp(rng.uniform(math.log(20), math.log(200)))) for _ in range(3)]
        return {"kind": "kfield", "nx": n[0], "ny": n[1], "nz": n[2], "sigma2": sigma2, "lam": lam,
                "lam_z": round(lam * rng.choice([0.25, 1.0]), 2), "modes": rng.choice([500, 1000, 1000, 2000])}
    n = [8 * rng.randint(4, 16) for _ in range(3)]
    c = {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "sigma2": sigma2, "lam": lam}
    return dict(c, count=rng.randint(1, 4)) if kind == "train" else c


# ---- inputs -----------------------------------------------------------------------------------

def _bc(name):
    faces = [M.BCFace(M.DIRICHLET, 1.0), M.BCFace(M.DIRICHLET, 0.0)]
    t = M.PERIODIC if name == "periodic_yz" else M.NEUMANN
    return M.BCSpec(faces + [M.BCFace(t, 0.0) for _ in range(4)])


def _gaussian(shape, lam, gen):
    """Zero-mean, unit-variance Gaussian field with exponential covariance, float64 (nz, ny, nx):
    white noise filtered with the square root of the covariance's spectrum; lam = (x, y, z)."""
    nz, ny, nx = shape
    w = torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)
    f = torch.fft.rfftn(w)
    k = [2 * math.pi * torch.fft.fftfreq(nz, dtype=torch.float64, device="cuda").view(-1, 1, 1) * lam[2],
         2 * math.pi * torch.fft.fftfreq(ny, dtype=torch.float64, device="cuda").view(1, -1, 1) * lam[1],
         2 * math.pi * torch.fft.rfftfreq(nx, dtype=torch.float64, device="cuda").view(1, 1, -1) * lam[0]]
    f /= 1.0 + k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    g = torch.fft.irfftn(f, s=shape)
    g -= g.mean()
    return g / g.std()


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) % (1 << 62))
    return g


def _shape(c):
    return (c["nz"], c["ny"], c["nx"])


def _K(shape, c, seed, salt=0):
    lam = (c["lam"], c["lam"], c.get("lam_z", c["lam"]))
    return torch.exp(math.sqrt(c["sigma2"]) * _gaussian(shape, lam, _gen(seed, salt)))


def _edges(c, seed):
    """The realisations' grids: edges picked per axis (the same for every seed of a case)."""
    e = [int(v) for v in c["edges"].split(",")]
    r = np.random.RandomState(c["pick"])
    return [tuple(e[int(i)] for i in r.randint(0, len(e), 3)) for _ in range(c["count"])]


def _config(c):
    return M.HeadSolveConfig(mg_levels=16, cg_rtol=1e-10, cg_check_every=1, conv_norm=M.CONV_B,
                             precision=PREC[c["prec"]])


def _empty(n):
    return torch.empty(n, dtype=torch.float64, device="cuda")


def _head_like(shape, seed):
    """A head between 1 and 0 along x with a rough correction, as an iterate or a transient one has."""
    nx = shape[2]
    lin = 1.0 - (torch.arange(nx, dtype=torch.float64, device="cuda") + 0.5) / nx
    return lin + 0.05 * _gaussian(shape, (8.0, 8.0, 8.0), _gen(seed, 17))


def _training_pair(shape, c, seed, i):
    lnk = math.sqrt(c["sigma2"]) * _gaussian(shape, (c["lam"],) * 3, _gen(seed, 2 * i))
    lin = 1.0 - (torch.arange(shape[2], dtype=torch.float64, device="cuda") + 0.5) / shape[2]
    h = lin + 0.06 * _gaussian(shape, (24.0, 24.0, 24.0), _gen(seed, 2 * i + 1))
    return lnk.float().contiguous(), h.float().contiguous()


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"kind": kind, "stream": torch.cuda.Stream()}
    handle = s["stream"].cuda_stream
    if kind == "ensemble":
        shapes = _edges(c, seed)
        s["grids"] = [M.Grid3D(*e) for e in shapes]
        s["bc"] = _bc("darcy")
        s["K"] = [_K((e[2], e[1], e[0]), c, seed, r) for r, e in enumerate(shapes)]
        s["h"] = [torch.empty_like(k) for k in s["K"]]
        s["uvw"] = [tuple(_empty(n) for n in M.velocity_sizes(g)) for g in s["grids"]]
        s["solver"] = M.BatchSolver(s["grids"], s["bc"], _config(c), stream=handle)
        torch.cuda.synchronize()
        return s
    shape = _shape(c)
    s["grid"] = M.Grid3D(c["nx"], c["ny"], c["nz"], 1.0)
    s["bc"] = _bc(c.get("bc", "darcy"))
    if kind == "solve":
        s["K"] = _K(shape, c, seed)
        s["h"] = torch.empty_like(s["K"])
        s["uvw"] = tuple(_empty(n) for n in M.velocity_sizes(s["grid"]))
        s["solver"] = M.HeadSolver(s["grid"], s["bc"], _config(c), stream=handle)
    elif kind == "velocity":
        s["K"] = _K(shape, dict(c, sigma2=1.5, lam=6.0), seed)
        s["h"] = _head_like(shape, seed)
        s["uvw"] = tuple(torch.zeros(n, dtype=torch.float64, device="cuda")
                         for n in M.velocity_sizes(s["grid"], M.VEL_PADDED))
        s["fields"] = tuple(torch.empty_like(s["K"]) for _ in range(3))
    elif kind == "kfield":
        s["args"] = (c["sigma2"], (c["lam"], c["lam"], c["lam_z"]), int(seed), c["modes"])
    else:
        s["net"] = M.WarmStart.pretrained()
        if kind == "predict":
            s["K"] = _K(shape, c, seed)
            s["x0"] = torch.empty_like(s["K"])
        else:
            pairs = [_training_pair(shape, c, seed, i) for i in range(c["count"])]
            s["lnK"], s["heads"] = [p[0] for p in pairs], [p[1] for p in pairs]
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    with torch.cuda.stream(s["stream"]):
        if kind == "solve":
            s["solver"].set_K(s["K"])
            s["solver"].solve(s["h"])
            M.compute_velocity_from_head(*s["uvw"], s["h"], s["K"], s["grid"], s["bc"])
            return {"h": s["h"], "U": s["uvw"][0], "V": s["uvw"][1], "W": s["uvw"][2]}
        if kind == "ensemble":
            s["solver"].set_K(s["K"])
            s["solver"].solve(s["h"])
            for g, h, K, uvw in zip(s["grids"], s["h"], s["K"], s["uvw"]):
                M.compute_velocity_from_head(*uvw, h, K, g, s["bc"])
            return {"h": s["h"], "uvw": [list(v) for v in s["uvw"]]}
        if kind == "velocity":
            M.compute_velocity_from_head(*s["uvw"], s["h"], s["K"], s["grid"], s["bc"], layout=M.VEL_PADDED)
            div, om, he = s["fields"]
            st = M.velocity_diagnostics(*s["uvw"], s["grid"], layout=M.VEL_PADDED, div=div, omag=om, hel=he)
            return {"U": s["uvw"][0], "V": s["uvw"][1], "W": s["uvw"][2], "div": div, "omag": om, "hel": he,
                    "stats": np.array([st["div"][:2], st["vorticity_mag"][:2], st["helicity"][:2]])}
        if kind == "kfield":
            sigma2, lam, seed, modes = s["args"]
            return M.generate_K_field(s["grid"], sigma2, lam, seed=seed, n_modes=modes)
        if kind == "predict":
            s["net"].predict(s["grid"], s["bc"], s["K"], s["x0"])
            return s["x0"]
        loss = s["net"].train_step(s["grid"], s["bc"], s["lnK"], s["heads"], lr=0.0)
        return {"loss": loss, "grads": s["net"].get_grads()}


# ---- what a pass cannot do without --------------------------------------------------------------

def _iterations(sigma2):
    return 10.0 + 2.0 * sigma2


def work(case):
    c, kind = case, case["kind"]
    if kind in ("solve", "ensemble"):
        # K in; head and three velocities out.  Per cell and iteration: four smoothing sweeps, a residual
        # and the transfers on every level (8/7 of about 75), the matvec and the vector updates
        n = sum(a * b * d for a, b, d in _edges(c, 0)) if kind == "ensemble" else c["nx"] * c["ny"] * c["nz"]
        return {"bytes": 40.0 * n, "flops": n * (_iterations(c["sigma2"]) * 115.0 + 60.0)}
    n = float(c["nx"] * c["ny"] * c["nz"])
    if kind == "velocity":
        return {"bytes": 64.0 * n, "flops": 70.0 * n}  # K, h in; three velocities, three fields out
    if kind == "kfield":
        return {"bytes": 8.0 * n + 40.0 * c["modes"], "flops": 4.0 * n * c["modes"]}
    # the input has two live channels and the output one
    f = 2.0 * 27 * n * sum((2 if i == 0 else a) * (1 if i == 11 else b) / 8.0 ** l for i, (a, b, l) in enumerate(LAYERS))
    params = 774624
    if kind == "predict":
        return {"bytes": 16.0 * n + 2.0 * params, "flops": f}
    return {"bytes": c["count"] * 8.0 * n + 6.0 * params, "flops": 3.0 * f * c["count"]}


def tolerance(case):
    kind = case["kind"]
    if kind in ("solve", "ensemble"):
        # two solvers that stop at the same residual 1e-10 differ by what that residual leaves in
        # the head and its gradients (5e-8 from the 64-bit solution at variance 4)
        return {"rel": 2e-7, "max": 2e-5}
    if kind == "velocity":
        return {"rel": 4e-15, "max": 2e-13}  # 6e-16 from the 64-bit result
    if kind == "kfield":
        return {"rel": 1e-12, "max": 4e-11}  # 1e-13; phases k.x of the steepest modes reach 1e4
    if kind == "predict":
        return {"rel": 4e-4, "max": 1e-2}  # BF16 activations: 1e-4
    return {"rel": 4e-3, "max": 0.16}  # BF16 activations and their gradients: 1e-3


# ---- the same in 64 bits, in plain torch ---------------------------------------------------------

def _hm(a, b):
    return 2.0 / (1.0 / a + 1.0 / b)


class _Level:
    """The 7-point operator of one conductivity field: harmonic-mean faces, x faces Dirichlet, the
    others no-flow or periodic."""

    def __init__(self, K, periodic):
        self.K, self.per = K, periodic
        self.f = []
        for ax in (2, 1, 0):
            n = K.shape[ax]
            inner = _hm(K.narrow(ax, 0, n - 1), K.narrow(ax, 1, n - 1))
            lo, hi = K.narrow(ax, 0, 1), K.narrow(ax, n - 1, 1)
            if ax == 2:
                lo, hi = 2.0 * lo, 2.0 * hi
            elif periodic:
                lo = hi = _hm(lo, hi)
            else:
                lo, hi = torch.zeros_like(lo), torch.zeros_like(hi)
            self.f.append(torch.cat([lo, inner, hi], ax))
        self.D = sum(f.narrow(ax, 0, K.shape[ax]) + f.narrow(ax, 1, K.shape[ax]) for f, ax in zip(self.f, (2, 1, 0)))

    def apply(self, x):
        y = self.D * x
        for f, ax in zip(self.f, (2, 1, 0)):
            n = x.shape[ax]
            g = f.narrow(ax, 1, n - 1)
            y.narrow(ax, 1, n - 1).sub_(g * x.narrow(ax, 0, n - 1))
            y.narrow(ax, 0, n - 1).sub_(g * x.narrow(ax, 1, n - 1))
            if ax != 2 and self.per:
                g = f.narrow(ax, 0, 1)
                y.narrow(ax, 0, 1).sub_(g * x.narrow(ax, n - 1, 1))
                y.narrow(ax, n - 1, 1).sub_(g * x.narrow(ax, 0, 1))
        return y


def _halve(a):
    nz, ny, nx = a.shape
    return a.view(nz // 2, 2, ny // 2, 2, nx // 2, 2).mean((1, 3, 5))


def _double(a):
    return a.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)


def _cycle(levels, l, b):
    L = levels[l]
    if l == len(levels) - 1:
        x = 0.8 * b / L.D
        for _ in range(80):
            x = x + 0.8 * (b - L.apply(x)) / L.D
        return x
    x = 0.8 * b / L.D
    for _ in range(2):
        x = x + 0.8 * (b - L.apply(x)) / L.D
    x = x + _double(_cycle(levels, l + 1, 4.0 * _halve(b - L.apply(x))))
    for _ in range(3):
        x = x + 0.8 * (b - L.apply(x)) / L.D
    return x


def _exact_head(K, periodic):
    levels = [_Level(K, periodic)]
    while all(n % 2 == 0 and n >= 4 for n in levels[-1].K.shape) and len(levels) < 8:
        levels.append(_Level(torch.exp(_halve(torch.log(levels[-1].K))), periodic))
    A = levels[0]
    b = torch.zeros_like(K)
    b[:, :, 0] = 2.0 * K[:, :, 0]  # head 1 on the low x face, 0 on the high one
    x = torch.zeros_like(K)
    bn = float(b.norm())
    for _ in range(3):  # restarted on the true residual, until it stagnates
        r = b - A.apply(x)
        z = _cycle(levels, 0, r)
        p, rz = z.clone(), float((r * z).sum())
        for _ in range(150):
            if float(r.norm()) <= 1e-15 * bn:
                break
            Ap = A.apply(p)
            a = rz / float((p * Ap).sum())
            x += a * p
            r -= a * Ap
            z = _cycle(levels, 0, r)
            new = float((r * z).sum())
            p = z + (new / rz) * p
            rz = new
    return x


def _exact_velocity(h, K, periodic):
    """Compact face velocities (dx = 1), each with one more face along its axis."""
    out = []
    for ax in (2, 1, 0):
        n = K.shape[ax]
        a, b = (lambda t: t.narrow(ax, 0, n - 1)), (lambda t: t.narrow(ax, 1, n - 1))
        q = 2.0 * a(K) * b(K) / (a(K) + b(K)) * (a(h) - b(h))
        K0, K1, h0, h1 = K.narrow(ax, 0, 1), K.narrow(ax, n - 1, 1), h.narrow(ax, 0, 1), h.narrow(ax, n - 1, 1)
        if ax == 2:
            lo, hi = -2.0 * K0 * (h0 - 1.0), -2.0 * K1 * (0.0 - h1)
        elif periodic:
            lo = hi = 2.0 * K0 * K1 / (K0 + K1) * (h1 - h0)
        else:
            lo, hi = torch.zeros_like(K0), torch.zeros_like(K1)
        out.append(torch.cat([lo, q, hi], ax))
    return out


def _exact_solve(K, periodic):
    h = _exact_head(K, periodic)
    return h, [v.reshape(-1) for v in _exact_velocity(h, K, periodic)]


def _philox(seed, c0, c1):
    """Philox4x32-10 (Salmon et al. 2011), counter (c0, c1, 0, 0)."""
    c, k, m = [c0, c1, 0, 0], [seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF], 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [(p1 >> 32) ^ c[1] ^ k[0], p1 & m, (p0 >> 32) ^ c[3] ^ k[1], p0 & m]
        k = [(k[0] + 0x9E3779B9) & m, (k[1] + 0xBB67AE85) & m]
    return c


def _uniforms(seed, mode):
    d = 0
    while True:
        c = _philox(seed, mode, d)
        d += 1
        for a, b in ((c[0], c[1]), (c[2], c[3])):
            yield (((a >> 5) << 26 | (b >> 6)) + 0.5) / 9007199254740992.0


def _exact_kfield(c, seed):
    lam, rows = (c["lam"], c["lam"], c["lam_z"]), []
    for m in range(c["modes"]):
        u = _uniforms(int(seed), m)
        fi, theta = 2.0 * math.pi * next(u), math.acos(1.0 - 2.0 * next(u))
        while True:  # radial density k^2 / (1 + k^2)^2
            k = math.tan(math.pi * 0.5 * next(u))
            if next(u) < k * k / (1.0 + k * k):
                break
        kv = [k * math.sin(fi) * math.sin(theta) / lam[0], k * math.cos(fi) * math.sin(theta) / lam[1],
              k * math.cos(theta) / lam[2]]
        ab = []
        for _ in range(2):
            u1, u2 = next(u), next(u)
            ab.append(math.sqrt(-2.0 * math.log(u1)) * math.cos(2.0 * math.pi * u2))
        rows.append(kv + ab)
    t = torch.tensor(rows, dtype=torch.float64, device="cuda")
    wave = [torch.exp(1j * (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5).view(-1, 1) * t[:, a])
            for a, n in enumerate((c["nx"], c["ny"], c["nz"]))]
    amp = t[:, 4] - 1j * t[:, 3]  # a sin + b cos = Re((b - i a) exp(i k x))
    out = torch.empty(_shape(c), dtype=torch.float64, device="cuda")
    for k in range(c["nz"]):
        out[k] = ((wave[1] * (amp * wave[2][k])) @ wave[0].T).real
    return torch.exp(out * math.sqrt(c["sigma2"] / c["modes"]))


def _network(params, lnk):
    """The learned guess's output channel 0 for one log-conductivity field, in 64 bits."""
    import torch.nn.functional as F
    nz, ny, nx = lnk.shape
    lin = 1.0 - (torch.arange(nx, dtype=torch.float64, device="cuda") + 0.5) / nx
    x = torch.zeros((1, 16, nz, ny, nx), dtype=torch.float64, device="cuda")
    x[0, 0], x[0, 1] = 0.5 * lnk, (lin - 0.5).expand(nz, ny, nx)

    def conv(i, t):
        w, b = params[2 * i], params[2 * i + 1]
        cout, _, cin = w.shape
        y = torch.zeros((1, cout) + t.shape[2:], dtype=torch.float64, device="cuda")
        p = F.pad(t, (1, 1, 1, 1, 1, 1))
        d, e, f = t.shape[2:]
        for tap in range(27):
            z, yy, xx = tap // 9, (tap // 3) % 3, tap % 3
            y = y + torch.einsum("oc,bczyx->bozyx", w[:, tap], p[:, :, z:z + d, yy:yy + e, xx:xx + f])
        y = y + b.view(1, -1, 1, 1, 1)
        return y if i == 11 else torch.relu(y)

    def up(t):
        return t.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)

    e0 = conv(1, conv(0, x))
    e1 = conv(3, conv(2, F.avg_pool3d(e0, 2)))
    e2 = conv(5, conv(4, F.avg_pool3d(e1, 2)))
    e3 = conv(7, conv(6, F.avg_pool3d(e2, 2)))
    d2 = conv(8, torch.cat([up(e3), e2], 1))
    d1 = conv(9, torch.cat([up(d2), e1], 1))
    d0 = conv(10, torch.cat([up(d1), e0], 1))
    return conv(11, d0)[0, 0], lin


def _parameters():
    """The shipped parameters as the layers hold them: BF16 weights, 32-bit biases."""
    flat, out, at = torch.from_numpy(M.WarmStart.pretrained().get_params()), [], 0
    for cin, cout, _ in LAYERS:
        n = cout * 27 * cin
        out.append(flat[at:at + n].to(torch.bfloat16).double().view(cout, 27, cin).cuda())
        out.append(flat[at + n:at + n + cout].double().cuda())
        at += n + cout
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve":
        h, v = _exact_solve(_K(_shape(c), c, seed), c["bc"] == "periodic_yz")
        return {"h": h, "U": v[0], "V": v[1], "W": v[2]}
    if kind == "ensemble":
        got = [_exact_solve(_K((e[2], e[1], e[0]), c, seed, r), False) for r, e in enumerate(_edges(c, seed))]
        return {"h": [g[0] for g in got], "uvw": [g[1] for g in got]}
    if kind == "kfield":
        return _exact_kfield(c, seed)
    shape = _shape(c)
    if kind == "velocity":
        nz, ny, nx = shape
        h, per = _head_like(shape, seed), c["bc"] == "periodic_yz"
        u, v, w = _exact_velocity(h, _K(shape, dict(c, sigma2=1.5, lam=6.0), seed), per)
        div = (u[..., 1:] - u[..., :-1]) + (v[:, 1:] - v[:, :-1]) + (w[1:] - w[:-1])
        cu, cv, cw = 0.5 * (u[..., 1:] + u[..., :-1]), 0.5 * (v[:, 1:] + v[:, :-1]), 0.5 * (w[1:] + w[:-1])

        def d(a, ax):
            i = [slice(1, -1)] * 3
            lo, hi = list(i), list(i)
            lo[ax], hi[ax] = slice(0, -2), slice(2, None)
            return 0.5 * (a[tuple(hi)] - a[tuple(lo)])

        ox, oy, oz = d(cw, 1) - d(cv, 0), d(cu, 0) - d(cw, 2), d(cv, 2) - d(cu, 1)
        i = (slice(1, -1),) * 3
        om, he = torch.zeros_like(h), torch.zeros_like(h)
        om[i] = torch.sqrt(ox * ox + oy * oy + oz * oz)
        he[i] = cu[i] * ox + cv[i] * oy + cw[i] * oz
        pad = []
        for a in (u, v, w):
            t = torch.zeros((nz + 1, ny + 1, nx + 1), dtype=torch.float64, device="cuda")
            t[:a.shape[0], :a.shape[1], :a.shape[2]] = a
            pad.append(t.reshape(-1))
        st = np.array([[float(f.min()), float(f.max())] for f in (div, om, he)])
        return {"U": pad[0], "V": pad[1], "W": pad[2], "div": div, "omag": om, "hel": he, "stats": st}
    params = _parameters()
    if kind == "predict":
        with torch.no_grad():
            net, lin = _network(params, torch.log(_K(shape, c, seed)))
            return lin + 0.1 * net
    for p in params:
        p.requires_grad_(True)
    loss = 0.0
    for i in range(c["count"]):
        lnk, h = _training_pair(shape, c, seed, i)
        net, lin = _network(params, lnk.double())
        one = ((net - (h.double() - lin) / 0.1) ** 2).mean()
        one.backward()
        loss += float(one.detach())
    grads = torch.cat([p.grad.reshape(-1) for p in params])
    return {"loss": loss / c["count"], "grads": grads}
