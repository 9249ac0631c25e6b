"""GPU parity: the CUDA path (through the C-ABI) against the CPU oracle on seeded inputs.

Tolerances: single operator applications are compared element-wise at 1e-12 relative to
the array's max (the arithmetic differs only in rounding: stored vs recomputed harmonic
means, operation order, FMA); solves are compared by head relative max-norm <= 1e-9 and
mass balance <= 1e-10, the targets of the task statement for this path.
"""
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D, N, P = 0, 1, 2
BC_CASES = [
    ("darcy", [D, D, N, N, N, N], [1.0, 0.0, 0, 0, 0, 0], False),
    ("mixed", [D, N, N, D, N, D], [1.0, 0, 0, 0.5, 0, 0.25], False),
    ("neumann_pin", [N, N, N, N, N, N], [0.0] * 6, True),
    ("periodic", [P, P, N, N, D, D], [0, 0, 0, 0, 0.3, 0.7], False),
    ("all_dirichlet", [D] * 6, [1.0, 0.0, 0.2, 0.4, 0.6, 0.8], False),
]
SHAPES = [(8, 10, 6), (6, 8, 12), (12, 34, 40), (16, 16, 16)]


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def _np(t):
    return t.detach().cpu().numpy()


def _rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def _bcs(M, types, values):
    return M.BCSpec([M.BCFace(t, v) for t, v in zip(types, values)])


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("case", BC_CASES, ids=[c[0] for c in BC_CASES])
def test_operators_vs_oracle(mf3d, oracle_mod, shape, case):
    M, O = mf3d, oracle_mod
    name, types, values, pin = case
    rng = np.random.default_rng(zlib.crc32(repr((shape, name)).encode()))
    K = np.exp(rng.normal(size=shape))
    x, b = rng.normal(size=shape), rng.normal(size=shape)
    dx = 0.5
    g = M.Grid3D(shape[2], shape[1], shape[0], dx)
    bc, obc = _bcs(M, types, values), O.make_bc(types, values)
    Kt, xt, bt = _t(K), _t(x), _t(b)
    y = _t(np.zeros(shape))
    M.apply_A(g, bc, Kt, xt, y, pin)
    assert _rel(_np(y), O.apply_A(K, x, obc, dx, pin)) < 1e-12
    M.compute_residual_3d(g, xt, bt, Kt, y, bc, pin)
    assert _rel(_np(y), O.residual(K, x, b, obc, dx, pin)) < 1e-12
    for it in (1, 3):
        xs = xt.clone()
        M.gsrb_smooth_3d(g, xs, bt, Kt, it, bc, pin)
        assert _rel(_np(xs), O.gsrb(K, b, x, obc, it, dx, pin)) < 1e-11, it
    M.build_rhs_head(y, Kt, g, bc)
    assert _rel(_np(y), O.build_rhs(K, obc, dx)) < 1e-14 or np.abs(O.build_rhs(K, obc, dx)).max() == 0
    M.init_head_guess(y, g, bc)
    assert np.abs(_np(y) - O.init_guess(shape, obc)).max() < 1e-15
    for lay in (0, 1):
        su, sv, sw = M.velocity_sizes(g, lay)
        U, V, W = _t(np.zeros(su)), _t(np.zeros(sv)), _t(np.zeros(sw))
        M.compute_velocity_from_head(U, V, W, xt, Kt, g, bc, lay)
        Uo, Vo, Wo = O.velocity(x, K, obc, dx, lay)
        for a, o in ((U, Uo), (V, Vo), (W, Wo)):
            assert np.abs(_np(a) - o.ravel()).max() <= 1e-14 * np.abs(o).max()


# The x-pair sweep (kernels_sweep_pair.cuh) on the shapes that exercise its tile ring: partial
# tiles in x and y, periodic axes of whole tiles (x 32, y 16 cells), odd nz, nx = 2, and grids
# deep enough in z for several z chunks per tile.
PAIR_CASES = [
    ((12, 32, 64), [P, P, P, P, D, D], [0, 0, 0, 0, 0.3, 0.7], False),
    ((10, 16, 32), [P] * 6, [0.0] * 6, True),
    ((7, 20, 50), [D, N, N, D, N, D], [1.0, 0, 0, 0.5, 0, 0.25], False),
    ((40, 18, 34), [D, D, N, N, N, N], [1.0, 0.0, 0, 0, 0, 0], False),
    ((5, 3, 2), [D] * 6, [1.0, 0.0, 0.2, 0.4, 0.6, 0.8], False),
    ((96, 48, 96), [D, D, N, N, N, N], [1.0, 0.0, 0, 0, 0, 0], False),
    # 64 tiles: z chunks of several planes, so that the steady-state staging runs
    ((64, 128, 256), [D, D, N, N, N, N], [1.0, 0.0, 0, 0, 0, 0], False),
    ((48, 128, 128), [D, D, P, P, N, N], [1.0, 0.0, 0, 0, 0, 0], False),
]


@pytest.mark.parametrize("shape,types,values,pin", PAIR_CASES, ids=[str(c[0]) for c in PAIR_CASES])
def test_gsrb_pair_sweep_vs_oracle(mf3d, oracle_mod, shape, types, values, pin):
    M, O = mf3d, oracle_mod
    rng = np.random.default_rng(zlib.crc32(repr(("pair", shape)).encode()))
    K = np.exp(rng.normal(size=shape))
    x, b = rng.normal(size=shape), rng.normal(size=shape)
    g = M.Grid3D(shape[2], shape[1], shape[0], 0.5)
    bc, obc = _bcs(M, types, values), O.make_bc(types, values)
    for it in (1, 2, 3):
        xs = _t(x)
        M.gsrb_smooth_3d(g, xs, _t(b), _t(K), it, bc, pin)
        assert _rel(_np(xs), O.gsrb(K, b, x, obc, it, 0.5, pin)) < 1e-11, it


@pytest.mark.parametrize("shape,levels", [((32, 32, 32), 4), ((24, 16, 52), 3), ((64, 64, 64), 5)])
@pytest.mark.parametrize("case", BC_CASES[:4], ids=[c[0] for c in BC_CASES[:4]])
def test_fp32_vcycle_vs_oracle(mf3d, oracle_mod, shape, levels, case):
    """The FP32 V-cycle (x-pair sweeps in FP32, FP64 coarse tail) against the FP64 oracle: equal
    to FP32 rounding (1e-5 of the correction's max)."""
    M, O = mf3d, oracle_mod
    name, types, values, pin = case
    if types[0] == P and (shape[2] >> (levels - 1)) % 2:
        pytest.skip("periodic x with an odd count on the coarsest level: red-black order is undefined")
    rng = np.random.default_rng(zlib.crc32(repr((shape, name, 32)).encode()))
    K = np.exp(rng.normal(size=shape))
    r = rng.normal(size=shape)
    g = M.Grid3D(shape[2], shape[1], shape[0], 1.0)
    cfg = M.HeadSolveConfig(mg_levels=levels, precision=M.PREC_FP32, pin_mode=M.PIN_ON if pin else M.PIN_OFF)
    s = M.HeadSolver(g, _bcs(M, types, values), cfg)
    s.set_K(_t(K))
    z = _t(np.zeros(shape))
    s.vcycle(_t(r), z)
    zo, _ = O.vcycle(K, r, O.make_bc(types, values), levels, 2, 2, 50, 1.0, pin)
    assert _rel(_np(z), zo) < 1e-5


def test_transfer_vs_oracle(mf3d, oracle_mod):
    M, O = mf3d, oracle_mod
    rng = np.random.default_rng(5)
    fine = rng.normal(size=(8, 12, 16))
    coarse = rng.normal(size=(4, 6, 8))
    Kf = np.exp(rng.normal(size=(8, 12, 16)))
    cg = M.Grid3D(8, 6, 4, 2.0)
    out = _t(np.zeros((4, 6, 8)))
    M.restrict_3d(cg, _t(fine), out)
    assert _rel(_np(out), O.restrict(fine)) < 1e-15
    xf = _t(fine)
    M.prolong_3d_add(cg, _t(coarse), xf)
    assert _rel(_np(xf), O.prolong_add(coarse, fine)) < 1e-15
    M.coarsen_K(cg, _t(Kf), out)
    assert _rel(_np(out), O.coarsen_K(Kf)) < 1e-14


@pytest.mark.parametrize("shape,levels,pre,post,coarse", [
    ((16, 16, 16), 3, 2, 2, 50), ((32, 32, 32), 4, 2, 2, 50), ((64, 32, 32), 4, 1, 3, 20),
    ((8, 8, 8), 2, 2, 2, 50), ((64, 64, 64), 5, 2, 2, 50),
    # level 1 is 18 / 26 cells wide: 16-byte rows in FP64 but not whole 4-cell quads
    ((16, 20, 36), 3, 2, 2, 50), ((24, 16, 52), 3, 2, 2, 20)])
@pytest.mark.parametrize("case", BC_CASES[:4], ids=[c[0] for c in BC_CASES[:4]])
def test_vcycle_vs_oracle(mf3d, oracle_mod, shape, levels, pre, post, coarse, case):
    M, O = mf3d, oracle_mod
    name, types, values, pin = case
    if types[0] == P and (shape[2] >> (levels - 1)) % 2:
        pytest.skip("periodic x with an odd count on the coarsest level: red-black order is undefined")
    rng = np.random.default_rng(zlib.crc32(repr((shape, name, 1)).encode()))
    K = np.exp(rng.normal(size=shape))
    r = rng.normal(size=shape)
    g = M.Grid3D(shape[2], shape[1], shape[0], 1.0)
    cfg = M.HeadSolveConfig(mg_levels=levels, mg_pre_smooth=pre, mg_post_smooth=post,
                            mg_coarse_iters=coarse, pin_mode=M.PIN_ON if pin else M.PIN_OFF)
    s = M.HeadSolver(g, _bcs(M, types, values), cfg)
    s.set_K(_t(K))
    z = _t(np.zeros(shape))
    s.vcycle(_t(r), z)
    zo, nl = O.vcycle(K, r, O.make_bc(types, values), levels, pre, post, coarse, 1.0, pin)
    assert nl == s.num_levels
    assert _rel(_np(z), zo) < 1e-10


@pytest.mark.parametrize("shape,levels", [((64, 64, 64), 5), ((24, 16, 52), 3), ((32, 32, 32), 4),
                                          ((64, 48, 32), 4)])
@pytest.mark.parametrize("bcname", ["darcy", "periodic_yz"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("pre,post", [(2, 2), (1, 3)])
def test_cluster_coarse_end_matches_one_cta_tail(mf3d, monkeypatch, shape, levels, bcname, prec, pre, post):
    """The coarse end in one thread-block cluster (levels of up to 32^3 cells in z slabs over
    the cluster's CTAs, FP64; a coarsest level of at most 64 cells as its own map) against the same V-cycle
    with the one-CTA tail and x-pair sweeps above it: equal to rounding in FP64 (1e-12), to FP32 rounding of
    the levels it replaces in the FP32 V-cycle (1e-5).  The matrix of the coarsest levels, which would take the
    cluster's place here, is off, and in the tail's arm the bricks."""
    M = mf3d
    rng = np.random.default_rng(zlib.crc32(repr((shape, levels, bcname)).encode()))
    K = np.exp(rng.normal(size=shape))
    r = rng.normal(size=shape)
    g = M.Grid3D(shape[2], shape[1], shape[0], 1.0)
    if bcname == "darcy":
        bc = M.BCSpec.darcy_x()
    else:
        bc = _bcs(M, [D, D, P, P, P, P], [1.0, 0.0, 0, 0, 0, 0])
    P_ = {"fp64": M.PREC_FP64, "fp32": M.PREC_FP32}[prec]
    cfg = M.HeadSolveConfig(mg_levels=levels, mg_pre_smooth=pre, mg_post_smooth=post, precision=P_)
    z = {}
    for mode, off in (("cluster", ["MF3D_NO_MATRIX"]), ("tail", ["MF3D_NO_CLUSTER_TAIL", "MF3D_NO_BRICKS"])):
        for name in off:
            monkeypatch.setenv(name, "1")
        s = M.HeadSolver(g, bc, cfg)
        first, ctas = s.coarse_info
        if mode == "cluster":
            assert ctas >= 2, (first, ctas)
        else:
            assert ctas == 0
        s.set_K(_t(K))
        zz = _t(np.zeros(shape))
        s.vcycle(_t(r), zz)
        z[mode] = _np(zz)
        assert _coarse_way(s) == ["coarse_" + mode]
        s.close()
        for name in off:
            monkeypatch.delenv(name)
    assert _rel(z["cluster"], z["tail"]) < (1e-12 if prec == "fp64" else 1e-5)


@pytest.mark.parametrize("shape,levels", [((64, 64, 64), 5), ((32, 48, 64), 4), ((16, 16, 128), 3)])
@pytest.mark.parametrize("bcname", ["darcy", "all_dirichlet"])
def test_bf16_vcycle_staged_matches_unstaged(mf3d, monkeypatch, shape, levels, bcname):
    """The BF16-coefficient V-cycle on the TMA-staged x-pair sweep and the staged residual +
    restriction against the same V-cycle on the unstaged sweep (MF3D_NO_TMA): the same BF16
    coefficients and FP32 arithmetic, so equal to FP32 rounding (1e-5 of the max).  Both arms sweep: small
    levels would run in bricks, which stage nothing."""
    monkeypatch.setenv("MF3D_NO_BRICKS", "1")
    M = mf3d
    rng = np.random.default_rng(zlib.crc32(repr((shape, levels, bcname, "bf16")).encode()))
    K = np.exp(rng.normal(size=shape))
    r = rng.normal(size=shape)
    g = M.Grid3D(shape[2], shape[1], shape[0], 1.0)
    case = [c for c in BC_CASES if c[0] == bcname][0]
    bc = _bcs(M, case[1], case[2])
    cfg = M.HeadSolveConfig(mg_levels=levels, precision=M.PREC_BF16)
    z = {}
    for mode in ("staged", "unstaged"):
        if mode == "unstaged":
            monkeypatch.setenv("MF3D_NO_TMA", "1")
        s = M.HeadSolver(g, bc, cfg)
        s.set_K(_t(K))
        zz = _t(np.zeros(shape))
        s.vcycle(_t(r), zz)
        z[mode] = _np(zz)
        sweeps = {name.rsplit("_", 1)[1] for name, *_ in s.profile(1) if name.startswith("sweep_l0")}
        assert sweeps == {"pair" if mode == "staged" else "ldg"}
        s.close()
        monkeypatch.delenv("MF3D_NO_TMA", raising=False)
    assert _rel(z["staged"], z["unstaged"]) < 1e-5


def _lognormal(shape, sigma, seed):
    return np.exp(sigma * np.random.default_rng(seed).normal(size=shape))


@pytest.mark.parametrize("shape,sigma,levels", [((16, 16, 16), 1.0, 3), ((24, 40, 32), 2.0, 4),
                                                ((64, 64, 64), 1.0, 5)])
def test_pcg_reference_semantics_vs_oracle(mf3d, oracle_mod, shape, sigma, levels):
    """Reference stopping rule (||r||/||r0|| < rtol every check_every): same iteration count."""
    M, O = mf3d, oracle_mod
    K = _lognormal(shape, sigma, 11)
    g = M.Grid3D(shape[2], shape[1], shape[0], 1.0)
    bc = M.BCSpec.darcy_x()
    cfg = M.HeadSolveConfig(mg_levels=levels, cg_rtol=1e-10, cg_check_every=1)
    s = M.HeadSolver(g, bc, cfg)
    s.set_K(_t(K))
    h = _t(np.zeros(shape))
    res = s.solve(h)
    ho, ro = O.solve_head_pcg(K, O.baseline_bc(), levels, rtol=1e-10, check_every=1)
    assert res.converged and ro.converged
    assert abs(res.num_iterations - ro.iterations) <= 1
    assert _rel(_np(h), ho) < 1e-9
    assert res.true_rel_residual < 1e-9


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_mixed_precision_reaches_fp64_tolerance(mf3d, oracle_mod, prec):
    """FP32 / BF16-coefficient V-cycle inside flexible FP64 PCG to ||r||/||b|| <= 1e-10;
    the head agrees with a tightly solved FP64 oracle head."""
    M, O = mf3d, oracle_mod
    shape = (32, 32, 32)
    K = _lognormal(shape, 2.0, 12)
    g = M.Grid3D(32, 32, 32, 1.0)
    cfg = M.HeadSolveConfig(mg_levels=4, cg_rtol=1e-10, cg_check_every=1, conv_norm=M.CONV_B,
                            precision=prec)
    s = M.HeadSolver(g, M.BCSpec.darcy_x(), cfg)
    s.set_K(_t(K))
    h = _t(np.zeros(shape))
    res = s.solve(h)
    assert res.converged, res
    assert res.true_rel_residual <= 1.5e-10
    ho, _ = O.solve_head_pcg(K, O.baseline_bc(), 4, rtol=1e-15, check_every=1, max_iter=100)
    # measured 3.7e-9 (FP32, BF16) and 5.6e-9 (the FP64 reference algorithm) at 1e-10 on this
    # field of uncorrelated cell values, 1.04e-9 (FP32) at 1e-11: the head bound 1e-9 needs
    # ||r|| / ||b|| <= 1e-12 here (next assertion)
    assert _rel(_np(h), ho) < 1e-8
    s.close()
    cfg.cg_rtol = 1e-12
    s = M.HeadSolver(g, M.BCSpec.darcy_x(), cfg)
    s.set_K(_t(K))
    res = s.solve(h)
    assert res.converged and res.true_rel_residual <= 1.5e-12, res
    assert _rel(_np(h), ho) < 1e-9


def test_solvers_with_different_coarse_tails_coexist(mf3d):
    """A solver created later with a smaller coarse tail must not lower the tail kernel's
    shared-memory limit under an earlier solver's tail."""
    M = mf3d
    g = M.Grid3D(32, 32, 32, 1.0)
    K = _t(_lognormal((32, 32, 32), 1.0, 21))
    cfg = dict(cg_rtol=1e-10, cg_check_every=1, conv_norm=M.CONV_B)
    big = M.HeadSolver(g, M.BCSpec.darcy_x(), M.HeadSolveConfig(mg_levels=5, **cfg))
    small = M.HeadSolver(g, M.BCSpec.darcy_x(), M.HeadSolveConfig(mg_levels=2, **cfg))
    for s in (big, small, big):
        s.set_K(K)
        h = _t(np.zeros((32, 32, 32)))
        assert s.solve(h).converged


def test_graph_and_host_loop_identical(mf3d):
    M = mf3d
    shape = (32, 32, 32)
    K = _t(_lognormal(shape, 1.5, 13))
    g = M.Grid3D(32, 32, 32, 1.0)
    out = []
    for ug in (1, 0):
        cfg = M.HeadSolveConfig(mg_levels=4, cg_rtol=1e-10, cg_check_every=1, use_graph=ug)
        s = M.HeadSolver(g, M.BCSpec.darcy_x(), cfg)
        s.set_K(K)
        h = _t(np.zeros(shape))
        r = s.solve(h)
        out.append((r.num_iterations, _np(h)))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])  # deterministic reductions: bitwise equal


def test_repeated_solves_deterministic(mf3d):
    M = mf3d
    shape = (32, 32, 64)
    K = _t(_lognormal(shape, 1.0, 14))
    g = M.Grid3D(64, 32, 32, 1.0)
    s = M.HeadSolver(g, M.BCSpec.darcy_x(), M.HeadSolveConfig(mg_levels=4, cg_rtol=1e-10))
    s.set_K(K)
    hs = []
    for _ in range(3):
        h = _t(np.zeros(shape))
        s.solve(h)
        hs.append(_np(h))
    assert np.array_equal(hs[0], hs[1]) and np.array_equal(hs[1], hs[2])


def test_velocity_mass_balance_after_solve(mf3d, oracle_mod):
    M, O = mf3d, oracle_mod
    shape = (32, 32, 32)
    K = _lognormal(shape, 1.0, 15)
    g = M.Grid3D(32, 32, 32, 1.0)
    bc = M.BCSpec.darcy_x()
    s = M.HeadSolver(g, bc, M.HeadSolveConfig(mg_levels=4, cg_rtol=1e-12, cg_check_every=1,
                                              conv_norm=M.CONV_B))
    Kt = _t(K)
    s.set_K(Kt)
    h = _t(np.zeros(shape))
    s.solve(h)
    su, sv, sw = M.velocity_sizes(g)
    U, V, W = _t(np.zeros(su)), _t(np.zeros(sv)), _t(np.zeros(sw))
    mx, qin, qout = M.velocity_mass_balance(U, V, W, h, Kt, g, bc)
    assert mx / abs(qin) < 1e-10 and abs(qin - qout) / abs(qin) < 1e-10
    Uo, _, _ = O.velocity(_np(h), K, O.baseline_bc())
    assert _rel(_np(U), Uo.ravel()) < 1e-14


def test_warm_start_and_nonconvergence_reporting(mf3d):
    M = mf3d
    shape = (32, 32, 32)
    K = _t(_lognormal(shape, 1.0, 16))
    g = M.Grid3D(32, 32, 32, 1.0)
    s = M.HeadSolver(g, M.BCSpec.darcy_x(), M.HeadSolveConfig(mg_levels=4, cg_rtol=1e-10,
                                                              cg_check_every=1, conv_norm=M.CONV_B))
    s.set_K(K)
    h = _t(np.zeros(shape))
    r1 = s.solve(h)
    h2 = _t(np.zeros(shape))
    r2 = s.solve(h2, x0=h)  # warm start from the converged head
    assert r2.num_iterations <= 1 and r2.converged
    s3 = M.HeadSolver(g, M.BCSpec.darcy_x(), M.HeadSolveConfig(mg_levels=4, cg_rtol=1e-14,
                                                               cg_max_iter=3, cg_check_every=1))
    s3.set_K(K)
    r3 = s3.solve(h2)
    assert not r3.converged and r3.num_iterations == 3 and r1.converged


def test_nonfinite_K_reports_status(mf3d):
    M = mf3d
    shape = (16, 16, 16)
    Kn = _lognormal(shape, 1.0, 17)
    Kn[3, 4, 5] = np.nan
    g = M.Grid3D(16, 16, 16, 1.0)
    s = M.HeadSolver(g, M.BCSpec.darcy_x(), M.HeadSolveConfig(mg_levels=3, cg_rtol=1e-10))
    s.set_K(_t(Kn))
    res = s.solve(_t(np.zeros(shape)))
    assert not res.converged and res.status == 2


def test_kfield_vs_oracle(mf3d, oracle_mod):
    M, O = mf3d, oracle_mod
    g = M.Grid3D(37, 9, 5, 1.0)
    modes = M.kfield_modes(99, 1000, M.COV_EXPONENTIAL, (4.0, 4.0, 2.0))
    lnk = M.generate_K_field(g, 2.0, (4.0, 4.0, 2.0), seed=99, log_only=True)
    ref = O.lnk_eval((5, 9, 37), modes, np.sqrt(2.0))
    assert np.abs(_np(lnk) - ref).max() < 1e-9
    K = M.generate_K_field(g, 2.0, (4.0, 4.0, 2.0), seed=99)
    assert np.allclose(_np(K), np.exp(ref), rtol=1e-9)


def test_host_kfield_equals_device_kfield(mf3d, oracle_mod):
    """The oracle's host generator (the reference arm's K) and the product's device generator
    give the same field at the headline statistics (sigma^2 = 4, lambda = 8, 1000 modes)."""
    M, O = mf3d, oracle_mod
    g = M.Grid3D(64, 48, 40, 1.0)
    K = M.generate_K_field(g, 4.0, (8.0, 8.0, 8.0), seed=20240601, n_modes=1000)
    Ko = O.generate_K((40, 48, 64), 4.0, (8.0, 8.0, 8.0), seed=20240601, n_modes=1000)
    assert _rel(_np(K), Ko) < 1e-12


@pytest.mark.parametrize("prec", [0, 1])
def test_standalone_mg_solver_vs_oracle(mf3d, oracle_mod, prec):
    """solver = mg: V-cycles on the current head until ||r||/||r0|| < rtol
    (mg_solve, src/multigrid/cycle/v_cycle.cu:76-116)."""
    M, O = mf3d, oracle_mod
    shape = (32, 32, 32)
    K = _lognormal(shape, 1.0, 21)
    g = M.Grid3D(32, 32, 32, 1.0)
    cfg = M.HeadSolveConfig(solver_type=M.SOLVER_MG, mg_levels=4, mg_max_cycles=60, rtol=1e-10,
                            precision=prec)
    s = M.HeadSolver(g, M.BCSpec.darcy_x(), cfg)
    s.set_K(_t(K))
    h = _t(np.zeros(shape))
    res = s.solve(h)
    ho, ro = O.solve_head_mg(K, O.baseline_bc(), 4, max_cycles=60, rtol=1e-10)
    assert res.converged and ro.converged
    if prec == 0:
        assert abs(res.num_iterations - ro.iterations) <= 1
    assert _rel(_np(h), ho) < 1e-8


def test_plain_cg_solver_vs_oracle(mf3d, oracle_mod):
    """solver = cg: unpreconditioned CG (cg_solve, src/numerics/solvers/cg.cuh:14-171)."""
    M, O = mf3d, oracle_mod
    shape = (16, 16, 16)
    K = _lognormal(shape, 0.5, 22)
    g = M.Grid3D(16, 16, 16, 1.0)
    cfg = M.HeadSolveConfig(solver_type=M.SOLVER_CG, cg_max_iter=800, cg_check_every=1, cg_rtol=1e-9)
    s = M.HeadSolver(g, M.BCSpec.darcy_x(), cfg)
    s.set_K(_t(K))
    h = _t(np.zeros(shape))
    res = s.solve(h)
    ho, ro = O.solve_head_cg(K, O.baseline_bc(), max_iter=800, check_every=1, rtol=1e-9)
    assert res.converged and ro.converged
    assert abs(res.num_iterations - ro.iterations) <= 2
    assert _rel(_np(h), ho) < 1e-7


@pytest.mark.parametrize("case", BC_CASES, ids=[c[0] for c in BC_CASES])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_pcg_every_bc_case_vs_oracle(mf3d, oracle_mod, case, prec):
    """PCG (search-direction update fused with the matvec) on every boundary kind: periodic
    wrap, the pinned cell, all-Dirichlet; 40 x 20 x 12 leaves partial column tiles in x and y
    and halves evenly through the three levels (the CUDA hierarchy stops at an odd axis)."""
    M, O = mf3d, oracle_mod
    name, types, values, _ = case
    shape = (12, 20, 40)
    K = _lognormal(shape, 1.0, zlib.crc32(name.encode()))
    g = M.Grid3D(shape[2], shape[1], shape[0], 1.0)
    P = {"fp64": M.PREC_FP64, "fp32": M.PREC_FP32}[prec]
    cfg = M.HeadSolveConfig(mg_levels=3, cg_rtol=1e-10, cg_check_every=1, precision=P)
    # a random initial guess: with no Dirichlet face the right-hand side is zero, and the
    # pinned system then iterates from x0 towards h = 0
    x0 = np.random.default_rng(5).normal(size=shape)
    s = M.HeadSolver(g, _bcs(M, types, values), cfg)
    s.set_K(_t(K))
    h = _t(np.zeros(shape))
    res = s.solve(h, _t(x0))
    ho, ro = O.solve_head_pcg(K, O.make_bc(types, values), 3, rtol=1e-10, check_every=1, h0=x0)
    assert res.converged and ro.converged and ro.iterations > 3
    if prec == "fp64":
        assert abs(res.num_iterations - ro.iterations) <= 1
    assert np.abs(_np(h) - ho).max() / max(np.abs(ho).max(), np.abs(x0).max()) < 1e-8
    s.close()


@pytest.mark.parametrize("case", BC_CASES, ids=[c[0] for c in BC_CASES])
def test_plain_cg_every_bc_case_vs_oracle(mf3d, oracle_mod, case):
    """Plain CG (z = r, the FP64 form of the fused update) on every boundary kind."""
    M, O = mf3d, oracle_mod
    name, types, values, _ = case
    shape = (10, 18, 36)
    K = _lognormal(shape, 0.5, zlib.crc32(("cg" + name).encode()))
    g = M.Grid3D(shape[2], shape[1], shape[0], 1.0)
    cfg = M.HeadSolveConfig(solver_type=M.SOLVER_CG, cg_max_iter=3000, cg_check_every=1, cg_rtol=1e-10)
    s = M.HeadSolver(g, _bcs(M, types, values), cfg)
    s.set_K(_t(K))
    h = _t(np.zeros(shape))
    res = s.solve(h)
    ho, ro = O.solve_head_cg(K, O.make_bc(types, values), max_iter=3000, check_every=1, rtol=1e-10)
    assert res.converged and ro.converged
    assert abs(res.num_iterations - ro.iterations) <= 2
    assert _rel(_np(h), ho) < 1e-7
    s.close()


@pytest.mark.parametrize("shape", [(24, 20, 32), (2, 6, 8), (9, 5, 3)])
@pytest.mark.parametrize("layout", [0, 1])
def test_velocity_diagnostics_vs_oracle(mf3d, oracle_mod, shape, layout):
    """compute_velocity_diagnostics on the velocity of a solved head: divergence, |curl u| and
    helicity per cell and their min / max / mean, against the oracle (1e-12 of each field's
    max); (2, 6, 8) has a dimension below 3 (no curl)."""
    M, O = mf3d, oracle_mod
    K = _lognormal(shape, 1.0, 21)
    g = M.Grid3D(shape[2], shape[1], shape[0], 0.5)
    bc = M.BCSpec.darcy_x()
    s = M.HeadSolver(g, bc, M.HeadSolveConfig(mg_levels=2, cg_rtol=1e-12, cg_check_every=1))
    Kt = _t(K)
    s.set_K(Kt)
    h = _t(np.zeros(shape))
    s.solve(h)
    su, sv, sw = M.velocity_sizes(g, layout)
    U, V, W = _t(np.zeros(su)), _t(np.zeros(sv)), _t(np.zeros(sw))
    M.compute_velocity_from_head(U, V, W, h, Kt, g, bc, layout)
    div, om, he = _t(np.zeros(shape)), _t(np.zeros(shape)), _t(np.zeros(shape))
    st = M.velocity_diagnostics(U, V, W, g, layout, div, om, he)
    Un, Vn, Wn = _np(U), _np(V), _np(W)
    if layout == 0:
        Un = Un.reshape(shape[0], shape[1], shape[2] + 1)
        Vn = Vn.reshape(shape[0], shape[1] + 1, shape[2])
        Wn = Wn.reshape(shape[0] + 1, shape[1], shape[2])
    else:
        Un, Vn, Wn = (a.reshape(shape[0] + 1, shape[1] + 1, shape[2] + 1) for a in (Un, Vn, Wn))
    do, oo, ho, so = O.velocity_diagnostics(Un, Vn, Wn, shape, 0.5, layout)
    scale = max(np.abs(_np(U)).max(), 1e-300)
    for a, o in ((div, do), (om, oo), (he, ho)):
        assert np.abs(_np(a) - o).max() <= 1e-12 * max(np.abs(o).max(), scale)
    got = np.array(st["div"] + st["vorticity_mag"] + st["helicity"])
    assert np.allclose(got, so, rtol=1e-12, atol=1e-12 * scale ** 2)
    if min(shape) < 3:
        assert not _np(om).any() and not _np(he).any()
    # fields may be skipped; the statistics stay the same
    st2 = M.velocity_diagnostics(U, V, W, g, layout)
    assert st2 == st


@pytest.mark.parametrize("use_graph", [1, 0])
def test_time_budget_ends_the_loop_and_the_solver_recovers(mf3d, use_graph):
    """The device-time budget bounds a solve independently of the reductions: with a budget of
    one microsecond the loop's first kernel stops it (status 3, not converged) in the graph
    and in the host-driven loop; with the budget restored the same solver converges."""
    M = mf3d
    shape = (64, 64, 64)
    K = _lognormal(shape, 1.0, 31)
    g = M.Grid3D(64, 64, 64, 1.0)
    s = M.HeadSolver(g, M.BCSpec.darcy_x(), M.HeadSolveConfig(mg_levels=5, cg_rtol=1e-10, cg_check_every=1,
                                                             use_graph=use_graph))
    s.set_K(_t(K))
    h = _t(np.zeros(shape))
    s.set_time_budget(1e-6)
    res = s.solve(h)
    assert res.status == 3 and not res.converged, res
    assert res.num_iterations <= 2
    s.set_time_budget(120.0)
    res = s.solve(h)
    assert res.status == 0 and res.converged and res.true_rel_residual < 1e-9, res
    with pytest.raises(Exception):
        s.set_time_budget(0.0)


def test_bounded_mbarrier_waits_give_up_and_leave_the_context_usable(mf3d):
    """The bounded waits of the staged smoother and of the tensor-core convolution give up on a
    barrier that nothing completes and succeed on one that an arrival completes; the context
    then still runs a solve."""
    M = mf3d
    for which in (0, 1):
        assert M.diag_bounded_wait(which, False, 64)
        assert not M.diag_bounded_wait(which, True, 64)
    g = M.Grid3D(16, 16, 16, 1.0)
    s = M.HeadSolver(g, M.BCSpec.darcy_x(), M.HeadSolveConfig(mg_levels=3, cg_rtol=1e-10, cg_check_every=1))
    s.set_K(_t(_lognormal((16, 16, 16), 1.0, 3)))
    res = s.solve(_t(np.zeros((16, 16, 16))))
    assert res.converged


# the three tile shapes of the K generator (small fields; an even and an odd number of 32-cell column
# blocks), ragged rows and columns, single rows and columns, a mode count that is no multiple of the batch
@pytest.mark.parametrize("shape,modes", [((1, 1, 1), 1), ((3, 5, 31), 17), ((33, 40, 70), 100), ((90, 97, 64), 33),
                                         ((60, 71, 160), 48), ((200, 120, 33), 20)])
def test_kfield_tile_shapes_vs_oracle(mf3d, oracle_mod, shape, modes):
    """Phases reach about 1e4 here, so a mode is off by at most a few 1e-12 of its amplitude."""
    M, O = mf3d, oracle_mod
    g = M.Grid3D(shape[2], shape[1], shape[0], 0.7)
    table = M.kfield_modes(5, modes, M.COV_EXPONENTIAL, (4.0, 3.0, 2.0))
    lnk = _np(M.generate_K_field(g, 1.5, (4.0, 3.0, 2.0), seed=5, n_modes=modes, log_only=True))
    x = [(np.arange(n) + 0.5) * 0.7 for n in (shape[2], shape[1], shape[0])]
    ref = np.zeros(shape)
    for k1, k2, k3, a, b in table.T:
        ph = (k3 * x[2])[:, None, None] + (k2 * x[1])[None, :, None] + (k1 * x[0])[None, None, :]
        ref += a * np.sin(ph) + b * np.cos(ph)
    ref *= np.sqrt(1.5 / modes)
    assert np.abs(lnk - ref).max() < 1e-10
    K = _np(M.generate_K_field(g, 1.5, (4.0, 3.0, 2.0), seed=5, n_modes=modes, K_geo=2.0))
    assert np.allclose(K, 2.0 * np.exp(ref), rtol=1e-9)


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 3, 2), (5, 1, 33), (7, 9, 32), (6, 17, 65), (40, 8, 31)])
@pytest.mark.parametrize("per", [False, True])
def test_velocity_and_diagnostics_edges_vs_numpy(mf3d, shape, per):
    """Padded velocities and their diagnostics on tiles of one cell to ragged ones, against numpy's
    evaluation of the same formulas (a handful of roundings: 1e-13 of each field's largest value)."""
    M = mf3d
    nz, ny, nx = shape
    r = np.random.default_rng(nx + 10 * ny + 100 * nz)
    K, h, dx = np.exp(r.normal(size=shape)), r.normal(size=shape), 0.5
    faces = [M.BCFace(M.DIRICHLET, 1.0), M.BCFace(M.DIRICHLET, -0.5)]
    bc = M.BCSpec(faces + [M.BCFace(M.PERIODIC if per else M.NEUMANN, 0.0) for _ in range(4)])
    g = M.Grid3D(nx, ny, nz, dx)
    bufs = [_t(np.zeros(n)) for n in M.velocity_sizes(g, M.VEL_PADDED)]
    M.compute_velocity_from_head(*bufs, _t(h), _t(K), g, bc, M.VEL_PADDED)

    def flux(a, b, ha, hb):
        return 2.0 * a * b * (ha - hb) / ((a + b) * dx)

    ref = []
    for ax in (2, 1, 0):
        n = shape[ax]
        t = lambda v, lo, hi: np.take(v, np.arange(lo, hi), ax)  # noqa: E731
        q = flux(t(K, 0, n - 1), t(K, 1, n), t(h, 0, n - 1), t(h, 1, n))
        K0, K1, h0, h1 = t(K, 0, 1), t(K, n - 1, n), t(h, 0, 1), t(h, n - 1, n)
        if ax == 2:
            lo, hi = -K0 * (h0 - 1.0) / (dx / 2), -K1 * (-0.5 - h1) / (dx / 2)
        else:
            lo = hi = flux(K1, K0, h1, h0) if per else np.zeros_like(K0)
        ref.append(np.concatenate([lo, q, hi], ax))
    got = [_np(b).reshape(nz + 1, ny + 1, nx + 1) for b in bufs]
    for a, o in zip(got, ref):
        assert np.abs(a[:o.shape[0], :o.shape[1], :o.shape[2]] - o).max() <= 1e-13 * max(np.abs(o).max(), 1.0)
    u, v, w = ref
    div = ((u[..., 1:] - u[..., :-1]) + (v[:, 1:] - v[:, :-1]) + (w[1:] - w[:-1])) / dx
    om, he = np.zeros(shape), np.zeros(shape)
    if min(shape) >= 3:
        c = [0.5 * (u[..., 1:] + u[..., :-1]), 0.5 * (v[:, 1:] + v[:, :-1]), 0.5 * (w[1:] + w[:-1])]
        i = (slice(1, -1),) * 3

        def d(a, ax):
            s = [slice(1, -1)] * 3
            lo, hi = list(s), list(s)
            lo[ax], hi[ax] = slice(0, -2), slice(2, None)
            return (a[tuple(hi)] - a[tuple(lo)]) * (0.5 / dx)

        ox, oy, oz = d(c[2], 1) - d(c[1], 0), d(c[0], 0) - d(c[2], 2), d(c[1], 2) - d(c[0], 1)
        om[i] = np.sqrt(ox ** 2 + oy ** 2 + oz ** 2)
        he[i] = c[0][i] * ox + c[1][i] * oy + c[2][i] * oz
    out = [_t(np.full(shape, np.nan)) for _ in range(3)]
    st = M.velocity_diagnostics(*bufs, g, M.VEL_PADDED, *out)
    for a, o, s in zip(out, (div, om, he), (st["div"], st["vorticity_mag"], st["helicity"])):
        scale = max(np.abs(o).max(), np.abs(u).max() / dx)
        assert np.abs(_np(a) - o).max() <= 1e-13 * max(scale, scale ** 2)
        assert np.allclose(s, (o.min(), o.max(), o.mean()), rtol=1e-11, atol=1e-11 * max(scale, scale ** 2))


# the coarse end by its ways: bricks above a matrix with ragged bricks; the cluster with a coarsest level of 1680
# cells, and with a cell of each colour per thread (6175 cells); an odd periodic count on the coarsest level
# (bricks and matrix); a matrix from the coarsest of two levels on; a hierarchy that is one matrix
@pytest.mark.parametrize("shape,levels,per,way", [
    ((24, 40, 56), 4, False, "bricks_matrix"), ((20, 24, 28), 2, False, "cluster"), ((26, 38, 50), 2, False, "cluster"),
    ((48, 96, 80), 5, True, "bricks_matrix"), ((12, 20, 36), 3, True, "bricks_matrix"),
    ((8, 10, 12), 2, False, "bricks_matrix"), ((8, 8, 8), 2, False, "bricks_matrix")])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_coarse_end_ways_match_one_cta_tail(mf3d, monkeypatch, shape, levels, per, way, prec):
    """Against the same V-cycle with sweeps down to the one-CTA tail (no bricks either): the same arithmetic in
    another order, so equal to rounding (1e-12 in FP64, 1e-5 where FP32 levels are swept by another kernel)."""
    M = mf3d
    rng = np.random.default_rng(sum(shape) + levels)
    K, r = np.exp(rng.normal(size=shape)), rng.normal(size=shape)
    g = M.Grid3D(shape[2], shape[1], shape[0], 0.5)
    bc = _bcs(M, [D, D] + ([P, P, P, P] if per else [N, N, N, N]), [1.0, 0.0, 0, 0, 0, 0])
    cfg = M.HeadSolveConfig(mg_levels=levels, precision={"fp64": M.PREC_FP64, "fp32": M.PREC_FP32}[prec])
    z = []
    for tail in (False, True):
        if tail:
            monkeypatch.setenv("MF3D_NO_CLUSTER_TAIL", "1")
            monkeypatch.setenv("MF3D_NO_BRICKS", "1")
        s = M.HeadSolver(g, bc, cfg)
        s.set_K(_t(K))
        zz = _t(np.zeros(shape))
        s.vcycle(_t(r), zz)
        z.append(_np(zz))
        assert _coarse_way(s) == ["coarse_" + ("tail" if tail else way)]
        assert not tail or not [n for n, *_ in s.profile(1) if n.startswith("brick")]
        s.close()
    assert _rel(z[0], z[1]) < (1e-12 if prec == "fp64" else 1e-5)


def _coarse_way(s):
    """The way that the FP64 levels of a single solve go: the name of its entry in the profile."""
    return [name for name, *_ in s.profile(1) if name.startswith("coarse_")]


# where the matrix of the coarsest levels pays within a solve's own cycles and where it does not: too many cells
# (1728, 1100), a grid that is one level, few sweeps; at the limits (1000 coarsest cells; 1000 with levels below, and
# with many sweeps 125 of them; 512 of a full hierarchy; 20 sweeps)
@pytest.mark.parametrize("shape,levels,sweeps,way", [
    ((24, 24, 24), 2, 50, "cluster"), ((44, 40, 40), 3, 50, "cluster"), ((8, 16, 16), 1, 400, "cluster"),
    ((7, 7, 7), 1, 50, "cluster"), ((28, 28, 28), 3, 5, "cluster"),
    ((20, 20, 20), 2, 50, "bricks_matrix"), ((40, 40, 40), 3, 50, "bricks_matrix"),
    ((28, 28, 28), 3, 20, "bricks_matrix"), ((64, 64, 64), 16, 50, "bricks_matrix"), ((64, 64, 64), 16, 400, "bricks_matrix"),
    ((20, 20, 20), 3, 50, "bricks_matrix"), ((20, 20, 20), 3, 400, "bricks_matrix"),
    ((40, 44, 36), 3, 50, "bricks_matrix")])
def test_matrix_where_it_pays(mf3d, monkeypatch, shape, levels, sweeps, way):
    """The way chosen, its memory (a matrix of at most 1024 x 1024), and the V-cycle against the cluster's: the same
    cycle summed in another order, equal to rounding (1e-12 of the largest value)."""
    M = mf3d
    rng = np.random.default_rng(sum(shape) + levels + sweeps)
    K, r = np.exp(rng.normal(size=shape)), rng.normal(size=shape)
    g = M.Grid3D(shape[2], shape[1], shape[0], 0.5)
    cfg = M.HeadSolveConfig(mg_levels=levels, mg_coarse_iters=sweeps)
    z, size = [], []
    for off in (False, True):
        if off:
            monkeypatch.setenv("MF3D_NO_MATRIX", "1")
        s = M.HeadSolver(g, M.BCSpec.darcy_x(), cfg)
        s.set_K(_t(K))
        zz = _t(np.zeros(shape))
        s.vcycle(_t(r), zz)
        z.append(_np(zz))
        size.append(s.device_bytes)
        assert _coarse_way(s) == ["coarse_" + ("cluster" if off else way)]
        s.close()
    monkeypatch.delenv("MF3D_NO_MATRIX", raising=False)
    assert _rel(z[0], z[1]) < 1e-12
    assert size[0] - size[1] <= (10 << 20)
    if way == "cluster":
        assert size[0] == size[1]
    if shape == (20, 20, 20) and levels == 3:  # a matrix of 1000 x 1000, or of 125 x 125
        assert (size[0] - size[1] > (4 << 20)) == (sweeps == 50)


# several batches of modes (the last one ragged), several parts along one axis or all (ragged, of one cell), no
# tables at all
@pytest.mark.parametrize("shape,modes,table,axis", [((9, 14, 70), 50, 1, 1 << 16), ((21, 17, 33), 100, 3 * 8 * 16 * 102, 1 << 16),
                                                    ((20, 7, 150), 37, 1 << 20, 64), ((23, 40, 9), 24, 1 << 20, 11),
                                                    ((33, 20, 70), 41, 1, 32), ((5, 3, 4), 9, 1, 1),
                                                    ((9, 14, 70), 50, 0, 1 << 16), ((23, 40, 9), 24, 0, 11)])
def test_kfield_in_parts_vs_numpy(mf3d, shape, modes, table, axis):
    """lnK and K from every split of a field against the sum over the modes (as in the test of the tile shapes)."""
    import ctypes as C
    import torch
    M = mf3d
    from macroflow3d_b200 import _lib
    g = M.Grid3D(shape[2], shape[1], shape[0], 0.7)
    tab = M.kfield_modes(5, modes, M.COV_EXPONENTIAL, (4.0, 3.0, 2.0))
    x = [(np.arange(n) + 0.5) * 0.7 for n in (shape[2], shape[1], shape[0])]
    ref = np.zeros(shape)
    for k1, k2, k3, a, b in tab.T:
        ph = (k3 * x[2])[:, None, None] + (k2 * x[1])[None, :, None] + (k1 * x[0])[None, None, :]
        ref += a * np.sin(ph) + b * np.cos(ph)
    ref *= np.sqrt(1.5 / modes)
    dev = torch.from_numpy(np.ascontiguousarray(tab)).cuda()
    for want_exp in (0, 1):
        out = torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")
        M.check(_lib.lib().mf3d_diag_kfield_parts(C.byref(g.c()), modes, dev.data_ptr(), 1.5, float(np.log(2.0)), want_exp,
                                                  table, axis, out.data_ptr(), 0))
        if want_exp:
            assert np.allclose(_np(out), 2.0 * np.exp(ref), rtol=1e-9)
        else:
            assert np.abs(_np(out) - ref).max() < 1e-10


def test_kfield_keeps_little_device_memory(mf3d):
    """Tables of a 65536-cell axis and 2000 modes (2.1 GB at once) go in batches: the library keeps no more than
    32 MiB of the device afterwards, and 40 MiB with what the driver rounds up."""
    import torch
    M = mf3d
    g = M.Grid3D(65536, 4, 2, 0.7)
    M.generate_K_field(M.Grid3D(64, 4, 2, 0.7), 1.0, seed=1, n_modes=8)  # (context, module and pool)
    torch.cuda.synchronize()
    out = torch.empty((2, 4, 65536), dtype=torch.float64, device="cuda")
    del out  # (the cached block that the call below takes)
    free = torch.cuda.mem_get_info()[0]
    lnk = M.generate_K_field(g, 1.0, (4.0, 4.0, 4.0), seed=3, n_modes=2000, log_only=True)
    assert bool(torch.isfinite(lnk).all())
    assert free - torch.cuda.mem_get_info()[0] <= 40 << 20


@pytest.mark.parametrize("prec,ez", [("fp64", 8), ("fp32", 4)])
def test_profile_counts_the_head_update(mf3d, prec, ez):
    """The profile's matvec is the mean over iterations with and without the two steps of the head update (24 bytes
    a cell every second iteration, 12 on average), and a solve after it repeats the one before it."""
    M = mf3d
    n = (40, 48, 64)
    s = M.HeadSolver(M.Grid3D(64, 48, 40, 1.0), M.BCSpec.darcy_x(),
                     M.HeadSolveConfig(mg_levels=8, cg_rtol=1e-10, cg_check_every=1, precision=getattr(M, "PREC_" + prec.upper())))
    s.set_K(_t(_lognormal(n, 1.0, 7)))
    h0, h1 = _t(np.zeros(n)), _t(np.zeros(n))
    r0 = s.solve(h0)
    got = {name: (ms, nbytes, per) for name, ms, nbytes, per in s.profile(3)}["pupdate_matvec_dot"]
    assert got[0] > 0 and got[1] == (60 + ez) * 64 * 48 * 40 and got[2] == 1
    r1 = s.solve(h1)
    assert r0.num_iterations == r1.num_iterations and np.array_equal(_np(h0), _np(h1))
    s.close()
