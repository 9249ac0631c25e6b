"""Batched ensemble solves (mf3d_batch_*) against one HeadSolver per realisation.

A batch replaces the realisation loop of run_ensemble (src/runtime/ensemble/
EnsembleRunner.cu:259-317), so every realisation must come out as its own single solve would:
same iteration count (the batch changes only the summation order of the in-sweep <r, z>), the
same head to well below the solve tolerance, and the per-realisation stopping test must freeze
a realisation once it has converged while the others iterate.  Grids are uneven on purpose:
different level counts, levels with and without a staged (TMA) form, non-cubic coarse grids.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# both arms stop at ||r||/||b|| <= 1e-10; their iterates differ by rounding only
HEAD_TOL = 1e-8
# after a fixed number of iterations the iterates agree to rounding (the batch sums the
# in-sweep <r, z> per work item, the single solve per CTA).  In FP32 the single solve smooths
# with the x-pair sweep and the batch with the quad sweep, two kernels that round differently
# in FP32 (measured up to 2.4e-6 after six iterations on these grids); in FP64 both agree to
# 1e-14.  Converged heads are compared at HEAD_TOL, and with the oracle in test_batch_vs_oracle
ITERATE_TOL = {"fp32": 1e-4, "fp64": 1e-10}
# ||r|| after six iterations (1e-5 of ||r0||) relative to each other: a single solve takes
# the residual of the last pre-sweep in a kernel of its own, the batch inside the fused sweep;
# in FP32 the two sweep kernels also round differently, and a 1e-7 difference in the V-cycle's
# output becomes several per cent of a residual six digits below ||r0|| (measured up to 6%):
# FP32 only asks for the same convergence rate (within a factor 1.5)
RESID_TOL = {"fp32": 0.5, "fp64": 1e-6}
# near the stopping threshold the plain FP64 method (Fletcher-Reeves beta with the reference's
# non-symmetric V-cycle) converges unevenly, so a rounding difference can move the stop by an
# iteration or two; the flexible mixed-precision method does not
ITER_SLACK = {"fp32": 1, "bf16": 1, "fp64": 2}


def _grids(M):
    # 36: level 1 is 18 wide (not 16-byte aligned: L1 sweep); 48x40x24: three sweep levels
    shapes = [(32, 32, 32), (48, 40, 24), (36, 32, 32), (64, 32, 48), (32, 64, 40)]
    return [M.Grid3D(nx, ny, nz, 1.0) for nx, ny, nz in shapes]


def _cfg(M, prec, **kw):
    c = dict(mg_levels=8, cg_rtol=1e-10, cg_check_every=1, conv_norm=M.CONV_B, precision=prec)
    c.update(kw)
    return M.HeadSolveConfig(**c)


def _fields(M, grids, sigma2=2.0, lam=6.0, seed=100):
    return [M.generate_K_field(g, sigma2, (lam, lam, lam), seed=seed + r) for r, g in enumerate(grids)]


def _single(M, grids, bc, cfg, Ks):
    import torch
    out = []
    for g, K in zip(grids, Ks):
        s = M.HeadSolver(g, bc, cfg, stream=torch.cuda.current_stream().cuda_stream)
        s.set_K(K)
        h = torch.empty_like(K)
        res = s.solve(h)
        out.append((h.cpu().numpy(), res))
        s.close()
    return out


def _assert_batched(b):
    """The realisations are solved by batched launches: only these have sweeps to tune (ensembles of at most four
    small realisations, and large ones, are solved side by side by their own launches)."""
    assert b.autotune(1), "no realisation is batched"


def _batch(M, grids, bc, cfg, Ks, tune=False, x0s=None):
    import torch
    b = M.BatchSolver(grids, bc, cfg, stream=torch.cuda.current_stream().cuda_stream)
    b.set_K(Ks)
    tuning = b.autotune(2) if tune else None
    hs = [torch.full_like(K, float("nan")) for K in Ks]
    res = b.solve(hs, x0s)
    torch.cuda.synchronize()
    out = [(h.cpu().numpy(), r) for h, r in zip(hs, res)]
    return b, out, tuning


def _rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


@pytest.mark.parametrize("prec", ["fp32", "fp64", "bf16"])
def test_batch_matches_single_solves(mf3d, prec):
    M = mf3d
    P = {"fp32": M.PREC_FP32, "fp64": M.PREC_FP64, "bf16": M.PREC_BF16}[prec]
    grids = _grids(M)
    bc = M.BCSpec.darcy_x()
    cfg = _cfg(M, P)
    Ks = _fields(M, grids)
    ref = _single(M, grids, bc, cfg, Ks)
    b, got, _ = _batch(M, grids, bc, cfg, Ks)
    for (hr, rr), (hb, rb) in zip(ref, got):
        assert rr.converged and rb.converged, (rr, rb)
        assert np.all(np.isfinite(hb))
        assert abs(rb.num_iterations - rr.num_iterations) <= ITER_SLACK[prec], (rb.num_iterations, rr.num_iterations)
        assert rb.true_rel_residual <= 1e-10
        assert rb.num_levels == rr.num_levels
        assert _rel(hb, hr) < HEAD_TOL
    b.close()


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_batch_iterates_match_single_solves(mf3d, prec):
    """Six iterations, no convergence: the batched and the single iterates agree to rounding."""
    M = mf3d
    P = {"fp32": M.PREC_FP32, "fp64": M.PREC_FP64}[prec]
    grids = _grids(M)
    bc = M.BCSpec.darcy_x()
    cfg = _cfg(M, P, cg_max_iter=6)
    Ks = _fields(M, grids, seed=200)
    ref = _single(M, grids, bc, cfg, Ks)
    b, got, _ = _batch(M, grids, bc, cfg, Ks)
    for (hr, rr), (hb, rb) in zip(ref, got):
        assert rr.num_iterations == rb.num_iterations == 6 and not rb.converged
        assert _rel(hb, hr) < ITERATE_TOL[prec]
        assert abs(rb.final_residual - rr.final_residual) <= RESID_TOL[prec] * rr.final_residual, prec
    b.close()


def test_convergence_mask_freezes_finished_realisations(mf3d):
    """A homogeneous K converges in a few iterations, a sigma^2 = 4 field in many more; the
    easy realisation must report its own count and keep its own converged head."""
    import torch
    M = mf3d
    grids = [M.Grid3D(32, 32, 32, 1.0), M.Grid3D(48, 32, 32, 1.0), M.Grid3D(32, 48, 64, 1.0),
             M.Grid3D(32, 32, 40, 1.0), M.Grid3D(40, 32, 32, 1.0)]
    bc = M.BCSpec.darcy_x()
    cfg = _cfg(M, M.PREC_FP32)
    Ks = [torch.ones((32, 32, 32), dtype=torch.float64, device="cuda"),
          M.generate_K_field(grids[1], 4.0, (8.0, 8.0, 8.0), seed=5),
          M.generate_K_field(grids[2], 1.0, (4.0, 4.0, 4.0), seed=6),
          torch.ones((40, 32, 32), dtype=torch.float64, device="cuda"),
          M.generate_K_field(grids[4], 4.0, (8.0, 8.0, 8.0), seed=7)]
    for few in (False, True):  # all five as one batch; three of them side by side
        n = 3 if few else 5
        ref = _single(M, grids[:n], bc, cfg, Ks[:n])
        its = [r.num_iterations for _, r in ref]
        assert its[0] < its[1] - 3, its
        b, got, _ = _batch(M, grids[:n], bc, cfg, Ks[:n])
        for (hr, rr), (hb, rb) in zip(ref, got):
            assert rb.converged and abs(rb.num_iterations - rr.num_iterations) <= 1
            assert _rel(hb, hr) < HEAD_TOL
        if not few:
            _assert_batched(b)
        b.close()


def test_autotune_keeps_results(mf3d):
    M = mf3d
    grids = _grids(M)
    bc = M.BCSpec.darcy_x()
    cfg = _cfg(M, M.PREC_FP32)
    Ks = _fields(M, grids, seed=300)
    b0, base, _ = _batch(M, grids, bc, cfg, Ks)
    b1, tuned, tuning = _batch(M, grids, bc, cfg, Ks, tune=True)
    assert tuning and all(t["ms_best"] <= t["ms_default"] + 1e-9 for t in tuning)
    assert {t["path"] for t in tuning} <= {0, 1}  # quad, L1 (the batched x-pair sweep is off)
    for (h0, r0), (h1, r1) in zip(base, tuned):
        assert r1.converged and abs(r1.num_iterations - r0.num_iterations) <= 1
        assert _rel(h1, h0) < HEAD_TOL
    # solving again after tuning repeats the tuned result exactly (deterministic reductions)
    import torch
    hs = [torch.empty_like(K) for K in Ks]
    res = b1.solve(hs)
    torch.cuda.synchronize()
    for h, (h1, r1), r in zip(hs, tuned, res):
        assert r.num_iterations == r1.num_iterations
        assert np.array_equal(h.cpu().numpy(), h1)
    b0.close()
    b1.close()


@pytest.mark.parametrize("count", [5, 3])
def test_host_loop_equals_graph(mf3d, count):
    """Five realisations are one batch (its loop driven by the host polls the gate), three are side by side."""
    M = mf3d
    grids = _grids(M)[:count]
    bc = M.BCSpec.darcy_x()
    Ks = _fields(M, grids, seed=400)
    bg, g, _ = _batch(M, grids, bc, _cfg(M, M.PREC_FP32), Ks)
    bh, h, _ = _batch(M, grids, bc, _cfg(M, M.PREC_FP32, use_graph=0), Ks)
    for (ha, ra), (hb, rb) in zip(g, h):
        assert ra.num_iterations == rb.num_iterations
        assert np.array_equal(ha, hb)
    if count == 5:
        _assert_batched(bg)
        _assert_batched(bh)
    bg.close()
    bh.close()


@pytest.mark.parametrize("count", [5, 3])
def test_warm_start_and_iteration_cap(mf3d, count):
    """x0 per realisation (None entries use the reference guess); a cap of 3 iterations stops
    every realisation unconverged with 3 iterations.  Five realisations are one batch, three are side by side."""
    import torch
    M = mf3d
    grids = _grids(M)[:count]
    bc = M.BCSpec.darcy_x()
    Ks = _fields(M, grids, seed=500)
    b, got, _ = _batch(M, grids, bc, _cfg(M, M.PREC_FP32), Ks)
    x0s = [torch.from_numpy(got[0][0]).cuda(), None, torch.from_numpy(got[2][0]).cuda()] + [None] * (count - 3)
    hs = [torch.empty_like(K) for K in Ks]
    res = b.solve(hs, x0s)
    assert res[0].num_iterations <= 1 and res[2].num_iterations <= 1
    assert all(res[r].num_iterations == got[r][1].num_iterations for r in range(count) if x0s[r] is None)
    if count == 5:
        _assert_batched(b)
    b.close()
    bcap, capped, _ = _batch(M, grids, bc, _cfg(M, M.PREC_FP32, cg_max_iter=3), Ks)
    for _, r in capped:
        assert r.num_iterations == 3 and not r.converged
    bcap.close()


@pytest.mark.parametrize("count", [5, 3])
def test_nonfinite_realisation_does_not_stop_the_others(mf3d, count):
    """Five realisations are one batch, three are side by side."""
    import torch
    M = mf3d
    grids = _grids(M)[:count]
    bc = M.BCSpec.darcy_x()
    cfg = _cfg(M, M.PREC_FP32)
    Ks = _fields(M, grids, seed=600)
    Ks[1] = Ks[1].clone()
    Ks[1].view(-1)[17] = float("nan")
    rest = [r for r in range(count) if r != 1]
    ref = _single(M, [grids[r] for r in rest], bc, cfg, [Ks[r] for r in rest])
    b, got, _ = _batch(M, grids, bc, cfg, Ks)
    assert got[1][1].status == 2 and not got[1][1].converged
    for (hr, rr), (hb, rb) in zip(ref, [got[r] for r in rest]):
        assert rb.converged and abs(rb.num_iterations - rr.num_iterations) <= 1
        assert _rel(hb, hr) < HEAD_TOL
    if count == 5:
        _assert_batched(b)
    b.close()


def test_guesses_in_other_realisations_heads(mf3d):
    """Warm starts that lie in the arrays of other realisations' heads (arrays used in turn, a guess inside a larger
    head): every guess is read before any head is written, so each realisation starts from its converged head
    and is done after one step at most.  Six realisations are solved side by side, two on some streams, and
    five as one batch."""
    import torch
    M = mf3d
    grids = [M.Grid3D(64, 48, 80, 1.0)] * 6 + [M.Grid3D(32, 32, 32, 1.0)] * 5
    bc = M.BCSpec.darcy_x()
    cfg = _cfg(M, M.PREC_FP64)
    Ks = _fields(M, grids, seed=900)
    b, got, _ = _batch(M, grids, bc, cfg, Ks)
    _assert_batched(b)
    heads = [torch.from_numpy(h).cuda() for h, _ in got]
    hs = [torch.empty_like(K) for K in Ks]
    x0s = [None] * len(grids)
    for r in range(6):  # the head of r is in the array that realisation r + 1 writes
        x0s[r] = hs[(r + 1) % 6]
        x0s[r].copy_(heads[r])
    n = 32 ** 3
    for r in range(6, 9):  # a batched realisation's guess inside a larger array, from an odd cell on
        hs[r - 6].view(-1)[101:101 + n].copy_(heads[r].view(-1))
        x0s[r] = hs[r - 6].view(-1)[101:101 + n]
        x0s[(r - 7) % 6] = None  # (the guess that was there)
    x0s[9], x0s[10] = hs[10], hs[9]  # two batched ones crosswise
    x0s[9].copy_(heads[9])
    x0s[10].copy_(heads[10])
    assert sum(x is not None for x in x0s[:6]) == 3
    res = b.solve(hs, x0s)
    torch.cuda.synchronize()
    for r, one in enumerate(res):
        assert one.converged
        if x0s[r] is not None:
            assert one.num_iterations <= 1, r
        assert _rel(hs[r].cpu().numpy(), got[r][0]) < HEAD_TOL, r
    # all six crosswise, and a realisation's guess in its own head's array
    for r in range(6):
        x0s[r] = hs[(r + 1) % 6]
        x0s[r].copy_(heads[r])
    for r in range(6, 11):
        x0s[r] = hs[r]
    res = b.solve(hs, x0s)
    torch.cuda.synchronize()
    for r, one in enumerate(res):
        assert one.num_iterations <= 1 and _rel(hs[r].cpu().numpy(), got[r][0]) < HEAD_TOL, r
    b.close()


def test_missing_head_of_a_batched_realisation_refuses_the_call(mf3d):
    """A null head among the batched realisations is refused before a solve side by side starts: no other head
    is touched, and the next call works."""
    import torch
    M = mf3d
    from macroflow3d_b200 import _lib
    grids = [M.Grid3D(64, 48, 80, 1.0)] * 2 + [M.Grid3D(32, 32, 32, 1.0)] * 5
    Ks = _fields(M, grids, seed=950)
    b = M.BatchSolver(grids, M.BCSpec.darcy_x(), _cfg(M, M.PREC_FP64))
    b.set_K(Ks)
    hs = [torch.full_like(K, float("nan")) for K in Ks]
    torch.cuda.synchronize()
    ptrs = b._ptrs(hs, "h")
    ptrs[4] = None
    res = (_lib.SolveResult * len(grids))()
    assert _lib.lib().mf3d_batch_solve(b._h, ptrs, None, res) == _lib.MF3D_E_INVALID
    torch.cuda.synchronize()
    assert all(bool(torch.isnan(h).all()) for h in hs)
    assert all(r.converged for r in b.solve(hs))
    torch.cuda.synchronize()
    assert all(bool(torch.isfinite(h).all()) for h in hs)
    b.close()


def test_flags_of_several_realisations_end_one_call_only(mf3d):
    """Pipeline flags of two realisations solved side by side and of two batched ones: the call that meets them
    fails, and the next one has none left."""
    import torch
    M = mf3d
    from macroflow3d_b200 import _lib
    grids = [M.Grid3D(64, 48, 80, 1.0)] * 3 + [M.Grid3D(32, 32, 32, 1.0)] * 5
    Ks = _fields(M, grids, seed=970)
    b, got, _ = _batch(M, grids, M.BCSpec.darcy_x(), _cfg(M, M.PREC_FP64), Ks)
    hs = [torch.empty_like(K) for K in Ks]
    for which in ([0, 2], [1, 4, 6], [3, 7], [0, 1, 2, 3, 4, 5, 6, 7]):
        for r in which:
            M.check(_lib.lib().mf3d_diag_raise_pipeline_flag(b._h, r))
        with pytest.raises(M.Mf3dError, match="wait timed out"):
            b.solve(hs)
        res = b.solve(hs)
        torch.cuda.synchronize()
        for h, one, (hg, rg) in zip(hs, res, got):
            assert one.num_iterations == rg.num_iterations and np.array_equal(h.cpu().numpy(), hg)
    assert _lib.lib().mf3d_diag_raise_pipeline_flag(b._h, 8) == _lib.MF3D_E_INVALID
    b.close()


def test_reductions_of_successive_blocks_do_not_mix(mf3d):
    """Ninety-six small realisations: about four thousand virtual blocks of the r update and of the residual on
    at most eight CTAs a multiprocessor, so every CTA runs several blocks and the last block of one
    realisation's reduction is followed by a block of another.  Each solve must repeat the first one's counts,
    residual norms and heads to the last bit (the reductions are deterministic), and equal realisations must
    agree with each other: their blocks are cut alike and their sums ordered alike."""
    import torch
    M = mf3d
    base = [M.Grid3D(32, 32, 32, 1.0), M.Grid3D(48, 40, 24, 1.0), M.Grid3D(32, 64, 40, 1.0)]
    Kb = _fields(M, base, seed=800)
    grids, Ks = base * 32, Kb * 32
    b, first, _ = _batch(M, grids, M.BCSpec.darcy_x(), _cfg(M, M.PREC_FP64, cg_max_iter=30), Ks)
    _assert_batched(b)
    hs = [torch.empty_like(K) for K in Ks]
    b.solve(hs)  # (with the tuned sweeps, repeated below)
    tuned = None
    for _ in range(4):
        res = b.solve(hs)
        torch.cuda.synchronize()
        now = [(r.num_iterations, r.initial_residual, r.final_residual, r.true_rel_residual, r.b_norm) for r in res]
        heads = [h.cpu().numpy() for h in hs]
        if tuned is not None:
            assert now == tuned[0]
            assert all(np.array_equal(x, y) for x, y in zip(heads, tuned[1]))
        tuned = (now, heads)
        for r in range(3, len(grids)):
            assert now[r] == now[r % 3] and np.array_equal(heads[r], heads[r % 3]), r
    for r in range(3, len(grids)):
        assert first[r][1].final_residual == first[r % 3][1].final_residual, r
        assert np.array_equal(first[r][0], first[r % 3][0]), r
    ref = _single(M, base, M.BCSpec.darcy_x(), _cfg(M, M.PREC_FP64, cg_max_iter=30), Kb)
    for (hr, rr), (hb, rb) in zip(ref, first):
        assert rb.converged and abs(rb.num_iterations - rr.num_iterations) <= ITER_SLACK["fp64"]
        assert _rel(hb, hr) < HEAD_TOL
    b.close()


def test_grids_without_a_level_above_the_tail_are_refused(mf3d):
    """A grid that is all coarse tail is refused, batched or side by side."""
    M = mf3d
    for count in (1, 6):
        with pytest.raises(M.Mf3dError, match="above the coarse tail"):
            M.BatchSolver([M.Grid3D(8, 8, 8)] * count, M.BCSpec.darcy_x(), _cfg(M, M.PREC_FP32))


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_mixed_sizes_keep_their_places(mf3d, prec):
    """Realisations large enough to be solved side by side among seven small ones that are batched:
    every head, count and warm start belongs to its own realisation (compared with single solves, as
    above)."""
    import torch
    M = mf3d
    shapes = [(32, 32, 32), (96, 80, 64), (32, 40, 32), (40, 32, 32), (80, 64, 96), (32, 32, 40), (48, 32, 32),
              (32, 48, 32), (32, 32, 48)]
    grids = [M.Grid3D(*s) for s in shapes]
    bc = M.BCSpec.darcy_x()
    cfg = _cfg(M, getattr(M, "PREC_" + prec.upper()))
    Ks = _fields(M, grids, seed=700)
    ref = _single(M, grids, bc, cfg, Ks)
    b, got, _ = _batch(M, grids, bc, cfg, Ks)
    for (hr, rr), (hb, rb) in zip(ref, got):
        assert rb.converged and abs(rb.num_iterations - rr.num_iterations) <= ITER_SLACK[prec]
        assert rb.num_levels == rr.num_levels and _rel(hb, hr) < HEAD_TOL
    x0s = [None] * len(grids)
    for r in (0, 1, 7):
        x0s[r] = torch.from_numpy(got[r][0]).cuda()
    hs = [torch.empty_like(K) for K in Ks]
    res = b.solve(hs, x0s)
    for r, (h, one) in enumerate(zip(hs, res)):
        if x0s[r] is not None:
            assert one.num_iterations <= 1
        else:
            assert one.num_iterations == got[r][1].num_iterations
            assert np.array_equal(h.cpu().numpy(), got[r][0])
    b.close()


@pytest.mark.parametrize("way", ["batched", "side_by_side"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_batch_vs_oracle(mf3d, oracle_mod, prec, way):
    """Uneven realisations (non-cubic coarse grids), five small ones solved as one batch or three large ones side
    by side, each against the FP64 oracle at the same tolerance (the realisation loop the batch replaces:
    src/runtime/ensemble/EnsembleRunner.cu:259-317).  FP64: the reference algorithm, same
    iteration count, heads equal to rounding (measured 1e-14).  FP32 V-cycle: iterations within
    one, heads within the tolerance's reach (measured 1.2e-9)."""
    M, O = mf3d, oracle_mod
    shapes = {"batched": [(32, 48, 64), (48, 32, 64), (64, 32, 48), (64, 48, 32), (32, 32, 32)],
              "side_by_side": [(64, 96, 64), (96, 64, 128), (128, 64, 96)]}[way]
    grids = [M.Grid3D(*s) for s in shapes]
    Ks = _fields(M, grids, seed=500)
    cfg = _cfg(M, getattr(M, "PREC_" + prec.upper()))
    b, out, _ = _batch(M, grids, M.BCSpec.darcy_x(), cfg, Ks)
    if way == "batched":
        _assert_batched(b)
    else:
        assert not b.autotune(1)
    b.close()
    bc = O.baseline_bc()
    for (h, res), K, g in zip(out, Ks, grids):
        Kn = K.cpu().numpy()
        rhs = O.build_rhs(Kn, bc)
        r0 = np.linalg.norm(rhs - O.apply_A(Kn, O.init_guess(Kn.shape, bc), bc))
        ho, ro = O.solve_head_pcg(Kn, bc, 8, rtol=1e-10 * np.linalg.norm(rhs) / r0, check_every=1, max_iter=200)
        assert res.converged and ro.converged
        assert res.true_rel_residual <= 1e-10
        if prec == "fp64":
            assert res.num_iterations == ro.iterations
            assert _rel(h, ho) < 1e-12
        else:
            assert abs(res.num_iterations - ro.iterations) <= 1
            assert _rel(h, ho) < 5e-9
