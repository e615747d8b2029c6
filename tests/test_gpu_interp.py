"""GPU parity of the table gather / spread against the oracle.

Tolerances (FP32 arithmetic, FP64 table-index selection): relative L2
<= 1e-6 for the forward gather and <= 1e-5 for the adjoint spread, against the
reference's FP64 kernels (golden vectors, or oracle/_ref built from the
reference sources, or the bit-identical restatement when neither is here).
"""
from __future__ import annotations

import numpy as np
import pytest

import mirt_b200 as mb
import oracle
from conftest import load_golden, ref_impl, rel_l2

pytestmark = pytest.mark.gpu

FWD_TOL = 1e-6
ADJ_TOL = 1e-5


def _i32(v):
    return np.asarray(v, dtype=np.int32)


def _fwd(D, ck, h, J, L, tm, K, order):
    N = ck.shape[1]
    ckr = ck.reshape(tuple(K) + (N,), order="F")
    o = None if order is None else _i32([order])
    if D == 1:
        return mb.interp1_table_mex(ck, h[0], _i32(J), _i32(L), tm, o)
    if D == 2:
        return mb.interp2_table_mex(ckr, h[0], h[1], _i32(J), _i32(L), tm, o)
    if D == 3:
        return mb.interp3_table_mex(ckr, h[0], h[1], h[2], _i32(J), _i32(L), tm, o)
    return mb.interp4_table_mex(ckr, h[0], h[1], h[2], h[3], _i32(J), _i32(L), tm, o)


def _adj(D, fm, h, J, L, tm, K, order):
    o = None if order is None else _i32([order])
    if D == 1:
        return mb.interp1_table_adj_mex(fm, h[0], _i32(J), _i32(L), tm, _i32(K), o)
    if D == 2:
        return mb.interp2_table_adj_mex(fm, h[0], h[1], _i32(J), _i32(L), tm, _i32(K), o)
    if D == 3:
        return mb.interp3_table_adj_mex(fm, h[0], h[1], h[2], _i32(J), _i32(L), tm, _i32(K), o)
    return mb.interp4_table_adj_mex(fm, h[0], h[1], h[2], h[3], _i32(J), _i32(L), tm, _i32(K), o)


@pytest.mark.parametrize("i", range(24))
def test_mex_matches_golden(i):
    c = load_golden()[i]
    D = c["D"]
    fwd = _fwd(D, c["ck"], c["h"], c["J"], c["L"], c["tm"], c["K"], c["order"])
    assert fwd.shape == c["fwd"].shape
    assert rel_l2(fwd, c["fwd"]) <= FWD_TOL
    adj = _adj(D, c["fm"], c["h"], c["J"], c["L"], c["tm"], c["K"], c["order"])
    assert adj.shape == c["adj"].shape
    assert rel_l2(adj, c["adj"]) <= ADJ_TOL


def _radial(nspoke, nread):
    r = np.linspace(-np.pi, np.pi, nread, endpoint=False)
    ang = np.arange(nspoke) * np.pi / nspoke
    return np.stack([np.outer(np.cos(ang), r).ravel(), np.outer(np.sin(ang), r).ravel()], 1)


@pytest.mark.parametrize("case", [0, 1, 2], ids=["1d", "2d", "3d"])
def test_mex_delta_known_answer(case):
    """nufft/interp_table_test.m's inputs (a unit grid value, triangle-based
    complex tables, samples across +-2K) through the drop-ins: the known
    answer read straight from the tables (FP32 tables: within 1e-6), and the
    adjoint of single unit samples."""
    from conftest import delta_known_answer, interp_table_test_cases
    c = interp_table_test_cases()[case]
    K, J, L, h, k0, tm = c["K"], c["J"], c["L"], c["h"], c["k0"], c["tm"]
    D = len(K)
    ck = np.zeros((int(np.prod(K)), 1), dtype=np.complex128)
    kk = np.ravel_multi_index(k0, K, order="F")
    ck[kk, 0] = c["val"]
    ans = c["val"] * delta_known_answer(K, J, L, h, k0, tm)
    fm = _fwd(D, ck, h, J, L, tm, K, None)[:, 0]
    assert np.max(np.abs(fm - ans)) <= 1e-6
    ms = [0, len(tm) // 3, len(tm) - 1]
    e = np.zeros((len(tm), len(ms)), dtype=np.complex128)
    e[ms, range(len(ms))] = 1
    adj = _adj(D, e, h, J, L, tm, K, None)
    for i, m in enumerate(ms):
        want = np.conj(delta_known_answer(K, J, L, h, k0, tm[m:m + 1])[0])
        assert abs(adj[kk, i] - want) <= 1e-6


@pytest.mark.parametrize("N", [1, 3, 8, 32, 40])
def test_minmax_tables_2d_columns(N):
    """C1 geometry (K=128^2, J=6, L=1024, radial 64x128) with N columns,
    exercising every lane width of the kernels."""
    rng = np.random.default_rng(N)
    K, J, L = [128, 128], [6, 6], [1024, 1024]
    h = [mb.minmax_kb_table(64, 6, 128, 1024)] * 2
    om = _radial(64, 128)
    tm = om / (2 * np.pi / 128)
    ck = rng.standard_normal((128 * 128, N)) + 1j * rng.standard_normal((128 * 128, N))
    fm = rng.standard_normal((len(tm), N)) + 1j * rng.standard_normal((len(tm), N))
    ref_f = oracle.interp_for(ck, h, J, L, tm, K, 0, impl=ref_impl(), nthreads=8)
    ref_a = oracle.interp_adj(fm, h, J, L, tm, K, 0, impl=ref_impl(), nthreads=8)
    assert rel_l2(_fwd(2, ck, h, J, L, tm, K, None), ref_f) <= FWD_TOL
    assert rel_l2(_adj(2, fm, h, J, L, tm, K, None), ref_a) <= ADJ_TOL


@pytest.mark.parametrize("variant", ["cx0", "re0", "re1"])
@pytest.mark.parametrize("D", [1, 2, 3])
def test_random_geometry(D, variant):
    """Non-power-of-two grids, J != 6 (generic kernels), wrap far outside [0, K)."""
    rng = np.random.default_rng(100 + D)
    K = [37, 29, 19][:D]
    J = [5, 7, 4][:D]
    L = [128, 64, 256][:D]
    cx = variant == "cx0"
    order = 1 if variant == "re1" else 0
    h = [np.exp(-np.linspace(-j / 2, j / 2, j * l + 1) ** 2)
         * (np.exp(0.4j * np.linspace(-j / 2, j / 2, j * l + 1)) if cx else 1)
         for j, l in zip(J, L)]
    M = 3000
    tm = rng.uniform(-3 * max(K), 3 * max(K), (M, D))
    tm[:50] = np.round(tm[:50] * 2) / 2
    N = 5
    nk = int(np.prod(K))
    ck = rng.standard_normal((nk, N)) + 1j * rng.standard_normal((nk, N))
    fm = rng.standard_normal((M, N)) + 1j * rng.standard_normal((M, N))
    ref_f = oracle.interp_for(ck, h, J, L, tm, K, order, impl=ref_impl())
    ref_a = oracle.interp_adj(fm, h, J, L, tm, K, order, impl=ref_impl())
    assert rel_l2(_fwd(D, ck, h, J, L, tm, K, order), ref_f) <= FWD_TOL
    assert rel_l2(_adj(D, fm, h, J, L, tm, K, order), ref_a) <= ADJ_TOL


@pytest.mark.parametrize("variant", ["cx0", "re0", "re1"])
def test_4d_random_geometry(variant):
    """4D gateways (interp4_table1_for.c / interp4_table1_adj.c) on the 3D
    kernels: generic J, K4 < J4 (a 4th-dimension tap wraps twice),
    coordinates far outside [0, K), several columns."""
    rng = np.random.default_rng(404)
    K = [17, 13, 11, 5]
    J = [5, 6, 4, 6]
    L = [64, 128, 32, 64]
    cx = variant == "cx0"
    order = 1 if variant == "re1" else 0
    h = [np.exp(-np.linspace(-j / 2, j / 2, j * l + 1) ** 2)
         * (np.exp(0.4j * np.linspace(-j / 2, j / 2, j * l + 1)) if cx else 1)
         for j, l in zip(J, L)]
    M, N = 2000, 3
    tm = rng.uniform(-3 * max(K), 3 * max(K), (M, 4))
    tm[:40] = np.round(tm[:40] * 2) / 2
    nk = int(np.prod(K))
    ck = rng.standard_normal((nk, N)) + 1j * rng.standard_normal((nk, N))
    fm = rng.standard_normal((M, N)) + 1j * rng.standard_normal((M, N))
    ref_f = oracle.interp_for(ck, h, J, L, tm, K, order, impl=ref_impl())
    ref_a = oracle.interp_adj(fm, h, J, L, tm, K, order, impl=ref_impl())
    assert rel_l2(_fwd(4, ck, h, J, L, tm, K, order), ref_f) <= FWD_TOL
    assert rel_l2(_adj(4, fm, h, J, L, tm, K, order), ref_a) <= ADJ_TOL


def test_4d_plan_multislice_phase_autotuned():
    """4D device plan: uneven slices (one empty), 8 coils, a per-sample phase,
    J = 6 (the 3D plan underneath may pick its line sweep and TMA gather),
    against the oracle per slice before and after autotuning."""
    import torch
    rng = np.random.default_rng(44)
    K, J, L = [24, 20, 18, 9], [6, 6, 6, 6], [256, 256, 256, 256]
    h = [np.exp(-np.linspace(-3, 3, 6 * 256 + 1) ** 2 / 2)
         * np.exp(0.3j * d * np.linspace(-3, 3, 6 * 256 + 1)) for d in range(4)]
    counts = [1500, 0, 900]
    moff = np.concatenate([[0], np.cumsum(counts)])
    tm = np.concatenate([rng.uniform(-30, 30, (c, 4)) for c in counts])
    ph = np.exp(1j * rng.uniform(0, 2 * np.pi, len(tm)))
    C, S = 8, len(counts)
    plan = mb.InterpPlan(K, J, L, h, tm, C, slice_moff=moff, phase=ph)
    assert plan.grid_shape == (S, 9, 18, 20, 24, C)
    ck = rng.standard_normal(plan.grid_shape) + 1j * rng.standard_normal(plan.grid_shape)
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    ck_d = torch.from_numpy(ck.astype(np.complex64)).cuda()
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()

    def check():
        out_f = plan.forward(ck_d).cpu().numpy()
        out_a = plan.adjoint(fm_d).cpu().numpy()
        for s in range(S):
            sl = slice(moff[s], moff[s + 1])
            got_a = np.transpose(out_a[s], (3, 2, 1, 0, 4)).reshape(-1, C, order="F")
            if not counts[s]:
                assert not got_a.any()
                continue
            cks = np.transpose(ck[s], (3, 2, 1, 0, 4)).reshape(-1, C, order="F")
            ref_f = oracle.interp_for(cks, h, J, L, tm[sl], K, 0, impl=ref_impl())
            assert rel_l2(out_f[sl], ph[sl, None] * ref_f) <= FWD_TOL
            ref_a = oracle.interp_adj(np.conj(ph[sl, None]) * fm[sl], h, J, L, tm[sl], K, 0,
                                      impl=ref_impl())
            assert rel_l2(got_a, ref_a) <= ADJ_TOL
        return out_a

    before = check()
    plan.autotune()
    after = check()
    assert rel_l2(after, before) <= ADJ_TOL
    plan.close()


def test_3d_minmax_multicolumn():
    """3D J=6 (the fixed-J kernels), several columns (the reference's 3D
    gateway accepts only N = 1; this drop-in lifts that)."""
    rng = np.random.default_rng(5)
    K, J, L = [32, 32, 32], [6, 6, 6], [512, 512, 512]
    h = [mb.minmax_kb_table(16, 6, 32, 512)] * 3
    M = 4000
    om = rng.uniform(-np.pi, np.pi, (M, 3))
    tm = om / (2 * np.pi / 32)
    N = 8
    ck = rng.standard_normal((32 ** 3, N)) + 1j * rng.standard_normal((32 ** 3, N))
    fm = rng.standard_normal((M, N)) + 1j * rng.standard_normal((M, N))
    ref_f = oracle.interp_for(ck, h, J, L, tm, K, 0, impl=ref_impl(), nthreads=8)
    ref_a = oracle.interp_adj(fm, h, J, L, tm, K, 0, impl=ref_impl(), nthreads=8)
    assert rel_l2(_fwd(3, ck, h, J, L, tm, K, None), ref_f) <= FWD_TOL
    assert rel_l2(_adj(3, fm, h, J, L, tm, K, None), ref_a) <= ADJ_TOL


def test_adjoint_is_deterministic():
    """The spread has no atomics: two runs agree bit for bit."""
    rng = np.random.default_rng(9)
    K, J, L = [64, 64], [6, 6], [1024, 1024]
    h = [mb.minmax_kb_table(32, 6, 64, 1024)] * 2
    tm = rng.uniform(-40, 40, (20000, 2))
    fm = rng.standard_normal((20000, 4)) + 1j * rng.standard_normal((20000, 4))
    a = _adj(2, fm, h, J, L, tm, K, None)
    b = _adj(2, fm, h, J, L, tm, K, None)
    assert np.array_equal(a, b)


def test_empty_and_single_sample():
    h = [mb.minmax_kb_table(8, 6, 16, 64)] * 2
    J, L, K = [6, 6], [64, 64], [16, 16]
    ck = np.ones((256, 1), complex)
    out = _fwd(2, ck, h, J, L, np.zeros((0, 2)), K, None)
    assert out.shape == (0, 1)
    adj = _adj(2, np.zeros((0, 1), complex), h, J, L, np.zeros((0, 2)), K, None)
    assert adj.shape == (256, 1) and not adj.any()
    tm = np.array([[3.25, -7.5]])
    ref = oracle.interp_for(ck, h, J, L, tm, K, 0, impl=ref_impl())
    assert rel_l2(_fwd(2, ck, h, J, L, tm, K, None), ref) <= FWD_TOL


def test_plan_multislice_uneven():
    """Device plan over several slices of uneven length (one launch each way)
    against the oracle per slice."""
    import torch
    rng = np.random.default_rng(21)
    K, J, L = [96, 80], [6, 6], [512, 512]
    h = [mb.minmax_kb_table(48, 6, 96, 512), mb.minmax_kb_table(40, 6, 80, 512)]
    counts = [700, 0, 1300, 50, 2000]
    moff = np.concatenate([[0], np.cumsum(counts)])
    tm = np.concatenate([rng.uniform(-60, 60, (c, 2)) for c in counts])
    C = 8
    S = len(counts)
    plan = mb.InterpPlan(K, J, L, h, tm, C, slice_moff=moff)
    ck = (rng.standard_normal((S, 80, 96, C)) + 1j * rng.standard_normal((S, 80, 96, C)))
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    ck_d = torch.from_numpy(ck.astype(np.complex64)).cuda()
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    out_f = plan.forward(ck_d).cpu().numpy()
    out_a = plan.adjoint(fm_d).cpu().numpy()
    for s in range(S):
        sl = slice(moff[s], moff[s + 1])
        cks = np.transpose(ck[s], (1, 0, 2)).reshape(-1, C, order="F")
        ref_f = oracle.interp_for(cks, h, J, L, tm[sl], K, 0, impl=ref_impl())
        if counts[s]:
            assert rel_l2(out_f[sl], ref_f) <= FWD_TOL
        ref_a = oracle.interp_adj(fm[sl], h, J, L, tm[sl], K, 0, impl=ref_impl())
        got_a = np.transpose(out_a[s], (1, 0, 2)).reshape(-1, C, order="F")
        if counts[s]:
            assert rel_l2(got_a, ref_a) <= ADJ_TOL
        else:
            assert not got_a.any()
    plan.close()


@pytest.mark.parametrize("C", [1, 8, 32])
def test_autotuned_plan_keeps_parity(C):
    """Every tile shape the autotuner may pick gives the same (correct) result."""
    import torch
    rng = np.random.default_rng(31 + C)
    K, J, L = [128, 96], [6, 6], [1024, 1024]
    h = [mb.minmax_kb_table(64, 6, 128, 1024), mb.minmax_kb_table(48, 6, 96, 1024)]
    counts = [3000, 1700]
    moff = np.concatenate([[0], np.cumsum(counts)])
    tm = np.concatenate([rng.uniform(-70, 70, (c, 2)) for c in counts])
    plan = mb.InterpPlan(K, J, L, h, tm, C, slice_moff=moff)
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    before = plan.adjoint(fm_d).cpu().numpy()
    cfg = plan.autotune()
    assert cfg["spread_threads"] % 32 == 0
    after = plan.adjoint(fm_d).cpu().numpy()
    for s in range(2):
        sl = slice(moff[s], moff[s + 1])
        ref = oracle.interp_adj(fm[sl], h, J, L, tm[sl], K, 0, impl=ref_impl())
        got = np.transpose(after[s], (1, 0, 2)).reshape(-1, C, order="F")
        assert rel_l2(got, ref) <= ADJ_TOL
    assert rel_l2(after, before) <= ADJ_TOL
    ck = rng.standard_normal(plan.grid_shape) + 1j * rng.standard_normal(plan.grid_shape)
    out = plan.forward(torch.from_numpy(ck.astype(np.complex64)).cuda()).cpu().numpy()
    for s in range(2):
        sl = slice(moff[s], moff[s + 1])
        cks = np.transpose(ck[s], (1, 0, 2)).reshape(-1, C, order="F")
        ref = oracle.interp_for(cks, h, J, L, tm[sl], K, 0, impl=ref_impl())
        assert rel_l2(out[sl], ref) <= FWD_TOL
    plan.close()


@pytest.mark.parametrize("C", [1, 4, 8, 32])
def test_spread_tilings_padded_and_plain(C):
    """Every fixed tiling -- tile shape, warps per tile, spare tile columns
    (bounds-free row update) or none -- gives the oracle's adjoint."""
    import torch
    rng = np.random.default_rng(77 + C)
    K, J, L = [96, 80], [6, 6], [1024, 1024]
    h = [mb.minmax_kb_table(48, 6, 96, 1024), mb.minmax_kb_table(40, 6, 80, 1024)]
    tm = rng.uniform(-100, 100, (2500, 2))
    tm[:40] = np.round(tm[:40])
    plan = mb.InterpPlan(K, J, L, h, tm, C)
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    ref = oracle.interp_adj(fm, h, J, L, tm, K, 0, impl=ref_impl())
    for tile, threads in [((8, 8), 32), ((16, 16), 64), ((32, 8), 32), ((8, 32), 128)]:
        for padc in (0, 5):
            cfg = plan.set_spread(tile, threads, padc)
            assert cfg["spread_padc"] == padc and cfg["spread_tile"][:2] == list(tile)
            got = plan.adjoint(fm_d).cpu().numpy()[0]
            got = np.transpose(got, (1, 0, 2)).reshape(-1, C, order="F")
            assert rel_l2(got, ref) <= ADJ_TOL, (tile, threads, padc)
    plan.close()


def test_spread_tilings_3d_padded():
    import torch
    rng = np.random.default_rng(78)
    K, J, L = [24, 20, 16], [6, 6, 6], [256, 256, 256]
    h = [mb.minmax_kb_table(k // 2, 6, k, 256) for k in K]
    tm = rng.uniform(-40, 40, (1500, 3))
    C = 8
    plan = mb.InterpPlan(K, J, L, h, tm, C)
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    ref = oracle.interp_adj(fm, h, J, L, tm, K, 0, impl=ref_impl())
    for tile, threads in [((8, 8, 8), 32), ((16, 8, 8), 64)]:
        for padc in (0, 5):
            plan.set_spread(tile, threads, padc)
            got = plan.adjoint(fm_d).cpu().numpy()[0]
            got = np.transpose(got, (2, 1, 0, 3)).reshape(-1, C, order="F")
            assert rel_l2(got, ref) <= ADJ_TOL, (tile, threads, padc)
    plan.close()


@pytest.mark.parametrize("C", [1, 8, 32])
def test_atomic_spread_matches_oracle(C):
    """Non-deterministic mode: all warps of a tile take whole samples and add
    with shared-memory atomics; the result is the oracle's adjoint to the same
    tolerance, for several tilings, and the autotuner may pick it."""
    import torch
    rng = np.random.default_rng(91 + C)
    K, J, L = [96, 80], [6, 6], [1024, 1024]
    h = [mb.minmax_kb_table(48, 6, 96, 1024), mb.minmax_kb_table(40, 6, 80, 1024)]
    counts = [2000, 1500]
    moff = np.concatenate([[0], np.cumsum(counts)])
    tm = np.concatenate([rng.uniform(-100, 100, (c, 2)) for c in counts])
    plan = mb.InterpPlan(K, J, L, h, tm, C, slice_moff=moff)
    cfg = plan.set_deterministic(False)
    assert cfg["spread_atomic"] == 1
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    refs = [oracle.interp_adj(fm[moff[s]:moff[s + 1]], h, J, L, tm[moff[s]:moff[s + 1]], K, 0,
                              impl=ref_impl()) for s in range(2)]

    def check():
        out = plan.adjoint(fm_d).cpu().numpy()
        for s in range(2):
            got = np.transpose(out[s], (1, 0, 2)).reshape(-1, C, order="F")
            assert rel_l2(got, refs[s]) <= ADJ_TOL

    check()
    for tile, threads in [((8, 8), 128), ((16, 16), 256), ((32, 8), 256)]:
        plan.set_spread(tile, threads, 0)
        assert plan.config()["spread_atomic"] == 1
        check()
    plan.autotune()
    check()
    plan.close()


def test_atomic_spread_3d():
    import torch
    rng = np.random.default_rng(92)
    K, J, L = [24, 20, 16], [6, 6, 6], [256, 256, 256]
    h = [mb.minmax_kb_table(k // 2, 6, k, 256) for k in K]
    tm = rng.uniform(-40, 40, (1500, 3))
    C = 8
    plan = mb.InterpPlan(K, J, L, h, tm, C)
    plan.set_deterministic(False)
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    got = plan.adjoint(torch.from_numpy(fm.astype(np.complex64)).cuda()).cpu().numpy()[0]
    got = np.transpose(got, (2, 1, 0, 3)).reshape(-1, C, order="F")
    ref = oracle.interp_adj(fm, h, J, L, tm, K, 0, impl=ref_impl())
    assert rel_l2(got, ref) <= ADJ_TOL
    plan.close()


@pytest.mark.parametrize("C", [1, 8, 32])
def test_ownership_spread_matches_oracle(C):
    """Ownership spread (2D, J = 6): padded tiles in four colour launches.  A
    dense slice forces split tiles (partial tiles summed by the reduction);
    every tiling gives the oracle's adjoint, bitwise reproducibly."""
    import torch
    rng = np.random.default_rng(71 + C)
    K, J, L = [96, 96], [6, 6], [1024, 1024]
    h = [mb.minmax_kb_table(48, 6, 96, 1024)] * 2
    tms = [rng.uniform(-60, 60, (1500, 2)), rng.uniform(-3, 3, (5000, 2)),
           rng.uniform(-48, 48, (800, 2))]
    moff = np.concatenate([[0], np.cumsum([len(t) for t in tms])])
    tm = np.concatenate(tms)
    plan = mb.InterpPlan(K, J, L, h, tm, C, slice_moff=moff)
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    refs = [oracle.interp_adj(fm[moff[s]:moff[s + 1]], h, J, L, tms[s], K, 0, impl=ref_impl())
            for s in range(3)]
    for tile, threads in [((8, 8), 32), ((16, 8), 64), ((16, 16), 128)]:
        plan.set_spread(tile, threads, 0)
        cfg = plan.set_ownership(True)
        assert cfg["spread_own"] == 1 and cfg["spread_reductions"] > 0
        out = plan.adjoint(fm_d).cpu().numpy()
        for s in range(3):
            got = np.transpose(out[s], (1, 0, 2)).reshape(-1, C, order="F")
            assert rel_l2(got, refs[s]) <= ADJ_TOL, (tile, s)
        assert np.array_equal(out, plan.adjoint(fm_d).cpu().numpy())
    plan.close()


def test_ownership_spread_refused_where_colours_would_overlap():
    K, J, L = [80, 96], [6, 6], [256, 256]
    h = [mb.minmax_kb_table(40, 6, 80, 256), mb.minmax_kb_table(48, 6, 96, 256)]
    tm = np.random.default_rng(0).uniform(-40, 40, (300, 2))
    plan = mb.InterpPlan(K, J, L, h, tm, 4)
    plan.set_spread((16, 16), 32, 0)         # 5 tiles along K1 = 80: odd
    with pytest.raises(mb.MirtError, match="even number of tiles"):
        plan.set_ownership(True)
    plan.close()


@pytest.mark.parametrize("C", [1, 3, 8, 32, 40])
def test_sweep_spread_matches_oracle(C):
    """Row-sweep spread (2D, J = 6): three slices (one dense, one with
    coordinates far outside the grid, wrapping several times), a partial
    coil chunk at C = 3 and 40, bands of 1, 2 and 4 rows, whole rows, uniform
    row segments down to one column (K1 = 96 in 5 segments: a shorter last
    one) and balanced team lists (segments cut at equal visit counts); the oracle's adjoint, bitwise reproducible and
    independent of bands and segments, and the tiled spread's result to FP32
    rounding (another summation order)."""
    import torch
    rng = np.random.default_rng(171 + C)
    K, J, L = [96, 64], [6, 6], [1024, 1024]
    h = [mb.minmax_kb_table(48, 6, 96, 1024), mb.minmax_kb_table(32, 6, 64, 1024)]
    tms = [rng.uniform(-60, 60, (1500, 2)), rng.uniform(-3, 3, (5000, 2)),
           rng.uniform(-300, 300, (800, 2))]
    moff = np.concatenate([[0], np.cumsum([len(t) for t in tms])])
    tm = np.concatenate(tms)
    plan = mb.InterpPlan(K, J, L, h, tm, C, slice_moff=moff)
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    cfg = plan.config()                        # the default for 32-coil chunks: balanced teams
    assert (cfg["spread_sweep"], cfg["spread_sweep_rows"]) == ((-1, 1) if C >= 32 else (0, 1))
    # one-row bands with dense-bin patches (slice 1 is dense): oracle, and the
    # same bits for every segmentation
    plan.set_dense(True)
    dense_first = None
    for nseg in (-1, 1, 5, 96):
        plan.set_sweep(nseg, 1)
        out = plan.adjoint(fm_d).cpu().numpy()
        for s in range(3):
            got = np.transpose(out[s], (1, 0, 2)).reshape(-1, C, order="F")
            assert rel_l2(got, oracle.interp_adj(fm[moff[s]:moff[s + 1]], h, J, L, tms[s], K, 0,
                                                 impl=ref_impl())) <= ADJ_TOL, (nseg, s)
        dense_first = out if dense_first is None else dense_first
        assert np.array_equal(out, dense_first), nseg
    plan.set_dense(False)
    plan.set_sweep(0)
    tiled = plan.adjoint(fm_d).cpu().numpy()
    refs = [oracle.interp_adj(fm[moff[s]:moff[s + 1]], h, J, L, tms[s], K, 0, impl=ref_impl())
            for s in range(3)]
    first = None
    for nseg, rows in [(1, 1), (3, 2), (16, 4), (96, 4), (1, 4), (5, 2), (-1, 1), (-1, 2)]:
        cfg = plan.set_sweep(nseg, rows)
        assert cfg["spread_sweep"] == nseg and cfg["spread_sweep_rows"] == rows
        out = plan.adjoint(fm_d).cpu().numpy()
        for s in range(3):
            got = np.transpose(out[s], (1, 0, 2)).reshape(-1, C, order="F")
            assert rel_l2(got, refs[s]) <= ADJ_TOL, (nseg, rows, s)
        assert np.array_equal(out, plan.adjoint(fm_d).cpu().numpy())
        assert rel_l2(out, tiled) <= 5e-6      # two FP32 summation orders
        if first is None:
            first = out
        assert np.array_equal(out, first)      # neither segments nor bands change the sums
    with pytest.raises(mb.MirtError, match="segments"):
        plan.set_sweep(97)
    with pytest.raises(mb.MirtError, match="rows per band"):
        plan.set_sweep(1, 3)
    plan.set_sweep(False)
    assert np.array_equal(plan.adjoint(fm_d).cpu().numpy(), tiled)
    plan.close()


@pytest.mark.parametrize("order", [0, 1])
def test_sweep_spread_real_tables_phase_small_grid(order):
    """Real tables (order 0 and 1) with a per-sample phase, on grids down to
    K = 6 x 7 where every tap row and column wraps; bands of 2 and 4 rows
    with a partial last band (K2 = 7, 9)."""
    import torch
    rng = np.random.default_rng(5 + order)
    for K in ([6, 7], [12, 9], [40, 24]):
        J, L = [6, 6], [64, 64]
        h = [np.cos(np.linspace(-1.2, 1.2, 6 * 64 + 1)), np.exp(-np.linspace(-2, 2, 6 * 64 + 1) ** 2)]
        tm = rng.uniform(-20, 20, (700, 2))
        ph = np.exp(1j * rng.uniform(-np.pi, np.pi, len(tm)))
        C = 4
        plan = mb.InterpPlan(K, J, L, h, tm, C, order=order, phase=ph)
        plan.set_sweep(1, 4 if K[1] > 7 else 2)
        fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
        got = plan.adjoint(torch.from_numpy(fm.astype(np.complex64)).cuda()).cpu().numpy()[0]
        got = np.transpose(got, (1, 0, 2)).reshape(-1, C, order="F")
        ref = oracle.interp_adj(fm * np.conj(ph)[:, None], h, J, L, tm, K, order, impl=ref_impl())
        assert rel_l2(got, ref) <= ADJ_TOL, K
        plan.close()


@pytest.mark.parametrize("C", [32, 40, 64])
def test_staged_sweep_same_bits(C):
    """The row sweep staged per bin column (mirt_interp_plan_set_staged 1: after
    the ordering pass; 2: reading the caller's samples through the sort
    permutation) gives the unstaged sweep's bits for bands of 1, 2 and 4 rows,
    uniform segments and balanced teams, on three slices (a dense one, one
    wrapping several times) with a per-sample phase, a partial coil chunk at
    C = 40; and the oracle's adjoint.  Dense-bin patches take precedence over
    staging (one-row bands): the same bits as without staging."""
    import torch
    rng = np.random.default_rng(29 + C)
    K, J, L = [96, 64], [6, 6], [1024, 1024]
    h = [mb.minmax_kb_table(48, 6, 96, 1024), mb.minmax_kb_table(32, 6, 64, 1024)]
    tms = [rng.uniform(-60, 60, (1500, 2)), rng.uniform(-3, 3, (5000, 2)),
           rng.uniform(-300, 300, (800, 2))]
    moff = np.concatenate([[0], np.cumsum([len(t) for t in tms])])
    tm = np.concatenate(tms)
    ph = np.exp(1j * rng.uniform(-np.pi, np.pi, len(tm)))
    plan = mb.InterpPlan(K, J, L, h, tm, C, slice_moff=moff, phase=ph)
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    refs = [oracle.interp_adj((fm * np.conj(ph)[:, None])[moff[s]:moff[s + 1]], h, J, L, tms[s],
                              K, 0, impl=ref_impl()) for s in range(3)]
    plan.set_dense(False)
    first = None
    for nseg, rows in [(1, 1), (5, 2), (16, 4), (-1, 1), (-1, 4)]:
        plan.set_sweep(nseg, rows)
        plan.set_staged(0)
        base = plan.adjoint(fm_d).cpu().numpy()
        for s in range(3):
            got = np.transpose(base[s], (1, 0, 2)).reshape(-1, C, order="F")
            assert rel_l2(got, refs[s]) <= ADJ_TOL, (nseg, rows, s)
        for mode in (1, 2):
            plan.set_staged(mode)
            assert plan.config()["spread_staged"] == mode
            out = plan.adjoint(fm_d).cpu().numpy()
            assert np.array_equal(out, base), (nseg, rows, mode)
        first = base if first is None else first
        assert np.array_equal(base, first)
    plan.set_dense(True)
    plan.set_sweep(-1, 1)
    plan.set_staged(0)
    dense = plan.adjoint(fm_d).cpu().numpy()
    plan.set_staged(2)
    assert np.array_equal(plan.adjoint(fm_d).cpu().numpy(), dense)
    with pytest.raises(mb.MirtError, match="staged mode"):
        plan.set_staged(3)
    plan.close()
    small = mb.InterpPlan(K, J, L, h, tms[0], 8)
    with pytest.raises(mb.MirtError, match="32-coil"):
        small.set_staged(1)
    small.close()


@pytest.mark.parametrize("order", [0, 1])
def test_staged_sweep_real_tables_phase(order):
    """The staged row sweep with real tables (order 0 and 1) and a per-sample
    phase, 32 coils, grids down to K = 6 x 7 (every tap row and column wraps):
    the unstaged sweep's bits for both staged modes, and the oracle's adjoint."""
    import torch
    rng = np.random.default_rng(41 + order)
    for K in ([6, 7], [40, 24]):
        J, L = [6, 6], [64, 64]
        h = [np.cos(np.linspace(-1.2, 1.2, 6 * 64 + 1)), np.exp(-np.linspace(-2, 2, 6 * 64 + 1) ** 2)]
        tm = rng.uniform(-20, 20, (900, 2))
        ph = np.exp(1j * rng.uniform(-np.pi, np.pi, len(tm)))
        C = 32
        plan = mb.InterpPlan(K, J, L, h, tm, C, order=order, phase=ph)
        plan.set_dense(False)
        rows = 4 if K[1] > 7 else 2
        plan.set_sweep(1, rows)
        plan.set_staged(0)
        fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
        fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
        base = plan.adjoint(fm_d).cpu().numpy()
        for mode in (1, 2):
            plan.set_staged(mode)
            assert np.array_equal(plan.adjoint(fm_d).cpu().numpy(), base), (K, mode)
        got = np.transpose(base[0], (1, 0, 2)).reshape(-1, C, order="F")
        ref = oracle.interp_adj(fm * np.conj(ph)[:, None], h, J, L, tm, K, order, impl=ref_impl())
        assert rel_l2(got, ref) <= ADJ_TOL, K
        plan.close()


def test_sweep_spread_refused_where_it_does_not_apply():
    h = [mb.minmax_kb_table(8, 4, 16, 64)] * 2
    plan = mb.InterpPlan([16, 16], [4, 4], [64, 64], h, np.zeros((10, 2)), 2)
    with pytest.raises(mb.MirtError, match="row-sweep"):
        plan.set_sweep(True)
    plan.close()


@pytest.mark.parametrize("C,K", [(32, (96, 64)), (40, (13, 27)), (64, (40, 33))])
def test_tma_gather_matches_plain_gather_and_oracle(C, K):
    """Gather over TMA-staged tiles and records (2D, J = 6, even C >= 32):
    bitwise the plain gather (same arithmetic and order), the oracle's
    forward to FP32 rounding, coil chunks (C = 40, 64), grids from 13 points
    (where most blocks wrap and read the grid directly), a dense slice (blocks
    split into several work items), coordinates far outside the grid, three
    slices; the plan's fault flag stays clear."""
    import torch
    rng = np.random.default_rng(11 + C)
    J, L = [6, 6], [1024, 1024]
    h = [mb.minmax_kb_table(max(K[0] // 2, 6), 6, K[0], 1024),
         mb.minmax_kb_table(max(K[1] // 2, 6), 6, K[1], 1024)]
    tms = [rng.uniform(-40, 40, (2000, 2)), rng.uniform(-3, 3, (3000, 2)),
           rng.uniform(-300, 300, (700, 2))]
    moff = np.concatenate([[0], np.cumsum([len(t) for t in tms])])
    plan = mb.InterpPlan(K, J, L, h, np.concatenate(tms), C, slice_moff=moff)
    assert plan.config()["gather_tma"] == 1      # the default where it applies
    ck = (rng.standard_normal((3, K[1], K[0], C)) + 1j * rng.standard_normal((3, K[1], K[0], C)))
    ckd = torch.from_numpy(ck.astype(np.complex64)).cuda()
    a = plan.forward(ckd).cpu().numpy()
    assert plan.fault() == 0
    assert plan.set_gather(2)["gather_tma"] == 2  # tiles of 16 coils, a half-warp per sample
    assert np.array_equal(plan.forward(ckd).cpu().numpy(), a)
    assert plan.fault() == 0
    plan.set_gather(False)
    b = plan.forward(ckd).cpu().numpy()
    assert np.array_equal(a, b)
    with pytest.raises(mb.MirtError, match="gather mode"):
        plan.set_gather(3)
    for s in range(3):
        ref = oracle.interp_for(np.transpose(ck[s], (1, 0, 2)).reshape(-1, C, order="F"), h, J, L,
                                tms[s], K, 0, impl=ref_impl())
        assert rel_l2(a[moff[s]:moff[s + 1]], ref) <= FWD_TOL, s
    plan.close()


@pytest.mark.parametrize("C,K", [(16, (64, 48)), (18, (13, 30)), (24, (40, 33)), (30, (17, 96))])
def test_tma_gather_of_16_to_31_columns(C, K):
    """Tiles of 16 columns below 32 (one full chunk, a chunk of 2, of 8, of 14;
    wrapped blocks as rows or point by point): the plain gather's bits, in its
    arithmetic, from a grid at an odd multiple of 8 bytes too; the forms of 32
    columns stay refused."""
    import torch
    rng = np.random.default_rng(C)
    h = [mb.minmax_kb_table(max(k // 2, 6), 6, k, 256) for k in K]
    tms = [rng.uniform(-20, 20, (900, 2)), rng.uniform(-2, 2, (1500, 2)), rng.uniform(-90, 90, (77, 2))]
    moff = np.concatenate([[0], np.cumsum([len(t) for t in tms])])
    plan = mb.InterpPlan(K, [6, 6], [256, 256], h, np.concatenate(tms), C, slice_moff=moff)
    assert plan.config()["gather_tma"] == 2
    ck = rng.standard_normal((3, K[1], K[0], C)) + 1j * rng.standard_normal((3, K[1], K[0], C))
    buf = torch.zeros(ck.size + 1, dtype=torch.complex64, device="cuda")
    odd = buf[1:].view(ck.shape)
    odd.copy_(torch.from_numpy(ck.astype(np.complex64)))
    even = odd.clone()
    a = plan.forward(even).cpu().numpy()
    assert np.array_equal(plan.forward(odd).cpu().numpy(), a)
    for mode in (1, 2):
        with pytest.raises(mb.MirtError, match="TMA gather"):
            plan.set_gather(mode)
    plan.set_gather(False)
    assert np.array_equal(plan.forward(even).cpu().numpy(), a)
    for s in range(3):
        ref = oracle.interp_for(np.transpose(ck[s], (1, 0, 2)).reshape(-1, C, order="F"), h, [6, 6],
                                [256, 256], tms[s], K, 0, impl=ref_impl())
        assert rel_l2(a[moff[s]:moff[s + 1]], ref) <= FWD_TOL, s
    assert plan.fault() == 0
    plan.close()


@pytest.mark.parametrize("C,K", [(8, (32, 24, 20)), (10, (12, 9, 16))])
def test_tma_gather_3d_matches_plain_gather_and_oracle(C, K):
    """3D gather over TMA-staged 9 x 9 x 9 tiles of 8 coils (4 x 4 x 4 blocks
    of first taps, items of up to 32 samples): bitwise the plain 3D gather,
    the oracle's forward to FP32 rounding; a partial coil chunk (C = 10), grids
    down to K = 9 (most blocks wrap and read the grid directly), a dense slice
    (blocks split into several items), coordinates far outside the grid, three
    slices; a per-sample phase; the bounded waits' fault path."""
    import torch
    rng = np.random.default_rng(91 + C)
    J, L = [6, 6, 6], [256, 256, 256]
    h = [mb.minmax_kb_table(max(k // 2, 6), 6, k, 256) for k in K]
    tms = [rng.uniform(-20, 20, (1500, 3)), rng.uniform(-2, 2, (3000, 3)),
           rng.uniform(-100, 100, (500, 3))]
    moff = np.concatenate([[0], np.cumsum([len(t) for t in tms])])
    tm = np.concatenate(tms)
    ph = np.exp(1j * rng.uniform(-np.pi, np.pi, len(tm)))
    plan = mb.InterpPlan(K, J, L, h, tm, C, slice_moff=moff, phase=ph)
    assert plan.config()["gather_tma"] == 1      # the default where it applies
    ck = (rng.standard_normal((3, K[2], K[1], K[0], C)) +
          1j * rng.standard_normal((3, K[2], K[1], K[0], C)))
    ckd = torch.from_numpy(ck.astype(np.complex64)).cuda()
    a = plan.forward(ckd).cpu().numpy()
    assert plan.fault() == 0
    plan.set_gather(False)
    assert np.array_equal(plan.forward(ckd).cpu().numpy(), a)
    for s in range(3):
        ref = oracle.interp_for(np.transpose(ck[s], (2, 1, 0, 3)).reshape(-1, C, order="F"), h, J,
                                L, tms[s], K, 0, impl=ref_impl()) * ph[moff[s]:moff[s + 1], None]
        assert rel_l2(a[moff[s]:moff[s + 1]], ref) <= FWD_TOL, s
    with pytest.raises(mb.MirtError, match="2D only"):
        plan.set_gather(2)
    plan.set_gather(True)
    plan.set_fault_test(True)                   # no copies: every wait runs out, nothing in flight
    plan.forward(ckd)
    assert plan.fault() == 1
    plan.close()                                # a faulted plan is discarded
    p6 = mb.InterpPlan(K, J, L, h, tms[0], 6)   # C < 8: no 3D TMA blocks
    assert p6.config()["gather_tma"] == 0
    p6.close()


def _median_ms(f, n=15):
    import torch
    for _ in range(3):
        f()
    ms = []
    for _ in range(n):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(100000)                # the launches queue up behind it
        a.record()
        f()
        b.record()
        b.synchronize()
        ms.append(a.elapsed_time(b))
    return float(np.median(ms))


@pytest.mark.parametrize("C", [16, 20])
def test_3d_gather_time_follows_the_coil_chunks(C):
    """A 3D gather of two or three chunks of eight coils takes no more than its chunks' share of
    one chunk's time (30 % allowed), although the tiles of the blocks whose taps wrap, a
    third of these, are not contiguous in a grid of more than eight coils."""
    import torch
    rng = np.random.default_rng(C)
    K = [64, 64, 64]
    tm = rng.uniform(-32, 32, (100000, 3))
    ms = {}
    for c in (8, C):
        plan = mb.InterpPlan(K, [6] * 3, [64] * 3, [mb.newfft_kb_table(6, 64)] * 3, tm, c, order=1)
        assert plan.config()["gather_tma"] == 1
        ck = torch.randn(plan.grid_shape, dtype=torch.complex64, device="cuda")
        out = torch.empty(plan.sample_shape, dtype=torch.complex64, device="cuda")
        ms[c] = _median_ms(lambda: plan.forward(ck, out=out))
        plan.close()
    assert ms[C] <= 1.3 * -(-C // 8) * ms[8], ms


@pytest.mark.parametrize("C", [16, 18, 34, 40, 64])
def test_tma_gather_of_wrapped_tiles_by_their_samples(C):
    """Wrapped tiles of one to 30 samples, around the number from which they are copied to
    shared memory, at the grid's right end, its top and its corner: the plain gather's bits."""
    import torch
    rng = np.random.default_rng(C)
    K = [40, 48]
    slices = []
    for n in (1, 2, 22, 23, 24, 25, 30):
        corner = np.array([[36.0, 20.0], [20.0, 44.0], [36.0, 44.0], [12.0, 20.0]])
        slices.append(np.concatenate([c + rng.uniform(0, 2, (n, 2)) for c in corner]))
    if C < 32:  # samples enough for the tiles to be the default
        slices.append(rng.uniform(8, 30, (6000, 2)))
    moff = np.concatenate([[0], np.cumsum([len(s) for s in slices])])
    plan = mb.InterpPlan(K, [6, 6], [64, 64], [mb.newfft_kb_table(6, 64)] * 2,
                         np.concatenate(slices), C, order=1, slice_moff=moff)
    assert plan.config()["gather_tma"] == (2 if C < 32 else 1)
    ck = torch.randn(plan.grid_shape, dtype=torch.complex64, device="cuda")
    got = {mode: plan.forward(ck) for mode in ((None,) if C < 32 else (None, 2))
           if mode is None or plan.set_gather(mode)}
    plan.set_gather(False)
    ref = plan.forward(ck)
    assert all(torch.equal(g, ref) for g in got.values())
    assert plan.fault() == 0
    plan.close()


@pytest.mark.parametrize("C,sparse,dense", [(16, 1000, 30000), (18, 20000, 200000), (20, 8000, 60000),
                                            (24, 8000, 60000), (30, 5000, 40000)])
def test_gather_of_16_to_30_columns_by_density(C, sparse, dense):
    """Few samples a block of 8 x 8 first taps (1024 blocks): the plain gather, which goes by samples
    and columns; many: the staged tiles; the autotuner may choose the tiles for either."""
    import torch
    rng = np.random.default_rng(C)
    for M, tma in ((sparse, 0), (dense, 2)):
        tm = rng.uniform(-128, 128, (M, 2))
        plan = mb.InterpPlan([256, 256], [6, 6], [64, 64], [mb.newfft_kb_table(6, 64)] * 2, tm, C,
                             order=1)
        assert plan.config()["gather_tma"] == tma
        ck = torch.randn(plan.grid_shape, dtype=torch.complex64, device="cuda")
        a = plan.forward(ck)
        assert plan.autotune()["gather_tma"] in (0, 2)
        assert torch.equal(plan.forward(ck), a)
        plan.close()


@pytest.mark.parametrize("order", [0, 1])
def test_tma_gather_3d_real_tables(order):
    """3D TMA gather with real tables (order 0 and 1): the plain 3D gather's
    bits and the oracle's forward."""
    import torch
    rng = np.random.default_rng(61 + order)
    K, J, L = [16, 12, 10], [6, 6, 6], [64, 64, 64]
    t = np.linspace(-2, 2, 6 * 64 + 1)
    h = [np.exp(-t ** 2), np.cos(0.6 * t), np.exp(-0.5 * t ** 2)]
    tm = rng.uniform(-12, 12, (2500, 3))
    C = 8
    plan = mb.InterpPlan(K, J, L, h, tm, C, order=order)
    assert plan.config()["gather_tma"] == 1
    ck = rng.standard_normal((1, K[2], K[1], K[0], C)) + 1j * rng.standard_normal((1, K[2], K[1], K[0], C))
    ckd = torch.from_numpy(ck.astype(np.complex64)).cuda()
    a = plan.forward(ckd).cpu().numpy()
    plan.set_gather(False)
    assert np.array_equal(plan.forward(ckd).cpu().numpy(), a)
    ref = oracle.interp_for(np.transpose(ck[0], (2, 1, 0, 3)).reshape(-1, C, order="F"), h, J, L,
                            tm, K, order, impl=ref_impl())
    assert rel_l2(a, ref) <= FWD_TOL
    assert plan.fault() == 0
    plan.close()


def test_tma_gather_real_tables_phase_and_refusal():
    """Real tables, first order, with a per-sample phase: the TMA gather equals
    the plain gather and the oracle; a plan with C = 8 has no TMA blocks."""
    import torch
    rng = np.random.default_rng(3)
    K, J, L = [48, 40], [6, 6], [256, 256]
    h = [np.cos(np.linspace(-1.2, 1.2, 6 * 256 + 1)), np.exp(-np.linspace(-2, 2, 6 * 256 + 1) ** 2)]
    tm = rng.uniform(-30, 30, (4000, 2))
    ph = np.exp(1j * rng.uniform(-np.pi, np.pi, len(tm)))
    plan = mb.InterpPlan(K, J, L, h, tm, 32, order=1, phase=ph)
    plan.set_gather(True)
    ck = rng.standard_normal((1, K[1], K[0], 32)) + 1j * rng.standard_normal((1, K[1], K[0], 32))
    ckd = torch.from_numpy(ck.astype(np.complex64)).cuda()
    a = plan.forward(ckd).cpu().numpy()
    plan.set_gather(2)
    assert np.array_equal(a, plan.forward(ckd).cpu().numpy())
    plan.set_gather(False)
    assert np.array_equal(a, plan.forward(ckd).cpu().numpy())
    ref = oracle.interp_for(np.transpose(ck[0], (1, 0, 2)).reshape(-1, 32, order="F"), h, J, L, tm,
                            K, 1, impl=ref_impl()) * ph[:, None]
    assert rel_l2(a, ref) <= FWD_TOL
    assert plan.fault() == 0
    plan.close()
    p8 = mb.InterpPlan(K, J, L, h, tm, 8, order=1)
    assert p8.config()["gather_tma"] == 0
    with pytest.raises(mb.MirtError, match="TMA gather"):
        p8.set_gather(True)
    p8.close()


@pytest.mark.parametrize("C", [8, 16, 32, 40])
def test_3d_line_sweep_matches_oracle(C):
    """3D line sweep (J = 6; warps own 2 x 2, 2 x 1 or single lines for coil
    chunks of 8, 16, 32; C = 40: a partial second chunk): two slices, one dense
    and one wrapping far outside the grid, on a grid of 12 x 10 x 9 points (so
    tap rows and planes wrap); against the oracle, bitwise the same for 1, 2
    and 5 segments and on repeated calls, and the tiled spread to FP32
    rounding."""
    import torch
    rng = np.random.default_rng(300 + C)
    K, J, L = [12, 10, 9], [6, 6, 6], [512, 512, 512]
    h = [mb.minmax_kb_table(k // 2, 6, k, 512) for k in K]
    # slice 0: a cluster of ~100 samples per bin (dense bins, summed into
    # patches before the sweep) around sparse ones
    tms = [np.concatenate([rng.uniform(-1.5, 1.5, (3000, 3)), rng.uniform(-3, 3, (900, 3))]),
           rng.uniform(-60, 60, (700, 3))]
    moff = np.concatenate([[0], np.cumsum([len(t) for t in tms])])
    tm = np.concatenate(tms)
    plan = mb.InterpPlan(K, J, L, h, tm, C, slice_moff=moff)
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    assert plan.config()["spread_sweep"] > 0          # the default for 3D, J = 6
    refs = [oracle.interp_adj(fm[moff[s]:moff[s + 1]], h, J, L, tms[s], K, 0, impl=ref_impl())
            for s in range(2)]
    first = None
    for nseg in (1, 2, 5):
        plan.set_sweep(nseg)
        out = plan.adjoint(fm_d).cpu().numpy()
        for s in range(2):
            got = np.transpose(out[s], (2, 1, 0, 3)).reshape(-1, C, order="F")
            assert rel_l2(got, refs[s]) <= ADJ_TOL, (nseg, s)
        assert np.array_equal(out, plan.adjoint(fm_d).cpu().numpy())
        if first is None:
            first = out
        assert np.array_equal(out, first), nseg
    plan.set_sweep(0)
    tiled = plan.adjoint(fm_d).cpu().numpy()
    assert rel_l2(tiled, first) <= 5e-6
    plan.close()


@pytest.mark.parametrize("C", [8, 9, 17])
def test_3d_line_sweep_parts_and_tails(C):
    """Lines cut into parts of few columns (crowded columns, some side by side, some
    alone, at both ends of the lines): the parts' five columns past their last meet
    in one column, wrap, and cross further parts; odd column counts (rows at odd
    multiples of 8 bytes); an empty slice between two; a sample of infinities stays
    within its own taps."""
    import torch
    rng = np.random.default_rng(5 + C)
    K, J, L = [40, 11, 9], [6, 6, 6], [64, 64, 64]
    h = [mb.minmax_kb_table(k // 2, 6, k, 64) for k in K]

    def cluster(x, n):
        return np.stack([x + rng.uniform(0, 1, n), rng.uniform(-4, 4, n), rng.uniform(-4, 4, n)], 1)
    tms = [np.concatenate([cluster(x, n) for x, n in
                           ((0, 700), (1, 600), (2, 30), (3, 900), (17, 500), (36, 10), (39, 800))]),
           np.zeros((0, 3)), np.concatenate([cluster(38, 900), rng.uniform(-30, 30, (50, 3))])]
    moff = np.concatenate([[0], np.cumsum([len(t) for t in tms])])
    plan = mb.InterpPlan(K, J, L, h, np.concatenate(tms), C, slice_moff=moff)
    plan.set_sweep(2)
    fm = rng.standard_normal((moff[-1], C)) + 1j * rng.standard_normal((moff[-1], C))
    fd = torch.from_numpy(fm.astype(np.complex64)).cuda()
    out = plan.adjoint(fd).cpu().numpy()
    assert np.array_equal(out, plan.adjoint(fd).cpu().numpy())
    assert not out[1].any()
    for s in (0, 2):
        ref = oracle.interp_adj(fm[moff[s]:moff[s + 1]], h, J, L, tms[s], K, 0, impl=ref_impl())
        got = np.transpose(out[s], (2, 1, 0, 3)).reshape(-1, C, order="F")
        assert rel_l2(got, ref) <= ADJ_TOL, s
    # the last sample's taps alone turn non-finite
    fd[-1] = float("inf")
    bad = ~np.isfinite(plan.adjoint(fd).cpu().numpy()[..., 0])
    assert not bad[:2].any() and 0 < bad[2].sum() <= 216
    plan.close()


@pytest.mark.parametrize("order", [0, 1])
def test_3d_line_sweep_real_tables_phase(order):
    """3D line sweep with real tables (order 0 and 1) and a per-sample phase,
    8 coils, on the smallest grids it takes (6 x 7 x 6)."""
    import torch
    rng = np.random.default_rng(310 + order)
    for K in ([6, 7, 6], [16, 12, 20]):
        J, L = [6, 6, 6], [64, 64, 64]
        h = [np.cos(np.linspace(-1.2, 1.2, 6 * 64 + 1)),
             np.exp(-np.linspace(-2, 2, 6 * 64 + 1) ** 2),
             np.cos(np.linspace(-0.9, 0.9, 6 * 64 + 1))]
        tm = np.concatenate([rng.uniform(-20, 20, (900, 3)), rng.uniform(2, 3, (500, 3))])
        ph = np.exp(1j * rng.uniform(-np.pi, np.pi, len(tm)))
        C = 8
        plan = mb.InterpPlan(K, J, L, h, tm, C, order=order, phase=ph)
        plan.set_sweep(3)
        fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
        got = plan.adjoint(torch.from_numpy(fm.astype(np.complex64)).cuda()).cpu().numpy()[0]
        got = np.transpose(got, (2, 1, 0, 3)).reshape(-1, C, order="F")
        ref = oracle.interp_adj(fm * np.conj(ph)[:, None], h, J, L, tm, K, order, impl=ref_impl())
        assert rel_l2(got, ref) <= ADJ_TOL, K
        plan.close()


def test_tma_gather_bounded_wait_fault_path():
    """The TMA gather's bounded waits, made to run out without a GPU fault:
    the test hook arms every stage's barrier for bytes that no copy delivers
    and issues no copy, so each wait ends at its limit with nothing in flight.
    The launch returns, the plan's fault flag reads 1 (and is cleared by the
    read), and the device keeps working: a new plan's gather of the same
    problem matches the oracle."""
    import torch
    rng = np.random.default_rng(404)
    K, J, L = [96, 64], [6, 6], [1024, 1024]
    h = [mb.minmax_kb_table(48, 6, 96, 1024), mb.minmax_kb_table(32, 6, 64, 1024)]
    tm = rng.uniform(-40, 40, (6000, 2))
    C = 32
    ck = rng.standard_normal((96 * 64, C)) + 1j * rng.standard_normal((96 * 64, C))
    ck_d = torch.from_numpy(ck.reshape(64, 96, C).astype(np.complex64)).cuda()[None]
    for mode in (1, 2):                         # tiles of 32 and of 16 coils
        plan = mb.InterpPlan(K, J, L, h, tm, C)
        plan.set_gather(mode)
        plan.set_fault_test(True)
        plan.forward(ck_d)
        assert plan.fault() == 1
        assert plan.fault() == 0
        plan.close()                            # a faulted plan is discarded
    plan = mb.InterpPlan(K, J, L, h, tm, C)
    got = plan.forward(ck_d).cpu().numpy()
    assert plan.fault() == 0
    ref = oracle.interp_for(ck, h, J, L, tm, K, 0, impl=ref_impl(), nthreads=8)
    assert rel_l2(got, ref) <= FWD_TOL
    plan.close()


POINT_CASES = [
    # K, J, columns, table kind: blocks of four points cut at the grid's end, J = K,
    # odd and unequal J, every lane shape (1..4, 6, 8, 12, 16, 24, 32 columns a
    # chunk, idle columns, several chunks)
    ([64], [6], 1, "cx0"), ([7], [7], 3, "cx0"), ([130], [5], 33, "re1"),
    ([64, 48], [6, 6], 1, "cx0"), ([63, 50], [6, 6], 2, "re1"), ([6, 6], [6, 6], 4, "cx0"),
    ([66, 41], [5, 4], 5, "cx0"), ([48, 33], [7, 6], 7, "re0"), ([37, 64], [6, 6], 12, "cx0"),
    ([40, 44], [6, 6], 15, "re1"), ([45, 38], [6, 6], 24, "cx0"), ([34, 30], [6, 6], 31, "cx0"),
    ([33, 35], [5, 5], 49, "cx0"),
    ([20, 18, 16], [6, 6, 6], 1, "cx0"), ([6, 7, 9], [6, 6, 6], 2, "re1"),
    ([13, 14, 17], [5, 6, 4], 3, "cx0"), ([16, 12, 10], [4, 5, 3], 9, "re0"),
]


@pytest.mark.parametrize("K,J,C,variant", POINT_CASES)
def test_point_spread_matches_oracle(K, J, C, variant):
    """The point spread (the default where the sweeps are not): a sparse slice
    with coordinates that wrap several times, an empty one and one so dense that
    bricks are shared by the groups of a CTA and by several CTAs; with a
    per-sample phase; the oracle's adjoint, the same bits on a second call, and
    the tiled spread's result to FP32 rounding."""
    import torch
    D = len(K)
    rng = np.random.default_rng(sum(K) + 100 * C)
    L = [256] * D
    n = [max(2, k // 2) for k in K]
    if variant == "cx0":
        h = [mb.minmax_kb_table(n[d], J[d], K[d], L[d]) for d in range(D)]
    else:
        h = [mb.newfft_kb_table(J[d], L[d]) for d in range(D)]
    order = 1 if variant == "re1" else 0
    tms = [rng.uniform(-3 * max(K), 3 * max(K), (300, D)), np.zeros((0, D)),
           rng.uniform(-1.5, 1.5, (4000, D))]
    moff = np.concatenate([[0], np.cumsum([len(t) for t in tms])])
    tm = np.concatenate(tms)
    ph = np.exp(1j * rng.uniform(0, 6, len(tm)))
    plan = mb.InterpPlan(K, J, L, h, tm, C, order=order, slice_moff=moff, phase=ph)
    assert plan.config()["spread_points"] > 0
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    out = plan.adjoint(fm_d).cpu().numpy()
    assert np.array_equal(out, plan.adjoint(fm_d).cpu().numpy())
    for s in range(3):
        sl = slice(moff[s], moff[s + 1])
        got = np.transpose(out[s], tuple(range(D - 1, -1, -1)) + (D,)).reshape(-1, C, order="F")
        if not len(tms[s]):
            assert not got.any()
            continue
        ref = oracle.interp_adj(fm[sl] * np.conj(ph[sl])[:, None], h, J, L, tms[s], K, order,
                                impl=ref_impl())
        assert rel_l2(got, ref) <= ADJ_TOL, s
    plan.set_spread([min(8, k) for k in K])
    assert plan.config()["spread_points"] == 0
    assert rel_l2(plan.adjoint(fm_d).cpu().numpy(), out) <= 5e-6
    plan.close()


@pytest.mark.parametrize("K,J,C", [
    # base tiles 8 points wide along dimension 1 (2D from 17 columns, 3D from 5): J1 - 1 taps
    # within the first tile, up to its end, past it into the second
    ((64, 40), (9, 6), 17), ((64, 40), (10, 10), 24), ((40, 33), (13, 5), 32), ((64, 40), (16, 16), 33),
    ((19, 21), (16, 3), 24), ((16, 16), (16, 16), 20), ((24, 20, 18), (9, 4, 3), 5),
    ((24, 20, 18), (10, 5, 4), 9), ((25, 18, 14), (13, 3, 6), 17), ((24, 16, 13), (16, 2, 5), 5),
    ((16, 17, 18), (16, 16, 16), 3), ((40, 30), (16, 4), 1), ((70,), (16,), 33),
])
def test_point_spread_of_wide_kernels(K, J, C):
    """Up to 16 taps: coordinates whose first-dimension taps wrap from the grid's end, which
    then reach the tiles after the first one, spread over the grid and crowded at its start."""
    import torch
    D = len(K)
    rng = np.random.default_rng(sum(K) + 7 * C)
    L = [64] * D
    h = [mb.newfft_kb_table(j, 64) for j in J]
    tm = np.concatenate([rng.uniform(-2 * max(K), 2 * max(K), (500, D)),
                         rng.uniform(-9, 9, (300, D))])
    plan = mb.InterpPlan(list(K), list(J), L, h, tm, C, order=1)
    assert plan.config()["spread_points"] > 0
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    out = plan.adjoint(torch.from_numpy(fm.astype(np.complex64)).cuda()).cpu().numpy()[0]
    got = np.transpose(out, tuple(range(D - 1, -1, -1)) + (D,)).reshape(-1, C, order="F")
    ref = oracle.interp_adj(fm, h, list(J), L, tm, list(K), 1, impl=ref_impl())
    assert rel_l2(got, ref) <= ADJ_TOL
    plan.close()


@pytest.mark.parametrize("C", [32, 34, 64])
@pytest.mark.parametrize("kind,K,M,form", [
    ("even", (64, 48), 0, "points"), ("even", (64, 48), 4000, "points"), ("even", (128, 128), 16000, "points"),
    ("even", (256, 200), 16001, "split"), ("even", (64, 48), 20000, "points"),
    ("even", (200, 150), 40000, "row"), ("dense", (96, 80), 70000, "row"),
    ("dense", (96, 80), 60000, "split"), ("radial", (512, 512), 204800, "split"),
])
def test_default_spread_of_32_columns(C, kind, K, M, form):
    """The default of 2D plans of 32 columns and more by the samples in dense bins and in dense
    tiles: the point spread alone, the split spread or the row sweep; each the oracle's adjoint,
    the same bits again, and the row sweep when a row-sweep setting is chosen."""
    import torch
    rng = np.random.default_rng(M + C)
    if kind == "even":
        tm = rng.uniform(-1, 1, (M, 2)) * np.array(K)
    elif kind == "dense":                       # nine tenths of them within a few points
        tm = np.concatenate([rng.uniform(-5, 5, (M - M // 10, 2)), rng.uniform(-90, 90, (M // 10, 2))])
    else:
        tm = _radial(M // 512, 512) * 512 / (2 * np.pi)
    h = [mb.newfft_kb_table(6, 64)] * 2
    plan = mb.InterpPlan(list(K), [6, 6], [64, 64], h, tm, C, order=1)
    cfg = plan.config()
    assert cfg["spread_sweep"] == -1
    got = "split" if cfg["spread_split"] else "points" if cfg["spread_points"] else "row"
    assert got == form
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fd = torch.from_numpy(fm.astype(np.complex64)).cuda()
    out = plan.adjoint(fd)
    assert torch.equal(out, plan.adjoint(fd))
    plan.set_staged(2)
    assert plan.config()["spread_points"] == 0 and plan.config()["spread_split"] == 0
    row = plan.adjoint(fd).cpu().numpy()
    out = out.cpu().numpy()
    if M:
        cols = [0, C - 1]
        ref = oracle.interp_adj(fm[:, cols], h, [6, 6], [64, 64], tm, list(K), 1, impl=ref_impl())
        for o in (out, row):
            assert rel_l2(np.transpose(o[0], (1, 0, 2)).reshape(-1, C, order="F")[:, cols], ref) <= ADJ_TOL
    else:
        assert not out.any() and not row.any()
    plan.close()


@pytest.mark.parametrize("K,C,M", [((64, 48), 8, 3000), ((41, 50), 32, 7500), ((96, 80), 40, 1000),
                                   ((64, 60), 26, 5000)])
def test_ownership_off_leaves_the_spread(K, C, M):
    """set_ownership(False) on a plan whose spread is another one changes nothing; after
    set_ownership(True) it is the tiled spread."""
    import torch
    rng = np.random.default_rng(C)
    tm = np.concatenate([rng.uniform(-60, 60, (M // 2, 2)), rng.uniform(-3, 3, (M - M // 2, 2))])
    h = [mb.newfft_kb_table(6, 64)] * 2
    plan = mb.InterpPlan(list(K), [6, 6], [64, 64], h, tm, C, order=1)
    fm = rng.standard_normal((M, C)) + 1j * rng.standard_normal((M, C))
    fd = torch.from_numpy(fm.astype(np.complex64)).cuda()
    cfg, out = plan.config(), plan.adjoint(fd)
    plan.set_ownership(False)
    assert plan.config() == cfg
    got = torch.full_like(out, float("nan"))
    assert torch.equal(plan.adjoint(fd, out=got), out)
    ref = oracle.interp_adj(fm, h, [6, 6], [64, 64], tm, list(K), 1, impl=ref_impl())
    assert rel_l2(np.transpose(out.cpu().numpy()[0], (1, 0, 2)).reshape(-1, C, order="F"), ref) <= ADJ_TOL
    if all(k % 16 == 0 for k in K):             # an even number of 8-point tiles per dimension
        plan.set_spread((8, 8))
        plan.set_ownership(True)
        plan.set_ownership(False)
        assert plan.config()["spread_own"] == plan.config()["spread_sweep"] == 0
        assert rel_l2(plan.adjoint(fd).cpu().numpy(), out.cpu().numpy()) <= 5e-6
    plan.close()


def _each_failing_allocation(f, steps=range(400)):
    """Yields f's result, or None where it raised for want of memory, with the n-th device
    allocation failing for the n of steps, until one run needs fewer."""
    lib = mb.load()
    for n in steps:
        lib.mirt_test_fail_alloc(n)
        try:
            out = f()
        except mb.MirtError as e:
            out = None
            assert "memory" in str(e), e
        finally:
            left = lib.mirt_test_fail_alloc(-1)
        yield n, out
        if left >= 0:
            return
    raise AssertionError("allocations without end")


ALLOC_PLANS = [((64, 48), 26, 1500), ((64, 48), 32, 1500), ((96, 80), 32, 30000), ((128, 100), 34, 60000),
               ((16, 14, 12), 8, 6000)]


@pytest.mark.parametrize("K,C,M,what", [
    p + (w,) for p in ALLOC_PLANS for w in ("sweep", "balanced", "dense", "staged", "autotune")
    if not (w == "staged" and p[1] < 32 or w == "autotune" and p[2] > 6000)])
def test_failed_allocations_leave_the_plan_working(K, C, M, what):
    """A setter or the autotuner whose device allocation fails, whichever it is, returns an error
    or does without; the plan computes the adjoint and the forward as before either way, and the
    same call succeeds with memory again."""
    import torch
    D = len(K)
    rng = np.random.default_rng(C + M)
    tm = np.concatenate([rng.uniform(-60, 60, (M // 2, D)), rng.uniform(-3, 3, (M - M // 2, D))])
    h = [mb.newfft_kb_table(6, 64)] * D

    def call(plan):
        if what == "sweep":
            plan.set_sweep(3, 2)
        elif what == "balanced":
            plan.set_sweep(-1 if D == 2 else 1, 4)
        elif what == "dense":
            plan.set_dense(True)
        elif what == "staged":
            plan.set_staged(2)
        else:
            plan.autotune()
        return True
    first = mb.InterpPlan(list(K), [6] * D, [64] * D, h, tm, C, order=1)
    fm = torch.randn(first.sample_shape, dtype=torch.complex64, device="cuda")
    ck = torch.randn(first.grid_shape, dtype=torch.complex64, device="cuda")
    adj, fwd = first.adjoint(fm).cpu().numpy(), first.forward(ck)
    first.close()
    plan = mb.InterpPlan(list(K), [6] * D, [64] * D, h, tm, C, order=1)
    # (the autotuner builds hundreds of tile lists: its first allocations, then one in 197)
    steps = range(400) if what != "autotune" else list(range(8)) + list(range(8, 9999, 197))
    for n, ok in _each_failing_allocation(lambda: call(plan), steps):
        out = torch.full(first.grid_shape, float("nan"), dtype=torch.complex64, device="cuda")
        assert rel_l2(plan.adjoint(fm, out=out).cpu().numpy(), adj) <= 5e-6, (n, ok)
        assert torch.equal(plan.forward(ck), fwd), (n, ok)
        if what != "autotune" and ok is None:   # a plan that has its lists needs none again
            plan.close()
            plan = mb.InterpPlan(list(K), [6] * D, [64] * D, h, tm, C, order=1)
    assert ok
    assert rel_l2(plan.adjoint(fm).cpu().numpy(), adj) <= 5e-6
    plan.close()


_BUFFERS = """
import numpy as np, torch, mirt_b200 as mb
rng = np.random.default_rng(1)
M, C, K = 500000, 256, [256, 256]
tm = rng.uniform(-128, 128, (M, 2))
torch.zeros(1, device='cuda')
mb.InterpPlan([8], [4], [64], [mb.newfft_kb_table(4, 64)], np.zeros((1, 1)), 1, order=1).close()
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
plan = mb.InterpPlan(K, [6, 6], [64, 64], [mb.newfft_kb_table(6, 64)] * 2, tm, C, order=1)
used = free - torch.cuda.mem_get_info()[0]
split = plan.config()["spread_split"]
plan.set_staged(2)
print(split, used, free - torch.cuda.mem_get_info()[0], 8 * M * C)
"""


def test_plan_holds_the_row_sweeps_buffers_when_it_is_selected():
    """500,000 samples of 256 columns whose default is the split spread: the row sweep's copy of
    them, a gigabyte, is there once the row sweep is (in a process of its own, whose allocator
    has no blocks to reuse)."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", _BUFFERS], cwd=root, capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr
    split, used, selected, copy = map(int, out.stdout.split()[-4:])
    assert split == 1 and used < 0.9 * copy and selected > copy


@pytest.mark.parametrize("K,J,C,M", [((64, 48), 6, 26, 7000), ((64, 48), 6, 32, 1500), ((96, 80), 6, 32, 20000),
                                     ((128, 100), 6, 34, 60000), ((40, 36), 6, 5, 900), ((70,), 4, 2, 500),
                                     ((16, 14, 12), 6, 8, 6000), ((16, 14, 12), 5, 3, 600)])
def test_plans_without_room_for_their_spreads_lists(K, J, C, M):
    """Plan creation with each of its device allocations failing in turn: an error or a plan whose
    adjoint and forward are right; a plan where one of the lists, which come last, has found
    no room."""
    import torch
    D = len(K)
    rng = np.random.default_rng(C + M)
    tm = np.concatenate([rng.uniform(-60, 60, (M // 2, D)), rng.uniform(-3, 3, (M - M // 2, D))])
    h = [mb.newfft_kb_table(J, 64)] * D
    make = lambda: mb.InterpPlan(list(K), [J] * D, [64] * D, h, tm, C, order=1)   # noqa: E731
    plan = make()
    fm = torch.randn(plan.sample_shape, dtype=torch.complex64, device="cuda")
    ck = torch.randn(plan.grid_shape, dtype=torch.complex64, device="cuda")
    adj, fwd = plan.adjoint(fm).cpu().numpy(), plan.forward(ck)
    plan.close()
    made = []
    for n, plan in _each_failing_allocation(make):
        made.append(plan is not None)
        if plan is not None:
            out = torch.full(plan.grid_shape, float("nan"), dtype=torch.complex64, device="cuda")
            assert rel_l2(plan.adjoint(fm, out=out).cpu().numpy(), adj) <= 5e-6, n
            assert torch.equal(plan.forward(ck), fwd), n
            plan.close()
    # (the last run needed no failing allocation; before it, the last list's last one failed)
    assert made[-1] and made[-2] and not made[0]


def test_point_spread_counts_stay_sound_after_overlapping_calls():
    """Adjoints of one plan on two streams at once, which a caller is told to order: whatever they
    gave, a later call gives its result, so the counts of the shared bricks are at zero again."""
    import torch
    rng = np.random.default_rng(6)
    tm = np.concatenate([rng.uniform(-32, 32, (2000, 2)), rng.uniform(-2, 2, (60000, 2))])
    plan = mb.InterpPlan([64, 64], [6, 6], [64, 64], [mb.newfft_kb_table(6, 64)] * 2, tm, 8, order=1)
    fm = torch.randn(plan.sample_shape, dtype=torch.complex64, device="cuda")
    ref = plan.adjoint(fm)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [torch.empty_like(ref), torch.empty_like(ref)]
    torch.cuda.synchronize()
    for _ in range(50):
        for st, out in zip(streams, outs):
            plan.adjoint(fm, out=out, stream=st)
    torch.cuda.synchronize()
    assert torch.equal(plan.adjoint(fm), ref)
    plan.close()


def _taps_of(t, J, K):
    """Mask [K_D, ..., K_1] of the grid points that a sample at t reaches."""
    m = np.ones((), bool)
    for d in range(len(K)):
        row = np.zeros(K[d], bool)
        row[(1 + int(np.floor(t[d] - J[d] / 2)) + np.arange(J[d])) % K[d]] = True
        m = np.multiply.outer(row, m)
    return m


@pytest.mark.parametrize("K,J,C", [
    ((50,), (6,), 2), ((64, 48), (6, 6), 1), ((33, 35), (5, 4), 3), ((40, 41), (6, 6), 7),
    ((48, 40), (6, 6), 16), ((48, 40), (6, 6), 26), ((48, 40), (6, 6), 33), ((40, 36), (12, 5), 32),
    ((20, 18, 16), (6, 6, 6), 1), ((17, 14, 13), (5, 4, 3), 5), ((16, 12, 14), (4, 6, 5), 18),
])
@pytest.mark.parametrize("value", ["inf", "nan", "large", "large taps"])
def test_point_spread_keeps_non_finite_samples_to_their_taps(K, J, C, value):
    """A sample that is infinite, NaN or overflows times its taps changes the grid points of its
    own taps alone, all other points keep their bits: the point spread and the split spread
    sum blocks of four points."""
    import torch
    D = len(K)
    rng = np.random.default_rng(sum(K) + C)
    L = [64] * D
    h = [mb.newfft_kb_table(j, 64) for j in J]
    if value == "large taps":
        h[-1] = h[-1] * 2.0 ** 100
    tm = np.concatenate([rng.uniform(-40, 40, (400, D)), rng.uniform(-2, 2, (1500, D))])
    plan = mb.InterpPlan(list(K), list(J), L, h, tm, C, order=1)
    assert plan.config()["spread_points"] > 0
    fm = torch.from_numpy((rng.standard_normal((len(tm), C)) +
                           1j * rng.standard_normal((len(tm), C))).astype(np.complex64)).cuda()
    v = {"inf": complex(np.inf, -np.inf), "nan": complex(np.nan, 0), "large": 3e38 * (1 + 1j),
         "large taps": 2.0 ** 40 * (1 + 1j)}[value]
    for m in (0, 17, 399, 400, 1899):
        fm0, fm1 = fm.clone(), fm.clone()
        fm0[m] = 0
        fm1[m] = v
        a, b = plan.adjoint(fm0).cpu().numpy()[0], plan.adjoint(fm1).cpu().numpy()[0]
        own = _taps_of(tm[m], J, K)
        assert np.array_equal(a[~own], b[~own]), m
        if not value.startswith("large"):
            assert not np.isfinite(b[own]).any(), m
    plan.close()


@pytest.mark.parametrize("K,C,order", [((64, 48), 25, 0), ((41, 50), 32, 1), ((96, 80), 33, 0),
                                       ((6, 7), 64, 0)])
def test_split_spread_matches_oracle(K, C, order):
    """The split spread (the default from 25 columns in 2D, J = 6): a slice of
    even density, an empty one and one with a dense centre, so that some tiles go
    to the point spread and the bands between them to the row sweep; odd grids
    (bands and tiles cut at the end), idle columns and several chunks; the
    oracle's adjoint, bitwise reproducible, and the row sweep's result."""
    import torch
    rng = np.random.default_rng(C + K[0])
    J, L = [6, 6], [256, 256]
    h = ([mb.newfft_kb_table(6, 256)] * 2 if order else
         [mb.minmax_kb_table(max(2, k // 2), 6, k, 256) for k in K])
    tms = [rng.uniform(-60, 60, (900, 2)), np.zeros((0, 2)),
           np.concatenate([rng.uniform(-2, 2, (6000, 2)), rng.uniform(-30, 30, (600, 2))])]
    moff = np.concatenate([[0], np.cumsum([len(t) for t in tms])])
    tm = np.concatenate(tms)
    ph = np.exp(1j * rng.uniform(0, 6, len(tm)))
    plan = mb.InterpPlan(K, J, L, h, tm, C, order=order, slice_moff=moff, phase=ph)
    assert plan.config()["spread_split"] == 1
    fm = rng.standard_normal((len(tm), C)) + 1j * rng.standard_normal((len(tm), C))
    fm_d = torch.from_numpy(fm.astype(np.complex64)).cuda()
    out = plan.adjoint(fm_d).cpu().numpy()
    assert np.array_equal(out, plan.adjoint(fm_d).cpu().numpy())
    for s in range(3):
        sl = slice(moff[s], moff[s + 1])
        got = np.transpose(out[s], (1, 0, 2)).reshape(-1, C, order="F")
        if not len(tms[s]):
            assert not got.any()
            continue
        ref = oracle.interp_adj(fm[sl] * np.conj(ph[sl])[:, None], h, J, L, tms[s], K, order,
                                impl=ref_impl())
        assert rel_l2(got, ref) <= ADJ_TOL, s
    plan.set_sweep(1, 1)
    assert plan.config()["spread_split"] == 0
    assert rel_l2(plan.adjoint(fm_d).cpu().numpy(), out) <= 5e-6
    plan.close()
