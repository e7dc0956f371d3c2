"""The subtree-task programs of the factorization (task_plan.cpp), run by a
plain restatement of the kernel on the CPU: every arena access lies inside the
task's arena and reads what the task wrote there, every front is factored by
exactly one task, after its children, and the U rows and contribution blocks
are those of a dense unpivoted LU of the permuted matrix."""
from pathlib import Path

import numpy as np
import pytest

import cupf
from cupf import grids as G

GOLD = Path(__file__).resolve().parent / "golden"
WORDS = 12  # words of a front record before its lists


class _Arena:
    """Values with an owner tag per element: reading an element that was not
    written since its region was handed out is an error (NaN)."""

    def __init__(self, n):
        self.v = np.full(n, np.nan)


def _lists(w):
    nj, nz = w[7] & 0xffff, (w[7] >> 16) & 0xffff
    npass = w[8]
    cnt = w[WORDS:WORDS + npass]
    ext = w[WORDS + npass:WORDS + npass + 3 * w[9]].reshape(-1, 3)
    a = WORDS + npass + 3 * w[9]
    jsrc = w[a:a + nj]
    terms = w[a + nj:a + nj + cnt.sum()].copy().view(np.uint32).astype(np.int64)
    assert w[11] == a + nj + cnt.sum()
    h = w[w[11]:w[10]].copy().view(np.uint16).astype(np.int64)
    jdst, zdst = h[:nj], h[nj:nj + nz]
    dst, src, o = terms[:cnt[0] if npass else 0] & 0xffff, [], 0
    for c in cnt:
        assert (terms[o:o + c] & 0xffff == dst[:c]).all()
        src.append(terms[o:o + c] >> 16)
        o += c
    return cnt, ext, jsrc, jdst, zdst, dst, src


def run_tasks(s, vals, rhs, cls):
    """Factor vals (CSR order) with right-hand side rhs (pivot order) by the
    task programs; returns {element: value} arrays U, CB (NaN where not
    written), y, and the fronts' count per stage."""
    meta = s.plan_array(f"task_meta:{cls}").reshape(-1, 4)
    words = s.plan_array(f"task_words:{cls}")
    stages = s.plan_array(f"task_stages:{cls}").reshape(-1, 5)
    u_off, cb_off = s.plan_array64("u_off"), s.plan_array64("cb_off")
    U, CB = np.full(u_off[-1], np.nan), np.full(cb_off[-1], np.nan)
    y = np.full(rhs.size, np.nan)
    assert [int(b) for b in stages[:, 0]] == list(np.cumsum(np.r_[0, stages[:-1, 1]])) and stages[:, 1].sum() == len(meta)
    for b, n, max_words, max_arena, _ in stages:
        cb_new = CB.copy()  # a stage sees the blocks of earlier stages only
        for off, nw, nf, _ in meta[b:b + n]:
            assert off % 4 == 0 and nw % 4 == 0 and nw <= max_words
            w0 = words[off:off + nw]
            recs, at = [], 0
            for _ in range(nf):
                recs.append(w0[at:])
                at += w0[at + 10]
            assert at <= nw
            A = np.full(max_arena, np.nan)

            def fetch(w):
                fs, nc = w[0] & 0xff, (w[0] >> 8) & 0xff
                rs = 9 if fs <= 8 else (fs + 1) | 1
                _, ext, jsrc, jdst, zdst, _, _ = _lists(w)
                F = w[5]
                assert F + fs * rs <= max_arena
                seen = np.zeros(fs * rs, bool)
                for d in (jdst, zdst, np.arange(nc) * rs + fs):
                    assert not seen[d].any() and (d < fs * rs).all()
                    seen[d] = True
                assert seen.reshape(fs, rs)[:, :fs + 1].all()
                A[F:F + fs * rs] = np.nan
                A[F + jdst] = vals[jsrc]
                A[F + zdst] = 0.0
                A[F + np.arange(nc) * rs + fs] = rhs[w[1]:w[1] + nc]
                for co, k, to in ext:
                    assert to + k <= max_arena
                    A[to:to + k] = CB[co:co + k]

            fetch(recs[0])
            for i, w in enumerate(recs):
                fs, nc, leaves = w[0] & 0xff, (w[0] >> 8) & 0xff, w[0] >> 16
                rs, uc, F = 9 if fs <= 8 else (fs + 1) | 1, fs - nc, w[5]
                assert leaves or i < nf - 1
                cnt, _, _, _, _, dst, src = _lists(w)
                assert (np.diff(cnt) <= 0).all() and (cnt.size == 0 or cnt[0] == dst.size)
                assert np.unique(dst).size == dst.size
                for p, q in enumerate(src):
                    assert not np.isnan(A[q]).any()
                    A[F + dst[:q.size]] += A[q]
                if i + 1 < nf:
                    fetch(recs[i + 1])
                M = A[F:F + fs * rs].reshape(fs, rs)[:, :fs + 1].copy()
                assert not np.isnan(M).any()
                for k in range(nc):
                    M[k + 1:, k] /= M[k, k]
                    M[k + 1:, k + 1:] -= np.outer(M[k + 1:, k], M[k, k + 1:])
                assert np.isnan(U[w[2]:w[2] + nc * fs]).all()  # once
                U[w[2]:w[2] + nc * fs] = M[:nc, :fs].ravel()
                y[w[1]:w[1] + nc] = M[:nc, fs]
                if uc:
                    if leaves:
                        cb_new[w[4]:w[4] + uc * (uc + 1)] = M[nc:, nc:].ravel()
                    else:
                        assert 0 <= w[6] and w[6] + uc * (uc + 1) <= max_arena
                        A[w[6]:w[6] + uc * (uc + 1)] = M[nc:, nc:].ravel()
        CB = cb_new
    return U, CB, y


def _check(s, n, rp, ci, vals, cls):
    rng = np.random.default_rng(0)
    perm = s.plan_array("perm")
    rhs = rng.standard_normal(n)
    U, CB, y = run_tasks(s, vals, rhs[perm], cls)
    A = np.zeros((n, n))
    A[np.repeat(np.arange(n), np.diff(rp)), ci] = vals
    M = np.c_[A[perm][:, perm], rhs[perm]]
    for k in range(n):  # dense unpivoted LU in the engine's order
        r = np.flatnonzero(M[k + 1:, k]) + k + 1
        M[r, k] /= M[k, k]
        M[np.ix_(r, np.arange(k + 1, n + 1))] -= np.outer(M[r, k], M[k, k + 1:])
    fsz, nc, first = s.plan_array("fp_fsz"), s.plan_array("fp_nc"), s.plan_array("panel_first")
    fptr, frows, u_off = s.plan_array("front_ptr"), s.plan_array("front_rows"), s.plan_array64("u_off")
    done = ~np.isnan(y)
    for p in range(fsz.size):
        if not done[first[p]]:
            continue
        rows = frows[fptr[p]:fptr[p + 1]]
        got = U[u_off[p]:u_off[p] + nc[p] * fsz[p]].reshape(nc[p], fsz[p])
        want = M[np.ix_(np.arange(first[p], first[p] + nc[p]), rows)]
        np.testing.assert_allclose(got, want, rtol=1e-9, atol=1e-9 * np.abs(want).max())
        np.testing.assert_allclose(y[first[p]:first[p] + nc[p]], M[first[p]:first[p] + nc[p], n], rtol=1e-7, atol=1e-9)
    return done


def run_sweep(s, mode, U, L, rhs, cls):
    """One sweep (0 L y = b, 1 U^T w = g, 2 L^T z = w) by the task
    programs on factor elements U and L21 (flat); pivot order throughout."""
    meta = s.plan_array(f"task_sweep_meta:{cls}").reshape(-1, 4)
    words = s.plan_array(f"task_sweep_words:{cls}")
    stages = s.plan_array(f"task_sweep_stages:{cls}").reshape(-1, 9)
    uc_all = (s.plan_array("fp_fsz") - s.plan_array("fp_nc")).astype(np.int64)
    TV = np.full(uc_all.sum(), np.nan)
    W, X = rhs.copy(), np.full(rhs.size, np.nan)
    solved = np.zeros(rhs.size, bool)
    assert stages[:, 1].sum() == len(meta)
    for b, n, max_words, max_local, max_arena, max_rows, max_u, max_l, warps in (stages if mode < 2 else stages[::-1]):
        tv_new, x_new = TV.copy(), X.copy()  # a stage sees earlier stages only
        for off, nw, nf, nx in meta[b:b + n]:
            assert off % 4 == 0 and nw % 4 == 0 and nw <= max_words
            prog = words[off:off + nw]
            recs = [prog[o:] for o in prog[:nf]]
            x = np.full(max_local, np.nan)
            A = np.full(max_arena, np.nan)

            def fetch(w):
                e = w[12 + w[7]:12 + w[7] + 3 * w[8]].reshape(-1, 3)
                for to, k, at in e:
                    assert at + k <= max_arena
                    A[at:at + k] = TV[to:to + k]

            root = recs[-1]
            e0 = root[4] + (root[0] >> 16)
            assert e0 + nx <= max_local
            x[e0:e0 + nx] = X[prog[nf:nf + nx]]
            ahead = 1 if warps == 1 else 3  # fronts between a child vector's request and its use
            if mode < 2:
                for w in recs[:ahead]:
                    fetch(w)
            for i, w in (list(enumerate(recs)) if mode < 2 else list(enumerate(recs))[::-1]):
                fs, nc = w[0] & 0xffff, w[0] >> 16
                uc, first, npass = fs - nc, w[1], w[7]
                assert nc * fs <= max_u and uc * nc <= max_l and fs <= max_rows
                Uf, Lf = U[w[2]:w[2] + nc * fs].reshape(nc, fs), L[w[3]:w[3] + uc * nc].reshape(uc, nc)
                h = prog[prog[i] + w[9]:].copy().view(np.uint16).astype(np.int64)
                loc, rows = h[:uc], h[uc:uc + fs]
                assert not solved[first:first + nc].any()
                solved[first:first + nc] = True
                if mode < 2:
                    t, o = np.zeros(fs), uc + fs
                    assert sorted(rows) == list(range(fs))
                    for c in w[12:12 + npass]:
                        assert not np.isnan(A[h[o:o + c]]).any()
                        t[rows[:c]] += A[h[o:o + c]]
                        o += c
                    if i + ahead < nf:
                        fetch(recs[i + ahead])
                    r = W[first:first + nc] - t[:nc]
                    if mode == 0:
                        v = np.linalg.solve(np.tril(Uf[:, :nc], -1) + np.eye(nc), r)
                        tv = t[nc:] + Lf @ v
                    else:
                        v = np.linalg.solve(np.triu(Uf[:, :nc]).T, r)
                        tv = t[nc:] + Uf[:, nc:].T @ v
                    W[first:first + nc] = v
                    if w[6] < 0:
                        tv_new[w[5]:w[5] + uc] = tv
                    elif uc:
                        assert i < nf - 1 and w[6] + uc <= max_arena
                        A[w[6]:w[6] + uc] = tv
                else:
                    assert not np.isnan(x[loc]).any()
                    r = W[first:first + nc] - Lf.T @ x[loc]
                    v = np.linalg.solve((np.tril(Uf[:, :nc], -1) + np.eye(nc)).T, r)
                    assert w[4] + nc <= e0
                    x[w[4]:w[4] + nc] = x_new[first:first + nc] = v
        TV, X = tv_new, x_new
    assert solved.all()
    return W if mode < 2 else X


@pytest.mark.parametrize("cls", [0, 3])  # the classes' stages, of which 1 and 2 share class 0's
@pytest.mark.parametrize("buses", [5, 118, 500, 2000])
def test_sweep_programs_solve_like_dense_triangles(buses, cls):
    """The three sweeps against dense triangular solves with random factors of
    the plan's own pattern."""
    import scipy.linalg as sla

    g = G.make_grid(buses, buses * 3 // 2, buses // 5, seed=1000 + buses)
    s = cupf.NewtonSolver(cupf.NewtonOptions(backend=cupf.BackendKind.CUDA))
    s.analyze_host(g.indptr, g.indices, g.n_bus, g.pv, g.pq)
    fsz, nc, first = s.plan_array("fp_fsz"), s.plan_array("fp_nc"), s.plan_array("panel_first")
    fptr, frows, u_off = s.plan_array("front_ptr"), s.plan_array("front_rows"), s.plan_array64("u_off")
    n = int(nc.sum())
    rng = np.random.default_rng(2)
    U = 0.2 * rng.standard_normal(u_off[-1])
    l_off = np.r_[0, np.cumsum((fsz - nc).astype(np.int64) * nc)]
    L = 0.2 * rng.standard_normal(l_off[-1])
    Ud, Ld = np.zeros((n, n)), np.eye(n)
    for p in range(fsz.size):
        rows = frows[fptr[p]:fptr[p + 1]]
        Uf = U[u_off[p]:u_off[p + 1]].reshape(nc[p], fsz[p])
        Uf[np.arange(nc[p]), np.arange(nc[p])] += 4.0
        for k in range(nc[p]):
            Ud[first[p] + k, rows[k:]] = Uf[k, k:]
            Ld[first[p] + k, rows[:k]] = Uf[k, :k]
        Ld[np.ix_(rows[nc[p]:], rows[:nc[p]])] = L[l_off[p]:l_off[p + 1]].reshape(-1, nc[p])
    b = rng.standard_normal(n)
    for mode, (M, lower, trans) in enumerate([(Ld, True, 0), (Ud, False, 1), (Ld, True, 1)]):
        want = sla.solve_triangular(M, b, lower=lower, trans=trans)
        np.testing.assert_allclose(run_sweep(s, mode, U, L, b, cls), want, rtol=1e-8, atol=1e-9 * np.abs(want).max())


@pytest.mark.parametrize("cls", [0, 1, 2, 3])  # the batch classes' stages
@pytest.mark.parametrize("buses", [5, 118, 500])
def test_task_programs_factor_like_a_dense_lu(buses, cls):
    g = G.make_grid(buses, buses * 3 // 2, buses // 5, seed=1000 + buses)
    o = cupf.NewtonOptions()
    o.backend = cupf.BackendKind.CUDA
    o.custom.serial_nd = True
    s = cupf.NewtonSolver(o)
    s.analyze_host(g.indptr, g.indices, g.n_bus, g.pv, g.pq)
    rp, ci = s.plan_array("jac_row_ptr"), s.plan_array("jac_col_idx")
    n = rp.size - 1
    vals = np.random.default_rng(1).standard_normal(ci.size)
    rows = np.repeat(np.arange(n), np.diff(rp))
    vals[rows == ci] += 8.0
    assert _check(s, n, rp, ci, vals, cls).all()


@pytest.mark.parametrize("limit", [0, 9])
def test_task_programs_of_a_reference_system(limit):
    """case118's Jacobian; with fronts of 9 rows and more (and their
    ancestors) left to the any-size tier."""
    d = np.load(GOLD / "linsys_case118.npz")
    ls = cupf.LinearSolver(cupf.SolverConfig(precision=int(cupf.CustomPrecision.FP64), wide_min_front=limit))
    ls.set_data(d["row_ptr"], d["col_idx"])
    ls.analyze_host()
    n = d["row_ptr"].size - 1
    vals = np.random.default_rng(1).standard_normal(d["col_idx"].size)
    rows = np.repeat(np.arange(n), np.diff(d["row_ptr"]))
    vals[rows == d["col_idx"]] += 8.0
    nc, uc = ls.plan_array("fp_nc").astype(np.int64), ls.plan_array("fp_fsz") - ls.plan_array("fp_nc")
    ls.plan_array64 = {"u_off": np.r_[0, np.cumsum(nc * (nc + uc))], "cb_off": np.r_[0, np.cumsum(uc * (uc + 1))]}.get
    done = _check(ls, n, d["row_ptr"], d["col_idx"], vals, 1)
    fsz, first, parent = ls.plan_array("fp_fsz"), ls.plan_array("panel_first"), ls.plan_array("panel_parent")
    for p in range(fsz.size):
        kept_out = limit and fsz[p] >= limit
        assert not (kept_out and done[first[p]])
        if parent[p] >= 0 and done[first[parent[p]]]:
            assert done[first[p]]
    assert done.all() if not limit else (done.any() and not done.all())


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [(cupf.CustomPrecision.FP64, 1e-12), (cupf.CustomPrecision.FP32, 2e-4)])
@pytest.mark.parametrize("n", [1, 3, 24, 70, 130])
def test_dense_systems_factor_and_solve(n, precision, tol):
    """Dense diagonally dominant systems of one chain of fronts, up to 130 rows:
    small trees, on the single-system tree, the level launches and, from 65
    rows on, the any-size tier.  Residuals to the rounding of an LU of
    these matrices (condition below 10; n x the unit roundoff x a factor of
    about 50)."""
    import torch

    rng = np.random.default_rng(n)
    rp = (np.arange(n + 1) * n).astype(np.int32)
    ci = np.tile(np.arange(n, dtype=np.int32), n)
    for B in (1, 2, 33):
        A = rng.standard_normal((B, n, n)) + 4.0 * np.sqrt(n) * np.eye(n)
        b = rng.standard_normal((B, n))
        ls = cupf.LinearSolver(cupf.SolverConfig(precision=int(precision), autotune=False))
        ls.set_data(rp, ci)
        ls.analyze()
        ls.setup(B)
        dt = torch.float64 if precision == cupf.CustomPrecision.FP64 else torch.float32
        ls.factorize(torch.tensor(A.reshape(B, -1), dtype=dt, device="cuda"))
        rhs = torch.tensor(b, device="cuda")
        x, xt = ls.solve(rhs).cpu().numpy(), ls.solve_transpose(rhs).cpu().numpy()
        assert not ls.singular_flags().any()
        for M, v in ((A, x), (A.transpose(0, 2, 1), xt)):
            r = np.linalg.norm(np.einsum("bij,bj->bi", M, v) - b, axis=1) / np.linalg.norm(b, axis=1)
            assert r.max() <= tol, (B, r.max())


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 2, 31, 32, 33, 130, 500])
@pytest.mark.parametrize("policy", ["FP64", "Mixed", "FP32"])
def test_tasks_give_the_level_kernels_factors(batch, policy):
    """Solves of a 420-front grid on its schedule (the tree launch for one system,
    class 1's tasks for more) against the any-size tier (wide_min_front = 1
    leaves every front to it): the factors are the same bits, and so are the
    voltages of the first updates.  test_gpu_task_stages.py has every class."""
    import torch

    g = G.grid_500()
    out = []
    for wide in (0, 1):
        o = cupf.NewtonOptions(backend=cupf.BackendKind.CUDA, compute=cupf.ComputePolicy[policy])
        o.custom.serial_nd = True
        o.custom.autotune = False
        o.custom.wide_min_front = wide
        s = cupf.NewtonSolver(o)
        s.initialize(g.indptr, g.indices, g.data, g.n_bus, g.n_bus, g.pv, g.pq)
        S = torch.tensor(g.scenarios(batch, seed=batch), device="cuda")
        V0 = torch.tensor(g.flat_start(batch), device="cuda")
        out.append(s.solve_batch_device(S, V0, config=cupf.NRConfig(tolerance=1e-12, max_iter=2))[0])
    assert torch.equal(out[0], out[1])


def test_task_arrays_have_exact_names():
    """Names of plan arrays are not prefixes, and a class is one of 0 to 3."""
    g = G.make_grid(60, 90, 12, seed=1060)
    s = cupf.NewtonSolver(cupf.NewtonOptions(backend=cupf.BackendKind.CUDA))
    s.analyze_host(g.indptr, g.indices, g.n_bus, g.pv, g.pq)
    for name in ("task_meta", "task_meta:3", "task_words:0", "task_sweep_stages:1"):
        assert s.plan_array(name).size
    assert s.plan_array("task_class").tolist() == [-1] and s.plan_array("task_classes").size == 0
    for name in ("task_metadata", "task_stages_", "task_sweep_", "task_words:4", "task_words:", "task_words:0x"):
        with pytest.raises(Exception):
            s.plan_array(name)
