"""The subtree-task kernels on the GPU (kernels_task.cuh, kernels_sweep.cuh)
and what the engine keeps around them."""
import numpy as np
import pytest

import cupf
from cupf import grids as G
from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

POLICIES = {p: cupf.ComputePolicy[p] for p in ("FP64", "Mixed", "FP32")}


def _grid(buses):
    return G.make_grid(buses, buses * 3 // 2, buses // 5, seed=1000 + buses)


def _newton(g, policy, graph=False, **custom):
    o = cupf.NewtonOptions(backend=cupf.BackendKind.CUDA, compute=POLICIES[policy])
    o.use_cuda_graph = graph
    o.custom.serial_nd = True
    for k, v in custom.items():
        setattr(o.custom, k, v)
    s = cupf.NewtonSolver(o)
    s.initialize(g.indptr, g.indices, g.data, g.n_bus, g.n_bus, g.pv, g.pq)
    return s


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("policy", ["FP64", "Mixed", "FP32"])
@pytest.mark.parametrize("buses", [118, 400, 2000])  # tree launch; tasks with level sweeps; tasks
def test_padding_columns_of_a_batch_of_one_copy_the_scenario(buses, policy, graph):
    """The tasks of a single system write one of the 32 columns of the factors;
    the padding columns of the state still follow the scenario: every column of
    the padded batch ends with the same mismatch norm."""
    import torch

    g = _grid(buses)
    s = _newton(g, policy, graph)
    tol = 1e-4 if policy == "FP32" else 1e-8
    S = torch.tensor(g.scenarios(1, seed=buses), device="cuda")
    _, fm, _ = s.solve_batch_device(S, torch.tensor(g.flat_start(1), device="cuda"),
                                    config=cupf.NRConfig(tolerance=tol, max_iter=12))
    norms = s.plan_array64("mismatch_norm_bits").view(np.float64)
    assert norms.size == 32 and norms[0] <= tol
    assert (norms == norms[0]).all(), norms


def test_first_solves_on_a_side_stream_wait_for_their_plans():
    """What a solve uploads at the first batch of a class is on the device
    before its kernels run, whatever the default stream has queued."""
    import torch

    g = _grid(500)
    busy = torch.randn(4096, 4096, device="cuda")
    solver, other = _newton(g, "Mixed", autotune=False), torch.cuda.Stream()
    for batch in (300, 1, 200, 20):  # largest first, then the other classes on its workspace
        S = torch.tensor(g.scenarios(batch, seed=batch), device="cuda")
        V0 = torch.tensor(g.flat_start(batch), device="cuda")
        cfg = cupf.NRConfig(tolerance=1e-8, max_iter=10)
        want = _newton(g, "Mixed", autotune=False).solve_batch_device(S, V0, config=cfg)[0]
        torch.cuda.synchronize()
        for _ in range(8):
            busy @ busy
        with torch.cuda.stream(other):
            got = solver.solve_batch_device(S, V0, config=cfg)[0]
        torch.cuda.synchronize()
        assert torch.equal(got, want)


def test_smaller_batches_plan_and_allocate_nothing():
    """The plans of every class a workspace serves come with it; a tree below
    the thresholds gets none."""
    import torch

    def solve(s, g, batch):
        S = torch.tensor(g.scenarios(batch, seed=batch), device="cuda")
        s.solve_batch_device(S, torch.tensor(g.flat_start(batch), device="cuda"),
                             config=cupf.NRConfig(tolerance=1e-8, max_iter=10))
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    small = _newton(_grid(118), "Mixed", autotune=False)
    solve(small, _grid(118), 300)
    assert small.plan_array("task_classes").size == 0
    g = _grid(4000)
    s = _newton(g, "Mixed", autotune=False)
    solve(s, g, 288)
    assert s.plan_array("task_classes").tolist() == [0, 1, 3]
    for batch in (1, 20, 160):  # inputs of these sizes first, so that torch's pool holds them
        torch.tensor(g.scenarios(batch, seed=batch), device="cuda"), torch.tensor(g.flat_start(batch), device="cuda")
    free = solve(s, g, 288)
    for batch in (160, 20, 1):  # the other classes
        assert solve(s, g, batch) == free
    assert s.plan_array("task_classes").tolist() == [0, 1, 3]


@pytest.mark.parametrize("policy", ["FP64", "Mixed"])
@pytest.mark.parametrize("buses,wide", [(200, 0), (2000, 12)])
def test_autotuner_times_the_launches_that_factor(buses, wide, policy):
    """Plans that do run level launches: a tree below the tasks' threshold, and
    the fronts of 12 rows and more (with their ancestors) beside the tasks.
    The tuner times every one of them, and the solves keep their bits."""
    import torch

    g = _grid(buses)
    base = _newton(g, policy, autotune=False, wide_min_front=wide)
    tuned = _newton(g, policy, autotune=True, wide_min_front=wide)
    for batch in (96, 256, 96):
        S = torch.tensor(g.scenarios(batch, seed=9), device="cuda")
        V0 = torch.tensor(g.flat_start(batch), device="cuda")
        cfg = cupf.NRConfig(tolerance=1e-8, max_iter=12)
        a, b = (h.solve_batch_device(S, V0, config=cfg)[0] for h in (base, tuned))
        assert torch.equal(a, b)
        n = tuned.plan_array("factor_rest_warps" if wide else "factor_level_warps").size
        assert n > 0 and tuned.plan_array("factor_tuned_launches").tolist() == ([n, 0] if wide else [0, n])
        assert (tuned.plan_array("task_class")[0] >= 0) == bool(wide)
        if wide:
            assert (tuned.plan_array("factor_rest_tiers") == 1).any()


@pytest.mark.parametrize("schedule_first", [True, False])
def test_batches_of_one_and_of_many_tune_their_own_launches(schedule_first):
    """A batch of one on the lane kernels (batch1_schedule = 1) runs the level
    launches, a batch of 20 the tasks and their rest: neither passes for the
    other's tuning, though their padded batch is the same."""
    import torch

    g = _grid(500)
    s = _newton(g, "Mixed", autotune=True, batch1_schedule=1, wide_min_front=12)
    for batch in ((1, 20) if schedule_first else (20, 1)):
        S = torch.tensor(g.scenarios(batch, seed=9), device="cuda")
        s.solve_batch_device(S, torch.tensor(g.flat_start(batch), device="cuda"),
                             config=cupf.NRConfig(tolerance=1e-8, max_iter=12))
        rest, level = s.plan_array("factor_tuned_launches").tolist()
        assert (level > 0 and rest == 0) if batch == 1 else (rest > 0 and level == 0)


def test_static_scratch_factorization_keeps_its_tuning():
    """cls_factorize_static_scratch runs the level launches, so cls_factorize
    tunes those beside what it runs itself."""
    import torch

    g = _grid(500)
    ls, rp, ci = _linear(g, cupf.CustomPrecision.FP32, autotune=True)
    A, b = _systems(rp, ci, 64, 7, torch.float32)
    ls.setup(64)
    ls.factorize(A)
    want = ls.solve(b)
    assert ls.plan_array("factor_tuned_launches")[1] == ls.plan_array("factor_level_warps").size > 0
    ls.factorize_static_scratch(A)
    assert torch.equal(ls.solve(b), want)


@pytest.mark.parametrize("first,second", [(1290, 1311), (1311, 1290)])
def test_one_padded_batch_has_one_class(first, second):
    """500 buses are 420 fronts: 420 x 1,309 systems is where class 2 begins, and
    1,290 and 1,311 systems have the same padded batch, whose captured solve and
    tuned shapes they share."""
    import torch

    g = _grid(500)
    s = _newton(g, "Mixed", graph=True, autotune=False)
    cls = []
    for batch in (first, second):
        S = torch.tensor(g.scenarios(batch, seed=batch), device="cuda")
        s.solve_batch_device(S, torch.tensor(g.flat_start(batch), device="cuda"),
                             config=cupf.NRConfig(tolerance=1e-8, max_iter=10))
        cls += s.plan_array("task_class").tolist()
    assert cls == [2, 2]


def _linear(g, precision, **config):
    h = cupf.NewtonSolver(cupf.NewtonOptions(backend=cupf.BackendKind.CUDA))
    h.analyze_host(g.indptr, g.indices, g.n_bus, g.pv, g.pq)
    rp, ci = h.plan_array("jac_row_ptr"), h.plan_array("jac_col_idx")
    ls = cupf.LinearSolver(cupf.SolverConfig(precision=int(precision), serial_nd=True, **config))
    ls.set_data(rp, ci)
    ls.analyze()
    return ls, rp, ci


def _systems(rp, ci, batch, seed, dtype):
    """Diagonally dominant values on a pattern, and right-hand sides."""
    import torch

    rng = np.random.default_rng(seed)
    vals = rng.standard_normal((batch, ci.size))
    rows = np.repeat(np.arange(rp.size - 1), np.diff(rp))
    vals[:, rows == ci] += 8.0
    return (torch.tensor(vals, dtype=dtype, device="cuda"),
            torch.tensor(rng.standard_normal((batch, rp.size - 1)), device="cuda"))


@pytest.mark.parametrize("precision", [cupf.CustomPrecision.FP64, cupf.CustomPrecision.FP32])
# task factors under level sweeps (344 fronts); the tree launch under sweep tasks (420); tasks throughout
@pytest.mark.parametrize("buses", [400, 500, 2000])
def test_batch_of_one_sweeps_equal_the_lane_kernels(buses, precision):
    """Solve and transpose solve of a batch of one on the factors its tasks
    left in column 0, against the lane kernels' factors of every column
    (batch1_schedule = 1): the same bits."""
    import torch

    g = _grid(buses)
    dtype = torch.float64 if precision == cupf.CustomPrecision.FP64 else torch.float32
    out = []
    for schedule in (0, 1):
        ls, rp, ci = _linear(g, precision, batch1_schedule=schedule, autotune=False)
        A, b = _systems(rp, ci, 1, 5, dtype)
        ls.setup(1)
        ls.factorize(A)
        if schedule == 0:
            assert (ls.plan_array("task_class")[0] >= 0) == (buses != 500)
            assert ls.plan_array("task_sweeps")[0] == (buses != 400)
        out.append((ls.solve(b), ls.solve_transpose(b)))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


def test_launches_beside_tasks_fit_the_front_scratch():
    """Fronts that an option keeps off the tasks run in launches of their own,
    cut anew.  Dense blocks of 18, 20 and 28 rows in panels of 4: the leaf
    level's launches are 70 fronts of 18 and 20 rows and 64 of 28; without the
    blocks of 18, which the tasks take, the 40 and the 64 are one launch of 104
    at 28 rows, which needs more scratch than either."""
    import scipy.sparse as sp
    import torch

    rng = np.random.default_rng(3)
    sizes = [18] * 30 + [20] * 40 + [28] * 64
    A = sp.block_diag([sp.coo_array(np.ones((n, n))) for n in sizes]).tocsr()
    A.sort_indices()
    n = A.shape[0]
    ls = cupf.LinearSolver(cupf.SolverConfig(precision=int(cupf.CustomPrecision.FP64), serial_nd=True,
                                             max_panel_width=4, wide_min_front=20, autotune=False))
    ls.set_data(A.indptr.astype(np.int32), A.indices.astype(np.int32))
    ls.analyze()
    fsz = ls.plan_array("fp_fsz")
    assert fsz.size >= 300 and fsz.max() == 28
    B = 2
    vals = rng.standard_normal((B, A.nnz))
    rows = np.repeat(np.arange(n), np.diff(A.indptr))
    vals[:, rows == A.indices] += 24.0
    b = rng.standard_normal((B, n))
    ls.setup(B)
    ls.factorize(torch.tensor(vals, device="cuda"))
    x = ls.solve(torch.tensor(b, device="cuda")).cpu().numpy()
    for k in range(B):
        M = sp.csr_matrix((vals[k], A.indices, A.indptr), shape=(n, n))
        # diagonally dominant: growth below 2, n = 28 rows to a block
        assert np.linalg.norm(M @ x[k] - b[k]) <= 1e-13 * np.linalg.norm(b[k])


# batches of every class, odd ones among them: on 2,000 buses (1,671 fronts) a
# single system, little and much work (FP64 from 431 systems on, FP32 539; the
# sweeps 599 and 838), on 500 buses (420 fronts) those in between
@pytest.mark.parametrize("buses,batch,cls", [(2000, 1, 0), (2000, 2, 1), (2000, 33, 1), (2000, 128, 1), (2000, 161, 1),
                                             (2000, 449, (3, 1)), (2000, 517, 3), (2000, 850, 3), (500, 1601, 2)])
@pytest.mark.parametrize("precision", [cupf.CustomPrecision.FP64, cupf.CustomPrecision.FP32])
def test_tasks_solve_like_the_general_kernels(precision, buses, batch, cls):
    """Factor, solve and transpose solve by subtree tasks against the general
    kernels (wide_min_front = 1: the any-size tier and the level sweeps): the
    same solutions, bit for bit."""
    import torch

    g = _grid(buses)
    dtype = torch.float64 if precision == cupf.CustomPrecision.FP64 else torch.float32
    if isinstance(cls, tuple):
        cls = cls[dtype == torch.float32]
    out = []
    for wide in (0, 1):
        ls, rp, ci = _linear(g, precision, autotune=False, wide_min_front=wide)
        A, b = _systems(rp, ci, batch, batch, dtype)
        ls.setup(batch)
        ls.factorize(A)
        assert ls.plan_array("task_class")[0] == (-1 if wide else cls)
        out.append((ls.solve(b), ls.solve_transpose(b)))
        assert not ls.singular_flags().any()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    # and they solve the systems: diagonally dominant rows, so to a few hundred
    # times the unit roundoff
    if batch <= 33:
        rows = torch.tensor(np.repeat(np.arange(rp.size - 1), np.diff(rp)), device="cuda")
        cols = torch.tensor(ci.astype(np.int64), device="cuda")
        eps = torch.finfo(dtype).eps
        for x, r, c in ((out[0][0], rows, cols), (out[0][1], cols, rows)):
            y = torch.zeros_like(b).index_add_(1, r, A.double() * x.double()[:, c])
            assert float((y - b).norm() / b.norm()) <= 300 * eps


@pytest.mark.parametrize("buses,batch,cls", [(2000, 1, 0), (2000, 31, 1), (2000, 161, 1), (2000, 540, 3),
                                             (500, 1500, 2)])
@pytest.mark.parametrize("policy", ["FP64", "Mixed", "FP32"])
def test_newton_and_gradients_of_every_class_keep_the_general_kernels_bits(policy, buses, batch, cls):
    """Two Newton updates, and the gradients at the state they reach, against
    the general kernels."""
    import torch

    g = _grid(buses)
    S, V0 = g.scenarios(batch, seed=batch), g.flat_start(batch)
    grads = np.random.default_rng(batch).standard_normal((2, batch, g.n_bus))
    out = []
    for wide in (0, 1):
        s = _newton(g, policy, autotune=False, wide_min_front=wide)
        so = cupf.SolveOptions(prepare_adjoint_cache=policy != "FP32")  # (the adjoint needs an FP64 state)
        r = s.solve_batch(g.indptr, g.indices, g.data, g.n_bus, g.n_bus, S, V0, g.pv, g.pq,
                          cupf.NRConfig(tolerance=1e-12, max_iter=2), so)
        assert s.plan_array("task_class")[0] == (-1 if wide else cls)
        out.append([r.V_numpy])
        if policy != "FP32":
            a = s.solve_adjoint(*grads, g.pv, g.pq)
            out[-1] += [a.lambda_numpy, a.grad_load_p_numpy, a.grad_load_q_numpy]
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.parametrize("precision", [cupf.CustomPrecision.FP64, cupf.CustomPrecision.FP32])
# buses, batch, factored by tasks, swept by tasks: trees on both sides of each
# rule (tasks_pay, sweep_tasks_pay)
@pytest.mark.parametrize("buses,batch,factor,sweep", [
    (300, 64, False, False),   # 254 fronts
    (500, 1, False, True),     # the tree launch is faster than a long chain of fronts
    (700, 1, True, False),
    (480, 2, False, False),    # a heaviest chain of more than twice the tree's longest path
    (480, 33, True, False),    # one sweep task of 37 fronts, 12 levels
    (600, 2, True, True),
    (480, 2048, True, True),   # much work: the levels' cost grows with the batch, the chain's does not
])
def test_small_trees_take_the_faster_schedule_with_the_same_bits(buses, batch, factor, sweep, precision):
    import torch

    g = _grid(buses)
    dtype = torch.float64 if precision == cupf.CustomPrecision.FP64 else torch.float32
    out = []
    for wide in (0, 1):
        ls, rp, ci = _linear(g, precision, autotune=False, wide_min_front=wide)
        A, b = _systems(rp, ci, batch, batch, dtype)
        ls.setup(batch)
        ls.factorize(A)
        if not wide:
            assert (ls.plan_array("task_class")[0] >= 0) == factor and ls.plan_array("task_sweeps")[0] == sweep
        out.append((ls.solve(b), ls.solve_transpose(b)))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("batch", [1, 33, 1700])  # the classes' team shapes
@pytest.mark.parametrize("width", [8, 3])
@pytest.mark.parametrize("precision", [cupf.CustomPrecision.FP64, cupf.CustomPrecision.FP32])
def test_fronts_of_every_size_factor_and_solve(precision, width, batch):
    """Dense diagonally dominant blocks of 1 to 66 rows: fronts of every size a
    task takes, with every number of pivots, and those beside the tasks; the
    general kernels' bits, and residuals to the rounding of an LU of such
    blocks."""
    import scipy.sparse as sp
    import torch

    rng = np.random.default_rng(width)
    sizes = list(range(1, 67)) * (2 if width == 8 else 1)
    A = sp.block_diag([sp.coo_array(np.ones((n, n))) for n in sizes]).tocsr()
    A.sort_indices()
    n = A.shape[0]
    rp, ci = A.indptr.astype(np.int32), A.indices.astype(np.int32)
    dtype = torch.float64 if precision == cupf.CustomPrecision.FP64 else torch.float32
    rows = np.repeat(np.arange(n), np.diff(rp))
    gen = torch.Generator(device="cuda").manual_seed(batch)
    vals = torch.randn(batch, ci.size, device="cuda", generator=gen, dtype=dtype)
    vals[:, torch.tensor(rows == ci, device="cuda")] += 40.0
    b = torch.tensor(rng.standard_normal((batch, n)), device="cuda")
    out = []
    for wide in (0, 1):
        ls = cupf.LinearSolver(cupf.SolverConfig(precision=int(precision), serial_nd=True, max_panel_width=width,
                                                 wide_min_front=wide, autotune=False))
        ls.set_data(rp, ci)
        ls.analyze()
        ls.setup(batch)
        ls.factorize(vals)
        assert not ls.singular_flags().any()
        out.append((ls.solve(b), ls.solve_transpose(b)))
        del ls
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    # unpivoted LU of diagonally dominant blocks: growth below 2, so the backward
    # error is at most a few times the rows of a block x the unit roundoff
    r, c = torch.tensor(rows, device="cuda"), torch.tensor(ci.astype(np.int64), device="cuda")
    for x, i, j in ((out[0][0][:4], r, c), (out[0][1][:4], c, r)):
        y = torch.zeros_like(b[:4]).index_add_(1, i, vals[:4].double() * x.double()[:, j])
        assert float((y - b[:4]).norm() / b[:4].norm()) <= 4 * 66 * torch.finfo(dtype).eps
