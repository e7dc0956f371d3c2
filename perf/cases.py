"""The measured work of this framework, through its public entry points.

The listed cases are what its users have it do: one power flow as an operator
asks for it (batch 1), scenario batches of thousands of load draws in each
precision, an odd-sized branch sweep with its own admittances per scenario,
the learned warm start's network (inference and a training step), solves
started near the solution, gradients through torch, and the linear solver on
its own.  Grids, load draws and tolerances are those of the repository's
benchmark and tests (cupf.grids).  draw() gives further sizes of the same
ranges.  exact() solves the same problems in 64 bits with plain torch.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parent.parent / "gpu-powerflow_b200"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

import cupf  # noqa: E402
from cupf import grids  # noqa: E402
from cupf.warm_start import WarmStart, nominal_state  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # one interactive power flow on a small grid, FP64, the reference's basic call: latency and launches
        {"name": "one_118_fp64", "kind": "newton", "buses": 118, "batch": 1, "compute": "FP64", "graph": True},
        # the same on a medium transmission grid in the default precision
        {"name": "one_2000_mixed", "kind": "newton", "buses": 2000, "batch": 1, "compute": "Mixed", "graph": True},
        # a contingency-style sweep: an odd batch with its own branch admittances per scenario, default options
        {"name": "sweep_500x77_ybus", "kind": "newton", "buses": 500, "batch": 77, "compute": "Mixed",
         "graph": False, "ybus": True},
        # a host caller of the reference's batch entry point, all-FP32 policy at its reachable tolerance
        {"name": "host_118x256_fp32", "kind": "host", "buses": 118, "batch": 256, "compute": "FP32", "graph": False},
        # the headline workload: thousands of load scenarios of one grid, plain FP64 ...
        {"name": "batch_2000x1024_fp64", "kind": "newton", "buses": 2000, "batch": 1024, "compute": "FP64",
         "graph": True},
        # ... and in the default precision
        {"name": "batch_2000x1024_mixed", "kind": "newton", "buses": 2000, "batch": 1024, "compute": "Mixed",
         "graph": True},
        # the same scenarios started from a prediction of the state
        {"name": "warm_2000x1024_mixed", "kind": "warm", "buses": 2000, "batch": 1024, "compute": "Mixed",
         "graph": True},
        # the differentiable large grid: forward and backward through torch.autograd
        {"name": "grad_10000x64", "kind": "grad", "buses": 10000, "batch": 64, "compute": "Mixed", "graph": True},
        # the sparse direct solver on its own: factorize, solve and transpose solve of a batch of Jacobians
        {"name": "linear_2000x1024_fp32", "kind": "linear", "buses": 2000, "batch": 1024, "precision": "FP32"},
        {"name": "linear_500x200_fp64", "kind": "linear", "buses": 500, "batch": 200, "precision": "FP64"},
        # the warm-start network: predictions for a batch, and one training step
        {"name": "predict_2000x1024", "kind": "predict", "buses": 2000, "batch": 1024, "hidden": 1024},
        {"name": "train_2000x1024", "kind": "train", "buses": 2000, "batch": 1024, "hidden": 1024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["newton", "newton", "newton", "host", "warm", "grad", "linear", "linear", "predict", "train"])
    buses = _log_int(rng, 60, 2500)
    batch = min(_log_int(rng, 1, 2048), 2_000_000 // buses)
    if kind == "newton":
        compute = rng.choice(["FP64", "Mixed", "Mixed", "FP32"])
        return {"kind": kind, "buses": buses, "batch": batch, "compute": compute, "graph": rng.random() < 0.6,
                "ybus": compute != "FP32" and rng.random() < 0.25}
    if kind == "host":
        return {"kind": kind, "buses": buses, "batch": min(batch, 300_000 // buses + 1),
                "compute": rng.choice(["FP64", "Mixed"]), "graph": rng.random() < 0.5}
    if kind == "warm":
        return {"kind": kind, "buses": buses, "batch": batch, "compute": rng.choice(["FP64", "Mixed"]), "graph": True}
    if kind == "grad":
        if rng.random() < 0.3:  # the large grid with fewer scenarios
            return {"kind": kind, "buses": 10000, "batch": _log_int(rng, 1, 60), "compute": "Mixed", "graph": True}
        return {"kind": kind, "buses": buses, "batch": min(batch, 512), "compute": rng.choice(["FP64", "Mixed"]),
                "graph": rng.random() < 0.5}
    if kind == "linear":
        return {"kind": kind, "buses": buses, "batch": min(batch, 1_000_000 // buses),
                "precision": rng.choice(["FP32", "FP64"])}
    buses = _log_int(rng, 100, 2000)
    hidden = rng.choice([256, 512, 1024])
    if kind == "predict":  # any number of scenarios
        return {"kind": kind, "buses": buses, "batch": _log_int(rng, 1, 1024), "hidden": hidden}
    return {"kind": kind, "buses": buses, "batch": 128 * rng.randint(1, 8), "hidden": hidden}


# ---------------------------------------------------------------------------
# What a user's program keeps: the grid, and one solver handle per workload.
# ---------------------------------------------------------------------------
_GRIDS: dict = {}
_SOLVERS: dict = {}


def _grid(buses):
    if buses not in _GRIDS:
        pv = 53 if buses == 118 else buses // 5
        br = 186 if buses == 118 else buses * 3 // 2
        _GRIDS[buses] = grids.make_grid(buses, br, pv, seed=1000 + buses)
    return _GRIDS[buses]


def _solver(case):
    key = (case["kind"], case["buses"], case["batch"], case["compute"], case["graph"])
    if key not in _SOLVERS:
        while len(_SOLVERS) >= 3:  # a handle holds the arenas of its batch
            _SOLVERS.pop(next(iter(_SOLVERS)))
        g = _grid(case["buses"])
        o = cupf.NewtonOptions()
        o.backend = cupf.BackendKind.CUDA
        o.compute = cupf.ComputePolicy[case["compute"]]
        o.use_cuda_graph = case["graph"]
        o.custom.serial_nd = True
        s = cupf.NewtonSolver(o)
        s.initialize(g.indptr, g.indices, g.data, g.n_bus, g.n_bus, g.pv, g.pq)
        _SOLVERS[key] = s
    return _SOLVERS[key]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _loads(g, batch, seed):
    """Every bus load scaled by its own U(0.8, 1.2) factor: complex128 [batch, n]."""
    f = 0.8 + 0.4 * torch.rand(batch, g.n_bus, generator=_gen(seed), device=DEV, dtype=torch.float64)
    return f * torch.tensor(g.sload, device=DEV)


def _scenarios(g, batch, seed):
    return torch.tensor(g.sgen, device=DEV) - _loads(g, batch, seed)


def _ybus(g, batch, seed):
    """Per-scenario Ybus values [batch, nnz]: the series admittance of every
    bus pair scaled by its own U(0.9, 1.1) factor, shunts kept."""
    rows, cols = _coo(g)
    off = torch.nonzero(rows != cols).flatten()
    lo, hi = torch.minimum(rows[off], cols[off]), torch.maximum(rows[off], cols[off])
    _, pair = torch.unique(lo * g.n_bus + hi, return_inverse=True)
    f = 0.9 + 0.2 * torch.rand(batch, int(pair.max()) + 1, generator=_gen(seed), device=DEV, dtype=torch.float64)
    fo = f[:, pair]
    base = torch.tensor(g.data, device=DEV)
    y = base.repeat(batch, 1)
    y[:, off] = base[off] * fo
    d = torch.zeros_like(y)
    d[:, off] = -(fo - 1.0) * base[off]
    delta = _row_sums(g.indptr, d)
    dpos = torch.nonzero(rows == cols).flatten()
    y[:, dpos] += delta[:, rows[dpos]]
    return y.contiguous()


def _tol(case):
    return 1e-4 if case.get("compute") == "FP32" else 1e-8


def prepare(case, seed):
    g = _grid(case["buses"])
    kind, B = case["kind"], case["batch"]
    s = {"kind": kind}
    if kind in ("newton", "warm", "host", "grad"):
        s["solver"] = _solver(case)
        s["config"] = cupf.NRConfig(tolerance=_tol(case), max_iter=10)
    if kind == "newton":
        s["S"] = _scenarios(g, B, seed)
        s["V0"] = torch.tensor(g.v0, device=DEV).repeat(B, 1)
        s["ybus"] = _ybus(g, B, seed + 1) if case.get("ybus") else None
    elif kind == "host":
        s["grid"] = g
        s["S"] = _scenarios(g, B, seed).cpu().numpy()
        s["V0"] = g.flat_start(B)
    elif kind == "warm":
        s["S"] = _scenarios(g, B, seed)
        s["v0"] = torch.tensor(g.v0, device=DEV)
        pvpq = torch.tensor(np.r_[g.pv, g.pq].astype(np.int64), device=DEV)
        pq = torch.tensor(g.pq.astype(np.int64), device=DEV)
        vref = nominal_state(s["solver"], g)
        x = torch.cat([torch.angle(vref)[pvpq], torch.abs(vref)[pq]]).float()
        s["pred"] = x.repeat(B, 1)  # the state of the nominal load, predicted for every scenario
    elif kind == "grad":
        ld = _loads(g, B, seed)
        s["p"] = ld.real.float().contiguous().requires_grad_()
        s["q"] = ld.imag.float().contiguous().requires_grad_()
        f32 = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device=DEV)  # noqa: E731
        s["kw"] = {"sbus_base_re": f32(g.sgen.real), "sbus_base_im": f32(g.sgen.imag),
                   "v0_va": f32(np.angle(g.v0)), "v0_vm": f32(np.abs(g.v0)), "config": s["config"]}
    elif kind == "linear":
        key = (kind, case["buses"], B, case["precision"])
        rp, ci, _, _, _ = _jacobian_pattern(g)
        if key not in _SOLVERS:
            while len(_SOLVERS) >= 3:
                _SOLVERS.pop(next(iter(_SOLVERS)))
            ls = cupf.LinearSolver(cupf.SolverConfig(precision=int(cupf.CustomPrecision[case["precision"]])))
            ls.set_data(rp, ci)
            ls.analyze()
            ls.setup(B)
            _SOLVERS[key] = ls
        s["ls"] = _SOLVERS[key]
        gen = _gen(seed)
        r = lambda k: torch.randn(B, k, generator=gen, device=DEV, dtype=torch.float64)  # noqa: E731
        V = torch.polar(torch.tensor(np.abs(g.v0), device=DEV) * (1 + 0.02 * r(g.n_bus)), 0.02 * r(g.n_bus))
        dt = torch.float64 if case["precision"] == "FP64" else torch.float32
        s["A"] = _jacobian_values(g, V).to(dt)
        s["b"] = r(rp.size - 1)
    else:
        ws = WarmStart(g, hidden=case["hidden"], layers=3, seed=seed)
        gen = _gen(seed)
        f = lambda *k: torch.rand(*k, generator=gen, device=DEV)  # noqa: E731
        X = ws.features(_scenarios(g, 256, seed + 2))
        ws.x_mean, ws.x_istd = X.mean(0), 1.0 / X.std(0).clamp_min(1e-6)
        ws.y_mean, ws.y_std = 0.1 * f(ws.n_out), 0.05 + 0.1 * f(ws.n_out)
        s["ws"] = ws
        if kind == "predict":
            m = ws.mlp
            ws.mlp.set_output_layer(m.W[m.layers][: m.n_out].clone(), 0.01 * f(m.n_out))
            s["S"] = _scenarios(g, B, seed)
        else:
            s["X"] = ws.features(_scenarios(g, B, seed))
            s["Y"] = torch.randn(B, ws.n_out, generator=gen, device=DEV)
            s["h"] = ws.mlp.buffers(B)
    return s


def run(s):
    kind = s["kind"]
    if kind == "newton":
        V, _, it = s["solver"].solve_batch_device(s["S"], s["V0"], config=s["config"], ybus=s["ybus"])
        return {"V": V, "iterations": it}
    if kind == "host":
        g = s["grid"]
        r = s["solver"].solve_batch(g.indptr, g.indices, g.data, g.n_bus, g.n_bus, s["S"], s["V0"], g.pv, g.pq,
                                    s["config"])
        return {"V": r.V_numpy, "iterations": r.iterations_numpy}
    if kind == "warm":
        V, _, it = s["solver"].solve_batch_warm_device(s["S"], s["v0"], s["pred"], config=s["config"])
        return {"V": V, "iterations": it}
    if kind == "grad":
        s["p"].grad = s["q"].grad = None
        va, vm = cupf.solve(s["p"], s["q"], s["solver"], **s["kw"])
        ((vm - 1.0) ** 2).sum().backward()
        return {"va": va, "vm": vm, "grad_p": s["p"].grad, "grad_q": s["q"].grad}
    if kind == "linear":
        s["ls"].factorize(s["A"])
        return {"x": s["ls"].solve(s["b"]), "xt": s["ls"].solve_transpose(s["b"])}
    ws = s["ws"]
    if kind == "predict":
        return {"state": ws.predict(s["S"])}
    m, h = ws.mlp, s["h"]
    h["loss"].zero_()
    m.standardize(h, s["X"], ws.x_mean, ws.x_istd)
    m.train_step(h, s["Y"], 1e-4)
    return {"loss": h["loss"], "out": h["p"], "gW": h["gW"], "gb": h["gb"], "W": m.W, "b": m.b}


# ---------------------------------------------------------------------------
# What a pass cannot do without.
# ---------------------------------------------------------------------------
def work(case):
    n, B, kind = case["buses"], case["batch"], case["kind"]
    pv = 53 if n == 118 else n // 5
    dim = 2 * (n - 1) - pv
    nnz_y = n + 3 * n if n != 118 else 490
    nnz_j = 6.9 * dim  # Jacobian entries of these grids, counted: 6.2 to 6.9 per row
    lu = 132.0 * n     # operations of one sparse LU in nested-dissection order, counted: 80 to 150 per bus
    sweep = 4.0 * 11.0 * n
    if kind in ("newton", "warm", "host"):
        its = {"FP64": 5, "Mixed": 5, "FP32": 3}[case["compute"]] if kind != "warm" else 3
        by = 16.0 * n * B + 16.0 * n * B + (4.0 * dim * B if kind == "warm" else 16.0 * n * B)
        if case.get("ybus"):
            by += 16.0 * nnz_y * B
        return {"bytes": by, "flops": B * its * (lu + sweep + 16.0 * nnz_y + 30.0 * nnz_y)}
    if kind == "grad":
        return {"bytes": 4.0 * n * B * 6, "flops": B * (7 * (lu + sweep + 46.0 * nnz_y) + 3 * sweep)}
    if kind == "linear":
        e = 8.0 if case["precision"] == "FP64" else 4.0
        return {"bytes": B * (e * nnz_j + 3 * 8.0 * dim), "flops": B * (lu + 2 * sweep)}
    h = case["hidden"]
    n_in, n_out = 2 * n + pv, dim
    par = n_in * h + 2 * h * h + (h + n_in) * n_out
    if kind == "predict":
        return {"bytes": 16.0 * n * B + 4.0 * n_out * B + 2.0 * par, "flops": 2.0 * B * par}
    return {"bytes": 4.0 * (n_in + 2 * n_out) * B + par * (4 * 7 + 2), "flops": 6.0 * B * par}


def tolerance(case):
    kind = case["kind"]
    if kind in ("newton", "warm", "host"):
        # where Newton stops: up to 2.6e-9 from the exact state at 1e-8, 1.7e-6 in 32 bits at 1e-4
        return {"rel": 1e-5, "max": 4e-4} if case["compute"] == "FP32" else {"rel": 1e-8, "max": 4e-7}
    if kind == "grad":
        return {"rel": 4e-6, "max": 4e-4}
    if kind == "linear":
        # solutions with unpivoted factors: 6e-14 and 3.7e-5 from exact on the listed grids
        return {"rel": 4e-12, "max": 4e-10} if case["precision"] == "FP64" else {"rel": 4e-4, "max": 2e-2}
    return {"rel": 1.5e-2, "max": 0.6}  # bf16 activations: gradients up to 4.6e-3 from exact


# ---------------------------------------------------------------------------
# The same in 64 bits with plain torch.
# ---------------------------------------------------------------------------
def _coo(g):
    rows = torch.tensor(np.repeat(np.arange(g.n_bus), np.diff(g.indptr)), device=DEV)
    return rows, torch.tensor(g.indices.astype(np.int64), device=DEV)


def _jacobian_pattern(g):
    """CSR pattern of [dP/dVa dP/dVm; dQ/dVa dQ/dVm] over the Ybus entries,
    and each entry's (Ybus entry, block) and (row, column)."""
    n = g.n_bus
    fa, fm = np.full(n, -1), np.full(n, -1)
    npvpq = g.pv.size + g.pq.size
    fa[g.pv] = np.arange(g.pv.size)
    fa[g.pq] = g.pv.size + np.arange(g.pq.size)
    fm[g.pq] = npvpq + np.arange(g.pq.size)
    rows = np.repeat(np.arange(n), np.diff(g.indptr))
    cols = g.indices
    rr, cc, src = [], [], []
    for blk, (a, b) in enumerate(((fa, fa), (fa, fm), (fm, fa), (fm, fm))):
        k = np.flatnonzero((a[rows] >= 0) & (b[cols] >= 0))
        rr.append(a[rows[k]])
        cc.append(b[cols[k]])
        src.append(blk * rows.size + k)
    rr, cc, src = np.concatenate(rr), np.concatenate(cc), np.concatenate(src)
    o = np.lexsort((cc, rr))
    rp = np.zeros(npvpq + g.pq.size + 1, np.int32)
    np.add.at(rp, rr + 1, 1)
    return np.cumsum(rp).astype(np.int32), cc[o].astype(np.int32), src[o], rr[o], cc[o]


def _row_sums(ptr, x):
    """Sums of x [B, nnz] over the rows of a CSR pattern: [B, rows], added in order."""
    deg = np.diff(ptr)
    idx = np.full((deg.size, int(deg.max())), ptr[-1], np.int64)
    for j in range(idx.shape[1]):
        k = np.flatnonzero(deg > j)
        idx[k, j] = ptr[k] + j
    xp = torch.cat([x, torch.zeros_like(x[:, :1])], dim=1)
    out = xp[:, torch.tensor(idx[:, 0], device=DEV)]
    for j in range(1, idx.shape[1]):
        out = out + xp[:, torch.tensor(idx[:, j], device=DEV)]
    return out


def _current(g, V, y):
    return _row_sums(g.indptr, y * V[:, _coo(g)[1]])


def _jacobian_values(g, V, y=None):
    """Jacobian values [B, nnz] at the states V, in _jacobian_pattern's order."""
    rows, cols = _coo(g)
    y = torch.tensor(g.data, device=DEV)[None, :] if y is None else y
    I = _current(g, V, y)
    Vi, Vc = V[:, rows], V[:, cols]
    t = Vi * (y * Vc).conj()
    da = -1j * t
    dm = t / Vc.abs()
    dpos = torch.nonzero(rows == cols).flatten()
    Vd, Id = V[:, rows[dpos]], I[:, rows[dpos]]
    da[:, dpos] += 1j * Vd * Id.conj()
    dm[:, dpos] += Id.conj() * Vd / Vd.abs()
    blocks = torch.cat([da.real, dm.real, da.imag, dm.imag], dim=1)
    return blocks[:, torch.tensor(_jacobian_pattern(g)[2], device=DEV)].contiguous()


def _dense(g, vals):
    _, _, _, rr, cc = _jacobian_pattern(g)
    dim = g.dim_f
    A = torch.zeros(dim, dim, dtype=torch.float64, device=DEV)
    A[torch.tensor(rr, device=DEV), torch.tensor(cc, device=DEV)] = vals.double()
    return A


class _Anderson:
    """Anderson acceleration of x <- x - d(x), per row of x [B, k] (Anderson 1965), over 8 steps."""

    def __init__(self):
        self.x, self.d = [], []

    def next(self, x, d):
        self.x, self.d = (self.x + [x])[-9:], (self.d + [d])[-9:]
        y = x - d
        if len(self.x) > 1:
            dD = torch.stack([d - e for e in self.d[:-1]], dim=2)
            dY = torch.stack([y - (a - e) for a, e in zip(self.x[:-1], self.d[:-1])], dim=2)
            A = dD.transpose(1, 2) @ dD
            A = A + 1e-14 * A.diagonal(dim1=1, dim2=2).sum(1)[:, None, None] * torch.eye(A.shape[1], device=DEV) + \
                1e-300 * torch.eye(A.shape[1], device=DEV, dtype=A.dtype)
            c = torch.linalg.solve(A, dD.transpose(1, 2) @ d[:, :, None])
            y = y - (dY @ c)[:, :, 0]
        return y


def _newton_exact(g, S, v0, y=None):
    """(Va, Vm, LU of the nominal Jacobian) of every scenario to rounding:
    Newton steps with dense LU for the nominal load, then accelerated steps
    with that fixed LU for all scenarios; None where those do not converge."""
    pvpq = torch.tensor(np.r_[g.pv, g.pq].astype(np.int64), device=DEV)
    pq = torch.tensor(g.pq.astype(np.int64), device=DEV)
    base = torch.tensor(g.data, device=DEV)[None, :]

    def mismatch(va, vm, S, y):
        V = torch.polar(vm, va)
        m = V * _current(g, V, y).conj() - S
        return V, torch.cat([m[:, pvpq].real, m[:, pq].imag], dim=1)

    def step(va, vm, dx):
        va[:, pvpq] -= dx[:, : pvpq.numel()]
        vm[:, pq] -= dx[:, pvpq.numel():]

    S0 = torch.tensor(g.sbus, device=DEV)[None, :]
    va, vm = torch.angle(v0)[None, :].clone(), torch.abs(v0)[None, :].clone()
    for _ in range(15):
        V, F = mismatch(va, vm, S0, base)
        lu = torch.linalg.lu_factor(_dense(g, _jacobian_values(g, V)[0]))
        if float(F.abs().max()) < 1e-11:
            break
        step(va, vm, torch.linalg.lu_solve(*lu, F.T).T)
    yb = base if y is None else y
    B = S.shape[0]
    va, vm = va.repeat(B, 1), vm.repeat(B, 1)
    x, mix = torch.cat([va[:, pvpq], vm[:, pq]], dim=1), _Anderson()
    r = math.inf
    for k in range(150):
        va[:, pvpq], vm[:, pq] = x[:, : pvpq.numel()], x[:, pvpq.numel():]
        _, F = mismatch(va, vm, S, yb)
        r, last = float(F.abs().max()), r
        if not math.isfinite(r):
            return None
        if r < 2e-13 or (r < 1e-11 and r >= last):
            return va, vm, lu
        x = mix.next(x, torch.linalg.lu_solve(*lu, F.T.contiguous()).T.contiguous())
    return None


def _gelu(z):
    return 0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0)))


def _gelu_grad(z):
    return 0.5 * (1.0 + torch.erf(z / math.sqrt(2.0))) + z * torch.exp(-0.5 * z * z) / math.sqrt(2.0 * math.pi)


def _network_exact(s, kind):
    ws = s["ws"]
    m = ws.mlp
    L, n_in, H = m.layers, m.n_in, m.hidden
    raw = ws.features(s["S"]) if kind == "predict" else s["X"]
    x = torch.zeros(raw.shape[0], m.k0, dtype=torch.float64, device=DEV)
    x[:, :n_in] = (raw.double() - ws.x_mean.double()) * ws.x_istd.double()
    last = m.W[L].double() if kind == "predict" else m.W16[L].double()
    a, zs, acts = x, [], []
    for i in range(L):
        acts.append(a)
        z = a @ m.W16[i].double().T + m.b[i].double()
        zs.append(z)
        a = _gelu(z)
    cat = torch.cat([a, x], dim=1)
    acts.append(cat)
    p = cat @ last.T + m.b[L].double()
    if kind == "predict":
        return {"state": p[:, : m.n_out] * ws.y_std.double() + ws.y_mean.double()}
    B = p.shape[0]
    d = torch.zeros_like(p)
    d[:, : m.n_out] = p[:, : m.n_out] - s["Y"].double()
    out = {"loss": (d * d).sum().reshape(1) / (B * m.n_out), "out": p, "gW": [None] * (L + 1), "gb": [None] * (L + 1),
           "W": [None] * (L + 1), "b": [None] * (L + 1)}
    grad = 2.0 * d / (B * m.n_out)
    for i in range(L, -1, -1):
        gW, gb = grad.T @ acts[i], grad.sum(0)
        out["gW"][i], out["gb"][i] = gW, gb
        # the first Adam step from zero moments: w - lr g / (|g| + eps)
        out["W"][i] = m.W[i].double() - 1e-4 * gW / (gW.abs() + 1e-8)
        out["b"][i] = None  # from zero, lr times a sign: says nothing where a gradient is near rounding
        if i > 0:
            grad = (grad @ m.W16[i].double()[:, :H]) * _gelu_grad(zs[i - 1])
    return out


def exact(case, seed):
    kind = case["kind"]
    g = _grid(case["buses"])
    s = prepare(case, seed)
    v0 = torch.tensor(g.v0, device=DEV)
    if kind in ("newton", "warm", "host"):
        S = torch.as_tensor(s["S"], device=DEV)
        r = _newton_exact(g, S, v0, s.get("ybus"))
        if r is None:
            return None
        V = torch.polar(r[1], r[0])
        return {"V": V.cpu().numpy() if kind == "host" else V, "iterations": None}
    if kind == "grad":
        kw = s["kw"]
        base = torch.complex(kw["sbus_base_re"].double(), kw["sbus_base_im"].double())
        S = base - torch.complex(s["p"].detach().double(), s["q"].detach().double())
        r = _newton_exact(g, S, torch.polar(kw["v0_vm"].double(), kw["v0_va"].double()))
        if r is None:
            return None
        va, vm, lu = r
        _, _, _, rr, cc = _jacobian_pattern(g)
        rr, cc = torch.tensor(rr, device=DEV), torch.tensor(cc, device=DEV)
        J = _jacobian_values(g, torch.polar(vm, va))
        npv, npq = g.pv.size, g.pq.size
        pv, pq = (torch.tensor(a.astype(np.int64), device=DEV) for a in (g.pv, g.pq))
        # the loss is taken in 32 bits from the rounded magnitudes
        gv = 2.0 * (vm.float() - 1.0)
        G = torch.zeros(J.shape[0], g.dim_f, dtype=torch.float64, device=DEV)
        G[:, npv + npq:] = gv.double()[:, pq]
        order = torch.argsort(cc, stable=True)
        cptr = np.concatenate([[0], np.cumsum(np.bincount(cc.cpu().numpy(), minlength=g.dim_f))])
        lam, mix, r = torch.zeros_like(G), _Anderson(), math.inf
        for _ in range(150):
            R = _row_sums(cptr, (J * lam[:, rr])[:, order]) - G
            r, last = float(R.abs().max()), r
            if r < 1e-14 or (r < 1e-11 and r >= last):
                break
            lam = mix.next(lam, torch.linalg.lu_solve(*lu, R.T.contiguous(), adjoint=True).T.contiguous())
        if not r < 1e-10:
            return None
        gp, gq = torch.zeros_like(va), torch.zeros_like(va)
        gp[:, pv], gp[:, pq], gq[:, pq] = -lam[:, :npv], -lam[:, npv:npv + npq], -lam[:, npv + npq:]
        return {"va": va.float(), "vm": vm.float(), "grad_p": gp.float(), "grad_q": gq.float()}
    if kind == "linear":
        x, xt = torch.empty_like(s["b"]), torch.empty_like(s["b"])
        for k in range(s["b"].shape[0]):
            lu = torch.linalg.lu_factor(_dense(g, s["A"][k]))
            b = s["b"][k][:, None]
            x[k] = torch.linalg.lu_solve(*lu, b)[:, 0]
            xt[k] = torch.linalg.lu_solve(*lu, b, adjoint=True)[:, 0]
        return {"x": x, "xt": xt}
    return _network_exact(s, kind)
