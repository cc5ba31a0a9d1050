"""The measured workloads of the PDLP engine, through its public entry points.

Solves run a fixed number of iterations (an iteration limit below what the tolerance would take),
so a pass is the same work on every input of a size: the device setup (equilibration, operator
norm, step size), the iterations with an evaluation, the termination test and the restart rule
every 64 of them, and the answer back in host memory.

``listed`` gives the cases, ``draw`` more of the same ranges, ``prepare`` builds a case's inputs
and the handle a program keeps, ``run`` is one pass, ``work`` its unavoidable bytes and
operations, ``exact`` the same outputs computed in 64 bits by plain torch.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

CHECK = 64  # iterations between evaluations
L2_BYTES = 126e6  # operators and vectors beyond this are read from memory again every iteration


def listed():
    return [
        # The smallest call: one product with device pointers, for callers that own their memory.
        {"name": "spmv_device_500x1200", "kind": "spmv", "lp": "random", "m": 500, "n": 1200},
        # A host-driven loop over the inner seam: eight single steps and an evaluation.
        {"name": "seam_steps_200x500", "kind": "seam", "lp": "random", "m": 200, "n": 500,
         "steps": 8},
        # A small LP of a test family, latency-bound.
        {"name": "solve_random_200x500", "kind": "solve", "lp": "random", "m": 200, "n": 500,
         "algorithm": "reference", "fp32": False, "iterations": 640},
        # The CPU-runnable configuration, the reference algorithm in FP64.
        {"name": "solve_random_2000x5000", "kind": "solve", "lp": "random", "m": 2000, "n": 5000,
         "algorithm": "reference", "fp32": False, "iterations": 1280},
        # Odd sizes, the FP32 phase of the precision switch, a limit inside a chunk.
        {"name": "solve_random_777x2049_fp32", "kind": "solve", "lp": "random", "m": 777,
         "n": 2049, "algorithm": "halpern", "fp32": True, "iterations": 300},
        # The headline LP: the FP32 phase that takes most of its iterations.
        {"name": "solve_transport_1000x2000_fp32", "kind": "solve", "lp": "transport", "m": 1000,
         "n": 2000, "algorithm": "halpern", "fp32": True, "iterations": 512},
        # A ragged transportation LP in FP64 with averaging.
        {"name": "solve_transport_301x703", "kind": "solve", "lp": "transport", "m": 301,
         "n": 703, "algorithm": "enhanced", "fp32": False, "iterations": 256},
        # Power-law rows: a few rows hold most of the nonzeros, most rows are empty.
        {"name": "solve_powerlaw_400kx800k", "kind": "solve", "lp": "powerlaw", "m": 400000,
         "n": 800000, "algorithm": "halpern", "fp32": False, "iterations": 192},
        # The one-off call: upload, row-major copy, setup, solve, download, release.
        {"name": "call_facility_40x150", "kind": "call", "lp": "facility", "m": 40, "n": 150,
         "algorithm": "enhanced", "fp32": False, "iterations": 192},
        # Many LPs of uneven sizes in one launch.
        {"name": "batch_uneven_160", "kind": "batch", "lp": "random", "count": 160, "m": 100,
         "n": 2500, "algorithm": "reference", "fp32": False, "iterations": 256},
        # Branch-and-bound node relaxations sharing one matrix, FP32 storage.
        {"name": "batch_nodes_256_fp32", "kind": "batch", "lp": "facility", "count": 256,
         "m": 40, "n": 160, "algorithm": "halpern", "fp32": True, "iterations": 512},
        # The differentiable layer's unrolled part: forward and adjoint.
        {"name": "unroll_64x500x1200", "kind": "unroll", "lp": "random", "count": 64, "m": 500,
         "n": 1200, "iterations": 256, "every": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "seam", "random", "random", "transport", "transport", "powerlaw",
                       "call", "batch", "batch", "nodes", "unroll"])
    if kind == "spmv":
        m = _log_int(rng, 200, 40000)
        return {"kind": "spmv", "lp": "random", "m": m, "n": int(m * rng.uniform(2, 3))}
    if kind == "seam":
        m = _log_int(rng, 50, 2000)
        return {"kind": "seam", "lp": "random", "m": m, "n": int(m * rng.uniform(2, 3)),
                "steps": rng.randint(2, 8)}
    fp32 = rng.random() < 0.4
    algorithm = "halpern" if fp32 else rng.choice(["reference", "enhanced", "halpern"])
    if kind == "random":
        m = _log_int(rng, 60, 2000)
        return {"kind": "solve", "lp": "random", "m": m, "n": int(m * rng.uniform(2, 3)),
                "algorithm": algorithm, "fp32": fp32,
                "iterations": rng.randint(100, 320 if fp32 else 1280)}
    if kind == "transport":
        return {"kind": "solve", "lp": "transport", "m": _log_int(rng, 40, 1000),
                "n": _log_int(rng, 80, 2000), "algorithm": algorithm, "fp32": fp32,
                "iterations": rng.randint(100, 400)}
    if kind == "powerlaw":
        m = _log_int(rng, 20000, 400000)
        return {"kind": "solve", "lp": "powerlaw", "m": m, "n": 2 * m + rng.randint(0, 9),
                "algorithm": rng.choice(["enhanced", "halpern"]), "fp32": False,
                "iterations": rng.randint(64, 192)}
    if kind == "call":
        return {"kind": "call", "lp": "facility", "m": rng.randint(10, 40),
                "n": rng.randint(40, 150), "algorithm": rng.choice(["reference", "enhanced"]),
                "fp32": False, "iterations": rng.randint(64, 192)}
    if kind == "batch":
        return {"kind": "batch", "lp": "random", "count": _log_int(rng, 4, 160), "m": 60,
                "n": _log_int(rng, 200, 2500),
                "algorithm": rng.choice(["reference", "enhanced", "halpern"]),
                "fp32": fp32, "iterations": rng.randint(100, 256)}
    if kind == "nodes":
        f = rng.randint(8, 40)
        return {"kind": "batch", "lp": "facility", "count": _log_int(rng, 16, 256), "m": f,
                "n": rng.randint(2, 4) * f + rng.randint(0, 3),
                "algorithm": rng.choice(["enhanced", "halpern"]), "fp32": fp32,
                "iterations": rng.randint(100, 384)}
    m = _log_int(rng, 40, 500)
    return {"kind": "unroll", "lp": "random", "count": _log_int(rng, 1, 64), "m": m,
            "n": int(m * rng.uniform(2, 2.4)), "iterations": rng.randint(64, 256),
            "every": rng.choice([16, 50, 64])}


# ---------------------------------------------------------------------------------------------
# Inputs: LpProblems min c'v, [A -I] v = 0, l <= v <= u (m, n, colptr, rowidx, vals, c, l, u).


def _distinct_rows(n, k, draw_rows):
    """(n, k) row numbers, increasing and distinct within each column."""
    rows = np.sort(draw_rows(n * k).reshape(n, k), axis=1)
    bad = np.flatnonzero((rows[:, 1:] == rows[:, :-1]).any(axis=1))
    while bad.size:
        part = rows[bad]
        twice = np.zeros(part.shape, dtype=bool)
        twice[:, 1:] = part[:, 1:] == part[:, :-1]
        part[twice] = draw_rows(int(twice.sum()))
        part.sort(axis=1)
        rows[bad] = part
        bad = bad[(part[:, 1:] == part[:, :-1]).any(axis=1)]
    return rows


def _from_columns(rng, m, n, rows, upper, slack_rows):
    """A feasible, bounded LP whose column j has entries N(0, 1) in rows[j]."""
    k = rows.shape[1]
    rowidx = rows.reshape(-1).astype(np.int32)
    vals = rng.standard_normal(n * k)
    x0 = rng.random(n) * (rng.random(n) < 0.5)
    ax = np.bincount(rowidx, weights=vals * np.repeat(x0, k), minlength=m)
    loose = rng.random(m) < slack_rows
    y0 = rng.standard_normal(m)
    y0[loose] = np.abs(y0[loose])
    cost = (vals * y0[rowidx]).reshape(n, k).sum(axis=1) + rng.random(n)
    return (m, n, np.arange(0, n * k + 1, k, dtype=np.int64), rowidx, vals,
            np.concatenate([cost, np.zeros(m)]),
            np.concatenate([np.zeros(n), np.where(loose, -np.inf, ax)]),
            np.concatenate([np.full(n, upper), ax + np.where(loose, rng.random(m), 0.0)]))


def _random_lp(rng, m, n, k=6):
    rows = _distinct_rows(n, min(k, m), lambda size: rng.integers(0, m, size=size))
    return _from_columns(rng, m, n, rows, 10.0, 0.0)


def _powerlaw_lp(rng, m, n, k=6):
    perm = rng.permutation(m)

    def ranks(size):  # P(rank >= z) = z ** -0.5, truncated at m
        z = np.zeros(size, dtype=np.int64)
        todo = np.arange(size)
        while todo.size:
            u = rng.random(todo.size)
            z[todo] = np.minimum(1.0 / (u * u), m + 1.0).astype(np.int64)
            todo = todo[z[todo] > m]
        return perm[z - 1]

    return _from_columns(rng, m, n, _distinct_rows(n, k, ranks), 5.0, 0.3)


def _transport_lp(rng, supplies, demands):
    n, m = supplies * demands, supplies + demands
    sup = rng.integers(500, 1501, size=supplies).astype(np.float64)
    dem = rng.integers(200, 801, size=demands).astype(np.float64)
    dem *= sup.sum() / dem.sum()
    rowidx = np.empty((supplies, demands, 2), dtype=np.int32)
    rowidx[:, :, 0] = np.arange(supplies)[:, None]
    rowidx[:, :, 1] = supplies + np.arange(demands)[None, :]
    b = np.concatenate([sup, dem])
    return (m, n, np.arange(0, 2 * n + 1, 2, dtype=np.int64), rowidx.reshape(-1),
            np.ones(2 * n),
            np.concatenate([rng.integers(1, 101, size=n).astype(np.float64), np.zeros(m)]),
            np.concatenate([np.zeros(n), b]), np.concatenate([np.full(n, np.inf), b]))


def _facility_lp(rng, facilities, customers):
    """Capacitated facility location relaxation: open variables, then assignments f x c; demand
    rows, then capacity rows."""
    n, m = facilities + facilities * customers, customers + facilities
    where, to = rng.random((facilities, 2)), rng.random((customers, 2))
    dem = rng.integers(5, 36, size=customers).astype(np.float64)
    cap = rng.uniform(2.0, 5.0, size=facilities) * dem.sum() / facilities
    dist = np.sqrt(((where[:, None, :] - to[None, :, :]) ** 2).sum(-1))
    scale = 1.0 / dem.mean()
    colptr = np.concatenate([np.arange(facilities),
                             facilities + 2 * np.arange(facilities * customers + 1)])
    rowidx = np.empty(facilities + 2 * facilities * customers, dtype=np.int32)
    vals = np.empty(rowidx.size)
    rowidx[:facilities] = customers + np.arange(facilities)
    vals[:facilities] = -cap * scale
    f, c = np.divmod(np.arange(facilities * customers), customers)
    rowidx[facilities::2], vals[facilities::2] = c, 1.0
    rowidx[facilities + 1::2], vals[facilities + 1::2] = customers + f, dem[c] * scale
    cost = np.concatenate([rng.uniform(50.0, 150.0, size=facilities),
                           (dist * dem[None, :]).reshape(-1), np.zeros(m)])
    lower = np.concatenate([np.zeros(n), np.ones(customers), np.full(facilities, -np.inf)])
    upper = np.concatenate([np.ones(n), np.ones(customers), np.zeros(facilities)])
    return m, n, colptr.astype(np.int64), rowidx, vals, cost, lower, upper


def _problem(case, rng):
    make = {"random": _random_lp, "powerlaw": _powerlaw_lp, "transport": _transport_lp,
            "facility": _facility_lp}[case["lp"]]
    return make(rng, case["m"], case["n"])


def _instances(case, seed):
    """(matrices, instances) of a batch: (m, n, colptr, rowidx, vals) and (matrix, c, l, u)."""
    rng = np.random.default_rng(seed)
    if case["lp"] == "facility":
        p = _problem(case, rng)
        inst = []
        for _ in range(case["count"]):
            lower, upper = p[6].copy(), p[7].copy()
            fixed = rng.choice(case["m"], size=max(1, case["m"] // 20), replace=False)
            lower[fixed] = upper[fixed] = rng.integers(0, 2, size=fixed.size)
            inst.append((0, p[5], lower, upper))
        return [p[:5]], inst
    mats, inst = [], []
    for k in range(case["count"]):
        m, n = _size(case, k)
        p = _random_lp(rng, m, n)
        mats.append(p[:5])
        inst.append((k, p[5], p[6], p[7]))
    return mats, inst


def _size(case, k):
    """(m, n) of matrix k of a batch of random LPs: a batch solve's rows spread evenly over
    [m, n] (the case's fields) with 2 to 3 columns each, an unroll's all alike."""
    if case["kind"] == "unroll":
        return case["m"], case["n"]
    m = case["m"] + (case["n"] - case["m"]) * ((k * 37) % case["count"]) // case["count"]
    return m, int(math.ceil(m * (2.0 + (k % 11) / 11.0)))


def _csr(p):
    """Row starts, column indices and values of A by rows."""
    m, n, colptr, rowidx, vals = p[:5]
    order = np.argsort(rowidx, kind="stable")
    ptr = np.zeros(m + 1, dtype=np.int32)
    np.cumsum(np.bincount(rowidx, minlength=m), out=ptr[1:])
    return ptr, np.repeat(np.arange(n, dtype=np.int32), np.diff(colptr))[order], vals[order]


def _vectors(case, p, seed):
    """A primal and a dual point for products and single steps."""
    rng = np.random.default_rng(seed + 1)
    return rng.random(p[1] + p[0]), 0.1 * rng.standard_normal(p[0])


# ---------------------------------------------------------------------------------------------


def _options(case):
    import samaya_gb300 as sg
    algorithm = {"reference": sg.REFERENCE, "enhanced": sg.ENHANCED,
                 "halpern": sg.HALPERN}[case["algorithm"]]
    if case["kind"] == "batch":  # FP32 storage is the batch's reduced precision
        precision = sg.FP32_REFINED if case["fp32"] else sg.FP64
    else:
        precision = sg.FP32_THEN_FP64 if case["fp32"] else sg.FP64
    return sg.PdlpOptions(tol=1e-11, max_iterations=case["iterations"], inner_tol=1e-11,
                          algorithm=algorithm, precision=precision)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "unroll"):
        from samaya_gb300.batch import BatchSolver
        mats, inst = _instances(case, seed)
        if kind == "batch":
            return {"kind": kind, "fp32": case["fp32"],
                    "solver": BatchSolver(mats, inst, _options(case))}
        from samaya_gb300.diff import UnrolledPdhg
        unroll = UnrolledPdhg(BatchSolver(mats, inst), case["iterations"], case["every"])
        return {"kind": kind, "unroll": unroll,
                "grad": np.random.default_rng(seed + 2).standard_normal(unroll.total)}
    p = _problem(case, np.random.default_rng(seed))
    if kind == "spmv":
        from samaya_gb300 import _native
        v, _ = _vectors(case, p, seed)
        ptr, idx, val = (torch.from_numpy(a).cuda() for a in _csr(p))
        x = torch.from_numpy(v[:p[1]].copy()).cuda()
        f = _native.load().sg_spmv_noalloc
        f.restype = ctypes.c_int
        f.argtypes = [ctypes.c_int, ctypes.c_longlong] + [ctypes.c_void_p] * 6
        return {"kind": kind, "f": f, "m": p[0], "nnz": int(p[4].size), "ptr": ptr, "idx": idx,
                "val": val, "x": x, "y": torch.empty(p[0], dtype=torch.float64, device="cuda")}
    if kind == "seam":
        from samaya_gb300 import PdhgDevice
        v, y = _vectors(case, p, seed)
        d = PdhgDevice(*p)
        d.set_original(np.ones(p[1]), np.ones(p[0]), *p[5:])
        return {"kind": kind, "device": d, "steps": case["steps"], "v": v, "y": y,
                "eta": _seam_step_size(p)}
    from samaya_gb300 import LpProblem, PdlpSolver
    lp = LpProblem(*p)
    state = {"kind": kind, "fp32": case["fp32"]}
    if kind == "call":
        return state | {"lp": lp, "options": _options(case)}
    x = torch.empty(lp.n + lp.m, dtype=torch.float64, pin_memory=True)
    y = torch.empty(lp.m, dtype=torch.float64, pin_memory=True)
    return state | {"solver": PdlpSolver(lp, _options(case)), "x": x, "y": y,
                    "buffers": (x.numpy(), y.numpy())}


def _answer(r, x, y, fp32):
    """An answer's vectors (in the storage type's precision) and scalars."""
    kkt = [r.primal_residual, r.dual_residual, r.gap, r.primal_objective, r.dual_objective]
    if fp32:
        return {"x": torch.as_tensor(x).float(), "y": torch.as_tensor(y).float(),
                "kkt": torch.tensor(kkt, dtype=torch.float32), "iterations": r.iterations}
    return {"x": x, "y": y, "kkt": torch.tensor(kkt, dtype=torch.float64),
            "iterations": r.iterations}


def run(state):
    kind = state["kind"]
    if kind == "spmv":
        rc = state["f"](state["m"], state["nnz"], state["ptr"].data_ptr(),
                        state["idx"].data_ptr(), state["val"].data_ptr(), state["x"].data_ptr(),
                        state["y"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError(f"sg_spmv_noalloc: {rc}")
        return state["y"]
    if kind == "seam":
        d = state["device"]
        d.set_state(state["v"], state["y"], state["v"], state["y"])
        for k in range(state["steps"]):
            d.step(state["eta"], state["eta"], 1.0, k)
            d.advance()
        out = d.download()
        return {"v": out["v"], "y": out["y"], "v_average": out["v_erg"],
                "y_average": out["y_erg"], "sums": d.evaluate(1)}
    if kind == "unroll":
        u = state["unroll"]
        v = u.forward()
        gc, gl, gu = u.adjoint(state["grad"])
        return {"v": v, "grad_cost": gc, "grad_lower": gl, "grad_upper": gu}
    if kind == "batch":
        items = state["solver"].solve()
        dtype = np.float32 if state["fp32"] else np.float64
        return {"x": np.concatenate([r.x for r in items], dtype=dtype, casting="same_kind"),
                "y": np.concatenate([r.y for r in items], dtype=dtype, casting="same_kind"),
                "objective": np.array([r.primal_objective for r in items], dtype=dtype),
                "iterations": np.array([r.iterations for r in items])}
    if kind == "call":
        from samaya_gb300 import solve_pdlp
        r = solve_pdlp(state["lp"], state["options"])
        return _answer(r, r.x, r.y, state["fp32"])
    r = state["solver"].solve(*state["buffers"])
    return _answer(r, state["x"], state["y"], state["fp32"])


def _shape(case):
    """(rows, columns, nonzeros of the distinct matrices, rows and columns of all instances,
    nonzeros over all instances)."""
    kind, m, n = case["lp"], case["m"], case["n"]
    if kind == "transport":
        return m + n, m * n, 2 * m * n, 2 * m * n
    if kind == "facility":
        count, nnz = case.get("count", 1), m + 2 * m * n
        return count * (m + n), count * (m + m * n), nnz, count * nnz
    if case["kind"] in ("batch", "unroll"):
        sizes = [_size(case, k) for k in range(case["count"])]
        rows, cols = sum(s[0] for s in sizes), sum(s[1] for s in sizes)
        return rows, cols, 6 * cols, 6 * cols
    return m, n, 6 * n, 6 * n


def work(case):
    """Operators by rows and by columns (values and 32-bit indices), the problem's vectors, the
    iterates and the answer: once, or once an iteration where they exceed the L2 cache. Two
    operations per nonzero and product, about ten per entry of the iterate."""
    rows, cols, nnz, all_nnz = _shape(case)
    s = 4 if case.get("fp32") else 8
    if case["kind"] == "spmv":
        return {"bytes": nnz * 12 + 4 * (rows + 1) + 8 * (rows + cols), "flops": 2 * nnz}
    steps = case.get("iterations") or case["steps"]
    passes = steps * (3 if case["kind"] == "unroll" else 1)  # the adjoint recomputes, then steps
    state = 2 * nnz * (s + 4) + 4 * (rows + cols) + 8 * s * (rows + cols)
    once = nnz * 12 + 3 * 8 * (rows + cols) + 8 * (rows + cols) + 8 * rows
    again = passes * state if state > L2_BYTES else 0
    return {"bytes": once + again, "flops": passes * (4 * all_nnz + 10 * (rows + cols))}


# ---------------------------------------------------------------------------------------------
# The same outputs in 64 bits: torch on whole batches, per-instance scalars.


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _mt19937_64(count, seed=12345):
    """The first `count` outputs of the 64-bit Mersenne Twister."""
    mask = (1 << 64) - 1
    s = [seed]
    for i in range(1, 312):
        s.append((6364136223846793005 * (s[-1] ^ (s[-1] >> 62)) + i) & mask)
    out = []
    while len(out) < count:
        for i in range(312):
            x = (s[i] & 0xFFFFFFFF80000000) | (s[(i + 1) % 312] & 0x7FFFFFFF)
            s[i] = s[(i + 156) % 312] ^ (x >> 1) ^ (0xB5026F5AA96619E9 if x & 1 else 0)
        for x in s:
            x ^= (x >> 29) & 0x5555555555555555
            x ^= (x << 17) & 0x71D67FFFEDA60000
            x ^= (x << 37) & 0xFFF7EEE000000000
            out.append(x ^ (x >> 43))
    return out[:count]


class _Lps:
    """All instances' LPs side by side: entry k of A in row `i[k]`, column `j[k]`, instance of
    every column (`gc`) and row (`gr`); v = (all columns, then all rows)."""

    def __init__(self, mats, inst):
        dev = _dev()
        i, j, a, gc, gr, c, lo, up, r0, c0 = [], [], [], [], [], [], [], [], 0, 0
        self.dims = []
        for k, (g, cost, lower, upper) in enumerate(inst):
            m, n, colptr, rowidx, vals = mats[g]
            i.append(rowidx.astype(np.int64) + r0)
            j.append(np.repeat(np.arange(n), np.diff(colptr)) + c0)
            a.append(vals)
            gc.append(np.full(n, k))
            gr.append(np.full(m, k))
            for dst, src in ((c, cost), (lo, lower), (up, upper)):
                dst.append((src[:n], src[n:]))
            self.dims.append((m, n))
            r0 += m
            c0 += n

        def cat(parts):
            return torch.from_numpy(np.concatenate(parts)).to(dev)

        self.m, self.n, self.count = r0, c0, len(inst)
        self.i, self.j, self.a, self.gc, self.gr = cat(i), cat(j), cat(a), cat(gc), cat(gr)
        self.g = torch.cat([self.gc, self.gr])
        self.c, self.lo, self.up = (torch.cat([cat([p[0] for p in v]), cat([p[1] for p in v])])
                                    for v in (c, lo, up))

    def rows(self, w):
        """Per row, the sum of w over its entries."""
        return torch.zeros(self.m, dtype=w.dtype, device=w.device).index_add(0, self.i, w)

    def cols(self, w):
        return torch.zeros(self.n, dtype=w.dtype, device=w.device).index_add(0, self.j, w)

    def total(self, w, g):
        return torch.zeros(self.count, dtype=w.dtype, device=w.device).index_add(0, g, w)

    def largest(self, w, g):
        z = torch.zeros(self.count, dtype=w.dtype, device=w.device)
        return z.scatter_reduce(0, g, w, "amax")

    def split(self, v):
        """A vector over (columns, rows) instance by instance, host order."""
        v = v.cpu()
        out, c0, r0 = [], 0, self.n
        for m, n in self.dims:
            out += [v[c0:c0 + n], v[r0:r0 + m]]
            c0, r0 = c0 + n, r0 + m
        return torch.cat(out)

    def scale(self, enhanced):
        """Equilibration: column scales, row scales."""
        cs = torch.ones(self.n, dtype=torch.float64, device=self.a.device)
        rs = torch.ones(self.m, dtype=torch.float64, device=self.a.device)
        if enhanced:
            mag = self.a.abs()
            for k in range(11):
                w = mag * cs[self.j] * rs[self.i]
                if k < 10:
                    cn = torch.zeros_like(cs).scatter_reduce(0, self.j, w, "amax")
                    rn = torch.zeros_like(rs).scatter_reduce(0, self.i, w, "amax")
                else:
                    cn, rn = self.cols(w), self.rows(w)
                cs = torch.where(cn > 0, cs / cn.sqrt(), cs)
                rs = torch.where(rn > 0, rs / rn.sqrt(), rs)
            return cs, rs
        live = torch.ones(self.count, dtype=torch.bool, device=self.a.device)
        for _ in range(10):
            w = (self.a * cs[self.j] * rs[self.i]) ** 2
            new = []
            moved = torch.zeros(self.count, dtype=torch.float64, device=self.a.device)
            for s, nrm, g in ((cs, self.cols(w).sqrt(), self.gc), (rs, self.rows(w).sqrt(),
                                                                  self.gr)):
                t = torch.where(nrm > 0, (s / nrm).clamp(1e-8, 1e8), s)
                big = ((t - s).abs() / s.abs().clamp(min=1.0) > 0.1).double()
                moved = torch.maximum(moved, self.largest(big, g))
                new.append(torch.where(live[g], t, s))
            cs, rs = new
            live = live & (moved > 0)
        return cs, rs

    def equilibrated(self, enhanced):
        """Scales, A_eq's entries, the scaled cost and bounds, the step size."""
        cs, rs = self.scale(enhanced)
        a = self.a * cs[self.j] * rs[self.i]
        inv = torch.cat([1 / cs, rs])
        c, lo, up = self.c * torch.cat([cs, rs]), self.lo * inv, self.up * inv
        most = max(m for m, _ in self.dims)
        start = torch.tensor([float(x) / 2.0 ** 64 * 2.0 - 1.0 for x in _mt19937_64(most)],
                             dtype=torch.float64, device=a.device)
        u = torch.cat([start[:m] for m, _ in self.dims])
        u = u / self.total(u * u, self.gr).sqrt()[self.gr]
        for _ in range(20):
            v = self.cols(a * u[self.i])
            vn = self.total(v * v, self.gc).sqrt()
            u = self.rows(a * v[self.j])
            un = self.total(u * u, self.gr).sqrt()
            u = u / un[self.gr]
        eta = 0.99 / torch.sqrt((un / vn * 1.01) ** 2 + 1.0)
        return cs, rs, a, c, lo, up, eta


def _measures(P, a, cs, rs, c, lo, up, norms, v, y):
    """Relative primal and dual residuals and gap, and both objectives, per instance, of the
    point (v, y) mapped back by the scales (cs, rs)."""
    n = P.n
    value = torch.cat([v[:n] * cs, v[n:] / rs])
    yo = y * rs
    e = P.rows(a * v[P.j]) / rs - value[n:]
    g = torch.cat([c[:n] + P.cols(a * y[P.i]) / cs, c[n:] - yo])
    hl, hu = lo > -math.inf, up < math.inf
    lam = torch.where(hl & hu, g, torch.where(hl, g.clamp(min=0), torch.where(
        hu, g.clamp(max=0), torch.zeros_like(g))))
    finite_lo, finite_up = torch.where(hl, lo, 0.0 * g), torch.where(hu, up, 0.0 * g)
    pobj = P.total(c * value, P.g)
    dobj = P.total(lam.clamp(min=0) * finite_lo + lam.clamp(max=0) * finite_up, P.g)
    rp = P.total(e * e, P.gr).sqrt() / (
        1 + norms[0] * P.total(value[:n] ** 2, P.gc).sqrt()
        + P.total(value[n:] ** 2, P.gr).sqrt())
    rd = P.total((g - lam) ** 2, P.g).sqrt() / (
        1 + norms[1] * P.total(yo * yo, P.gr).sqrt() + norms[2])
    return rp, rd, (pobj - dobj) / (1 + pobj.abs() + dobj.abs()), pobj, dobj


def _pdlp64(P, algorithm, iterations, forced, scaled_measures):
    """`iterations` iterations of the restarted method on every instance: the answer (v, y) in
    the LpProblem's space and its measures."""
    halpern = algorithm == "halpern"
    cs, rs, a, c, lo, up, eta = P.equilibrated(algorithm != "reference")
    n, gc, gr, g = P.n, P.gc, P.gr, P.g

    def norms_of(w, cost):
        return (P.largest(P.cols(w * w).sqrt(), gc), P.largest(P.rows(w * w).sqrt(), gr),
                P.total(cost * cost, g).sqrt())

    given = (P.a, P.c)
    measure = (a, cs, rs, P.c, P.lo, P.up, norms_of(*given))
    if scaled_measures:  # the FP32 phase measures the equilibrated problem
        decide = (a, torch.ones_like(cs), torch.ones_like(rs), c, lo, up, norms_of(a, c))
    else:
        decide = measure
    omega = torch.ones_like(eta)
    if algorithm != "reference":
        b = torch.maximum(torch.where(lo[n:].isfinite(), lo[n:].abs(), 0 * lo[n:].nan_to_num()),
                          torch.where(up[n:].isfinite(), up[n:].abs(), 0 * up[n:].nan_to_num()))
        cn, bn = P.total(c[:n] ** 2, gc).sqrt(), P.total(b * b, gr).sqrt()
        omega = torch.where((cn > 1e-10) & (bn > 1e-10), cn / bn, omega)
    v = torch.zeros_like(c)
    vbar, verg, v0 = v, v, v
    y = torch.zeros(P.m, dtype=v.dtype, device=v.device)
    yerg, y0 = y, y
    k = torch.zeros_like(eta)
    kar, kprev = torch.full_like(eta, math.inf), torch.full_like(eta, math.inf)
    for t in range(1, iterations + 1):
        tau, sigma = eta / omega, eta * omega
        if halpern:
            grad = torch.cat([c[:n] + P.cols(a * y[P.i]), c[n:] - y])
            verg = torch.minimum(torch.maximum(v - tau[g] * grad, lo), up)
            refl = 2 * verg - v
            yerg = y + sigma[gr] * (P.rows(a * refl[P.j]) - refl[n:])
            w = 1 / (k + 2)
            v = refl + w[g] * (v0 - refl)
            yr = 2 * yerg - y
            y = yr + w[gr] * (y0 - yr)
        else:
            y = y + sigma[gr] * (P.rows(a * vbar[P.j]) - vbar[n:])
            grad = torch.cat([c[:n] + P.cols(a * y[P.i]), c[n:] - y])
            vn = torch.minimum(torch.maximum(v - tau[g] * grad, lo), up)
            vbar, v = 2 * vn - v, vn
            al = 1 / (k + 1)
            verg = (1 - al)[g] * verg + al[g] * v
            yerg = (1 - al)[gr] * yerg + al[gr] * y
        k = k + 1
        if t % CHECK and t != iterations:
            continue

        def kkt(mm):
            return ((omega * mm[0]) ** 2 + (mm[1] / omega) ** 2 + mm[2] ** 2).sqrt()

        avg = _measures(P, *decide, verg, yerg)
        cur = avg if halpern else _measures(P, *decide, v, y)
        final = _measures(P, *measure, verg, yerg) if halpern else cur
        ka, kc = kkt(avg), kkt(cur)
        to_avg = (ka < kc) | halpern
        cand = torch.where(to_avg, ka, kc)
        kar = torch.where(kar.isinf(), cand, kar)
        again = (cand <= 0.2 * kar) | ((cand <= 0.8 * kar) & (cand > kprev)) | (k >= forced * t)
        kprev = torch.where(again, torch.full_like(cand, math.inf), cand)
        kar = torch.where(again, cand, kar)
        vc = torch.where(to_avg[g], verg, v)
        yc = torch.where(to_avg[gr], yerg, y)
        dx = P.total((vc - v0) ** 2, g).sqrt()
        dy = P.total((yc - y0) ** 2, gr).sqrt()
        omega = torch.where(again & (dx > 1e-10) & (dy > 1e-10), (dy / dx * omega).sqrt(), omega)
        v, vbar, v0 = (torch.where(again[g], vc, o) for o in (v, vbar, v0))
        y, y0 = (torch.where(again[gr], yc, o) for o in (y, y0))
        k = torch.where(again, torch.zeros_like(k), k)
    if halpern:
        v, y = verg, yerg
    return torch.cat([v[:n] * cs, v[n:] / rs]), y * rs, final


def _seam_step_size(p):
    """0.9 over a bound of ||[A -I]||: sqrt of the largest column sum times the largest row sum
    of magnitudes, and 1 for the identity."""
    m, n, colptr, rowidx, vals = p[:5]
    by_row = np.bincount(rowidx, weights=np.abs(vals), minlength=m).max()
    by_col = np.bincount(np.repeat(np.arange(n), np.diff(colptr)), weights=np.abs(vals)).max()
    return 0.9 / math.sqrt(by_row * by_col + 1.0)


def _exact_seam(case, p, v, y):
    P = _Lps([p[:5]], [(0, *p[5:])])
    eta, n = _seam_step_size(p), p[1]
    v, y = torch.from_numpy(v).to(P.a.device), torch.from_numpy(y).to(P.a.device)
    vbar, verg, yerg = v, torch.zeros_like(v), torch.zeros_like(y)
    for k in range(case["steps"]):
        y = y + eta * (P.rows(P.a * vbar[P.j]) - vbar[n:])
        grad = torch.cat([P.c[:n] + P.cols(P.a * y[P.i]), P.c[n:] - y])
        vn = torch.minimum(torch.maximum(v - eta * grad, P.lo), P.up)
        vbar, v = 2 * vn - v, vn
        al = 1.0 / (k + 1)
        verg, yerg = (1 - al) * verg + al * v, (1 - al) * yerg + al * y
    return {"v": v.cpu(), "y": y.cpu(), "v_average": verg.cpu(), "y_average": yerg.cpu(),
            "sums": None}


def _exact_unroll(case, seed):
    P = _Lps(*_instances(case, seed))
    cs, rs, a, c, lo, up, eta = P.equilibrated(False)
    c, lo, up = (t.detach().requires_grad_() for t in (c, lo, up))
    n, step, step_rows = P.n, eta[P.g], eta[P.gr]
    v = torch.zeros_like(c)
    vbar, y = v, torch.zeros(P.m, dtype=v.dtype, device=v.device)
    for _ in range(case["iterations"]):
        y = y + step_rows * (P.rows(a * vbar[P.j]) - vbar[n:])
        z = v - step * torch.cat([c[:n] + P.cols(a * y[P.i]), c[n:] - y])
        vn = torch.where(z <= lo, lo, torch.where(z >= up, up, z))
        vbar, v = 2 * vn - v, vn
    out = torch.cat([v[:n] * cs, v[n:] / rs])
    w = np.random.default_rng(seed + 2).standard_normal(P.n + P.m)
    parts, off = [[], []], 0
    for m, nn in P.dims:
        parts[0].append(w[off:off + nn])
        parts[1].append(w[off + nn:off + nn + m])
        off += nn + m
    grad = torch.from_numpy(np.concatenate(parts[0] + parts[1])).to(v.device)
    gc, gl, gu = torch.autograd.grad(out, (c, lo, up), grad)
    by_cost, by_bound = torch.cat([cs, rs]), torch.cat([1 / cs, rs])
    return {"v": P.split(out.detach()), "grad_cost": P.split(gc * by_cost),
            "grad_lower": P.split(gl * by_bound), "grad_upper": P.split(gu * by_bound)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "unroll":
        return _exact_unroll(case, seed)
    if kind == "batch":
        P = _Lps(*_instances(case, seed))
        forced = 0.1 if case["algorithm"] == "halpern" else 0.36
        v, y, final = _pdlp64(P, case["algorithm"], case["iterations"], forced, False)
        return {"x": P.split(v), "y": y.cpu(), "objective": final[3].cpu(), "iterations": None}
    p = _problem(case, np.random.default_rng(seed))
    if kind == "spmv":
        x, _ = _vectors(case, p, seed)
        w = p[4] * x[np.repeat(np.arange(p[1]), np.diff(p[2]))]
        return torch.from_numpy(np.bincount(p[3], weights=w, minlength=p[0]))
    if kind == "seam":
        return _exact_seam(case, p, *_vectors(case, p, seed))
    P = _Lps([p[:5]], [(0, *p[5:])])
    forced = 0.36 if case["algorithm"] == "reference" else 0.1
    v, y, final = _pdlp64(P, case["algorithm"], case["iterations"], forced, case["fp32"])
    return {"x": v.cpu(), "y": y.cpu(), "kkt": torch.cat(final).cpu(), "iterations": None}
