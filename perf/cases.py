"""What is timed: the work a user of this framework has it do, through its public entry points.

Every case is a dict of plain values; `kind` says which entry points it calls:

- role: Sampler.sample and Bounder.bound on one box, the two calls a driver makes per expanded box, with the
  role handles built once per composition (host box in, host verdicts and candidate out).
- aggregate: Bounder.bound_children, the aggregate driver's call: the regions' verdicts folded per child.
- eval_host / eval_device: the batched evaluator on boxes a caller holds on the host (a model with shared
  subexpressions, divisions and roots) or on the device (quadratic models, FP64 or the FP32 enclosure).
- solve: one device-resident solve up to an iteration limit: create, step, outcome, close.
- batch: batch_solve of many problems of uneven sizes.
- serve: a running server given a group of mixed requests, until the last one is answered.

The models are the (mixed-integer) QCQPs of the repository's benchmark shapes (n = 4, 32 and 64, uneven
n in 4..48, serving sizes 8..64) and sizes between them, with coefficients and boxes drawn from the seed.
"""

from __future__ import annotations

import numpy as np
import torch

from cuminlp_gb300 import Bounder, DeviceProblem, Problem, Sampler, Server, Solver, abi, sqr, sqrt
from cuminlp_gb300.solver import batch_solve, eval_boxes, eval_boxes_device

COUNTERS = ("iterations", "expansions", "fathomed", "fathomed_points", "bounded", "sampled", "enqueued",
            "pruned_duplicate", "pruned_infeasible", "pruned_dominated", "dropped_viable", "dropped_dominated",
            "screened_fp32", "certified_fp64", "peak_frontier", "certify_pruned")


# ---- the listed cases and their ranges --------------------------------------------------------------------
def listed():
    return [
        # the reference driver's smallest expansion: one n=4 box into 4 regions, all latency
        dict(name="role_n4_4", kind="role", n=4, m=1, n_int=0, qd=1.0, ad=1.0, bits=2, points=1),
        # an ordinary expansion of the n=32 MIQCQP: 2^12 regions, several sample points each
        dict(name="role_n32_4k", kind="role", n=32, m=16, n_int=4, qd=1.0, ad=0.2, bits=12, points=3),
        # the largest: the n=64 MIQCQP box into 2^17 regions in one call
        dict(name="role_n64_128k", kind="role", n=64, m=32, n_int=8, qd=0.3, ad=0.1, bits=17, points=1),
        # the aggregate driver's bound: n=24, 2^14 regions folded into 8 children
        dict(name="aggregate_n24_16k", kind="aggregate", n=24, m=8, n_int=3, qd=0.6, ad=0.4, bits=14, children=8),
        # host boxes of a general model (divisions, roots, shared subexpressions), an odd count
        dict(name="eval_host_n17_3001", kind="eval_host", n=17, boxes=3001),
        # device boxes, FP64: the evaluator over a frontier of the n=64 MIQCQP, an odd count
        dict(name="eval_dev_n64_50001", kind="eval_device", n=64, m=32, n_int=8, qd=0.3, ad=0.1, boxes=50001,
             precision=0),
        # device boxes, the FP32 enclosure of the screen: n=32
        dict(name="eval_dev32_n32_200k", kind="eval_device", n=32, m=16, n_int=4, qd=1.0, ad=0.2, boxes=200000,
             precision=1),
        # a plain FP64 solve of the n=4 QCQP with large iterations: the pool and the launches count
        dict(name="solve_n4_fp64", kind="solve", n=4, m=1, n_int=0, qd=1.0, ad=1.0, precision="fp64", bits=2,
             parents=1 << 20, cap=1 << 24, points=1, iters=32),
        # a plain FP64 solve of the n=32 MIQCQP
        dict(name="solve_n32_fp64", kind="solve", n=32, m=16, n_int=4, qd=1.0, ad=0.2, precision="fp64", bits=4,
             parents=1 << 14, cap=1 << 18, points=1, iters=12),
        # the benchmark's headline: the lazy form on the n=64 MIQCQP, 2^16 parents x 2^4 children per iteration
        dict(name="solve_n64_lazy", kind="solve", n=64, m=32, n_int=8, qd=0.3, ad=0.1, precision="lazy", bits=4,
             parents=1 << 16, cap=1 << 20, points=1, iters=12),
        # uneven problems advanced together (n ~ U{4..48}), the lazy form
        dict(name="batch_uneven_lazy", kind="batch", count=24, n_lo=4, n_hi=48, precision="lazy", bits=4,
             parents=256, cap=4096, iters=12),
        # a group of serving requests, n in {8, 16, 32, 64}
        dict(name="serve_16", kind="serve", count=16, precision="lazy", bits=4, parents=64, cap=1024, expansions=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: n log-uniform over 4..64, constraints, integers, densities and
    launch sizes spread, and the work held below the largest listed case of the kind."""
    kind = rng.choice(["role", "role", "aggregate", "eval_host", "eval_device", "solve", "solve", "batch", "serve"])
    if kind == "eval_host":
        return dict(kind=kind, n=_log_int(rng, 5, 40), boxes=_log_int(rng, 17, 4000))
    if kind == "batch":
        lo = rng.randint(4, 16)
        return dict(kind=kind, count=rng.randint(3, 24), n_lo=lo, n_hi=rng.randint(lo + 4, 40),
                    precision=rng.choice(["lazy", "lazy", "fp64"]), bits=rng.randint(2, 4),
                    parents=rng.randint(16, 160), cap=rng.randint(300, 4096), iters=rng.randint(4, 10))
    if kind == "serve":
        return dict(kind=kind, count=rng.randint(4, 14), precision=rng.choice(["lazy", "lazy", "fp64"]),
                    bits=rng.randint(2, 4), parents=rng.randint(16, 64), cap=rng.randint(256, 1024),
                    expansions=rng.randint(100, 400))
    n = _log_int(rng, 4, 64)
    m = rng.randint(0, max(1, n // 2))
    c = dict(kind=kind, n=n, m=m, n_int=rng.randint(0, n // 4), qd=round(rng.uniform(0.1, 1.0), 3),
             ad=round(rng.uniform(0.1, 0.6), 3))
    while _terms(c) > 9000:
        c["m"] = c["m"] // 2
        c["qd"] = round(max(0.1, c["qd"] * 0.8), 3)
    most = 9500 * (1 << 17)  # terms x regions of the largest listed role
    if kind in ("role", "aggregate"):
        bits = rng.randint(2, 17 if kind == "role" else 14)
        while (_terms(c) << bits) > most:
            bits -= 1
        if kind == "role":
            points = rng.randint(1, 3)
            if (_terms(c) << bits) * points > most:
                points = 1
            return dict(c, bits=bits, points=points)
        return dict(c, bits=bits, children=1 << rng.randint(1, min(bits, 4)))
    if kind == "eval_device":
        return dict(c, boxes=_log_int(rng, 33, min(200000, 50000 * 9500 // _terms(c))), precision=rng.randint(0, 1))
    bits = rng.randint(1, 4)
    parents = _log_int(rng, 64, min(1 << 16, max(128, (1 << 28) // (_terms(c) << bits))))
    return dict(c, precision=rng.choice(["fp64", "lazy", "fp32"]), bits=bits, parents=parents,
                cap=max(16, int(parents * rng.uniform(2.0, 12.0))), points=rng.randint(1, 2), iters=rng.randint(6, 12))


# ---- models ------------------------------------------------------------------------------------------------
def _terms(c):
    """Expected terms of a case's model: the objective's and every constraint's quadratic and linear ones."""
    pairs = c["n"] * (c["n"] + 1) / 2
    return int(pairs * c["qd"] + c["n"] + c["m"] * (pairs * c["ad"] + c["n"]))


def _quadratic_data(rng, n, density):
    """Upper-triangle terms (i, j, coefficient) and the linear coefficients of x^T Q x + c^T x."""
    i, j = np.triu_indices(n)
    q = rng.standard_normal(len(i))
    keep = rng.random_sample(len(i)) < density
    i, j, q = i[keep], j[keep], q[keep]
    return i, j, np.where(i == j, q, 2.0 * q), rng.standard_normal(n)


def _qcqp_data(n, m, n_int, qd, ad, seed):
    """Coefficients, variable kinds and root box of a QCQP: continuous in [-10, 10], integers in [0, 15]."""
    rng = np.random.RandomState(seed & 0x7FFFFFFF)
    kinds = np.array([abi.VAR_INTEGER] * n_int + [abi.VAR_CONTINUOUS] * (n - n_int))
    lo = np.where(kinds == abi.VAR_INTEGER, 0.0, -10.0)
    hi = np.where(kinds == abi.VAR_INTEGER, 15.0, 10.0)
    obj = _quadratic_data(rng, n, qd)
    cons = [(_quadratic_data(rng, n, ad), rng.uniform(1.0, 10.0)) for _ in range(m)]
    return dict(n=n, kinds=kinds, lo=lo, hi=hi, obj=obj, cons=cons, rng=rng)


def _expression(x, data):
    i, j, q, lin = data
    acc = None
    for a, b, c in zip(i.tolist(), j.tolist(), q.tolist()):
        t = c * (x[a] * x[b])
        acc = t if acc is None else acc + t
    for v, c in enumerate(lin.tolist()):
        t = c * x[v]
        acc = t if acc is None else acc + t
    return acc


def _problem(d):
    p = Problem()
    x = [p.int_var(lo, hi) if k == abi.VAR_INTEGER else p.var(lo, hi)
         for k, lo, hi in zip(d["kinds"].tolist(), d["lo"].tolist(), d["hi"].tolist())]
    p.set_objective(_expression(x, d["obj"]))
    for data, rhs in d["cons"]:
        p.add_constraint(_expression(x, data), abi.CMP_LE, float(rhs))
    return p


def _model(case, seed):
    return _qcqp_data(case["n"], case["m"], case["n_int"], case["qd"], case["ad"], seed)


def _boxes(d, count):
    """`count` boxes inside the root box as (n, count) planes: uniform centres, half-widths up to a quarter of
    the root's, integers on the lattice."""
    rng = d["rng"]
    span = (d["hi"] - d["lo"])[:, None]
    c = d["lo"][:, None] + span * rng.random_sample((d["n"], count))
    w = 0.25 * span * rng.random_sample((d["n"], count))
    lo, hi = np.maximum(c - w, d["lo"][:, None]), np.minimum(c + w, d["hi"][:, None])
    ints = d["kinds"] == abi.VAR_INTEGER
    lo[ints] = np.ceil(lo[ints])
    hi[ints] = np.maximum(np.floor(hi[ints]), lo[ints])
    return np.ascontiguousarray(lo), np.ascontiguousarray(hi)


def _composition(d, lo, hi, bits):
    """Slots of one box for 2^bits regions, as a bisecting driver picks them: integers enumerated while their
    lattice fits the budget, then the widest continuous variables halved.  (kinds, var_ids, widths)."""
    kinds, vids, widths = [], [], []
    for v in np.flatnonzero(d["kinds"] == abi.VAR_INTEGER).tolist():
        need = int(hi[v] - lo[v]).bit_length()
        if 0 < need <= bits:
            kinds.append(abi.SLOT_INTEGER_ENUMERATE)
            vids.append(v)
            widths.append(1 << need)
            bits -= need
    cont = np.flatnonzero(d["kinds"] != abi.VAR_INTEGER)
    w = (hi - lo)[cont].copy()
    halved = np.zeros(len(cont), dtype=int)
    for _ in range(bits):
        k = int(np.argmax(w))
        w[k] /= 2.0
        halved[k] += 1
    for k in np.flatnonzero(halved).tolist():
        kinds.append(abi.SLOT_CONTINUOUS)
        vids.append(int(cont[k]))
        widths.append(1 << int(halved[k]))
    return kinds, vids, widths


def _region_planes(d, lo, hi, kinds, vids, widths):
    """The boxes of every region of a composition, (n, regions) planes: slot 0 varies fastest."""
    count = int(np.prod(widths))
    plo, phi = np.repeat(lo[:, None], count, 1), np.repeat(hi[:, None], count, 1)
    r = np.arange(count)
    for k, v, w in zip(kinds, vids, widths):
        part = r % w
        r = r // w
        if k == abi.SLOT_INTEGER_ENUMERATE:
            plo[v] = phi[v] = np.minimum(np.ceil(lo[v]) + part, hi[v])
        else:
            step = (hi[v] - lo[v]) / w
            plo[v], phi[v] = lo[v] + step * part, np.where(part + 1 == w, hi[v], lo[v] + step * (part + 1))
    return plo, phi


# ---- prepare / run -----------------------------------------------------------------------------------------
def _general(n, seed):
    """A model with shared subexpressions, divisions and roots: its variable pairs."""
    rng = np.random.RandomState(seed & 0x7FFFFFFF)
    perm = rng.permutation(n)
    return dict(n=n, kinds=np.zeros(n, dtype=int), lo=np.full(n, -2.0), hi=np.full(n, 3.0), rng=rng,
                perm=perm.tolist(), w=rng.uniform(0.5, 2.0, n).tolist())


def _general_problem(d):
    p = Problem()
    x = [p.var(lo, hi) for lo, hi in zip(d["lo"].tolist(), d["hi"].tolist())]
    obj = con = None
    for k in range(d["n"]):
        a, b, c = x[k], x[d["perm"][k]], x[(k + 1) % d["n"]]
        s = sqr(a) + 1.0  # shared by the quotient and the root
        t = sqr(b - c) / s + d["w"][k] * sqrt(s)
        obj = t if obj is None else obj + t
        u = (a + b) * c
        con = u if con is None else con + u
    p.set_objective(obj)
    p.add_constraint(con, abi.CMP_LE, 0.5 * d["n"])
    return p


def _slot_args(case, d):
    lo, hi = _boxes(d, 1)
    lo, hi = lo[:, 0], hi[:, 0]
    wide = d["kinds"] != abi.VAR_INTEGER  # an open box: a driver's expanded node is wide in most variables
    lo[wide] = np.maximum(lo[wide] - 2.0, d["lo"][wide])
    hi[wide] = np.minimum(hi[wide] + 2.0, d["hi"][wide])
    return lo, hi, _composition(d, lo, hi, case["bits"])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("role", "aggregate"):
        d = _model(case, seed)
        lo, hi, (kinds, vids, widths) = _slot_args(case, d)
        dp = DeviceProblem(_problem(d))
        regions = int(np.prod(widths))
        s = dict(case=case, dp=dp, box=np.stack([lo, hi], 1).reshape(-1).copy(), vids=vids, widths=widths,
                 salt=1 + seed % 1000, bounder=Bounder(dp, kinds, regions))
        if kind == "role":
            s["sampler"] = Sampler(dp, kinds, regions, sample_points=case["points"])
        return s
    if kind == "eval_host":
        d = _general(case["n"], seed)
        lo, hi = _boxes(d, case["boxes"])
        return dict(case=case, dp=DeviceProblem(_general_problem(d)), lo=lo, hi=hi)
    if kind == "eval_device":
        d = _model(case, seed)
        lo, hi = _boxes(d, case["boxes"])
        n = case["boxes"]
        return dict(case=case, dp=DeviceProblem(_problem(d)), lo=torch.from_numpy(lo).cuda(),
                    hi=torch.from_numpy(hi).cuda(), lb=torch.empty(n, dtype=torch.float64, device="cuda"),
                    ub=torch.empty(n, dtype=torch.float64, device="cuda"),
                    feasible=torch.empty(n, dtype=torch.uint8, device="cuda"))
    if kind == "solve":
        return dict(case=case, dp=DeviceProblem(_problem(_model(case, seed))))
    if kind == "batch":
        rng = np.random.RandomState(seed & 0x7FFFFFFF)
        dps = []
        for k in range(case["count"]):
            n = int(rng.randint(case["n_lo"], case["n_hi"] + 1))
            c = dict(n=n, m=int(rng.randint(0, 13)), n_int=int(rng.uniform(0.0, 0.25) * n),
                     qd=rng.uniform(0.1, 1.0), ad=rng.uniform(0.1, 0.6))
            dps.append(DeviceProblem(_problem(_model(c, seed * 64 + k))))
        return dict(case=case, dps=dps)
    dps = []
    sizes = [8] * 4 + [16] * 3 + [32] * 2 + [64]  # the serving mix's weights
    rng = np.random.RandomState(seed & 0x7FFFFFFF)
    for k in range(case["count"]):
        n = sizes[k % len(sizes)]
        c = dict(n=n, m=n // 4, n_int=n // 10, qd=rng.uniform(0.1, 1.0), ad=rng.uniform(0.1, 0.4))
        dps.append(DeviceProblem(_problem(_model(c, seed * 64 + k))))
    server = Server([(8, 8), (16, 8), (32, 8), (64, 4)], bisection_budget=case["bits"],
                    batch_parents=case["parents"], frontier_cap=case["cap"],
                    precision=abi.precision_code(case["precision"]))
    return dict(case=case, dps=dps, server=server)


def _outcome(o, n):
    found = bool(o["found_incumbent"])
    return dict(bounds=np.array([o["lower_bound"], o["upper_bound"] if found else np.inf]),
                best_point=np.asarray(o["best_point"]) if found else np.full(n, np.nan),
                counts=np.array([o["counters"][c] for c in COUNTERS] + [o["frontier_size"], o["viable"],
                                int(o["proven_optimal"]), int(found)], dtype=np.int64))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "role":
        cand = state["sampler"].sample(state["box"], state["vids"], state["widths"], state["salt"])
        feasible, lb = state["bounder"].bound(state["box"], state["vids"], state["widths"])
        return dict(feasible=feasible, lb=lb, found=cand.found, value=cand.value, point=cand.point, index=cand.index)
    if kind == "aggregate":
        lb, ub, feasible = state["bounder"].bound_children(state["box"], state["vids"], state["widths"],
                                                           case["children"])
        return dict(lb=lb, ub=ub, feasible=feasible)
    if kind == "eval_host":
        lb, ub, feasible = eval_boxes(state["dp"], state["lo"], state["hi"])
        return dict(lb=lb, ub=ub, feasible=feasible)
    if kind == "eval_device":
        n = case["boxes"]
        eval_boxes_device(state["dp"], state["lo"].data_ptr(), state["hi"].data_ptr(), n, n, state["lb"].data_ptr(),
                          state["ub"].data_ptr(), state["feasible"].data_ptr(), case["precision"],
                          torch.cuda.current_stream().cuda_stream)
        return dict(lb=state["lb"], ub=state["ub"], feasible=state["feasible"])
    if kind == "solve":
        s = Solver(state["dp"], precision=case["precision"], bisection_budget=case["bits"],
                   batch_parents=case["parents"], frontier_cap=case["cap"], sample_points=case["points"],
                   batch_iter_limit=case["iters"], iter_limit=1 << 40)
        try:
            s.step(0)
            return _outcome(s.outcome(), case["n"])
        finally:
            s.close()
    if kind == "batch":
        outs = batch_solve(state["dps"], precision=abi.precision_code(case["precision"]),
                           bisection_budget=case["bits"], batch_parents=case["parents"], frontier_cap=case["cap"],
                           batch_iter_limit=case["iters"], iter_limit=1 << 40)
    else:
        server = state["server"]
        ids = [server.submit(dp, iter_limit=case["expansions"]) for dp in state["dps"]]
        outs = [server.wait(i) for i in ids]
    outs = [_outcome(o, dp.n_vars) for o, dp in zip(outs, state["dps"])]
    points = np.full((len(outs), 64), np.nan)  # one row per problem, past its variables NaN
    for row, o in zip(points, outs):
        row[:len(o["best_point"])] = o["best_point"]
    return dict(bounds=np.stack([o["bounds"] for o in outs]), points=points,
                counts=np.stack([o["counts"] for o in outs]))


# ---- what a pass cannot do without -------------------------------------------------------------------------
def work(case):
    """Bytes: every box or region verdict crosses memory once.  Flops: one product, one scaling and one add per
    term of every bound that is returned or that decides feasibility, and of every sample point."""
    kind = case["kind"]
    if kind == "eval_host":
        return {"bytes": case["boxes"] * (16.0 * case["n"] + 17), "flops": case["boxes"] * 40.0 * case["n"]}
    if kind in ("batch", "serve"):
        n = 0.5 * (case["n_lo"] + case["n_hi"]) if kind == "batch" else 20.0
        boxes = case["count"] * (case["parents"] * case["iters"] if kind == "batch" else case["expansions"])
        boxes = float(boxes << case["bits"])
        return {"bytes": boxes * 16 * n, "flops": boxes * 3 * (n * (n + 1) / 2 * 0.5 + n)}
    terms = _terms(case)
    if kind in ("role", "aggregate"):
        regions = float(1 << case["bits"])
        passes = 1 + (case["points"] if kind == "role" else 0)
        return {"bytes": 16.0 * case["n"] + 9 * regions, "flops": regions * passes * 3 * terms}
    if kind == "eval_device":
        return {"bytes": case["boxes"] * (16.0 * case["n"] + 17), "flops": case["boxes"] * 3.0 * terms}
    boxes = float((case["parents"] << case["bits"]) * case["iters"])
    return {"bytes": boxes * (16.0 * case["n"] + 26), "flops": boxes * 3 * terms * (1 + case["points"])}


# ---- the same in plain numpy, 64 bits ----------------------------------------------------------------------
def _product(al, ah, bl, bh):
    p = (al * bl, al * bh, ah * bl, ah * bh)
    return np.minimum(np.minimum(p[0], p[1]), np.minimum(p[2], p[3])), \
        np.maximum(np.maximum(p[0], p[1]), np.maximum(p[2], p[3]))


def _square(lo, hi):
    a, b = lo * lo, hi * hi
    return np.where((lo <= 0) & (hi >= 0), 0.0, np.minimum(a, b)), np.maximum(a, b)


def _quadratic_range(data, lo, hi):
    i, j, q, lin = data
    rl, rh = np.zeros(lo.shape[1]), np.zeros(lo.shape[1])
    for a, b, c in zip(i.tolist(), j.tolist(), q.tolist()):
        pl, ph = _square(lo[a], hi[a]) if a == b else _product(lo[a], hi[a], lo[b], hi[b])
        rl += c * (pl if c >= 0 else ph)
        rh += c * (ph if c >= 0 else pl)
    for v, c in enumerate(lin.tolist()):
        rl += c * (lo[v] if c >= 0 else hi[v])
        rh += c * (hi[v] if c >= 0 else lo[v])
    return rl, rh


def exact(case, seed):
    kind = case["kind"]
    if kind == "role":
        d = _model(case, seed)
        lo, hi, slots = _slot_args(case, d)
        lb, _ = _quadratic_range(d["obj"], *_region_planes(d, lo, hi, *slots))
        return dict(feasible=None, lb=lb, found=None, value=None, point=None, index=None)
    if kind == "aggregate":
        d = _model(case, seed)
        lo, hi, slots = _slot_args(case, d)
        plo, phi = _region_planes(d, lo, hi, *slots)
        keep = np.ones(plo.shape[1], dtype=bool)
        for data, rhs in d["cons"]:
            keep &= _quadratic_range(data, plo, phi)[0] <= rhs
        rl, rh = _quadratic_range(d["obj"], plo, phi)
        lb = np.where(keep, rl, np.inf).reshape(case["children"], -1).min(1)
        ub = np.where(keep, rh, -np.inf).reshape(case["children"], -1).max(1)
        return dict(lb=lb, ub=np.where(ub > -np.inf, ub, np.inf), feasible=None)
    if kind == "eval_device":
        d = _model(case, seed)
        lb, ub = _quadratic_range(d["obj"], *_boxes(d, case["boxes"]))
        return dict(lb=lb, ub=ub, feasible=None)
    if kind == "eval_host":
        d = _general(case["n"], seed)
        lo, hi = _boxes(d, case["boxes"])
        rl, rh = np.zeros(case["boxes"]), np.zeros(case["boxes"])
        for k in range(case["n"]):
            b, c = d["perm"][k], (k + 1) % case["n"]
            sl, sh = _square(lo[k], hi[k])
            sl, sh = sl + 1.0, sh + 1.0
            ql, qh = _square(lo[b] - hi[c], hi[b] - lo[c])
            rl += ql / sh + d["w"][k] * np.sqrt(sl)
            rh += qh / sl + d["w"][k] * np.sqrt(sh)
        return dict(lb=rl, ub=rh, feasible=None)
    return None
