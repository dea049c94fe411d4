"""What the presolve engine's speed is measured on: calls that a user's program
makes through the public entry points, on LPs of the families and sizes that
this repository's tests and benchmark use.

Kinds of case:

* ``pipeline``: preprocess, then postprocess of a reduced point into host
  x, y, z (gpp_preprocess, gpp_postprocess): what a solver's caller pays.
* ``postsolve``: the tape replayed into device x, y, z alone
  (gpp_postsolve_device), the presolved model at hand.
* ``load``: a model in page-locked host memory brought to the device, A^T built
  there (gpp_lp_from_host).
* ``batch``: many LPs in one call (gpp_preprocess_batch, gpp_postprocess_batch).
* ``sort``: the engine's stable sort of (64-bit key, 32-bit value) device pairs
  (gpp_sort_pairs).

Families: ``random`` (the benchmark's random LPs, optionally with hub rows),
``slack`` (the same with singleton columns), ``qap`` (Adams-Johnson QAP
relaxations), ``replicated`` (symmetric LPs, which colour refinement folds) and
``auxiliary`` (LPs on which the Startup projection rules fire).  All values
are FP64 and all indices int32: the engine has no other types.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "gpu-preprocessor-ijoc_b200"))
from gpp_b200 import capi, device, lpgen  # noqa: E402

INF = math.inf


def listed():
    return [
        # A model of the smoke test's size: launches and waits only.
        {"name": "tiny pipeline", "kind": "pipeline", "family": "slack", "m": 400, "n": 1000},
        # The 2,000 x 5,000 model, the standard small instance.
        {"name": "small pipeline", "kind": "pipeline", "family": "random", "m": 2000, "n": 5000, "hubs": 0},
        # A mid-size model whose singleton columns get substituted out.
        {"name": "slack pipeline", "kind": "pipeline", "family": "slack", "m": 20000, "n": 50000},
        # The largest model of the batched workload, presolved by itself; odd sizes.
        {"name": "medium pipeline", "kind": "pipeline", "family": "random", "m": 199999, "n": 500001, "hubs": 0},
        # The benchmark's single-GPU scale model (about 29.8M nonzeros, 2,000 long rows).
        {"name": "scale pipeline", "kind": "pipeline", "family": "random", "m": 2000000, "n": 5000000, "hubs": 2000},
        # The benchmark's QAP linearisation: parallel rows and columns.
        {"name": "qap pipeline", "kind": "pipeline", "family": "qap", "size": 30},
        # A symmetric model: presolve, folding, postsolve and unfolding.
        {"name": "folded pipeline", "kind": "pipeline", "family": "replicated", "m": 3000, "n": 7500, "copies": 16},
        # A model on which the structure-specific Startup rules fire.
        {"name": "startup pipeline", "kind": "pipeline", "family": "auxiliary", "m": 20000, "n": 50000},
        # Primal and dual recovery of a solver's point, on the device.
        {"name": "postsolve", "kind": "postsolve", "family": "random", "m": 500000, "n": 1250000, "hubs": 500},
        # A model loaded from host memory.
        {"name": "load", "kind": "load", "family": "random", "m": 200000, "n": 500000, "hubs": 0},
        # A batch of small and mid-size LPs, log-uniform in size as in the batched workload.
        {"name": "batch", "kind": "batch", "count": 32, "low": 1000, "high": 20000, "workers": 8},
        # The sort of hashed rows, as the parallel-row rule's callers use it; an odd count.
        {"name": "sort", "kind": "sort", "pairs": 2000003},
    ]


def _log_between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["pipeline"] * 6 + ["postsolve", "load", "batch", "sort"])
    if kind == "sort":
        return {"kind": kind, "pairs": _log_between(rng, 1000, 5000000)}
    if kind == "batch":
        low = _log_between(rng, 500, 4000)
        return {"kind": kind, "count": rng.randint(8, 40), "low": low, "high": low * rng.randint(4, 16),
                "workers": rng.choice([0, 4, 8, 16])}
    family = rng.choice(["random", "random", "slack", "qap", "replicated", "auxiliary"])
    if kind != "pipeline":
        family = "random"
    if family == "qap":
        return {"kind": kind, "family": family, "size": rng.randint(5, 28)}
    if family == "replicated":
        m = _log_between(rng, 200, 4000)
        return {"kind": kind, "family": family, "m": m, "n": int(m * rng.uniform(2.0, 3.0)),
                "copies": rng.randint(4, 16)}
    if family in ("slack", "auxiliary"):
        m = _log_between(rng, 400 if family == "slack" else 4000, 30000)
        return {"kind": kind, "family": family, "m": m, "n": int(m * rng.uniform(2.0, 3.0))}
    m = _log_between(rng, 400, 1000000)
    return {"kind": kind, "family": family, "m": m, "n": int(m * rng.uniform(2.0, 3.0)),
            "hubs": m // 1000 if rng.random() < 0.5 else 0}


# ---- models ---------------------------------------------------------------


class GeneratedLp(device.DeviceLp):
    """An LP whose device arrays were made on the GPU."""

    def __init__(self, m, n, arrays):
        self.host = None
        self.m, self.n, self.nnz = m, n, int(arrays["A_idx"].numel())
        self.t = arrays
        self.obj_constant = 0.0


def _segments(start, length):
    """The positions start[k] .. start[k] + length[k] - 1 of every k, one after the other."""
    ends = torch.cumsum(length, 0)
    first = torch.repeat_interleave(start - (ends - length), length)
    return first + torch.arange(first.numel(), device=first.device)


def _pointers(items, count):
    p = torch.zeros(count + 1, dtype=torch.int64, device=items.device)
    torch.cumsum(torch.bincount(items, minlength=count), 0, out=p[1:])
    return p


def random_lp(m, n, hubs, seed):
    """The random family of gpp_b200.lpgen made on the GPU: per regular column
    1 + Poisson(4) entries at uniform rows, values in [-10, 10] on a 1e-3 grid;
    5% singleton rows, 5% two-entry equality rows, 3% scaled copies of rows, 2%
    scaled copies of columns, 2% empty columns; `hubs` rows of 500 to 5,000
    further entries.  Row sides come from a planted point, so the LP is
    feasible.  Sums are formed on integers, so one seed gives one model."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dev = {"device": "cuda", "generator": g}

    def integers(high, size, low=0):
        return torch.randint(low, high, (size,), **dev)

    def uniform(size, low=0.0, high=1.0):
        return torch.rand(size, dtype=torch.float64, **dev) * (high - low) + low

    def grid(size):   # nonzero integers of a 1e-3 grid
        v = integers(10001, size, 1)
        return torch.where(integers(2, size) == 0, v, -v)

    perm = torch.randperm(m, **dev)
    single, two, copied = round(0.05 * m), round(0.05 * m), round(0.03 * m)
    s_rows, d_rows, c_rows = perm[:single], perm[single:single + two], perm[single + two:single + two + copied]
    normal = perm[single + two + copied:]
    cperm = torch.randperm(n, **dev)
    c_cols, regular = cperm[:round(0.02 * n)], cperm[round(0.02 * n) + round(0.02 * n):]

    # Entries of the regular columns and of the hub rows (each (row, col) once),
    # by column; then the scaled copies of columns.
    per = 1 + torch.poisson(torch.full((regular.numel(),), 4.0, device="cuda"), generator=g).long()
    cols = torch.repeat_interleave(regular, per)
    rows = normal[integers(normal.numel(), cols.numel())]
    if hubs:
        length = torch.exp(uniform(hubs, math.log(500.0), math.log(5000.0))).long().clamp(max=regular.numel())
        h_rows = torch.repeat_interleave(normal[:hubs], length)
        rows = torch.cat([rows, h_rows])
        cols = torch.cat([cols, regular[integers(regular.numel(), h_rows.numel())]])
    key = torch.unique(cols * m + rows)
    cols, rows = key // m, key % m
    vals = grid(key.numel()) * 1000   # from here on in units of 1e-6
    ptr = _pointers(cols, n)
    source = regular[integers(regular.numel(), c_cols.numel())]
    factor = integers(4001, c_cols.numel(), 500)
    factor = torch.where(integers(2, c_cols.numel()) == 0, factor, -factor)
    size = ptr[source + 1] - ptr[source]
    take = _segments(ptr[source], size)
    rows = torch.cat([rows, rows[take]])
    vals = torch.cat([vals, vals[take] // 1000 * torch.repeat_interleave(factor, size)])
    cols = torch.cat([cols, torch.repeat_interleave(c_cols, size)])
    # Singleton rows and two-entry equality rows over regular columns.
    first = integers(regular.numel(), two)
    second = (first + integers(regular.numel(), two, 1)) % regular.numel()
    rows = torch.cat([rows, s_rows, d_rows, d_rows])
    cols = torch.cat([cols, regular[integers(regular.numel(), single)], regular[first], regular[second]])
    vals = torch.cat([vals, grid(single + 2 * two) * 1000])
    order = torch.argsort(rows * n + cols)
    rows, cols, vals = rows[order], cols[order], vals[order]

    # Bounds, a planted point on a 1e-3 grid and its row activities.
    u = uniform(n, 1.0, 100.0)
    unbounded = uniform(n) < 0.2
    x0 = torch.where(unbounded, uniform(n, 0.0, 10000.0), torch.floor(uniform(n) * u * 1000.0)).long()
    u = torch.where(unbounded, INF, u)
    act = torch.zeros(m, dtype=torch.int64, device="cuda").index_add_(0, rows, vals * x0[cols]).double() / 1e9

    # Scaled copies of rows.
    ptr = _pointers(rows, m)
    source = normal[integers(normal.numel(), copied)]
    factor = uniform(copied, 0.5, 4.0)
    size = ptr[source + 1] - ptr[source]
    take = _segments(ptr[source], size)
    vals = vals.double() / 1e6
    vals = torch.cat([vals, vals[take] * torch.repeat_interleave(factor, size)])
    cols = torch.cat([cols, cols[take]])
    rows = torch.cat([rows, torch.repeat_interleave(c_rows, size)])
    act[c_rows] = act[source] * factor

    by_row, by_col = torch.argsort(rows * n + cols), torch.argsort(cols * m + rows)
    equal = torch.zeros(m, dtype=torch.bool, device="cuda")
    equal[d_rows] = True
    AL = torch.where(uniform(m) < 0.5, act - uniform(m, 0.0, 5.0), -INF)
    AU = torch.where(uniform(m) < 0.5, act + uniform(m, 0.0, 5.0), INF)
    c = torch.randn(n, dtype=torch.float64, **dev)
    return GeneratedLp(m, n, {
        "A_ptr": _pointers(rows, m).int(), "A_idx": cols[by_row].int(), "A_val": vals[by_row],
        "AT_ptr": _pointers(cols, n).int(), "AT_idx": rows[by_col].int(), "AT_val": vals[by_col],
        "c": torch.where(unbounded, c.abs(), c), "AL": torch.where(equal, act, AL), "AU": torch.where(equal, act, AU),
        "l": torch.zeros(n, dtype=torch.float64, device="cuda"), "u": u})


def _model(case, seed):
    family = case["family"]
    if family == "random":
        return random_lp(case["m"], case["n"], case["hubs"], seed)
    if family == "qap":
        return device.DeviceLp(lpgen.qap_lp(case["size"], seed))
    if family == "replicated":
        return device.DeviceLp(lpgen.replicated_lp(case["m"], case["n"], case["copies"], seed))
    if family == "auxiliary":
        return device.DeviceLp(lpgen.auxiliary_lp(case["m"], case["n"], seed))
    return device.DeviceLp(lpgen.random_lp(case["m"], case["n"], seed, slack_frac=0.3))


def _point(lp, seed):
    """A solver's point, long enough for any reduction of `lp`: x, y, z."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    kw = {"dtype": torch.float64, "device": "cuda", "generator": g}
    return torch.rand(lp.n, **kw), torch.randn(lp.m, **kw), torch.randn(lp.n, **kw)


def _reduced_point(point, s):
    x, y, z = point
    return x[:s.reduced_cols], y[:s.reduced_rows], z[:s.reduced_cols]


# ---- results --------------------------------------------------------------


class _Memory:
    """`count` values at a device address inside a summary."""

    def __init__(self, address, count, kind):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": kind, "data": (address, False), "version": 2}


def _view(address, count, kind):
    if not count or not address:
        return torch.empty(0, dtype=torch.int32 if kind == "<i4" else torch.float64, device="cuda")
    return torch.as_tensor(_Memory(address, count, kind), device="cuda")


def _reduced(s):
    """Views of the reduced model's arrays."""
    if s.has_infeasible or s.has_unbounded:
        return {}
    m, n, nnz, L = s.reduced_rows, s.reduced_cols, s.reduced_nnz, s.reduced_lp
    return {name: _view(address, count, kind) for name, address, count, kind in (
        ("A_ptr", L.A.rowPtr, m + 1, "<i4"), ("A_idx", L.A.colVal, nnz, "<i4"), ("A_val", L.A.nzVal, nnz, "<f8"),
        ("AT_ptr", L.AT.rowPtr, n + 1, "<i4"), ("AT_idx", L.AT.colVal, nnz, "<i4"), ("AT_val", L.AT.nzVal, nnz, "<f8"),
        ("c", L.c, n, "<f8"), ("AL", L.AL, m, "<f8"), ("AU", L.AU, m, "<f8"), ("l", L.l, n, "<f8"),
        ("u", L.u, n, "<f8"))}


def _said(s):
    """What a summary says of the reduced model."""
    return [s.reduced_rows, s.reduced_cols, s.reduced_nnz, s.iterations, s.has_infeasible, s.has_unbounded,
            s.folding_applied]


def _model_buffers(nnz, m, n):
    """A solver's arrays for a model of at most these sizes; what a model does not fill stays zero."""
    sizes = {"A_ptr": m + 1, "A_idx": nnz, "A_val": nnz, "AT_ptr": n + 1, "AT_idx": nnz, "AT_val": nnz, "c": n,
             "AL": m, "AU": m, "l": n, "u": n}
    return {k: torch.zeros(v, dtype=torch.int32 if k.endswith(("ptr", "idx")) else torch.float64, device="cuda")
            for k, v in sizes.items()}


def _fill(buffers, parts):
    """The solver's copy of the parts' arrays, one after the other."""
    for k, buffer in buffers.items():
        at = 0
        for part in parts:
            if k in part:
                buffer[at:at + part[k].numel()].copy_(part[k])
                at += part[k].numel()
    return buffers


def _capacity(case):
    """Entries, rows and columns that every model of a case stays below."""
    if case["family"] == "qap":
        return tuple(map(int, _entries(case)))
    entries, m, n = (int(1.15 * v) + 400 for v in _entries(case))
    return entries + int(4000 * math.sqrt(case.get("hubs", 0))), m, n


# ---- cases ----------------------------------------------------------------


class State:
    summary = None

    def __del__(self):
        if self.summary is not None:
            device.free_summary(self.summary)


_HOST_ARRAYS = ("A_ptr", "A_idx", "A_val", "c", "AL", "AU", "l", "u")


def _batch_sizes(case):
    """Rows of every LP of a batch: an even spread over the logarithm of the size."""
    k = max(1, case["count"] - 1)
    return [int(case["low"] * (case["high"] / case["low"]) ** (i / k)) for i in range(case["count"])]


def prepare(case, seed):
    s = State()
    s.case, s.params = case, capi.Params.defaults()
    if case["kind"] == "sort":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = case["pairs"]
        # 64-bit hashes, a few percent of them held twice.
        s.keys = torch.randint(-2**63, 2**63 - 1, (n,), device="cuda", generator=g)
        s.keys[n - n // 32:] = s.keys[:n // 32]
        s.values = torch.arange(n, dtype=torch.int32, device="cuda")
        s.out = torch.empty_like(s.keys), torch.empty_like(s.values)
        return s
    if case["kind"] == "batch":
        s.lps = [random_lp(m, int(2.5 * m), 0, 1000 * seed + k) for k, m in enumerate(_batch_sizes(case))]
        s.points = [_point(lp, 1000 * seed + k) for k, lp in enumerate(s.lps)]
        sizes = [_capacity(dict(case, family="random", m=lp.m, n=lp.n)) for lp in s.lps]
        s.model = _model_buffers(*map(sum, zip(*sizes)))
        return s
    s.lp = _model(case, seed)
    if case["kind"] == "load":
        s.host = {k: s.lp.t[k].cpu().pin_memory() for k in _HOST_ARRAYS}
        s.model = _model_buffers(*_capacity(case))
        s.lp = GeneratedLp(s.lp.m, s.lp.n, {k: s.model[k][:v.numel()] for k, v in s.lp.t.items()})
        return s
    s.point = _point(s.lp, seed)
    if case["kind"] == "postsolve":
        s.summary = device.preprocess(s.lp, s.params)
        s.point = _reduced_point(s.point, s.summary)
        return s
    entries, m, n = _capacity(case)
    s.model = _model_buffers(entries, m, n)
    s.solution = [torch.zeros(k, dtype=torch.float64).pin_memory() for k in (n, m, n)]
    return s


def run(s):
    kind = s.case["kind"]
    if kind == "pipeline":
        summary = device.preprocess(s.lp, s.params)
        said, obj = _said(summary), summary.obj_constant_delta
        _fill(s.model, [_reduced(summary)])
        if not summary.has_infeasible and not summary.has_unbounded:
            x, y, z = s.solution
            device.postprocess(*_reduced_point(s.point, summary), summary, s.lp,
                               out=(x[:s.lp.n], y[:s.lp.m], z[:s.lp.n]))
        device.free_summary(summary)
        return s.model, s.solution, said, obj
    if kind == "postsolve":
        return device.postsolve_device(*s.point, s.summary, s.lp)
    if kind == "load":
        s.lp.load_from_host(s.host)
        return s.model
    if kind == "batch":
        summaries, _ = device.preprocess_batch(s.lps, s.params, s.case["workers"])
        said = np.array([_said(x) for x in summaries])
        _fill(s.model, [_reduced(x) for x in summaries])
        reduced = [_reduced_point(p, x) for p, x in zip(s.points, summaries)]
        xs, ys, zs = ([r[k] for r in reduced] for k in range(3))
        solutions = device.postprocess_batch(xs, ys, zs, summaries, s.lps, s.case["workers"])
        for x in summaries:
            device.free_summary(x)
        return s.model, [np.concatenate([v[k] for v in solutions]) for k in range(3)], said
    keys, values = s.out
    keys.copy_(s.keys)
    values.copy_(s.values)
    capi.check(capi.load().gpp_sort_pairs(C.c_void_p(keys.data_ptr()), C.c_void_p(values.data_ptr()), keys.numel()))
    return keys, values


def _entries(case):
    """Stored entries, rows and columns of a case's model (the random ones by expectation)."""
    family = case["family"]
    if family == "qap":
        N = case["size"]
        return 5 * N ** 4 + 2 * N ** 3 + N ** 2, 2 * N ** 4 + 2 * N ** 3 + N ** 2 + 2 * N, N ** 4 + N ** 2
    m, n = case["m"], case["n"]
    per_row = 4.8 * n / (0.87 * m)
    nnz = 0.90 * m * per_row * 1.02 + 0.15 * m + case.get("hubs", 0) * 1950
    if family == "replicated":
        k = case["copies"]
        return nnz * k + n * k, m * k + 1, n * k
    if family == "slack":
        return nnz + 0.3 * m, m, n + 0.3 * m
    if family == "auxiliary":
        return nnz + 0.26 * n, m + 0.1 * n, n + 0.126 * n
    return nnz, m, n


def work(case):
    """Each input read once and each output written once; the reduced model
    counts as three quarters of the entries (one to three rows in ten go)."""
    if case["kind"] == "sort":
        return {"bytes": 24.0 * case["pairs"], "flops": 0.0}
    if case["kind"] == "batch":
        per = [dict(case, kind="pipeline", family="random", m=m, n=int(2.5 * m), hubs=0) for m in _batch_sizes(case)]
        return {"bytes": sum(work(p)["bytes"] for p in per), "flops": 0.0}
    nnz, m, n = _entries(case)
    model = 24.0 * nnz + 4.0 * (m + n) + 8.0 * (3 * n + 2 * m)
    point = 8.0 * (2 * n + m)
    if case["kind"] == "postsolve":
        return {"bytes": 2.0 * point + 12.0 * nnz, "flops": 0.0}
    if case["kind"] == "load":
        return {"bytes": 2.0 * model - 12.0 * nnz, "flops": 0.0}
    return {"bytes": 1.75 * model + 2.0 * point, "flops": 0.0}


def exact(case, seed):
    """A presolved model and a recovered point have no value apart from the
    rules that made them; a loaded model is its host arrays and their transpose."""
    if case["kind"] != "load":
        return None
    s = prepare(case, seed)
    t = {k: v.cpu() for k, v in s.host.items()}
    m, n = s.lp.m, s.lp.n
    cols, ptr = t["A_idx"].long(), t["A_ptr"].long()
    rows = torch.repeat_interleave(torch.arange(m), ptr[1:] - ptr[:-1])
    order = torch.argsort(cols, stable=True)
    t["AT_ptr"] = torch.cat([torch.zeros(1, dtype=torch.int64), torch.cumsum(torch.bincount(cols, minlength=n), 0)]).int()
    t["AT_idx"] = rows[order].int()
    t["AT_val"] = t["A_val"][order]
    return {k: torch.cat([t[k], torch.zeros(v.numel() - t[k].numel(), dtype=t[k].dtype)]) for k, v in s.model.items()}
