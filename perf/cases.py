"""The work that users of this library have it do, as cases that can be timed
and checked one by one: SpMV, lock() of a first and of a later epoch,
transpose, SpGEMM, addition and the batched multi-right-hand-side SpMV, each
through the Python binding, from small matrices to the largest configuration.

All matrices are seeded synthetic ones, drawn with torch on the device:
  stencil2d  5-point stencil on a g x g grid, coefficients uniform in [-1, 1)
  stencil3d  7-point stencil on a g^3 grid, coefficients uniform in [-1, 1)
  uniform    `per_row` uniform columns per row (a column may repeat: the last
             insert wins)
  zipf       row lengths Zipf(1.8) on [1, 10 000], scaled to a mean of 16,
             uniform columns
A case's random pattern is drawn once and turned by a number of rows and
columns that depends on the seed, so that every seed's outputs have the same
sizes; the values, vectors and insertion orders are drawn from the seed.
"""
import math

import numpy as np
import torch

import spira_gb300 as sg

ZIPF_ALPHA, ZIPF_CAP, ZIPF_MEAN = 1.8, 10_000, 16.0
KS = (1, 2, 4, 8, 16, 32)  # right-hand sides of the batched SpMV


def listed():
    return [
        # The small configuration (10 000 rows, 10 entries each), x and y in
        # host memory as the C++ facade's spmv() takes them: the call, its
        # copies and its launch are what is paid.
        {"name": "spmv_host_uniform_10k", "op": "spmv", "family": "uniform", "rows": 10_000, "cols": 10_000,
         "per_row": 10, "staging": "host"},
        # The large stencil configuration: 2 M rows of five entries.
        {"name": "spmv_stencil2d_1414", "op": "spmv", "family": "stencil2d", "grid": 1414,
         "staging": "device"},
        # The large power-law configuration: 64 M entries, columns anywhere.
        {"name": "spmv_zipf_4m", "op": "spmv", "family": "zipf", "rows": 4_000_000, "staging": "device"},
        # The small configuration's lock(): inserts staged on the host row by
        # row, the way the C++ facade's insert() hands them over.
        {"name": "lock_host_uniform_10k", "op": "lock", "family": "uniform", "rows": 10_000, "cols": 10_000,
         "per_row": 10, "order": "rows", "staging": "host"},
        # The large power-law configuration's first lock(): assembled on the
        # device row by row, columns in any order.
        {"name": "lock_zipf_4m", "op": "lock", "family": "zipf", "rows": 4_000_000, "order": "rows",
         "staging": "device"},
        # Assembly in any order (element by element, or merged from several
        # producers): the stencil's 10 M inserts shuffled.
        {"name": "lock_shuffled_stencil2d_1414", "op": "lock", "family": "stencil2d", "grid": 1414,
         "order": "shuffled", "staging": "device"},
        # A later epoch: 1 % new entries in 10 % of the rows, staged on the
        # host, locked into a copy of the matrix.
        {"name": "relock_stencil2d_1414", "op": "relock", "family": "stencil2d", "grid": 1414},
        # A rectangular interpolation-like operator, transposed for the
        # restriction; an odd size.
        {"name": "transpose_uniform_500k", "op": "transpose", "family": "uniform", "rows": 500_009, "cols": 200_003,
         "per_row": 8},
        # The SpGEMM configurations: products that collapse onto few columns
        # and products that hardly ever meet.
        {"name": "spgemm_stencil3d_100", "op": "spgemm", "family": "stencil3d", "grid": 100},
        {"name": "spgemm_uniform_200k", "op": "spgemm", "family": "uniform", "rows": 200_000, "cols": 200_000,
         "per_row": 8},
        # A + B of two power-law matrices (a quarter of the large one), B
        # being A after another epoch of 1 % new entries.
        {"name": "add_zipf_1m", "op": "add", "family": "zipf", "rows": 1_000_000, "pattern": "same"},
        # The batched configuration, a sixteenth of its matrices.
        {"name": "batched_256", "op": "batched", "matrices": 256, "rows_lo": 100, "rows_hi": 200_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_family(rng, op, entries):
    """A matrix of about `entries` entries; the shape is odd as often as not."""
    families = ["stencil2d", "stencil3d", "uniform"] + ([] if op == "spgemm" else ["zipf"])
    f = rng.choice(families)
    if f == "stencil2d":
        return {"family": f, "grid": max(20, int(math.sqrt(entries / 5.0)))}
    if f == "stencil3d":
        return {"family": f, "grid": max(8, int((entries / 7.0) ** (1.0 / 3.0)))}
    if f == "zipf":
        return {"family": f, "rows": max(2000, int(entries / ZIPF_MEAN))}
    per = rng.randint(4, 12 if op == "spgemm" else 24)
    rows = max(500, entries // per)
    square = op == "spgemm"
    cols = rows if square else max(500, int(rows * math.exp(rng.uniform(math.log(0.3), math.log(3.0)))))
    return {"family": f, "rows": rows, "cols": cols, "per_row": per}


def draw(rng):
    op = rng.choice(["spmv", "lock", "lock", "relock", "transpose", "spgemm", "spgemm", "add", "batched"])
    if op == "batched":
        return {"op": op, "matrices": _log_int(rng, 8, 256), "rows_lo": 100, "rows_hi": _log_int(rng, 5_000, 200_000)}
    top = {"spmv": 60_000_000, "lock": 30_000_000, "relock": 16_000_000, "transpose": 16_000_000,
           "spgemm": 3_000_000, "add": 16_000_000}[op]
    entries = _log_int(rng, 100_000, top)
    case = {"op": op, **_draw_family(rng, op, entries)}
    if op == "spmv":
        case["staging"] = "host" if entries < 1_000_000 else "device"
    if op == "lock":
        case["order"] = rng.choice(["rows", "shuffled"])
        case["staging"] = rng.choice(["device", "device", "host"])
    if op == "add":
        case["pattern"] = rng.choice(["same", "other"])
    return case


# ------------------------------------------------------------------- inputs
def _gen(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + stream) & 0x7FFFFFFFFFFFFFFF)
    return g


def _sym(n, g):
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2.0 - 1.0


def _shape(case):
    f = case["family"]
    if f == "stencil2d":
        return case["grid"] ** 2, case["grid"] ** 2
    if f == "stencil3d":
        return case["grid"] ** 3, case["grid"] ** 3
    return case["rows"], case.get("cols", case["rows"])


def _stencil(grid, dims):
    """(rows, cols) of a grid stencil in row order, columns ascending."""
    n = grid ** dims
    i = torch.arange(n, dtype=torch.int64, device="cuda")
    steps = [-grid ** d for d in range(dims - 1, -1, -1)] + [0] + [grid ** d for d in range(dims)]
    cols = torch.empty((n, len(steps)), dtype=torch.int64, device="cuda")
    ok = torch.empty((n, len(steps)), dtype=torch.bool, device="cuda")
    for k, s in enumerate(steps):
        cols[:, k] = i + s
        if s == 0:
            ok[:, k] = True
        else:
            pos = (i // abs(s)) % grid
            ok[:, k] = pos > 0 if s < 0 else pos < grid - 1
    rows = i[:, None].expand_as(cols)[ok]
    return rows.to(torch.int32), cols[ok].to(torch.int32)


def _zipf_lengths(n, g):
    k = torch.arange(1, ZIPF_CAP + 1, dtype=torch.float64, device="cuda")
    p = k ** -ZIPF_ALPHA
    cdf = torch.cumsum(p, 0) / p.sum()
    scale = ZIPF_MEAN / float((k * p).sum() / p.sum())
    u = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    z = (torch.searchsorted(cdf, u, right=True) + 1).clamp(max=ZIPF_CAP)
    return (z * scale).round().clamp(1, ZIPF_CAP).to(torch.int64)


def _turn(case, seed):
    """How far the seed turns a case's random pattern (a stencil: not)."""
    return 0 if "grid" in case else (int(seed) * 7919 + 1) % _shape(case)[0]


def _staged(case, seed, stream=0):
    """One epoch of inserts (rows, cols, vals) on the device, row by row."""
    f = case["family"]
    if f in ("stencil2d", "stencil3d"):
        rows, cols = _stencil(case["grid"], 2 if f == "stencil2d" else 3)
    else:
        n, m = _shape(case)
        g = _gen(0, stream + 100)
        if f == "zipf":
            lengths = _zipf_lengths(n, g)
            rows = torch.repeat_interleave(torch.arange(n, dtype=torch.int32, device="cuda"), lengths)
        else:
            rows = torch.arange(n, dtype=torch.int32, device="cuda").repeat_interleave(case["per_row"])
        cols = torch.randint(0, m, (rows.numel(),), dtype=torch.int32, device="cuda", generator=g)
        turn = _turn(case, seed)
        cut = int((rows < n - turn).sum())  # the rows after it come first now
        rows = torch.cat([rows[cut:] - (n - turn), rows[:cut] + turn])
        cols = (torch.cat([cols[cut:], cols[:cut]]) + turn) % m
    return rows, cols, _sym(rows.numel(), _gen(seed, stream))


def _epoch(case, seed, nnz, stream):
    """A later epoch: 1 % of nnz new entries in a random tenth of the rows."""
    g = _gen(0, stream + 100)
    n, m = _shape(case)
    dirty = torch.randperm(n, device="cuda", generator=g)[: max(1, n // 10)].to(torch.int32)
    k = max(1, int(round(0.01 * nnz)))
    rows = dirty[torch.randint(0, dirty.numel(), (k,), device="cuda", generator=g)]
    cols = torch.randint(0, m, (k,), dtype=torch.int32, device="cuda", generator=g)
    turn = _turn(case, seed)
    return (rows + turn) % n, (cols + turn) % m, _sym(k, _gen(seed, stream))


def _lock_inputs(case, seed):
    rows, cols, vals = _staged(case, seed)
    if case["order"] == "shuffled":
        p = torch.randperm(rows.numel(), device="cuda", generator=_gen(seed, 9))
        rows, cols, vals = rows[p], cols[p], vals[p]
    return rows, cols, vals


def _batch_shapes(case):
    r = np.random.RandomState(17)
    lo, hi = math.log(case["rows_lo"]), math.log(case["rows_hi"])
    rows = np.rint(np.exp(lo + r.random_sample(case["matrices"]) * (hi - lo))).astype(np.int64)
    ks = np.array(KS)[r.randint(0, len(KS), case["matrices"])].astype(np.int64)
    return rows, ks


def _batch_inputs(case, seed):
    """Every matrix's inserts (Poisson(12) uniform columns per row) and
    right-hand sides, each as one tensor with the matrices' bounds."""
    rows, ks = _batch_shapes(case)
    g = _gen(0, 20)
    n = torch.from_numpy(rows).cuda()
    total = int(rows.sum())
    lengths = torch.poisson(torch.full((total,), 12.0, device="cuda"), generator=g).to(torch.int64)
    mat_of_row = torch.repeat_interleave(torch.arange(len(rows), device="cuda"), n)
    first = torch.cumsum(n, 0) - n
    local = torch.arange(total, device="cuda") - first[mat_of_row]
    r = torch.repeat_interleave(local, lengths).to(torch.int32)
    width = n[torch.repeat_interleave(mat_of_row, lengths)]
    u = torch.rand(r.numel(), dtype=torch.float64, device="cuda", generator=g)
    c = ((torch.minimum((u * width).to(torch.int64), width - 1) + int(seed) * 7919) % width).to(torch.int32)
    g = _gen(seed, 21)
    v = _sym(r.numel(), g)
    per_mat = torch.zeros(len(rows), dtype=torch.int64, device="cuda").index_add_(0, mat_of_row, lengths).cpu().numpy()
    bounds = np.concatenate([[0], np.cumsum(per_mat)])
    xb = np.concatenate([[0], np.cumsum(rows * ks)])
    return rows, ks, (r, c, v), bounds, _sym(int(xb[-1]), g), xb


# ------------------------------------------------------------ states and runs
_CTX = []


def _ctx():
    """One context per process, as a program keeps it."""
    if not _CTX:
        _CTX.append(sg.Context(0))
    return _CTX[0]


def _locked(shape, staged):
    A = sg.Csr(_ctx(), *shape)
    torch.cuda.synchronize()
    A.lock_device(*staged, staged[0].numel())
    return A


class _Device:
    """An array of a matrix on the device, for torch; keeps the matrix."""

    def __init__(self, owner, ptr, n, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (ptr, False), "version": 3}


def _csr(A):
    """The whole CSR as tensors over the matrix's own arrays."""
    off, cols, vals = A.device_arrays()
    i = A.info()
    t = lambda p, n, kind: torch.as_tensor(_Device(A, p, n, kind), device="cuda")  # noqa: E731
    return {"off": t(off, i["n_rows"] + 1, "<i8"), "cols": t(cols, i["nnz"], "<i4"), "vals": t(vals, i["nnz"], "<f8")}


def _host(t):
    return t.cpu().numpy()


def prepare(case, seed):
    op = case["op"]
    ctx = _ctx()
    if op == "batched":
        rows, ks, (r, c, v), b, X, xb = _batch_inputs(case, seed)
        torch.cuda.synchronize()
        mats, Y = [], torch.zeros_like(X)
        for i, n in enumerate(rows):
            lo, hi = int(b[i]), int(b[i + 1])
            A = sg.Csr(ctx, int(n), int(n))
            A.lock_device(r[lo:hi], c[lo:hi], v[lo:hi], hi - lo)
            mats.append(A)
        Xs = [X[xb[i]:xb[i + 1]] for i in range(len(rows))]
        Ys = [Y[xb[i]:xb[i + 1]] for i in range(len(rows))]
        return {"op": op, "batch": sg.Batch(ctx, mats, Xs, Ys, [int(k) for k in ks]), "X": X, "Y": Y}
    shape = _shape(case)
    if op == "lock":
        staged = _lock_inputs(case, seed)
        if case["staging"] == "host":
            staged = (_host(staged[0]).view(np.uint32), _host(staged[1]).view(np.uint32), _host(staged[2]))
        return {"op": op, "shape": shape, "host": case["staging"] == "host", "staged": staged}
    A = _locked(shape, _staged(case, seed))
    if op == "spmv":
        x = _sym(shape[1], _gen(seed, 1))
        if case["staging"] == "host":
            return {"op": op, "host": True, "A": A, "x": _host(x), "y": np.zeros(shape[0])}
        return {"op": op, "host": False, "A": A, "x": x, "y": torch.zeros(shape[0], dtype=torch.float64, device="cuda")}
    if op == "relock":
        r, c, v = _epoch(case, seed, A.nnz, 2)
        return {"op": op, "shape": shape, "A": A,
                "staged": (_host(r).view(np.uint32), _host(c).view(np.uint32), _host(v))}
    if op == "add":
        if case["pattern"] == "same":
            B = sg.Csr(ctx, *shape)
            B.copy_from(A)
            e = _epoch(case, seed, A.nnz, 2)
            torch.cuda.synchronize()
            B.lock_device(*e, e[0].numel())
        else:
            B = _locked(shape, _staged(case, seed, 3))
        return {"op": op, "A": A, "B": B}
    return {"op": op, "A": A}  # transpose, spgemm


def run(state):
    op = state["op"]
    if op == "spmv":
        if state["host"]:
            return state["A"].spmv_host(state["x"], state["y"])
        state["A"].spmv(state["x"], state["y"])
        return state["y"]
    if op == "lock":
        A = sg.Csr(_ctx(), *state["shape"])
        if state["host"]:
            A.lock(*state["staged"])
        else:
            A.lock_device(*state["staged"], state["staged"][0].numel())
        return _csr(A)
    if op == "relock":
        A = sg.Csr(_ctx(), *state["shape"])
        A.copy_from(state["A"])
        A.lock(*state["staged"])
        return _csr(A)
    if op == "transpose":
        return _csr(state["A"].transpose())
    if op == "spgemm":
        return _csr(state["A"].spgemm(state["A"]))
    if op == "add":
        return _csr(state["A"].add(state["B"]))
    state["batch"].run()
    return state["Y"]


# ------------------------------------------------------------------- the work
def _entries(case):
    f = case["family"]
    if f == "stencil2d":
        g = case["grid"]
        return 5 * g * g - 4 * g
    if f == "stencil3d":
        g = case["grid"]
        return 7 * g ** 3 - 6 * g * g
    return int(case["rows"] * (ZIPF_MEAN if f == "zipf" else case["per_row"]))


def _csr_bytes(rows, nnz):
    return 12 * nnz + 8 * (rows + 1)


def work(case):
    """Inputs read once and outputs written once; entries of random families
    by their expected number."""
    op = case["op"]
    if op == "batched":
        mean_rows = (case["rows_hi"] - case["rows_lo"]) / math.log(case["rows_hi"] / case["rows_lo"])
        rows = case["matrices"] * mean_rows
        k = sum(KS) / len(KS)
        return {"bytes": 12 * 12 * rows + 8 * rows + 16 * k * rows, "flops": 2 * 12 * rows * k}
    n, m = _shape(case)
    z = _entries(case)
    if op == "spmv":
        return {"bytes": _csr_bytes(n, z) + 8 * (n + m), "flops": 2 * z}
    if op == "lock":
        return {"bytes": 16 * z + _csr_bytes(n, z), "flops": 0}
    if op == "relock":
        d = int(0.01 * z)
        return {"bytes": _csr_bytes(n, z) + 16 * d + _csr_bytes(n, z + d), "flops": 0}
    if op == "transpose":
        return {"bytes": _csr_bytes(n, z) + _csr_bytes(m, z), "flops": 0}
    if op == "add":
        same = case["pattern"] == "same"
        b = z * 1.01 if same else z
        return {"bytes": _csr_bytes(n, z) + _csr_bytes(n, b) + _csr_bytes(n, b if same else z + b),
                "flops": z if same else 0}
    per = {"stencil2d": 5, "stencil3d": 7}.get(case["family"]) or case["per_row"]
    out = {"stencil2d": 13, "stencil3d": 25}.get(case["family"]) or per * per
    return {"bytes": _csr_bytes(n, z) + _csr_bytes(n, out * n), "flops": 2 * per * z}


# ------------------------------------------------------------ the exact answers
def _last_writes(shape, *epochs):
    """What locking the epochs one after another leaves: sorted (keys, vals)."""
    m = shape[1]
    keys = torch.cat([e[0].to(torch.int64) * m + e[1].to(torch.int64) for e in epochs])
    vals = torch.cat([e[2] for e in epochs])
    keys, at = torch.sort(keys, stable=True)
    last = torch.ones(keys.numel(), dtype=torch.bool, device=keys.device)
    last[:-1] = keys[1:] != keys[:-1]
    keys, vals = keys[last], vals[at[last]]
    kept = vals != 0
    return keys[kept], vals[kept]


def _as_csr(shape, keys, vals):
    rows = torch.div(keys, shape[1], rounding_mode="floor")
    off = torch.zeros(shape[0] + 1, dtype=torch.int64, device=keys.device)
    off[1:] = torch.cumsum(torch.bincount(rows, minlength=shape[0]), 0)
    return {"off": off, "cols": (keys - rows * shape[1]).to(torch.int32), "vals": vals}


def _row_sums(data, off):
    """Each row's sum of `data`, one term after another."""
    return torch.segment_reduce(data, "sum", lengths=off[1:] - off[:-1], axis=0, unsafe=True, initial=0.0)


def _summed(shape, keys, vals):
    """Equal keys' values summed one after another, zero sums dropped."""
    keys, at = torch.sort(keys, stable=True)
    uniq, counts = torch.unique_consecutive(keys, return_counts=True)
    off = torch.zeros(counts.numel() + 1, dtype=torch.int64, device=keys.device)
    off[1:] = torch.cumsum(counts, 0)
    sums = _row_sums(vals[at], off)
    kept = sums != 0
    return _as_csr(shape, uniq[kept], sums[kept])


def exact(case, seed):
    op = case["op"]
    if op == "batched":
        rows, ks, (r, c, v), b, X, xb = _batch_inputs(case, seed)
        out = torch.empty_like(X)
        for i, n in enumerate(int(n) for n in rows):
            s = slice(int(b[i]), int(b[i + 1]))
            M = _as_csr((n, n), *_last_writes((n, n), (r[s], c[s], v[s])))
            x = X[xb[i]:xb[i + 1]].view(n, int(ks[i]))
            y = _row_sums(M["vals"][:, None] * x[M["cols"].to(torch.int64)], M["off"])
            out[xb[i]:xb[i + 1]] = y.reshape(-1)
        return out
    shape = _shape(case)
    if op == "lock":
        return _as_csr(shape, *_last_writes(shape, _lock_inputs(case, seed)))
    first = _staged(case, seed)
    keys, vals = _last_writes(shape, first)
    if op == "spmv":
        M = _as_csr(shape, keys, vals)
        return _row_sums(vals * _sym(shape[1], _gen(seed, 1))[M["cols"].to(torch.int64)], M["off"])
    if op == "transpose":
        rows = torch.div(keys, shape[1], rounding_mode="floor")
        turned, at = torch.sort((keys - rows * shape[1]) * shape[0] + rows)
        return _as_csr((shape[1], shape[0]), turned, vals[at])
    if op == "relock":
        return _as_csr(shape, *_last_writes(shape, first, _epoch(case, seed, keys.numel(), 2)))
    if op == "add":
        if case["pattern"] == "same":
            b = _last_writes(shape, first, _epoch(case, seed, keys.numel(), 2))
        else:
            b = _last_writes(shape, _staged(case, seed, 3))
        return _summed(shape, torch.cat([keys, b[0]]), torch.cat([vals, b[1]]))
    # C = A A: every product a_ik b_kj, in ascending k for each (i, j)
    M = _as_csr(shape, keys, vals)
    i = torch.div(keys, shape[1], rounding_mode="floor")
    k = M["cols"].to(torch.int64)
    lengths = (M["off"][1:] - M["off"][:-1])[k]
    e = torch.repeat_interleave(torch.arange(keys.numel(), device="cuda"), lengths)
    first_of = torch.cumsum(lengths, 0) - lengths
    f = M["off"][k][e] + torch.arange(e.numel(), device="cuda") - first_of[e]
    return _summed(shape, i[e] * shape[1] + k[f], vals[e] * vals[f])
