"""Performance cases of the framework's public entry points.

Each case is one call (or, for index growth, one short sequence of calls) of
the Python binding as a program would make it, on seeded synthetic data of
the benchmark workloads' distributions (``cuapss.synth.CONFIGS``):

* ``self``   ``Context.run`` / ``run_device``: the self-join of one matrix;
* ``join``   ``Context.join``: the cross-join of two matrices;
* ``batch``  ``Context.batch_run_device``: many uneven instances in one call;
* ``query``  ``Index.query``: a query batch against a resident index;
* ``grow``   building an index, appending rows and querying it;
* ``tools``  the reference's inverted index (``cuapss_build_index``) and the
  frequency remap (``cuapss_feature_remap``), through the C ABI.

``io`` is where the matrix and the pairs live: ``host`` (numpy arrays in and
out, the whole call with its copies) or ``device`` (CUDA tensors). Pairs come
back in buffers of a size that the case alone fixes, with their count.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "apss-cuda_b200"))

import cuapss  # noqa: E402
from cuapss import synth  # noqa: E402

PRECISIONS = {"fp32": cuapss.PREC_FP32, "mixed": cuapss.PREC_MIXED}


def listed():
    return [
        # one small instance by itself (a document set of a few hundred rows,
        # host arrays): launches, host round trips and copies
        {"name": "self_500_mixed", "kind": "self", "cfg": "batch_instance", "n": 500, "t": 0.8,
         "precision": "mixed", "io": "host"},
        # the 20,000-row workload at its own threshold, data already on the GPU
        {"name": "self_20k_mixed", "kind": "self", "cfg": "plain_20k", "n": 20_000, "t": 0.9,
         "precision": "mixed", "io": "device"},
        # the same through the default (plain FP32) context from host arrays
        {"name": "self_20k_fp32", "kind": "self", "cfg": "plain_20k", "n": 20_000, "t": 0.7,
         "precision": "fp32", "io": "host"},
        # plain FP32 at a larger, ragged size and the lowest threshold in use
        {"name": "self_60k_fp32", "kind": "self", "cfg": "plain_800k", "n": 60_001, "t": 0.5,
         "precision": "fp32", "io": "device"},
        # a 200,000-row prefix of the headline workload (d = 1M, Zipf 1.2)
        {"name": "self_200k_mixed", "kind": "self", "cfg": "mixed_1m", "n": 200_000, "t": 0.7,
         "precision": "mixed", "io": "device"},
        # the largest: half of the 800,000-row workload at its lowest threshold
        {"name": "self_400k_mixed", "kind": "self", "cfg": "plain_800k", "n": 400_000, "t": 0.5,
         "precision": "mixed", "io": "device"},
        # two partitions of one corpus against each other, odd sizes
        {"name": "join_mixed", "kind": "join", "cfg": "plain_800k", "n": 20_011, "m": 50_003,
         "t": 0.6, "precision": "mixed", "io": "host"},
        # an eighth of the batched workload: 512 instances of 64 .. 20,000 rows
        {"name": "batch_512_mixed", "kind": "batch", "k": 512, "n_lo": 64, "n_hi": 20_000,
         "precision": "mixed", "io": "device"},
        # the serving workload's request: 256 queries, here on 1M resident rows
        {"name": "query_256_mixed", "kind": "query", "cfg": "serve_5m", "n": 1_000_000, "q": 256,
         "precision": "mixed", "io": "host"},
        # one lookup: the smallest request of the serving mix
        {"name": "query_1_mixed", "kind": "query", "cfg": "serve_5m", "n": 200_000, "q": 1,
         "precision": "mixed", "io": "host"},
        # index growth: bulk load, one append of the serving mix, a lookup
        {"name": "grow_mixed", "kind": "grow", "cfg": "serve_5m", "n": 200_000, "m": 20_000,
         "q": 64, "precision": "mixed", "io": "host"},
        # the reference's inverted index and the frequency remap of a corpus
        {"name": "tools_100k", "kind": "tools", "cfg": "plain_800k", "n": 100_000, "p": 64,
         "precision": "fp32", "io": "device"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["self", "self", "self", "join", "batch", "query", "query", "grow", "tools"])
    prec = rng.choice(["mixed", "mixed", "fp32"])
    cfg = rng.choice(["plain_20k", "plain_800k", "mixed_1m", "batch_instance", "serve_5m"])
    mixed = prec == "mixed"
    t = round(rng.uniform(0.5, 0.95), 3)
    if kind == "self":
        return {"kind": kind, "cfg": cfg, "n": _log(rng, 200, 300_000 if mixed else 70_000),
                "t": t, "precision": prec, "io": rng.choice(["host", "device"])}
    if kind == "join":
        return {"kind": kind, "cfg": cfg, "n": _log(rng, 100, 60_000), "m": _log(rng, 100, 60_000),
                "t": t, "precision": prec, "io": "host"}
    if kind == "batch":
        n_hi = _log(rng, 500, 20_000)
        return {"kind": kind, "k": _log(rng, 4, 400), "n_lo": 64, "n_hi": n_hi, "precision": prec,
                "io": "device"}
    if kind == "query":
        return {"kind": kind, "cfg": "serve_5m", "n": _log(rng, 20_000, 1_000_000),
                "q": _log(rng, 1, 4096), "precision": prec, "io": "host"}
    if kind == "grow":
        return {"kind": kind, "cfg": "serve_5m", "n": _log(rng, 20_000, 200_000),
                "m": _log(rng, 1000, 50_000), "q": _log(rng, 1, 256), "precision": prec,
                "io": "host"}
    return {"kind": "tools", "cfg": cfg, "n": _log(rng, 500, 150_000),
            "p": rng.choice([0, 64, 1000, 4096]), "precision": "fp32", "io": "device"}


# ------------------------------------------------------------------ inputs
# A program keeps one context (stream, working memory) for all its calls of
# one precision.
_contexts = {}


def _context(precision):
    if precision not in _contexts:
        _contexts[precision] = cuapss.Context(device=0, precision=PRECISIONS[precision])
    return _contexts[precision]


def _seed(seed):
    return int(seed) % (1 << 62) + 1


def _rows(case, seed, n, offset=0):
    return synth.generate(case["cfg"], n=n, seed=_seed(seed), row_offset=offset)


def _on_device(x):
    return {"rowptr": torch.from_numpy(x.rowptr).cuda(), "col": torch.from_numpy(x.col).cuda(),
            "val": torch.from_numpy(x.val).cuda(), "d": x.d}


def _pair_slots(case):
    """Slots of a case's pair buffers: a few times the pairs that the
    distributions hold (the planted near-duplicates, and the share of random
    pairs that reach t, about 1e-4 at t = 0.5 and ten times less per 0.1)."""
    kind = case["kind"]
    if kind == "batch":
        rows, square = _batch_sizes(case)
        return 20_000 + int(2 * rows + 1e-4 * square)
    n = case["n"]
    if kind in ("query", "grow"):
        pairs, rows, t = (n + case.get("m", 0)) * case["q"], 8 * case["q"], 0.6
    elif kind == "join":
        pairs, rows, t = n * case["m"], n + case["m"], case["t"]
    else:
        pairs, rows, t = n * n / 2, n, case["t"]
    return 4096 + rows + int(3 * 1.5e-4 * 10 ** (-10 * (t - 0.5)) * pairs)


def _batch_sizes(case):
    """Expected rows, and squared rows, over a batch's instances."""
    span = max(math.log(case["n_hi"] / case["n_lo"]), 1e-9)
    return (case["k"] * (case["n_hi"] - case["n_lo"]) / span,
            case["k"] * (case["n_hi"] ** 2 - case["n_lo"] ** 2) / (2 * span))


def _tool_slots(case):
    return int(case["n"] * synth.CONFIGS[case["cfg"]].nnz_mean * 2) + 4096


def _thresholds(seed, q):
    return np.random.default_rng(_seed(seed)).uniform(0.6, 0.95, size=q).astype(np.float32)


def _queries(case, seed, x):
    """Lookups: every other query is a row the index holds (what are its near
    duplicates?), the rest are rows it has not seen."""
    fresh = _rows(case, seed, case["q"], 50_000_000)
    held = np.random.default_rng(_seed(seed)).integers(0, x.n, size=case["q"])
    both = _stack(fresh, x.take(held))
    k = np.arange(case["q"])
    return both.take(np.where(k % 2 == 0, k + case["q"], k))


def _stack(a, b):
    return synth.Csr(np.concatenate([a.rowptr, b.rowptr[1:] + a.nnz]), np.concatenate([a.col, b.col]),
                     np.concatenate([a.val, b.val]), a.d)


def _inputs(case, seed):
    """The host matrices and thresholds of a case."""
    kind = case["kind"]
    if kind == "batch":
        x, ptr, t = synth.generate_batch(k=case["k"], n_lo=case["n_lo"], n_hi=case["n_hi"],
                                         seed=_seed(seed))
        return {"x": x, "ptr": ptr, "t": t}
    got = {"x": _rows(case, seed, case["n"])}
    if kind == "self":
        got["t"] = case["t"]
    elif kind == "join":
        got["y"] = _rows(case, seed, case["m"], case["n"])
        got["t"] = case["t"]
    elif kind in ("query", "grow"):
        if kind == "grow":
            got["y"] = _rows(case, seed, case["m"], case["n"])
        got["q"] = _queries(case, seed, got["x"])
        got["t"] = _thresholds(seed, case["q"])
    return got


def _empty(slots, kind, device):
    if device:
        return torch.zeros(slots, dtype=getattr(torch, kind), device="cuda")
    return np.zeros(slots, dtype=kind)


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    s["ctx"] = _context(case["precision"])
    kind, device = case["kind"], case["io"] == "device"
    if kind == "query":
        s["index"] = cuapss.Index(s["ctx"], s["x"])
    x = s["x"]
    if device:
        s["x"] = _on_device(x)
    if kind == "tools":
        slots = _tool_slots(case)
        s["desc"] = cuapss.CsrDesc(x.n, x.d, x.nnz, s["x"]["rowptr"].data_ptr(),
                                   s["x"]["col"].data_ptr(), s["x"]["val"].data_ptr(), 1)
        s["out"] = {"ptr": _empty(x.d + 1, "int32", True), "rows": _empty(slots, "int32", True),
                    "vals": _empty(slots, "float32", True), "perm": _empty(x.d, "int32", True),
                    "counts": _empty(x.d, "int32", True)}
    else:
        slots = _pair_slots(case)
        s["out"] = {"i": _empty(slots, "int32", device), "j": _empty(slots, "int32", device),
                    "sim": _empty(slots, "float32", device)}
    return s


# -------------------------------------------------------------------- calls
def _found(s, pairs):
    """The pairs of a call that returns arrays, in the case's buffers."""
    count = len(pairs[0])
    for name, values in zip(("i", "j", "sim"), pairs):
        s["out"][name][:count] = values
    return dict(s["out"], count=count)


def _tools(s):
    lib, ctx, out, found = cuapss.lib(), s["ctx"], s["out"], ctypes.c_int64()
    x = ctypes.byref(s["desc"])
    status = lib.cuapss_build_index(ctx._h, x, s["case"]["p"], out["ptr"].data_ptr(),
                                    out["rows"].data_ptr(), out["vals"].data_ptr(),
                                    out["rows"].numel(), ctypes.byref(found))
    status = status or lib.cuapss_feature_remap(ctx._h, x, out["perm"].data_ptr(),
                                                out["counts"].data_ptr())
    if status:
        raise cuapss.CuapssError(status, "tools")
    return dict(out, count=found.value)


def run(s):
    case, ctx, out = s["case"], s["ctx"], s["out"]
    kind = case["kind"]
    if kind == "self" and case["io"] == "device":
        return dict(out, count=ctx.run_device(s["x"], s["t"], out))
    if kind == "batch":
        return dict(out, count=ctx.batch_run_device(s["x"], s["ptr"], s["t"], out))
    if kind == "tools":
        return _tools(s)
    room = len(out["i"])
    if kind == "self":
        return _found(s, ctx.run(s["x"], s["t"], capacity=room))
    if kind == "join":
        return _found(s, ctx.join(s["x"], s["y"], s["t"], capacity=room))
    if kind == "query":
        return _found(s, s["index"].query(s["q"], s["t"], capacity=room))
    with cuapss.Index(ctx, s["x"]) as index:
        index.append(s["y"])
        return _found(s, index.query(s["q"], s["t"], capacity=room))


# --------------------------------------------------------------------- work
_products = {}


def _shared_features(cfg):
    """Expected shared features of two rows of a distribution: the sum over
    features of the squared share of rows that hold the feature, rows being
    Zipf draws without replacement of the mean length."""
    if cfg not in _products:
        c = synth.CONFIGS[cfg]
        p = np.arange(1, c.d + 1, dtype=np.float64) ** -c.zipf_s
        p /= p.sum()
        lo, hi = 0.0, 1e9
        for _ in range(60):
            mid = 0.5 * (lo + hi)
            if -np.expm1(-mid * p).sum() < c.nnz_mean:
                lo = mid
            else:
                hi = mid
            if hi - lo < 1e-3 * hi:
                break
        _products[cfg] = float(np.square(np.expm1(-lo * p)).sum())
    return _products[cfg]


def work(case):
    """Bytes: the matrices once (8 bytes a non-zero, 8 a row). Operations: the
    multiply-adds of the shared features of every pair of rows asked for."""
    kind = case["kind"]
    cfg = case.get("cfg", "batch_instance")
    nnz = synth.CONFIGS[cfg].nnz_mean

    def csr(n):
        return n * (8.0 * nnz + 8.0)

    if kind == "tools":
        d = synth.CONFIGS[cfg].d
        return {"bytes": 4 * csr(case["n"]) + 12.0 * d, "flops": 0.0}
    shared = 2.0 * _shared_features(cfg)
    if kind == "self":
        n = case["n"]
        return {"bytes": csr(n), "flops": shared * n * (n - 1) / 2}
    if kind == "join":
        return {"bytes": csr(case["n"]) + csr(case["m"]), "flops": shared * case["n"] * case["m"]}
    if kind == "batch":
        rows, square = _batch_sizes(case)
        return {"bytes": csr(rows), "flops": shared * square / 2}
    n = case["n"] + case.get("m", 0)
    grown = 2 * csr(n) if kind == "grow" else 0.0
    return {"bytes": csr(n) + csr(case["q"]) + grown, "flops": shared * n * case["q"]}


# -------------------------------------------------------------------- exact
_EXACT_LIMIT = 1.2e12  # multiply-adds of the dense-by-sparse products below


def _sparse(x, device):
    return torch.sparse_csr_tensor(torch.from_numpy(x.rowptr), torch.from_numpy(x.col.astype(np.int64)),
                                   torch.from_numpy(x.val.astype(np.float64)),
                                   size=(x.n, x.d)).to(device)


def _above(a, b, t, upper, device):
    """(i, j, sim) of the pairs of rows of a and b with similarity >= t (one
    threshold or one per row of a), sorted; upper: only i < j."""
    sb = _sparse(b, device)
    step = max(1, min(1024, int(3e9 // (8 * max(a.d, b.n)))))
    got = []
    for lo in range(0, a.n, step):
        part = a.rows(lo, min(a.n, lo + step))
        dense = torch.zeros((a.d, part.n), dtype=torch.float64, device=device)
        r = np.repeat(np.arange(part.n), np.diff(part.rowptr))
        dense[torch.from_numpy(part.col.astype(np.int64)).to(device),
              torch.from_numpy(r).to(device)] = torch.from_numpy(part.val.astype(np.float64)).to(device)
        s = (sb @ dense).t()
        limit = torch.as_tensor(np.broadcast_to(np.asarray(t, np.float32).astype(np.float64),
                                                (a.n,))[lo:lo + part.n].copy(), device=device)
        hit = s >= limit[:, None]
        if upper:
            ids = torch.arange(b.n, device=device)
            hit &= ids[None, :] > torch.arange(lo, lo + part.n, device=device)[:, None]
        i, j = torch.nonzero(hit, as_tuple=True)
        got.append(torch.stack([(i + lo).double(), j.double(), s[i, j]]).cpu().numpy())
    return np.concatenate(got, axis=1) if got else np.zeros((3, 0))


def _exact_pairs(case, g):
    out = {"i": np.zeros(_pair_slots(case), np.int64), "j": np.zeros(_pair_slots(case), np.int64),
           "sim": np.zeros(_pair_slots(case))}
    for name, values in zip(("i", "j", "sim"), g):
        out[name][:g.shape[1]] = values
    return dict(out, count=g.shape[1])


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    s = _inputs(case, seed)
    x, kind = s["x"], case["kind"]
    if kind == "tools":
        rows = np.repeat(np.arange(x.n), np.diff(x.rowptr))
        keep = x.col >= case["p"]
        order = np.lexsort((rows[keep], x.col[keep]))
        counts = np.bincount(x.col, minlength=x.d)
        ptr = np.zeros(x.d + 1, np.int64)
        np.cumsum(np.where(np.arange(x.d) >= case["p"], counts, 0), out=ptr[1:])
        perm = np.empty(x.d, np.int64)
        perm[np.lexsort((np.arange(x.d), -counts))] = np.arange(x.d)
        index_rows, vals = np.zeros(_tool_slots(case), np.int64), np.zeros(_tool_slots(case))
        index_rows[:len(order)] = rows[keep][order]
        vals[:len(order)] = x.val[keep][order]
        return {"ptr": ptr, "rows": index_rows, "vals": vals, "perm": perm, "counts": counts,
                "count": len(order)}
    if kind == "batch":
        n = np.diff(s["ptr"])
        if float((np.diff(x.rowptr[s["ptr"]]) * n).sum()) > _EXACT_LIMIT:
            return None
        parts = []
        for q in range(len(n)):
            sub = x.rows(int(s["ptr"][q]), int(s["ptr"][q + 1]))
            g = _above(sub, sub, s["t"][q], True, device)
            g[:2] += float(s["ptr"][q])
            parts.append(g)
        return _exact_pairs(case, np.concatenate(parts, axis=1))
    if kind == "self":
        if float(x.nnz) * x.n > _EXACT_LIMIT:
            return None
        return _exact_pairs(case, _above(x, x, s["t"], True, device))
    if kind == "join":
        if float(s["y"].nnz) * x.n > _EXACT_LIMIT:
            return None
        return _exact_pairs(case, _above(x, s["y"], s["t"], False, device))
    index = _stack(x, s["y"]) if kind == "grow" else x
    return _exact_pairs(case, _above(s["q"], index, s["t"], False, device))
