"""GPU parity of the folded-bound joins against the FP64 oracle, where their
kernels change behaviour: one I block without a partner, a partial last
block, the sampled choice of widths (from 64 row blocks on) with rows long
enough for the streamed and the widest folds, signed values, and inputs whose
bound prunes nothing (the join falls back to the probing path).

Pair sets are exact; similarities are FP64 sums rounded once to FP32, so they
lie within 2^-24 (half an ulp below 1, values up to 1 + 1e-4) of the oracle's:
1.2e-7 allows for both roundings."""
import numpy as np
import pytest

import cuapss
from cuapss import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

SIM_TOL = 1.2e-7


def _check(got, want):
    gi, gj, gs = got
    wi, wj, ws = want
    assert len(gi) == len(wi)
    assert np.array_equal(gi, wi) and np.array_equal(gj, wj)
    if len(gs):
        assert float(np.max(np.abs(gs.astype(np.float64) - ws))) <= SIM_TOL


def _signed(x, seed):
    sign = np.random.default_rng(seed).choice(np.array([-1, 1], np.float32), size=x.nnz)
    return synth.Csr(x.rowptr, x.col, x.val * sign, x.d)


@pytest.fixture(scope="module", params=[cuapss.PREC_MIXED, cuapss.PREC_FP32],
                ids=["mixed", "fp32"])
def ctx(request):
    with cuapss.Context(precision=request.param) as c:
        yield c


@pytest.mark.parametrize("cfg,n,t", [
    ("plain_20k", 129, 0.5), ("plain_20k", 384, 0.6), ("batch_instance", 8064, 0.6),
    ("batch_instance", 8193, 0.5), ("mixed_1m", 8320, 0.5), ("plain_800k", 12_345, 0.3),
    ("serve_5m", 9999, 0.95)])
def test_self_join(ctx, cfg, n, t):
    x = synth.generate(cfg, n=n, seed=n)
    _check(ctx.run(x, t, capacity=1 << 22), oracle.apss(x, t))


@pytest.mark.parametrize("n,m", [(100, 9000), (9000, 100), (5001, 4097), (257, 129)])
def test_cross_join(ctx, n, m):
    x = synth.generate("plain_800k", n=n + m, seed=3)
    a, b = x.rows(0, n), x.rows(n, n + m)
    _check(ctx.join(a, b, 0.5, capacity=1 << 20), oracle.join(a, b, 0.5))


def test_signed_values(ctx):
    x = _signed(synth.generate("plain_20k", n=9000, seed=4), 5)
    _check(ctx.run(x, 0.3, capacity=1 << 20), oracle.apss(x, 0.3))


def test_device_capacity_and_determinism(ctx):
    x = synth.generate("plain_800k", n=9000, seed=6)
    a = ctx.run(x, 0.5, capacity=1)  # EOVERFLOW, then the required room
    b = ctx.run(x, 0.5, capacity=1 << 20)
    assert all(np.array_equal(p, q) for p, q in zip(a, b))


def test_no_pruning_falls_back(ctx):
    # 2,200 near-identical rows: 2.4M candidates, more than a small folded
    # join takes
    rng = np.random.default_rng(7)
    n, m = 2200, 20
    col = np.tile(np.arange(m, dtype=np.int32) * 3, n)
    val = (1.0 + 0.05 * rng.standard_normal((n, m)))
    val = (val / np.linalg.norm(val, axis=1, keepdims=True)).astype(np.float32).ravel()
    x = synth.Csr(np.arange(n + 1, dtype=np.int64) * m, col, val, 3 * m)
    _check(ctx.run(x, 0.95, capacity=1 << 22), oracle.apss(x, 0.95))


@pytest.mark.parametrize("t", [0.5, 0.9])
def test_rows_too_short_for_one_another(ctx, t):
    # 40,000 rows whose lengths run from 1 to 400 with a few dominant values:
    # tiles of short against long rows are skipped, and rows with one large
    # value match much longer ones
    rng = np.random.default_rng(11)
    n, d = 40_000, 3000
    lens = np.minimum(400, np.maximum(1, rng.lognormal(3.0, 1.3, size=n))).astype(np.int64)
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(lens, out=rp[1:])
    col = np.concatenate([np.sort(rng.choice(d, size=k, replace=False)) for k in lens]).astype(np.int32)
    val = rng.uniform(0.5, 1.5, size=int(rp[-1]))
    big = rng.random(n) < 0.3
    val[rp[:-1][big]] *= 30.0
    row = np.repeat(np.arange(n), lens)
    val = (val / np.sqrt(np.bincount(row, weights=val * val))[row]).astype(np.float32)
    x = synth.Csr(rp, col, val, d)
    rows = np.concatenate([rng.choice(n, size=120, replace=False), np.argsort(lens)[-8:],
                           np.argsort(lens)[:8]])
    rows = np.unique(rows).astype(np.int32)
    wi, wj, ws = oracle.rows(x, t, rows)
    assert len(wi) > 100
    gi, gj, gs = ctx.run(x, t, capacity=1 << 24)
    sel = np.isin(gi, rows) | np.isin(gj, rows)
    _check((gi[sel], gj[sel], gs[sel]), (wi, wj, ws))


@pytest.mark.parametrize("signed", [False, True])
def test_index_query_sampled_widths(ctx, signed):
    # 157 x 16 tiles of 128 x 128: the widths come from samples (from 2,048
    # tiles on); thresholds differ by query
    x = synth.generate("plain_800k", n=20_000, seed=8)
    q = synth.generate("plain_800k", n=2000, seed=8, row_offset=19_000)
    if signed:
        x, q = _signed(x, 9), _signed(q, 10)
    t = np.random.default_rng(12).uniform(0.3, 0.9, size=q.n).astype(np.float32)
    with cuapss.Index(ctx, x) as idx:
        gi, gj, gs = idx.query(q, t)
    wi, wj, ws = oracle.join(q, x, float(t.min()))
    keep = ws >= t[wi].astype(np.float64)
    assert keep.sum() >= 1000 * (not signed)  # 1,000 queries are index rows
    _check((gi, gj, gs), (wi[keep], wj[keep], ws[keep]))


def test_batch_signed_and_odd_blocks(ctx):
    # instances of 1 .. 5 blocks: odd last blocks are multiplied alone
    sizes = [1, 128, 129, 257, 384, 385, 640, 2]
    x = _signed(synth.generate("plain_20k", n=sum(sizes), seed=13), 14)
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    t = np.linspace(0.2, 0.6, len(sizes)).astype(np.float32)
    want = [oracle.apss(x.rows(a, b), float(tq)) for a, b, tq in zip(ptr, ptr[1:], t)]
    want = [np.concatenate([w[k] + (a if k < 2 else 0) for a, w in zip(ptr, want)])
            for k in range(3)]
    assert len(want[0]) > 0
    _check(ctx.batch_run(x, ptr, t), want)


@pytest.mark.parametrize("groups", [2047, 2048, 2049])
def test_result_sort_edge(ctx, groups):
    # two pairs a group of near-duplicates: 4,094 / 4,096 / 4,098 results
    # around the 4,096 that one launch ranks
    rng = np.random.default_rng(groups)
    d = 50_000
    rows, cols, vals = [0], [], []
    for g in range(groups):
        base = np.sort(rng.choice(d, size=12, replace=False)).astype(np.int32)
        v = rng.uniform(0.5, 1.5, size=12)
        # the outer two share half of the middle's squares each and no feature
        h = np.sqrt(np.sum(v[:6] ** 2) / np.sum(v[6:] ** 2))
        v[6:] *= h
        for sl in (slice(0, 6), slice(0, 12), slice(6, 12)):
            w = v[sl] / np.linalg.norm(v[sl])
            cols.append(base[sl])
            vals.append(w)
            rows.append(rows[-1] + len(w))
    x = synth.Csr(np.array(rows, np.int64), np.concatenate(cols),
                  np.concatenate(vals).astype(np.float32), d)
    want = oracle.apss(x, 0.7)
    assert len(want[0]) == 2 * groups
    _check(ctx.run(x, 0.7, capacity=1 << 14), want)


@pytest.mark.parametrize("n", [18_815, 18_817, 37_760, 37_761])
def test_threads_per_row(ctx, n):
    # folded rows take 32, 16 or 8 threads each from 148 and 296 blocks on
    x = synth.generate("batch_instance", n=n, seed=n)
    rows = np.unique(np.random.default_rng(n).choice(n, size=150)).astype(np.int32)
    wi, wj, ws = oracle.rows(x, 0.4, rows)
    assert len(wi) > 0
    gi, gj, gs = ctx.run(x, 0.4, capacity=1 << 24)
    sel = np.isin(gi, rows) | np.isin(gj, rows)
    _check((gi[sel], gj[sel], gs[sel]), (wi, wj, ws))
