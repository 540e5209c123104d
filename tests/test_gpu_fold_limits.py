"""Folded joins at the edges of what they take: such a call gives what the
probing path gives, whatever the size, the memory at hand and the calls made
before it."""
import os
import subprocess
import sys

import numpy as np
import pytest

import cuapss
from cuapss import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

# reported similarities of either route against the FP64 oracle
SIM_TOL = 1e-6


def _check(got, want):
    assert len(got[0]) == len(want[0])
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert np.max(np.abs(got[2].astype(np.float64) - want[2]), initial=0.0) <= SIM_TOL


@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
def test_batch_past_32_bit_offsets(precision):
    """4,300 single rows of 999,999 entries (no pairs) push the one real
    instance's entries past offset 2^32."""
    import torch
    m, d, k = 999_999, 1_000_000, 4300
    x = synth.generate("plain_20k", n=300, seed=21)
    want = oracle.apss(x, 0.5)
    assert len(want[0]) > 0
    free, _ = torch.cuda.mem_get_info()
    if free < 60e9:
        pytest.skip("needs 60 GB of device memory")
    nnz = m * k + x.nnz
    assert m * k > 2**32
    col = torch.empty(nnz, dtype=torch.int32, device="cuda")
    val = torch.full((nnz,), float(m) ** -0.5, dtype=torch.float32, device="cuda")
    col[:m * k].view(k, m)[:] = torch.arange(m, dtype=torch.int32, device="cuda")
    col[m * k:] = torch.from_numpy(x.col).cuda()
    val[m * k:] = torch.from_numpy(x.val).cuda()
    rowptr = np.concatenate([np.arange(k, dtype=np.int64) * m, m * k + x.rowptr])
    a = {"rowptr": torch.from_numpy(rowptr).cuda(), "col": col, "val": val, "d": d}
    ptr = np.concatenate([np.arange(k + 1), [k + x.n]]).astype(np.int64)
    t = np.full(k + 1, 0.5, np.float32)
    out = {"i": torch.empty(4096, dtype=torch.int32, device="cuda"),
           "j": torch.empty(4096, dtype=torch.int32, device="cuda"),
           "sim": torch.empty(4096, dtype=torch.float32, device="cuda")}
    assert len(want[0]) <= 4096
    with cuapss.Context(precision=precision) as ctx:
        c = ctx.batch_run_device(a, ptr, t, out)
    gi, gj, gs = (out[q][:c].cpu().numpy() for q in ("i", "j", "sim"))
    _check((gi - k, gj - k, gs), want)


def _near_identical(n, groups, m, seed):
    """n rows in groups of one support of m features each, values within 5%."""
    rng = np.random.default_rng(seed)
    g = np.arange(n) % groups
    col = (g[:, None] * m + np.arange(m)).astype(np.int32).ravel()
    val = 1.0 + 0.05 * rng.standard_normal((n, m))
    val = (val / np.linalg.norm(val, axis=1, keepdims=True)).astype(np.float32).ravel()
    return synth.Csr(np.arange(n + 1, dtype=np.int64) * m, col, val, groups * m)


@pytest.mark.parametrize("precision,n,t", [(cuapss.PREC_MIXED, 100_000, 0.4),
                                           (cuapss.PREC_FP32, 60_000, 0.5)], ids=["mixed", "fp32"])
def test_route_does_not_depend_on_earlier_calls(precision, n, t):
    """2,100 near-identical rows are 2.2M candidates, which a small folded join
    does not take, also where an earlier call left room for them."""
    x = _near_identical(2100, 1, 20, 7)
    runs = []
    for warm in (False, True):
        with cuapss.Context(precision=precision) as ctx:
            if warm:
                ctx.run(synth.generate("plain_800k", n=n, seed=1), t, capacity=1 << 22)
                assert ctx.last_stats["rescored"] == ctx.last_stats["candidates"] > 3_000_000
            got = ctx.run(x, 0.95, capacity=1 << 22)
            runs.append((got, ctx.last_stats["candidates"], ctx.last_stats["rescored"]))
    for a, b in zip(*(r[0] for r in runs)):
        assert np.array_equal(a, b)
    assert runs[0][1:] == runs[1][1:]


def _footprint(precision, x, t, **opts):
    """Device bytes a context holds after one self-join, and its result."""
    import torch
    with cuapss.Context(precision=precision, **opts) as ctx:
        got = ctx.run(x, t, capacity=1 << 22)
        held = torch.cuda.mem_get_info()[0]
    return torch.cuda.mem_get_info()[0] - held, got


@pytest.mark.parametrize("precision,t,head", [(cuapss.PREC_FP32, 0.5, 64),
                                              (cuapss.PREC_MIXED, 0.4, 512)], ids=["fp32", "mixed"])
def test_short_of_memory_probes(precision, t, head):
    """With room for the probing path's working memory but not for the folded
    join's candidates, the call probes instead of failing."""
    import torch
    x = synth.generate("plain_20k", n=120_000, seed=1)
    small = synth.generate("plain_20k", n=100, seed=1)
    _footprint(precision, small, 0.5)  # module loading
    probing, want = _footprint(precision, x, t, head_width=head)
    folding, same = _footprint(precision, x, t)
    leave = probing + (160 << 20)
    assert folding > leave + (160 << 20)
    free = torch.cuda.mem_get_info()[0]
    rest = torch.empty(free - leave, dtype=torch.uint8, device="cuda")
    try:
        with cuapss.Context(precision=precision) as ctx:
            got = ctx.run(x, t, capacity=1 << 22)
            probed = ctx.last_stats["rescored"] < ctx.last_stats["candidates"]
            again = ctx.run(x, t, capacity=1 << 22)
    finally:
        del rest
        torch.cuda.empty_cache()
    assert probed
    for k in range(2):
        assert np.array_equal(got[k], want[k]) and np.array_equal(got[k], same[k])
    assert np.max(np.abs(got[2] - same[2])) <= SIM_TOL
    assert all(np.array_equal(a, b) for a, b in zip(got, again))


@pytest.mark.parametrize("precision,head", [(cuapss.PREC_MIXED, 256), (cuapss.PREC_FP32, 64)],
                         ids=["mixed", "fp32"])
def test_batch_feature_limit(precision, head):
    """Batches of more features than 20-bit tail keys and the tuner's narrowest
    head hold are refused, as joins are; the last number of features is served."""
    x = synth.generate("plain_20k", n=400, seed=22)
    ptr = np.array([0, 150, 400], np.int64)
    t = np.array([0.5, 0.6], np.float32)
    top = (1 << 20) - 2 + head
    with cuapss.Context(precision=precision) as ctx:
        for d, ok in ((top, True), (top + 1, False), (top, True)):
            # the features used most keep their ids, the others move to the top
            wide = synth.Csr(x.rowptr, np.where(x.col < 100, x.col, x.col - x.d + d).astype(np.int32),
                             x.val, d)
            if not ok:
                with pytest.raises(cuapss.CuapssError) as e:
                    ctx.batch_run(wide, ptr, t)
                assert e.value.status == cuapss.EINVAL
                # instances of one row have no pairs and need no keys
                one = wide.rows(0, 2)
                assert len(ctx.batch_run(one, np.arange(3, dtype=np.int64), t)[0]) == 0
                continue
            got = ctx.batch_run(wide, ptr, t)
            parts = [oracle.apss(wide.rows(a, b), float(q)) for a, b, q in zip(ptr, ptr[1:], t)]
            want = [np.concatenate([w[q] + (a if q < 2 else 0) for a, w in zip(ptr, parts)])
                    for q in range(3)]
            assert len(want[0]) > 0
            _check(got, want)


def _in_process(program, *args):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.join(root, "apss-cuda_b200")]))
    r = subprocess.run([sys.executable, "-c", program, *args], env=env, cwd=root,
                       capture_output=True, text=True, timeout=240)
    assert r.returncode == 0 and "fine" in r.stdout, r.stdout + r.stderr


_SHORT_INDEX = """
import sys
import numpy as np, torch
import cuapss
from cuapss import synth
from oracle import oracle

MB = 1 << 20
n, m = 300_000, 60_000
x = synth.generate("serve_5m", n=n, seed=3)
q = synth.generate("serve_5m", n=40, seed=3, row_offset=n - 20)
more = synth.generate("serve_5m", n=m, seed=3, row_offset=n)
t = np.full(q.n, 0.6, np.float32)
want = oracle.join(q, x, 0.6)
want2 = oracle.join(q, more, 0.6)
free = lambda: torch.cuda.mem_get_info()[0]

def check(got, want):
    assert len(want[0]) >= 20
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert np.max(np.abs(got[2] - want[2])) <= 1e-6

small = x.rows(0, 3000)
for opts in ({}, {"head_width": 512}):  # module loading
    with cuapss.Context(precision=PRECISION, **opts) as c, cuapss.Index(c, small) as i:
        i.query(q, t)
with cuapss.Context(precision=PRECISION) as c, cuapss.Index(c, x) as i:
    check(i.query(q, t), want)
    i.query(q, 1.5 * t)
    assert c.last_stats["rescored"] == c.last_stats["candidates"] > 0
    full, p = i.info()["device_bytes"], i.info()["head_width"]

if sys.argv[1] == "create":
    # room for the probing layout, not for the folded rows beside it. The
    # device pool's unused memory counts as room: two indexes that stay take
    # what the first one left there
    contexts = [cuapss.Context(precision=PRECISION, head_width=p) for _ in range(2)]
    kept = [cuapss.Index(c, x) for c in contexts]
    f0 = free()
    with cuapss.Context(precision=PRECISION, head_width=p) as c, cuapss.Index(c, x) as i:
        check(i.query(q, t), want)
        used = f0 - free()
        bare = i.info()["device_bytes"]
    assert full > bare + 300 * MB, (full, bare)
    leave = used - (f0 - free()) + 100 * MB
    rest = torch.empty(free() - leave, dtype=torch.uint8, device="cuda")
    with cuapss.Context(precision=PRECISION) as c, cuapss.Index(c, x) as i:
        assert i.info()["device_bytes"] < bare * 1.02
        check(i.query(q, t), want)
else:
    # an append that needs more than is left takes the folded rows' memory
    with cuapss.Context(precision=PRECISION) as c, cuapss.Index(c, x) as i:
        i.query(q, t)
        got = []
        before = i.info()["device_bytes"]
        rest = torch.empty(free() - 30 * MB, dtype=torch.uint8, device="cuda")
        i.append(more)
        info = i.info()
        assert info["rows"] == n + m
        assert info["device_bytes"] < before
        gi, gj, gs = i.query(q, t)
        wi = np.concatenate([want[0], want2[0]])
        wj = np.concatenate([want[1], want2[1] + n])
        ws = np.concatenate([want[2], want2[2]])
        o = np.lexsort((wj, wi))
        check((gi, gj, gs), (wi[o], wj[o], ws[o]))
print("fine")
"""


@pytest.mark.parametrize("what", ["create", "append"])
@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
def test_index_short_of_memory(precision, what):
    """An index whose probing layout fits is built, and grown, without its
    folded rows where they do not fit (in a process of its own, whose device
    memory pool holds nothing yet)."""
    _in_process(f"PRECISION = {precision}\n" + _SHORT_INDEX, what)


_DEFAULT_POOL = """
import ctypes
import numpy as np, torch
import cuapss
from cuapss import synth

torch.cuda.init()
rt = ctypes.CDLL("libcudart.so.12")
pool = ctypes.c_void_p()
assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0

def attr(which):
    v = ctypes.c_uint64()
    assert rt.cudaMemPoolGetAttribute(pool, which, ctypes.byref(v)) == 0
    return v.value

before = attr(4), attr(5)  # release threshold, reserved bytes
x = synth.generate("plain_20k", n=3000, seed=1)
with cuapss.Context() as c:
    for _ in range(2):
        with cuapss.Index(c, x) as i:
            i.append(x.rows(0, 500))
            assert (attr(4), attr(5)) == before
    assert (attr(4), attr(5)) == before
print("fine")
"""


def test_default_pool_is_left_alone():
    """An index takes nothing from the device's default memory pool and changes
    none of its settings: the process's other users share it."""
    _in_process(_DEFAULT_POOL)


def _rows(n, nnz, seed):
    cfg = synth.CONFIGS["plain_800k"].replace(nnz_mean=nnz, nnz_sigma=0.7, nnz_max=8 * nnz, seed=seed)
    return synth.generate(cfg, n=n)


def _probed(ctx):
    return ctx.last_stats["rescored"] < ctx.last_stats["candidates"]


@pytest.mark.parametrize("precision,n,nnz,t,tried", [
    (cuapss.PREC_MIXED, 2000, 800, 0.5, False), (cuapss.PREC_MIXED, 2000, 200, 0.3, False),
    (cuapss.PREC_MIXED, 8000, 75, 0.4, True), (cuapss.PREC_FP32, 2000, 400, 0.6, False),
    (cuapss.PREC_FP32, 8000, 120, 0.5, False), (cuapss.PREC_FP32, 8000, 75, 0.8, True)])
def test_small_joins_that_folding_slows_down(precision, n, nnz, t, tried):
    """Unsampled joins with more candidates than are worth computing probe:
    expected (not tried) or found while the tiles run (given up)."""
    x = _rows(n, nnz, 31)
    rows = np.unique(np.random.default_rng(n).choice(n, size=100)).astype(np.int32)
    wi, wj, ws = oracle.rows(x, t, rows)
    with cuapss.Context(precision=precision) as ctx:
        got = ctx.run(x, t, capacity=1 << 20)
        assert _probed(ctx)
        launches = ctx.last_stats["launches"]
        again = ctx.run(x, t, capacity=1 << 20)
        p = ctx.last_stats["head_width"]
    assert all(np.array_equal(a, b) for a, b in zip(got, again))
    sel = np.isin(got[0], rows) | np.isin(got[1], rows)
    _check(tuple(g[sel] for g in got), (wi, wj, ws))
    with cuapss.Context(precision=precision, head_width=p) as ctx:
        same = ctx.run(x, t, capacity=1 << 20)
        assert (launches > ctx.last_stats["launches"]) == tried
    assert all(np.array_equal(a, b) for a, b in zip(got, same))


@pytest.mark.parametrize("precision,t", [(cuapss.PREC_MIXED, 0.1), (cuapss.PREC_FP32, 0.3)],
                         ids=["mixed", "fp32"])
def test_small_queries_that_folding_slows_down(precision, t):
    """The same for a query batch over an unsampled number of tiles."""
    x = synth.generate("serve_5m", n=30_000, seed=32)
    q = synth.generate("serve_5m", n=100, seed=32, row_offset=29_950)
    sign = np.random.default_rng(33).choice(np.array([-1, 1], np.float32), size=x.nnz + q.nnz)
    x = synth.Csr(x.rowptr, x.col, x.val * sign[:x.nnz], x.d)
    q = synth.Csr(q.rowptr, q.col, q.val * sign[x.nnz:], q.d)
    with cuapss.Context(precision=precision) as ctx, cuapss.Index(ctx, x) as idx:
        got = idx.query(q, np.full(q.n, t, np.float32))
        assert _probed(ctx)
        again = idx.query(q, np.full(q.n, 0.9, np.float32))
    want = oracle.join(q, x, t)
    assert len(want[0]) > 100
    _check(got, want)
    keep = want[2] >= np.float64(np.float32(0.9))
    _check(again, tuple(w[keep] for w in want))


def _batch(sizes, lens, d, seed):
    """Instances of the given rows, of rows of the given mean length each."""
    parts = []
    for k, (n, nnz) in enumerate(zip(sizes, lens)):
        cfg = synth.CONFIGS["batch_instance"].replace(d=d, nnz_mean=nnz, nnz_sigma=0.7,
                                                      nnz_max=8 * nnz, seed=seed + k)
        parts.append(synth.generate(cfg, n=n))
    off = np.cumsum([0] + [p.nnz for p in parts])
    rowptr = np.concatenate([[0]] + [p.rowptr[1:] + o for p, o in zip(parts, off)])
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    x = synth.Csr(rowptr.astype(np.int64), np.concatenate([p.col for p in parts]),
                  np.concatenate([p.val for p in parts]), d)
    return x, ptr, parts


# sampled batches: few and many instances for the sixteen threshold classes,
# instances of fewer rows than a sample takes, equal and different thresholds
@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
@pytest.mark.parametrize("sizes,lens,t", [
    ([4000], [30], [0.6]), ([200, 257], [30, 30], [0.5, 0.9]),
    ([40] * 30, [30] * 30, [0.4] * 30), ([700] * 20, [30] * 20, np.linspace(0.3, 0.9, 20)),
    ([4000] * 20 + [4000] * 10, [10] * 20 + [300] * 10, [0.7] * 30),
    ([4000] * 10 + [4000] * 20, [300] * 10 + [10] * 20, [0.7] * 30)],
    ids=["one", "two", "tiny", "spread", "short-long", "long-short"])
def test_sampled_batches(precision, sizes, lens, t):
    x, ptr, parts = _batch(sizes, lens, 30_000, 41)
    t = np.asarray(t, np.float32)
    want = [oracle.apss(p, float(q)) for p, q in zip(parts, t)]
    want = [np.concatenate([w[k] + (a if k < 2 else 0) for a, w in zip(ptr, want)])
            for k in range(3)]
    assert len(want[0]) > 0
    with cuapss.Context(precision=precision) as ctx:
        _check(ctx.batch_run(x, ptr, t, capacity=1 << 20), want)
        # rows of different instances never meet: a sample across instances
        # promised candidates that a fold of this batch does not have
        if precision == cuapss.PREC_MIXED:
            assert ctx.last_stats["rescored"] == ctx.last_stats["candidates"] > 0


@pytest.mark.parametrize("precision,n,nnz,t", [(cuapss.PREC_FP32, 500, 30, 0.6),
                                               (cuapss.PREC_MIXED, 400, 200, 0.6),
                                               (cuapss.PREC_MIXED, 400, 800, 0.9)])
def test_probing_cost_counts_its_preparation(precision, n, nnz, t):
    """Small batches, whose probing time is launches and preparation, and
    batches of long rows, whose probing tiles are slow, fold."""
    x, ptr, parts = _batch([n] * 12, [nnz] * 12, 30_000, 51)
    t = np.full(12, t, np.float32)
    want = [oracle.apss(p, float(q)) for p, q in zip(parts, t)]
    want = [np.concatenate([w[k] + (a if k < 2 else 0) for a, w in zip(ptr, want)])
            for k in range(3)]
    with cuapss.Context(precision=precision) as ctx:
        _check(ctx.batch_run(x, ptr, t, capacity=1 << 20), want)
        assert ctx.last_stats["rescored"] == ctx.last_stats["candidates"] > 0


# The routes themselves. cuapss_fold_tiles says which one a call took and what
# it multiplied.
@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
def test_fold_tiles_reports_the_route(precision):
    x = synth.generate("plain_800k", n=9000, seed=61)
    widths = {64, 128, 192, 256, 320, 384, 512, 768, 1024, 2048}
    if precision == cuapss.PREC_FP32:
        widths = {16, 32, 48, 64, 96, 128, 192, 256, 512, 1024}
    with cuapss.Context(precision=precision) as ctx:
        assert ctx.fold_tiles() == {}
        t = 0.95
        ctx.run(x.rows(0, 1000), t)  # 8 blocks, one width
        assert list(ctx.fold_tiles().values()) == [36]
        ctx.join(x.rows(0, 130), x.rows(0, 1000), t)
        assert list(ctx.fold_tiles().values()) == [16]
        ctx.run(x, t)  # sampled widths; 71 blocks, none skipped in so small a join
        tiles = ctx.fold_tiles()
        assert set(tiles) <= widths and sum(tiles.values()) == 71 * 72 // 2
        ctx.batch_run(x.rows(0, 1000), np.array([0, 300, 1000], np.int64),
                      np.array([t, t], np.float32))
        tiles = ctx.fold_tiles()
        assert set(tiles) <= widths and sum(tiles.values()) == 6 + 21
        with cuapss.Index(ctx, x.rows(0, 1000)) as idx:
            idx.query(x.rows(0, 130), np.full(130, t, np.float32))
            assert list(ctx.fold_tiles().values()) == [16]
            idx.query(x.rows(0, 130), np.full(130, 0.04, np.float32))
            assert ctx.fold_tiles() == {}
        ctx.run(x.rows(0, 1000), 0.04)
        assert ctx.fold_tiles() == {}
    with cuapss.Context(precision=precision, head_width=64) as ctx:
        ctx.run(x, t)
        assert ctx.fold_tiles() == {}


@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
@pytest.mark.parametrize("opts,low", [({"head_width": 128}, 0.3), ({}, 0.03)],
                         ids=["head_width", "low threshold"])
def test_probing_index_query(precision, opts, low):
    """The probing form of an index query, over appends and merges."""
    x = synth.generate("plain_20k", n=5000, seed=62)
    q = synth.generate("plain_20k", n=129, seed=62, row_offset=4950)
    t = np.random.default_rng(63).uniform(0.4, 0.9, size=q.n).astype(np.float32)
    t[77] = low
    with cuapss.Context(precision=precision, **opts) as ctx:
        with cuapss.Index(ctx, x.rows(0, 3000)) as idx:
            idx.append(x.rows(3000, 3100))
            idx.append(x.rows(3100, 5000))
            got = idx.query(q, t, capacity=1 << 20)
            assert ctx.fold_tiles() == {}
    wi, wj, ws = oracle.join(q, x, low)
    keep = ws >= t[wi].astype(np.float64)
    assert keep.sum() > 100
    _check(got, (wi[keep], wj[keep], ws[keep]))


@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
@pytest.mark.parametrize("opts,low", [({}, 0.04), ({"head_width": 64}, 0.3)],
                         ids=["low threshold", "head_width"])
def test_probing_batch(precision, opts, low):
    """The probing form of a batch, all three size buckets."""
    sizes = [1, 129, 1100, 0, 8300, 500]
    x, ptr, parts = _batch([s for s in sizes if s], [30] * 5, 30_000, 64)
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    t = np.array([0.5, low, 0.6, 0.7, 0.8, 0.4], np.float32)
    want = [oracle.apss(x.rows(a, b), float(q)) if b > a else [np.empty(0)] * 3
            for a, b, q in zip(ptr, ptr[1:], t)]
    want = [np.concatenate([w[k] + (a if k < 2 else 0) for a, w in zip(ptr, want)])
            for k in range(3)]
    with cuapss.Context(precision=precision, **opts) as ctx:
        got = ctx.batch_run(x, ptr, t, capacity=1 << 20)
        assert ctx.fold_tiles() == {} and (ctx.last_bucket_p > 0).all()
    _check(got, want)


@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
def test_probing_join_with_the_modelled_explicit_pairs(precision):
    """The plan of a default self-join, run by the probing path: the explicit
    pairs are built and added."""
    x = synth.generate("mixed_1m", n=40_000, seed=65)
    plan = cuapss.plan_self_join(x, precision)
    assert plan["explicit_pairs"] > 0
    rows = np.unique(np.random.default_rng(66).choice(x.n, size=120)).astype(np.int32)
    with cuapss.Context(precision=precision, rare_max_count=plan["rare_max_count"]) as ctx:
        got = ctx.run(x, 0.6, capacity=1 << 20)
        assert ctx.fold_tiles() == {}
        assert ctx.last_stats["explicit_pairs"] > 0
        assert ctx.last_stats["tail_products"] > 0
    wi, wj, ws = oracle.rows(x, 0.6, rows)
    sel = np.isin(got[0], rows) | np.isin(got[1], rows)
    assert len(wi) > 0
    _check(tuple(g[sel] for g in got), (wi, wj, ws))


def _clusters(n, size, count, within, seed):
    """n rows of 20 entries: `count` runs of `size` rows among the first
    `within` that share their features (every pair of a run is at 0.9 or more),
    the others unrelated."""
    rng = np.random.default_rng(seed)
    d = 200_000
    col = np.sort(rng.integers(0, d // 20, size=(n, 20)) + np.arange(20) * (d // 20), axis=1)
    for k in range(count):
        a = k * (within // count)
        col[a:a + size] = col[a]
    val = 1.0 + 0.1 * rng.standard_normal((n, 20))
    val = (val / np.linalg.norm(val, axis=1, keepdims=True)).astype(np.float32)
    return synth.Csr(np.arange(n + 1, dtype=np.int64) * 20, col.astype(np.int32).ravel(),
                     val.ravel(), d)


# rows of one length keep their order, and a sample takes every 195th of the
# first 125,000 of a join of 200,000 (every 234th of one instance of 60,000):
# runs shorter than that hide their pairs from it
@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
@pytest.mark.parametrize("n,size,count,batch,folds", [
    (200_000, 190, 170, False, True),   # 3.1M candidates: past the list, run again
    (200_000, 190, 640, False, False),  # 11.5M: past four times the list, probes
    (60_000, 230, 260, True, False)],   # 6.8M: the batch's tile kernel gives up
    ids=["retry", "fallback", "batch"])
def test_candidates_hidden_from_the_sample(precision, n, size, count, batch, folds):
    x = _clusters(n, size, count, n if batch else n * 5 // 8, 71)
    rows = np.unique(np.random.default_rng(72).choice(n, size=60)).astype(np.int32)
    wi, wj, ws = oracle.rows(x, 0.9, rows)
    with cuapss.Context(precision=precision) as ctx:
        if batch:
            got = ctx.batch_run(x, np.array([0, n], np.int64), np.array([0.9], np.float32),
                                capacity=1 << 24)
        else:
            got = ctx.run(x, 0.9, capacity=1 << 25)
        assert (ctx.fold_tiles() != {}) == folds
    assert len(got[0]) > 0.9 * count * size * (size - 1) / 2
    sel = np.isin(got[0], rows) | np.isin(got[1], rows)
    _check(tuple(g[sel] for g in got), (wi, wj, ws))


@pytest.mark.parametrize("cfg,n,t", [("plain_800k", 8320, 0.5), ("plain_800k", 8320, 0.6)])
def test_small_sampled_joins_take_wide_rows(cfg, n, t):
    """Just past the unsampled joins, long rows still get the widths that they
    need (mixed precision: at 256 columns half of the time went to candidates)."""
    x = synth.generate(cfg, n=n, seed=71)
    with cuapss.Context(precision=cuapss.PREC_MIXED) as ctx:
        got = ctx.run(x, t, capacity=1 << 16)
        assert max(ctx.fold_tiles()) > 256
    _check(got, oracle.apss(x, t))


# Forms of folded calls whose inputs elsewhere may probe: the route is checked.
def _signed(x, seed):
    sign = np.random.default_rng(seed).choice(np.array([-1, 1], np.float32), size=x.nnz)
    return synth.Csr(x.rowptr, x.col, x.val * sign, x.d)


@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
@pytest.mark.parametrize("cfg,n,t,sign", [
    ("batch_instance", 18_815, 0.7, False), ("batch_instance", 18_817, 0.7, False),
    ("batch_instance", 37_760, 0.8, False), ("batch_instance", 37_761, 0.8, False),
    ("plain_20k", 9000, 0.6, True)])
def test_folded_self_joins(precision, cfg, n, t, sign):
    """Folded rows by 32, 16 and 8 threads each, and signed ones, against the
    probing path (a fixed head width)."""
    x = synth.generate(cfg, n=n, seed=n)
    if sign:
        x = _signed(x, 5)
    with cuapss.Context(precision=precision, head_width=64) as ctx:
        want = ctx.run(x, t, capacity=1 << 16)
        assert ctx.fold_tiles() == {} and len(want[0]) > 0
    with cuapss.Context(precision=precision) as ctx:
        got = ctx.run(x, t, capacity=1 << 16)
        assert ctx.fold_tiles() != {}
    assert all(np.array_equal(a, b) for a, b in zip(got[:2], want[:2]))
    # both are within SIM_TOL of the oracle
    assert np.max(np.abs(got[2] - want[2])) <= 2 * SIM_TOL


@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
@pytest.mark.parametrize("sign", [False, True], ids=["unsigned", "signed"])
def test_folded_sampled_query(precision, sign):
    """Widths from samples, thresholds of their own, both sides signed or not."""
    x = synth.generate("batch_instance", n=20_000, seed=8)
    q = synth.generate("batch_instance", n=2000, seed=8, row_offset=19_000)
    if sign:
        x, q = _signed(x, 9), _signed(q, 10)
    t = np.random.default_rng(12).uniform(0.5, 0.9, size=q.n).astype(np.float32)
    with cuapss.Context(precision=precision) as ctx, cuapss.Index(ctx, x) as idx:
        got = idx.query(q, t)
        assert len(ctx.fold_tiles()) > 1
    wi, wj, ws = oracle.join(q, x, 0.5)
    keep = ws >= t[wi].astype(np.float64)
    assert keep.sum() > 100
    _check(got, (wi[keep], wj[keep], ws[keep]))


@pytest.mark.parametrize("precision", [cuapss.PREC_MIXED, cuapss.PREC_FP32], ids=["mixed", "fp32"])
def test_folded_unsampled_cross_join(precision):
    x = synth.generate("batch_instance", n=9098, seed=3)
    a, b = x.rows(0, 5001), x.rows(5001, 9098)
    with cuapss.Context(precision=precision) as ctx:
        got = ctx.join(a, b, 0.6, capacity=1 << 16)
        assert sum(ctx.fold_tiles().values()) == 40 * 33
    _check(got, oracle.join(a, b, 0.6))


@pytest.mark.parametrize("cfg,t", [("plain_800k", 0.5), ("batch_instance", 0.7)])
def test_small_batch_widths(cfg, t):
    """Small mixed batches sample wide rows only where the mean length calls for
    them: rows of 75 entries and of 30."""
    x = synth.generate(cfg, n=3000, seed=72)
    ptr = np.array([0, 300, 1500, 3000], np.int64)
    parts = [oracle.apss(x.rows(a, b), t) for a, b in zip(ptr, ptr[1:])]
    want = [np.concatenate([p[k] + (a if k < 2 else 0) for a, p in zip(ptr, parts)])
            for k in range(3)]
    with cuapss.Context(precision=cuapss.PREC_MIXED) as ctx:
        got = ctx.batch_run(x, ptr, np.full(3, t, np.float32), capacity=1 << 16)
        if cfg == "batch_instance":
            assert 0 < max(ctx.fold_tiles()) <= 256
    _check(got, want)
