"""Folded joins at the edges of what they take: such a call gives what the
probing path gives, whatever the size, the memory at hand and the calls made
before it."""
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
