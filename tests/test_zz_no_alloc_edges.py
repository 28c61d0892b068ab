"""The no-allocation entry point at the edges of its last kernel, a block to a
bitmap word: batches around 32 transactions, one operation and the most, scans,
and transactions that write a field several times.  Against the oracle, bit for
bit."""
import ctypes as C

import numpy as np
import pytest

import ltpg_gb300
import oracle
from ltpg_gb300 import YcsbBatch, abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 31, 32, 33, 1000])
@pytest.mark.parametrize("k", [1, 7, 32])
def test_edges(gpu, B, k):
    import torch
    n, seed = 3000, 9
    rng = np.random.RandomState(1000 * k + B)
    ops, values = [], []
    for _ in range(B):
        pool = rng.randint(0, n, max(1, k // 3))  # few keys, two fields: updates repeat
        txn = [(int(rng.choice(pool)), True, int(rng.randint(2))) if rng.randint(100) < 40
               else (int(rng.randint(n)), False, int(rng.randint(16)) if rng.randint(100) < 20 else 0) for _ in range(k)]
        ops.append(txn)
        values.append([int(rng.randint(1 << 30)) for op in txn if op[1]])
    b = YcsbBatch.from_ops(ops, values)
    o = oracle.YcsbOracle(seed, n)
    dev = torch.device("cuda", 0)
    to = lambda a, t: torch.from_numpy(np.ascontiguousarray(a).view(t)).to(dev)
    rows = to(o.rows.copy(), np.int64)
    d_ops, d_off, d_vals = to(b.ops, np.int32), to(b.val_off, np.int32), to(np.append(b.vals, np.uint64(0)), np.int64)
    flags = torch.empty(B, dtype=torch.uint8, device=dev)
    bitmap = torch.empty((B + 31) // 32, dtype=torch.int32, device=dev)
    results = torch.empty(B, dtype=torch.int64, device=dev)
    for _ in range(2):
        torch.cuda.synchronize()
        args = [C.c_void_p(x.data_ptr()) for x in (rows, d_ops, d_off, d_vals, flags, bitmap, results)]
        rc = ltpg_gb300.lib().ltpg_ycsb_batch_noalloc(0, args[0], n, *args[1:4], B, k, *args[4:], None)
        assert rc == abi.OK
        want = o.run(b)
        for got, w in zip((flags, bitmap, results), want):
            got = got.cpu().numpy()
            assert np.array_equal(got.view(w.dtype), w)
        assert np.array_equal(rows.cpu().numpy().view(np.uint64).reshape(o.rows.shape), o.rows)
