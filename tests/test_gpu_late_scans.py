"""Late reads of range scans, four scans of a warp at a time: any number of
scans among a warp's reads, every length, starts at every place in a 128-byte
line, ends at the table's end.  Results bit-exact against the oracle."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, YcsbBatch, abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("k", [1, 3, 8, 13, 32])
def test_scans_of_a_warp(gpu, threads, k):
    n, B = 5003, 600
    rng = np.random.RandomState(100 * k + threads)
    ops, values = [], []
    for t in range(B):
        share = rng.choice([0, 10, 50, 100])  # scans among the reads, in percent
        keys = np.where(rng.rand(k) < 0.05, n - 1 - rng.randint(0, 16, k), rng.randint(0, n, k))
        upd = rng.randint(0, 40 * k) == 0
        txn = [(int(q), False, int(rng.randint(1, 16)) if rng.randint(100) < share else 0) for q in keys]
        if upd:
            txn[0] = (txn[0][0], True, int(rng.randint(10)))
        ops.append(txn)
        values.append([int(rng.randint(1 << 30))] if upd else [])
    batch = YcsbBatch.from_ops(ops, values)
    e = Engine(device=0, n_slots=1, max_txn=B, max_ops_per_txn=k)
    try:
        e.load_ycsb(7, n)
        o = oracle.YcsbOracle(7, n)
        for late, mode in [(3, "fused"), (2, "graph"), (1, "fused"), (3, "persistent")]:
            e.set_launch("ycsb", late_reads=late, block_threads=threads)
            e.upload(0, batch)
            e.run_batch(0, mode)
            e.sync()
            flags, _, results, commits = o.run(batch)
            assert commits > B // 2
            assert np.array_equal(e.txn_flags(0, B), flags)
            assert np.array_equal(e.txn_results(0, B), np.where((flags & abi.FLAG_COMMIT) != 0, results, 0))
        assert np.array_equal(e.download_table(abi.TABLE_YCSB), o.rows)
    finally:
        e.close()
