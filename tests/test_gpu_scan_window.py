"""Write-first registration of range scans: the keys after a scan's first are
looked up in one or two words of the writer bitmap, so scans that start, end or
sit around a 32-key word boundary or the table's end are held to the oracle."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, YcsbBatch, abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fused", "persistent"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 100])
def test_scans_around_bitmap_words(gpu, n, mode):
    rng = np.random.RandomState(n)
    seed, B = 5, 700
    edges = [0, 1, 15, 16, 17, 30, 31, 32, 33, 47, 48, 62, 63, 64, 65, n - 16, n - 2, n - 1]
    edges = [e for e in edges if 0 <= e < n]
    ops, values = [], []
    for _ in range(B):
        txn, vals = [], []
        for _ in range(rng.randint(1, 6)):
            if rng.randint(100) < 15:
                txn.append((int(rng.randint(n)), True, int(rng.randint(10))))
                vals.append(int(rng.randint(1 << 30)))
            else:
                txn.append((int(rng.choice(edges)), False, int(rng.randint(16))))  # a read's field is its span
        ops.append(txn)
        values.append(vals)
    batch = YcsbBatch.from_ops(ops, values)
    e = Engine(device=0, n_slots=1, max_txn=B, max_ops_per_txn=batch.ops_per_txn)
    try:
        e.load_ycsb(seed, n)
        e.set_launch("ycsb", late_reads=3)
        o = oracle.YcsbOracle(seed, n)
        for _ in range(2):
            e.upload(0, batch)
            e.run_batch(0, mode)
            e.sync()
            flags, bitmap, results, _ = o.run(batch)
            com = (flags & abi.FLAG_COMMIT) != 0
            assert np.array_equal(e.txn_flags(0, B), flags)
            assert np.array_equal(e.commit_bitmap(0, B), bitmap)
            assert np.array_equal(e.txn_results(0, B), np.where(com, results, 0))
        assert np.array_equal(e.download_table(abi.TABLE_YCSB), o.rows)
    finally:
        e.close()
