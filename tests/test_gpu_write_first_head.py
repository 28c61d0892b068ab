"""Write-first registration whose smallest TIDs register in a launch of their
own (filtered batches of 8,192 transactions or more): batch sizes around the
threshold, every count of op vectors, against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, YcsbGenerator, abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [128, 512])
@pytest.mark.parametrize("k", [1, 6, 10, 16, 31])
def test_around_the_threshold(gpu, threads, k):
    n, most = 50_000, 9300
    e = Engine(device=0, n_slots=1, max_txn=most, max_ops_per_txn=k)
    try:
        e.set_launch("ycsb", block_threads=threads, filter=1, late_reads=3)
        for B, mode, scan in [(8191, "fused", 0), (8192, "graph", 0), (most, "fused", 5)]:
            e.load_ycsb(3, n)
            o = oracle.YcsbOracle(3, n)
            for i in range(2):
                b = YcsbGenerator(3, n, B, k, 20, 0.99, 0, scan).batch(i)
                e.upload(0, b)
                e.run_batch(0, mode)
                e.sync()
                flags, bitmap, results, _ = o.run(b)
                assert np.array_equal(e.txn_flags(0, B), flags)
                assert np.array_equal(e.commit_bitmap(0, B), bitmap)
                assert np.array_equal(e.txn_results(0, B), np.where((flags & abi.FLAG_COMMIT) != 0, results, 0))
            assert np.array_equal(e.download_table(abi.TABLE_YCSB), o.rows)
    finally:
        e.close()
