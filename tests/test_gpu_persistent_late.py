"""Persistent batches with late reads 1 and 2, whose grid is bounded by the
check's tiles and, at 128 threads, by the multiprocessors: batches with fewer
tiles than blocks, at the bounds and past them, against the oracle."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, YcsbGenerator, abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("k,B,scan", [(1, 40, 0), (32, 1217, 0), (32, 4864, 3), (3, 97_281, 0), (10, 6081, 5), (16, 19_457, 0)])
def test_grids(gpu, k, B, scan, threads):
    n = 40_000
    b = YcsbGenerator(9, n, B, k, 50, 0.9, 0, scan).batch(0)
    o = oracle.YcsbOracle(9, n)
    flags, bitmap, results, _ = o.run(b)
    com = (flags & abi.FLAG_COMMIT) != 0
    e = Engine(device=0, n_slots=1, max_txn=B, max_ops_per_txn=k)
    try:
        for late in (1, 2):
            for filt, cap in ((0, 0), (1, 0), (1, 1)):
                e.load_ycsb(9, n)
                e.set_launch("ycsb", block_threads=threads, ops_per_thread=1, blocks_per_sm=cap, stage_ways=4,
                             filter=filt, dedupe=0, late_reads=late)
                e.upload(0, b)
                e.run_batch(0, "persistent")
                e.sync()
                assert np.array_equal(e.txn_flags(0, B), flags)
                assert np.array_equal(e.commit_bitmap(0, B), bitmap)
                assert np.array_equal(e.txn_results(0, B), np.where(com, results, 0))
                assert np.array_equal(e.download_table(abi.TABLE_YCSB), o.rows)
    finally:
        e.close()
