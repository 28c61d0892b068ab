"""Batches just past the size up to which a block registers a key once (8,192
lanes of the cooperative execute kernel a multiprocessor): the kernels chosen by
the launch settings dedupe, filter and late_reads, with operation counts that
leave lanes of a warp's step idle, against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, YcsbGenerator, abi, key_bucket

pytestmark = pytest.mark.gpu


def _past_the_threshold(k):
    """The least number of transactions that the block table does not take."""
    import torch
    lanes = 8192 * torch.cuda.get_device_properties(0).multi_processor_count
    return lanes // 32 * (32 // k) + 1


@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("k", [3, 10, 16, 32])
def test_settings(gpu, threads, k):
    n, B = 100_000, _past_the_threshold(k)
    b = YcsbGenerator(5, n, B, k, 30, 0.9).batch(0)
    o = oracle.YcsbOracle(5, n)
    flags, bitmap, results, _ = o.run(b)
    com = (flags & abi.FLAG_COMMIT) != 0
    e = Engine(device=0, n_slots=1, max_txn=B, max_ops_per_txn=k)
    try:
        for late in (0, 1, 2):
            for filt in (0, 1):
                for dedupe in (0, 1):
                    e.load_ycsb(5, n)
                    e.set_launch("ycsb", block_threads=threads, ops_per_thread=1, blocks_per_sm=0, stage_ways=4,
                                 filter=filt, dedupe=dedupe, late_reads=late)
                    e.upload(0, b)
                    e.run_batch(0, "fused" if dedupe else "graph")
                    e.sync()
                    case = (late, filt, dedupe)
                    assert np.array_equal(e.txn_flags(0, B), flags), case
                    assert np.array_equal(e.commit_bitmap(0, B), bitmap), case
                    assert np.array_equal(e.txn_results(0, B), np.where(com, results, 0) if late else results), case
                    assert np.array_equal(e.download_table(abi.TABLE_YCSB), o.rows), case
    finally:
        e.close()


@pytest.mark.parametrize("k", [3, 10])
def test_scans(gpu, k):
    """Range scans in a second pass over the warp's steps."""
    n, B = 20_000, _past_the_threshold(k)
    b = YcsbGenerator(6, n, B, k, 10, 0.6, 0, 5).batch(0)
    o = oracle.YcsbOracle(6, n)
    want = o.run(b)
    e = Engine(device=0, n_slots=1, max_txn=B, max_ops_per_txn=k)
    try:
        for dedupe in (0, 1):
            e.load_ycsb(6, n)
            e.set_launch("ycsb", ops_per_thread=1, filter=1, dedupe=dedupe, late_reads=0)
            e.upload(0, b)
            e.run_batch(0, "fused")
            e.sync()
            assert np.array_equal(e.txn_flags(0, B), want[0])
            assert np.array_equal(e.txn_results(0, B), want[2])
            assert np.array_equal(e.download_table(abi.TABLE_YCSB), o.rows)
    finally:
        e.close()


@pytest.mark.parametrize("staged", [False, True])
@pytest.mark.parametrize("threads", [128, 512])
@pytest.mark.parametrize("k,scan", [(1, 0), (3, 2), (10, 0), (16, 5), (32, 0)])
def test_tiles(gpu, k, scan, threads, staged):
    """Eight ops per thread: block tiles, past the threshold or with staging."""
    n = 50_000
    B = 5001 if staged else _past_the_threshold(k)
    b = YcsbGenerator(7, n, B, k, 30, 0.99, 0, scan).batch(0)
    o = oracle.YcsbOracle(7, n)
    want = o.run(b)
    e = Engine(device=0, n_slots=1, max_txn=B, max_ops_per_txn=k)
    try:
        for filt in (0, 1):
            e.load_ycsb(7, n)
            e.set_launch("ycsb", block_threads=threads, ops_per_thread=8, filter=filt, dedupe=0, late_reads=0)
            if staged:
                e.stage_set(key_bucket(np.arange(100)))
            e.upload(0, b)
            e.run_batch(0, "graph" if filt else "fused")
            e.sync()
            assert np.array_equal(e.txn_flags(0, B), want[0])
            assert np.array_equal(e.commit_bitmap(0, B), want[1])
            assert np.array_equal(e.txn_results(0, B), want[2])
            assert np.array_equal(e.download_table(abi.TABLE_YCSB), o.rows)
            assert (e.stats(0)["staged_ops"] > 0) == staged
    finally:
        e.close()
