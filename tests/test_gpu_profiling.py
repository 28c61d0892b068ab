"""Batches with per-kernel events on, in every mode: events between kernels
whose launches may overlap, in the stream and in a captured graph.  Outcomes as
the oracle's, and a time for every kernel that ran on its own."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, TpccGenerator, YcsbGenerator

pytestmark = pytest.mark.gpu
# which of execute, check, reads, write-back have a time
SPLIT = {"plain": (1, 1, 0, 1), "fused": (1, 1, 0, 0), "graph": (1, 1, 0, 0), "persistent": (1, 0, 0, 0)}


def _run(e, o, batches, mode, split):
    for i, b in enumerate(batches):
        e.upload(i, b)
    for _ in range(2):  # graphs: captured, then replayed
        if mode == "graph":
            e.run_batches(0, len(batches), mode)
        else:
            for i in range(len(batches)):
                e.run_batch(i, mode)
        e.sync()
        for i, b in enumerate(batches):
            flags, bitmap, results, _ = o.run(b)
            assert np.array_equal(e.txn_flags(i, b.n_txn), flags)
            assert np.array_equal(e.commit_bitmap(i, b.n_txn), bitmap)
            assert np.array_equal(e.txn_results(i, b.n_txn), results)
            times = np.array(e.kernel_times(i))
            assert (times >= 0).all() and (times[np.array(split, dtype=bool)] > 1e-3).all(), times
            assert times.sum() < 50.0


@pytest.mark.parametrize("mode", SPLIT)
@pytest.mark.parametrize("B", [500, 20_000])
def test_ycsb(gpu, B, mode):
    n = 20_000
    e = Engine(device=0, n_slots=2, max_txn=B, max_ops_per_txn=10)
    try:
        e.load_ycsb(3, n)
        e.set_profiling(True)
        g = YcsbGenerator(3, n, B, 10, 50, 0.9)
        _run(e, oracle.YcsbOracle(3, n), [g.batch(0), g.batch(1)], mode, SPLIT[mode])
    finally:
        e.close()


@pytest.mark.parametrize("mode", SPLIT)
@pytest.mark.parametrize("W,B", [(2, 1000), (16, 1 << 17)])
def test_tpcc(gpu, W, B, mode):
    e = Engine(device=0, n_slots=2, max_txn=B, max_lines=15 * B)
    try:
        e.load_tpcc(3, W)
        e.set_profiling(True)
        g = TpccGenerator(3, W, B)
        _run(e, oracle.TpccOracle(3, W), [g.next(), g.next()], mode, SPLIT[mode])
    finally:
        e.close()
