"""YCSB batches made on the GPU by one thread per transaction or by refilled
slots: byte-identical to the host generator on both sides of the rule that
chooses (batch sizes, uniform keys in rank order, transactions that redraw most
of their keys), and where the permutation is not worth a table."""
import numpy as np
import pytest

from ltpg_gb300 import Engine, YcsbGenerator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n,theta,rot,sizes", [
    (1, 500, 0.9, 0, (4096, 4097)), (1, 3_000_000, 0.99, 8, (60, 4096, 4097)), (2, 70, 0.0, 0, (4096, 4097)),
    (2, 70, 0.6, 8, (4096,)), (10, 4000, 0.0, 0, (8192, 8193)), (32, 64, 0.0, 0, (20, 8193)),
    (32, 120, 0.9, 8, (8192, 8193)), (16, 60, 0.999, 0, (8193,)), (5, 9_000_000, 0.0, 4, (30, 20_000))])
def test_both_sides(gpu, k, n, theta, rot, sizes):
    e = Engine(device=0, n_slots=1, max_txn=max(sizes), max_ops_per_txn=k)
    try:
        e.load_ycsb(1, n)
        for B in sizes:
            g = YcsbGenerator(11, n, B, k, 40, theta, rot, 3 if k == 2 else 0)
            for bid in (0, 9):
                e.generate(0, g, bid)
                got, want = e.download_batch(0), g.batch(bid)
                assert np.array_equal(got.ops, want.ops)
                assert np.array_equal(got.val_off, want.val_off)
                assert np.array_equal(got.vals, want.vals)
    finally:
        e.close()
