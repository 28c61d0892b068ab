"""YCSB batches made on the GPU by tiles: byte-identical to the host generator
at the edges of a tile (batch sizes around it, operation counts from 1 to 32,
with and without padding words), where keys repeat often (skew, small tables),
and where the permutation is too wide to tabulate."""
import numpy as np
import pytest

from ltpg_gb300 import Engine, YcsbGenerator

pytestmark = pytest.mark.gpu


def _same(e, g, bid):
    e.generate(0, g, bid)
    got, want = e.download_batch(0), g.batch(bid)
    assert np.array_equal(got.ops, want.ops)
    assert np.array_equal(got.val_off, want.val_off)
    assert np.array_equal(got.vals, want.vals)


@pytest.mark.parametrize("k", [1, 2, 5, 13, 16, 31, 32])
@pytest.mark.parametrize("n,theta,rot", [(40, 0.0, 3), (300, 0.9, 0), (5000, 0.99, 2), (100_000, 0.9999, 1)])
def test_tiles(gpu, k, n, theta, rot):
    e = Engine(device=0, n_slots=1, max_txn=9000, max_ops_per_txn=k)
    try:
        e.load_ycsb(1, n)
        for B in (1, 15, 17, 511, 513, 4097, 9000):
            _same(e, YcsbGenerator(9, n, B, k, 37, theta, rot), B % 5)
    finally:
        e.close()


def test_wide_permutation(gpu):
    n = (1 << 24) + 5
    e = Engine(device=0, n_slots=1, max_txn=6000, max_ops_per_txn=16)
    try:
        e.load_ycsb(1, n)
        _same(e, YcsbGenerator(3, n, 6000, 16, 5, 0.99, 8), 9)
    finally:
        e.close()
