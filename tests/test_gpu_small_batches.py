"""The tuned YCSB kernels on batches of a few waves: hot keys registered once
per block, updates stored by the thread that holds them, tiles that shrink with
the batch.  Flags, bitmap, results and rows bit-exact against the oracle, at
every padded operation count, with repeated fields inside a transaction."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, YcsbBatch, YcsbGenerator, abi

pytestmark = pytest.mark.gpu


def _same(e, o, b, mode):
    e.upload(0, b)
    e.run_batch(0, mode)
    e.sync()
    flags, bitmap, results, _ = o.run(b)
    got = e.txn_flags(0, b.n_txn)
    assert np.array_equal(got, flags), np.nonzero(got != flags)[0][:10]
    assert np.array_equal(e.commit_bitmap(0, b.n_txn), bitmap)
    assert np.array_equal(e.txn_results(0, b.n_txn), results)
    assert np.array_equal(e.download_table(abi.TABLE_YCSB), o.rows)


@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("filt", [0, 1])
@pytest.mark.parametrize("k", [1, 7, 10, 17, 32])
def test_waves(gpu, threads, filt, k):
    """One transaction, one step, a few, and more than the ~1.2 M lanes up to
    which a block registers a key once."""
    n, lanes = 20_000, max(4, 1 << (k - 1).bit_length())
    most = (8192 * 152 + 8192) // lanes
    e = Engine(device=0, n_slots=1, max_txn=most, max_ops_per_txn=k)
    try:
        e.set_launch("ycsb", block_threads=threads, filter=filt, ops_per_thread=1, dedupe=0, late_reads=0)
        for B, mode, theta in [(1, "fused", 0.0), (4001, "graph", 0.99), (20_001, "persistent", 0.99), (most, "fused", 0.9)]:
            e.load_ycsb(3, n)
            o = oracle.YcsbOracle(3, n)
            _same(e, o, YcsbGenerator(3, n, min(B, most), k, 30, theta).batch(0), mode)
    finally:
        e.close()


@pytest.mark.parametrize("mode", ["fused", "persistent"])
def test_repeated_fields(gpu, mode):
    """A committed transaction that writes a field several times, in one
    16-byte vector and across vectors, leaves the last value."""
    n, k = 5000, 14
    rng = np.random.default_rng(9)
    n_txn, stride = 300, (k + 3) // 4 * 4
    ops = np.full((n_txn, stride), 0xFFFFFFFF, dtype=np.uint32)
    for t in range(n_txn):  # four keys of its own per transaction, two fields: most updates repeat
        key, fld, upd = 16 * t + rng.integers(0, 4, k), rng.integers(0, 2, k), rng.random(k) < 0.8
        ops[t, :k] = np.where(upd, 0x80000000 | (fld << 27), 0) | key
    count = ((ops != 0xFFFFFFFF) & (ops >> 31 != 0)).sum(1)
    off = np.concatenate([[0], np.cumsum(count)]).astype(np.uint32)
    vals = rng.integers(0, 1 << 63, int(off[-1]), dtype=np.uint64)
    b = YcsbBatch(ops.ravel(), off, vals, n_txn, k)
    e = Engine(device=0, n_slots=1, max_txn=n_txn, max_ops_per_txn=k)
    try:
        e.load_ycsb(3, n)
        _same(e, oracle.YcsbOracle(3, n), b, mode)
        assert (e.txn_flags(0, n_txn) & abi.FLAG_COMMIT).all()
    finally:
        e.close()
