"""The tuned TPC-C kernels at the edges of their dispatch: batch sizes around
which a block's tile grows, batches that claim their inserted rows in bitmaps
(large ones, many warehouses) with rows that several transactions touch, and
last names on both sides of the name directory's end.  Flags, bitmap, results
and tables bit-exact against the oracle."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, TpccBatch, TpccGenerator, abi

pytestmark = pytest.mark.gpu
MIX = dict(neworder_pct=45, orderstatus_pct=4, delivery_pct=4, stocklevel_pct=4)


def _same(e, o, b, slot, mode):
    e.upload(slot, b)
    e.run_batch(slot, mode)
    e.sync()
    flags, bitmap, results, _ = o.run(b)
    got = e.txn_flags(slot, b.n_txn)
    assert np.array_equal(got, flags), np.nonzero(got != flags)[0][:10]
    assert np.array_equal(e.commit_bitmap(slot, b.n_txn), bitmap)
    assert np.array_equal(e.txn_results(slot, b.n_txn), results)
    return flags


def _tables(e, o):
    for t in range(abi.TPCC_TABLES):
        assert np.array_equal(e.download_table(t), o.tables[t]), f"table {t}"


@pytest.mark.parametrize("threads", [128, 256, 512])
def test_tile_sizes(gpu, threads):
    """152 SMs x 1,536 threads: a block's tile grows at 29,184, 58,368 and 116,736 transactions."""
    W, edge = 4, 29184
    e = Engine(device=0, n_slots=1, max_txn=4 * edge + 1, max_lines=15 * (4 * edge + 1))
    try:
        e.set_launch("tpcc", block_threads=threads)
        e.load_tpcc(41, W)
        o = oracle.TpccOracle(41, W)
        for B, mode in [(1, "fused"), (edge, "graph"), (edge + 1, "persistent"), (2 * edge + 1, "fused"),
                        (4 * edge + 1, "graph")]:
            _same(e, o, TpccGenerator(41, W, B, **MIX).next(), 0, mode)
        _tables(e, o)
    finally:
        e.close()


@pytest.mark.parametrize("strict", [False, True])
def test_claimed_rows_that_collide(gpu, strict):
    """All kinds on a few shared ORDER, NEW-ORDER, HISTORY and ORDER-LINE rows
    (runs over word boundaries and the wrap at 450,000); the 64 records that
    the engine samples are NewOrders, so the batch claims its rows.  NEW-ORDER
    inserts meet no other op unless strict: the outcome is defined by the
    protocol only then."""
    W, B = 16, (1 << 17) + 77
    rng = np.random.default_rng(5)
    e = Engine(device=0, n_slots=2, max_txn=B, max_lines=15 * B, strict_insert=strict)
    try:
        e.load_tpcc(43, W)
        o = oracle.TpccOracle(43, W, strict=strict)
        g = TpccGenerator(43, W, B, **MIX)
        for i, mode in enumerate(["fused", "graph", "graph"]):
            b = g.next()
            t = b.txns.copy()
            kind = t["kind_info"] & 0xFF
            if not strict:
                t = np.where(kind == abi.TPCC_DELIVERY, t[np.nonzero(kind == abi.TPCC_PAYMENT)[0][0]], t)
                kind = t["kind_info"] & 0xFF
            near = rng.random(B) < 0.3
            c = rng.integers(0, 120, B)
            c = np.where(rng.random(B) < 0.5, 449_999 - c, c)
            has_order = kind != abi.TPCC_STOCKLEVEL
            t["a"] = np.where(near & has_order, rng.integers(0, 90, B), t["a"])
            insert = (kind == abi.TPCC_NEWORDER) | (kind == abi.TPCC_DELIVERY)
            t["b"] = np.where(near & insert & strict, rng.integers(0, 90, B), t["b"])
            t["b"] = np.where(near & (kind == abi.TPCC_ORDERSTATUS), c, t["b"])
            t["c"] = np.where(near & insert, c, t["c"])
            sampled = B * np.arange(64) // 64
            t[sampled] = t[np.nonzero(kind == abi.TPCC_NEWORDER)[0][:64]]
            if i == 2:  # nothing read or delivered, rows as generated
                t = np.where((kind == abi.TPCC_NEWORDER) | (kind == abi.TPCC_PAYMENT), b.txns, t[sampled[0]])
            flags = _same(e, o, TpccBatch(t, b.lines, b.txn_base), i % 2, mode)
            com = (flags & abi.FLAG_COMMIT) != 0
            assert 0 < com.sum() < B
        _tables(e, o)
    finally:
        e.close()


@pytest.mark.parametrize("first", [0, 1019, 1 << 20])
def test_names_around_the_directory(gpu, first):
    W, B = 2, 3000
    e = Engine(device=0, n_slots=1, max_txn=B, max_lines=15 * B)
    try:
        e.load_tpcc(47, W)
        o = oracle.TpccOracle(47, W)
        cust = o.tables[abi.T_CUSTOMER].reshape(-1, abi.TPCC_COLS[abi.T_CUSTOMER])
        cust[:, 13] = first + np.arange(len(cust)) % 10
        e.upload_table(abi.T_CUSTOMER, o.tables[abi.T_CUSTOMER])
        t = TpccGenerator(47, W, B, neworder_pct=0, by_name_pct=100).next().txns.copy()
        names = first + np.arange(B) % 12 - (1 if first else 0)  # names on both sides that no customer has
        t["c_id"] = (names << 8) | (t["c_id"] & 0xFF)
        flags = _same(e, o, TpccBatch(t, np.zeros(0, TpccBatch.LINE_DTYPE), 0), 0, "fused")
        missing = (flags & abi.FLAG_NOT_FOUND) != 0
        assert missing.any() and not missing.all()
        _tables(e, o)
    finally:
        e.close()
