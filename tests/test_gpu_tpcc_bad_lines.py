"""Order lines out of range (item past the ITEM table, supply warehouse past the
last one): reported as LTPG_ERR_BOUNDS, their NewOrders do not commit and write
nothing, and the batch's other transactions are as without them.  The bad
orders come last, so that no other transaction can meet them."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, LtpgError, TpccBatch, TpccGenerator, abi

pytestmark = pytest.mark.gpu
BAD = [(100_000, 0, 1), (131_071, 0, 5), (7, None, 1), (99_999, None, 10)]  # None: supply warehouse W


def _with_bad_orders(b, W):
    """b and, behind it, NewOrders of three lines with one bad line each."""
    good = b.txns[np.nonzero((b.txns["kind_info"] & 0xFF) == abi.TPCC_NEWORDER)[0][0]]
    txns, lines = [], []
    for i, (item, w, qty) in enumerate(BAD * 3):
        t = good.copy()
        t["kind_info"] = abi.TPCC_NEWORDER | (3 << 8) | ((i % 10) << 16)
        t["w"], t["c_id"], t["a"], t["b"], t["c"] = i % W, 2000 + i, 29_900 + i, 29_900 + i, 440_000 + 3 * i
        t["line_off"] = len(b.lines) + len(lines)
        own = [(50_000 + i, i % W, 3), (60_000 + i, i % W, 4)]
        own.insert(i // len(BAD), (item, W if w is None else w, qty))
        txns.append(t)
        lines += own
    return TpccBatch(np.concatenate([b.txns, np.array(txns, dtype=b.txns.dtype)]),
                     np.concatenate([b.lines, np.array(lines, dtype=b.lines.dtype)]), b.txn_base)


@pytest.mark.parametrize("mode", ["plain", "fused", "persistent", "graph"])
@pytest.mark.parametrize("W,B,kw", [(2, 3000, dict(orderstatus_pct=4, delivery_pct=4, stocklevel_pct=4)),
                                    (16, 1 << 17, {})])  # the larger claims its rows
def test_bad_lines(gpu, W, B, kw, mode):
    n = B + 3 * len(BAD)
    e = Engine(device=0, n_slots=1, max_txn=n, max_lines=15 * n)
    try:
        e.load_tpcc(61, W)
        o = oracle.TpccOracle(61, W)
        g = TpccGenerator(61, W, B, **kw)
        for packed in (False, True):
            b = g.next()
            bad = _with_bad_orders(b, W)
            e.upload(0, bad.with_packed_lines() if packed else bad)
            e.run_batch(0, mode)
            with pytest.raises(LtpgError) as ei:
                e.sync()
            assert ei.value.code == abi.ERR_BOUNDS
            flags, _, results, commits = o.run(b)
            got = e.txn_flags(0, n)
            assert np.array_equal(got[:B], flags)
            assert not (got[B:] & abi.FLAG_COMMIT).any()
            assert np.array_equal(e.txn_results(0, n)[:B], results)
            assert e.stats(0)["commits"] == commits
        for t in range(abi.TPCC_TABLES):
            assert np.array_equal(e.download_table(t), o.tables[t]), t
    finally:
        e.close()
