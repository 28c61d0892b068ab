"""TPC-C batches made on the GPU: byte-identical to the host generator where the
ranking's chunks, the block's order by kind and the scan of a warehouse's
Deliveries end unevenly (batch sizes around them, one warehouse and many,
Deliveries far more than the orders they deliver)."""
import numpy as np
import pytest

from ltpg_gb300 import Engine, TpccGenerator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 31, 127, 129, 257, 4097, 9000])
@pytest.mark.parametrize("W,kw", [
    (1, dict(neworder_pct=20, orderstatus_pct=20, delivery_pct=50, stocklevel_pct=5)),
    (2, dict(neworder_pct=90, orderstatus_pct=2, delivery_pct=4, stocklevel_pct=2, by_name_pct=60)),
    (9, dict(neworder_pct=45, orderstatus_pct=4, delivery_pct=4, stocklevel_pct=4, by_name_pct=60)),
])
def test_uneven_ends(gpu, B, W, kw):
    e = Engine(device=0, n_slots=1, max_txn=B, max_lines=15 * B)
    try:
        e.load_tpcc(7, W)
        host, dev = (TpccGenerator(7, W, B, **kw) for _ in range(2))
        for _ in range(3):
            e.generate(0, dev)
            got, want = e.download_batch(0), host.next()
            assert got.txn_base == want.txn_base
            assert np.array_equal(got.txns, want.txns)
            assert np.array_equal(got.lines, want.lines)
    finally:
        e.close()
