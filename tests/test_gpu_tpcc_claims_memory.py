"""Device memory of the claims (bitmaps and STOCK writers, 0.95 MB a warehouse):
a load takes none, nor does a batch that does not claim its rows; the first
batch that does takes it once, and a batch that is in a slot when other tables
are loaded claims on."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, TpccGenerator, abi

pytestmark = pytest.mark.gpu
MIX = dict(neworder_pct=45, orderstatus_pct=4, delivery_pct=4, stocklevel_pct=4)


def test_taken_when_used(gpu):
    import torch
    W, B = 128, (1 << 17) + 1
    claims = 950_000 * W

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    e = Engine(device=0, n_slots=1, max_txn=B, max_lines=15 * B)
    try:
        e.load_tpcc(3, 1)  # the first load brings the kernels onto the device too
        e.load_tpcc(3, 1)
        before = free()
        e.load_tpcc(3, W)
        tables = sum(r * c * 8 for r, c in (e.table_shape(t) for t in range(abi.TPCC_TABLES)))
        rows = sum(e.table_shape(t)[0] for t in range(abi.TPCC_TABLES))
        names = W * (30_000 * 8 + 10 * 1025 * 2)
        assert before - free() < tables + 16 * rows + names + claims // 2
        o = oracle.TpccOracle(3, W)
        e.upload(0, TpccGenerator(5, W, B, **MIX).next())
        at = free()
        e.upload(0, TpccGenerator(6, W, B, **MIX).next())
        assert abs(at - free()) < claims // 2
        e.upload(0, TpccGenerator(5, W, B - 1).next())
        after = free()
        assert at - after > claims // 2
        g = TpccGenerator(7, W, B - 1)
        for _ in range(2):
            b = g.next()
            e.upload(0, b)
            e.run_batch(0, "fused")
            e.sync()
            flags = o.run(b)[0]
            assert np.array_equal(e.txn_flags(0, B - 1), flags)
        assert after == free()
        e.load_tpcc(4, W)  # the slot's batch again, on other tables
        o = oracle.TpccOracle(4, W)
        before = e.counters()[1]
        e.run_batch(0, "fused")
        e.sync()
        assert e.counters()[1] - before == 3  # execute, the claimed rows that met others, check
        assert np.array_equal(e.txn_flags(0, B - 1), o.run(b)[0])
        for t in (abi.T_STOCK, abi.T_ORDERLINE, abi.T_CUSTOMER):
            assert np.array_equal(e.download_table(t), o.tables[t]), t
    finally:
        e.close()
