"""Large TPC-C batches of a mix whose order reads are rare, so that the engine's
look at 64 records finds one in some batches only: the slot keeps its kernels
once one was seen (a launch of three kernels where inserted rows are claimed,
two otherwise), instead of capturing its graph again for every other batch, and
a batch of another size is looked at anew."""
import numpy as np
import pytest

import oracle
from ltpg_gb300 import Engine, TpccBatch, TpccGenerator, abi

pytestmark = pytest.mark.gpu


def test_kernels_stay(gpu):
    W, B = 16, (1 << 17) + 1
    e = Engine(device=0, n_slots=1, max_txn=B, max_lines=15 * B)
    try:
        e.load_tpcc(71, W)
        o = oracle.TpccOracle(71, W)
        g = TpccGenerator(71, W, B)
        launches = []
        for sampled, n in [(False, B), (True, B), (False, B), (True, B), (False, B - 1), (False, B)]:
            b = g.next()
            t = b.txns[:n].copy()
            at = 0 if sampled else 1  # the first record is one of those looked at
            no = t[np.nonzero((t["kind_info"] & 0xFF) == abi.TPCC_NEWORDER)[0][at]]
            d = (int(no["kind_info"]) >> 16) & 0xFF
            t[at] = (abi.TPCC_ORDERSTATUS | (d << 16) | (d << 24), no["w"], no["w"], no["c_id"], no["a"], no["c"], 0, 0)
            b = TpccBatch(t, b.lines, b.txn_base)
            before = e.counters()[1]
            e.upload(0, b)
            e.run_batch(0, "graph")
            e.sync()
            launches.append(e.counters()[1] - before)
            flags, _, results, _ = o.run(b)
            assert np.array_equal(e.txn_flags(0, n), flags)
            assert np.array_equal(e.txn_results(0, n), results)
        assert launches == [3, 2, 2, 2, 3, 3]
    finally:
        e.close()
