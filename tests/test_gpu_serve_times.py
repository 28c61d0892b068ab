"""Submit times of the requests of one large submit: each counts from when the
call reached it, so their mean wait holds half of the call's own time, not all
of it."""
import ctypes as C
import time

import numpy as np
import pytest

import ltpg_gb300 as L
from ltpg_gb300 import Engine, abi

pytestmark = pytest.mark.gpu


def test_wait_of_a_large_submit(gpu):
    n, k = 300_000, 16
    c = Engine(device=0, n_slots=2, max_txn=n)
    y = Engine(device=0, n_slots=2, max_txn=n, max_ops_per_txn=k)
    try:
        c.load_tpcc(1, 1)
        y.load_ycsb(1, 1000)
        s = L.Server(c, y, max_batch=n, deadline_ms=1e6, slots=1, ycsb_ops=k)
        ops = np.arange(k, dtype=np.uint32)  # reads
        reqs = (abi.RequestC * n)(*([abi.RequestC(abi.WORKLOAD_YCSB, k, None, None, ops.ctypes.data, None)] * n))
        first = C.c_uint64()
        t0 = time.perf_counter()
        assert L.lib().ltpg_serve_submit(s._h, reqs, n - 1, C.byref(first)) == 0
        t1 = time.perf_counter()
        s.flush()
        t2 = time.perf_counter()
        wait = s.close()["wait_ms"] * 1e-3  # to the batch's closing, at the start of the flush
        assert wait < 0.75 * (t1 - t0) + min(t2 - t1, 0.1 * (t1 - t0))
        assert wait > 0.25 * (t1 - t0)
    finally:
        c.close()
        y.close()
