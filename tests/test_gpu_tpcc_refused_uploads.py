"""TPC-C uploads that are refused (more transactions than the slots take, a bad
slot, no tables) are refused before any of the batch's records is read: the
batch claims far more than its one record.  In a child process, which a read
past the record would end."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C
import numpy as np
from ltpg_gb300 import Engine, TpccBatch, abi, lib
e = Engine(device=0, n_slots=1, max_txn=1 << 18)
one = np.zeros(1, dtype=TpccBatch.TXN_DTYPE)
b = abi.TpccBatchC((1 << 32) - 1, 0, 0, one.ctypes.data, None)
few = abi.TpccBatchC(1 << 18, 0, 0, one.ctypes.data, None)
L = lib()
assert L.ltpg_batch_upload_tpcc(e._h, 0, C.byref(few)) == abi.ERR_STATE  # no tables
e.load_tpcc(1, 1)
for call in (lambda s: L.ltpg_batch_upload_tpcc(e._h, s, C.byref(b)),
             lambda s: L.ltpg_run_tpcc_host(e._h, s, C.byref(b), 0, None),
             lambda s: L.ltpg_submit_tpcc_host(e._h, s, C.byref(b), 0, None)):
    assert call(0) == abi.ERR_INVALID
    assert call(7) == abi.ERR_INVALID
e.close()
print("refused")
"""


def test_refused_unread(gpu):
    r = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "refused" in r.stdout, (r.returncode, r.stderr[-2000:])
