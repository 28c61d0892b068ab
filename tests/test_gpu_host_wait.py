"""ltpg_host_wait on a slot whose batch was waited for already, or that never
had one, does not wait for the work of other slots behind it on the stream; an
error that a batch left is still reported, once."""
import pytest

from ltpg_gb300 import Engine, LtpgError, YcsbBatch, YcsbGenerator, abi, pinned_copy, pinned_empty

pytestmark = pytest.mark.gpu


def test_no_wait_without_a_batch(gpu):
    import torch
    n, B = 5000, 1000
    e = Engine(device=0, n_slots=3, max_txn=B)
    try:
        e.load_ycsb(1, n)
        bits = pinned_empty((B + 31) // 32)
        b = pinned_copy(YcsbGenerator(1, n, B, 10).batch(0))
        e.submit_host(0, b, "fused", bits)
        e.host_wait(0)
        stream = torch.cuda.ExternalStream(e.stream())
        later = torch.cuda.Event()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1_000_000_000)  # about half a second
            later.record()
        for slot in (0, 2):
            e.host_wait(slot)
        assert not later.query()
        e.sync()
        # a batch with a key past the table, submitted and then waited for twice
        bad = pinned_copy(YcsbBatch.from_ops([[(n, False, 0)]], [[]]))
        e.submit_host(1, bad, "fused", bits)
        with pytest.raises(LtpgError) as ei:
            e.host_wait(1)
        assert ei.value.code == abi.ERR_BOUNDS
        e.host_wait(1)
        # and one whose error another slot's wait finds
        e.upload(1, YcsbBatch.from_ops([[(n, False, 0)]], [[]]))
        e.run_batch(1, "fused")
        torch.cuda.synchronize()
        with pytest.raises(LtpgError) as ei:
            e.host_wait(2)
        assert ei.value.code == abi.ERR_BOUNDS
        e.sync()
    finally:
        e.close()
