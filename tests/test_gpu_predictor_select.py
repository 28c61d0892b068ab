"""The predictor's choice of the staged buckets: exactly the top scores, ties in
bucket order, wherever the last one falls among the blocks that choose.  With
weights that make a bucket's score its last count, the staged share of the next
batch tells the set."""
import numpy as np
import pytest

from oracle import predictor_ref as R
from ltpg_gb300 import Engine, YcsbBatch, abi

pytestmark = pytest.mark.gpu
N, K = 400_000, 4


def _reads(keys):
    """A batch of point reads, K a transaction."""
    ops = np.resize(np.asarray(keys, dtype=np.uint32), (len(keys) + K - 1) // K * K)
    return YcsbBatch(ops, np.zeros(len(ops) // K + 1, np.uint32), np.zeros(0, np.uint64), len(ops) // K, K)


@pytest.mark.parametrize("ways", [1, 4])
@pytest.mark.parametrize("counts", [(300, 500, 700), (200, 50, 0), (0, 0, 3000), (1024, 256, 1)])
def test_top_scores_and_ties(gpu, ways, counts):
    rng = np.random.default_rng(sum(counts) + ways)
    bucket_of = ((np.arange(N, dtype=np.uint64) * 0x9E3779B1) & 0xFFFFFFFF) >> 16
    first = np.full(abi.STAGE_BUCKETS, -1, dtype=np.int64)
    first[bucket_of[::-1]] = np.arange(N)[::-1]
    buckets = rng.permutation(np.nonzero(first[1:] >= 0)[0] + 1)  # bucket 0 is staged to begin with
    last = np.zeros(abi.STAGE_BUCKETS, dtype=np.int64)
    at = 0
    for c, n in zip((3, 2, 1), counts):
        last[buckets[at:at + n]] = c
        at += n
    filler, at = first[buckets[at]], at + 1
    # one transaction in 16 is counted: the others read one key
    counted = np.repeat(first[np.nonzero(last)[0]], last[last > 0])
    counted = np.append(counted, np.full(-len(counted) % K, filler)).reshape(-1, K)
    txns = np.full((16 * len(counted), K), filler)
    txns[::16] = counted
    last[bucket_of[filler]] += -int(last.sum()) % K
    p = np.zeros(R.N_PARAM, dtype=np.float32)
    p[R.W1 + R.F - 1] = p[R.W2] = p[R.W3] = 1.0  # unit 0 of both layers passes the last count on
    e = Engine(device=0, n_slots=1, max_txn=1 << 16, max_ops_per_txn=K)
    try:
        e.load_ycsb(3, N)
        e.set_launch("ycsb", stage_ways=ways, ops_per_thread=1)
        e.predictor(enable=True, train=False, stage=True, seed=5)
        e.predictor_params(p)
        order = np.lexsort((np.arange(abi.STAGE_BUCKETS), -last))  # the larger count, then the smaller bucket
        staged = np.zeros(abi.STAGE_BUCKETS, dtype=bool)
        staged[order[:abi.STAGE_ENTRIES // ways]] = True
        probe = np.unique(np.concatenate([buckets[:at], buckets[at:at + 4000], np.nonzero(staged & (first >= 0))[0]]))
        probe = probe[: len(probe) // K * K]
        for b in (_reads(txns.ravel()), _reads(first[probe])):
            e.upload(0, b)
            e.run_batch(0, "fused")
            e.sync()
        assert e.stats(0)["staged_ops"] == int(staged[probe].sum())
    finally:
        e.close()
