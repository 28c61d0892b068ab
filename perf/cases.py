"""The engine's workloads as timed cases: what a program that embeds it has it do.

A case is a dict of plain values.  `prepare` makes what the program holds before
the call (tables in HBM, batches, a launch shape, a server), `run` is one pass
through the public entry points (ltpg_gb300, the C ABI of include/ltpg.h) and
returns what that program gets back: commit bitmaps, flags, results, and for the
calls that own them the table image or the predictor's weights.

The kinds of work:
  ycsb       YCSB batches resident in HBM, run back to back; the commit bitmaps
             stay on the GPU, the last batch's flags and results go to the host
  tpcc       the same for TPC-C batches
  host       one synchronous host-buffer call: copy, run, bitmap back
  pipeline   host batches through the pipelined calls (copies overlap kernels)
  generate   batches made on the GPU and run, pipelined
  serve      mixed caller-owned requests through the batching server
  caller     a YCSB batch on buffers the caller owns (no allocation)
  predictor  YCSB batches with the contention predictor training and staging
"""
import ctypes as C
import math

import numpy as np
import torch

import ltpg_gb300 as L
from ltpg_gb300 import abi, tune

MIX = dict(neworder_pct=45, orderstatus_pct=4, delivery_pct=4, stocklevel_pct=4, by_name_pct=60)


def listed():
    return [
        # A front end that sends its few hundred waiting transactions as soon as the
        # last call is back: copies, launches and synchronisation are all there is.
        dict(name="ycsb_host_tiny", kind="host", work="ycsb", n_records=100_000, n_txn=257, ops=5, update_pct=50,
             theta=0.9, scan_len=0, mode="fused", shape=""),
        # A host runtime that owns the GPU's memory runs a small batch on its own
        # buffers; 7 operations, so that no transaction fills its 16-byte vectors.
        dict(name="caller_small", kind="caller", n_records=100_000, n_txn=4099, ops=7, update_pct=30, theta=0.8),
        # One 2 ms window of the serving loop at a million requests a second: 70 %
        # TPC-C, 30 % YCSB, packed, run on two engines and polled.
        dict(name="serve_mixed", kind="serve", warehouses=64, n_records=1_000_000, n_req=2000, tpcc_pct=70,
             theta=0.9, mode="fused", shape="ycsb_small|theta=0.6", tpcc_shape="tpcc"),
        # The reference's shipped YCSB shape (10,000 x 9 reads + 1 update), in the
        # persistent mode that suits a batch of one wave.
        dict(name="ycsb_10k", kind="ycsb", n_records=1_000_000, n_txn=10_000, ops=10, update_pct=10, theta=0.99,
             scan_len=0, rotate_every=0, batches=8, mode="persistent", shape="ycsb_ref_10k|theta=0.99"),
        # Small batches, half updates, moderate skew, replayed from a graph.
        dict(name="ycsb_small", kind="ycsb", n_records=1_000_000, n_txn=65_536, ops=10, update_pct=50, theta=0.6,
             scan_len=0, rotate_every=0, batches=8, mode="graph", shape="ycsb_small|theta=0.6"),
        # The headline: a million transactions of 16 operations, 95/5, high skew, a
        # rotating hot set.
        dict(name="ycsb_hc", kind="ycsb", n_records=10_000_000, n_txn=1 << 20, ops=16, update_pct=5, theta=0.99,
             scan_len=0, rotate_every=8, batches=4, mode="graph", shape="ycsb_hc|theta=0.99"),
        # No skew, an odd batch and an operation count that leaves padding words,
        # sent from pinned host memory through the pipelined calls.
        dict(name="ycsb_uniform_pipe", kind="pipeline", work="ycsb", n_records=10_000_000, n_txn=700_001, ops=13,
             update_pct=10, theta=0.0, scan_len=0, batches=3, mode="fused", shape="ycsb_hc|theta=0.0"),
        # Range scans: every read covers 10 keys.
        dict(name="ycsb_scan", kind="ycsb", n_records=10_000_000, n_txn=1 << 18, ops=10, update_pct=5, theta=0.99,
             scan_len=10, rotate_every=8, batches=4, mode="graph", shape="ycsb_scan|theta=0.99"),
        # TPC-C NewOrder + Payment at 64 warehouses, a million transactions.
        dict(name="tpcc_50", kind="tpcc", warehouses=64, n_txn=1 << 20, mix=False, batches=4, mode="graph",
             shape="tpcc"),
        # The five-transaction mix with customers by last name, a full serving batch,
        # made on the GPU and run (the load driver has no host batches to copy).
        dict(name="tpcc_mix_generate", kind="generate", work="tpcc", warehouses=64, n_txn=1 << 18, mix=True,
             batches=4, mode="fused", shape="tpcc"),
        # The headline batches made on the GPU and run.
        dict(name="ycsb_generate", kind="generate", work="ycsb", n_records=10_000_000, n_txn=1 << 20, ops=16,
             update_pct=5, theta=0.99, scan_len=0, rotate_every=8, batches=2, mode="graph",
             shape="ycsb_hc|theta=0.99"),
        # Learned staging on the high-contention stream: every batch trains the
        # predictor and stages its buckets on the warp-aggregated path.
        dict(name="ycsb_predictor", kind="predictor", n_records=10_000_000, n_txn=1 << 18, ops=16, update_pct=5,
             theta=0.99, rotate_every=8, batches=4, mode="fused"),
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["ycsb", "ycsb", "tpcc", "tpcc", "host", "pipeline", "generate", "serve", "caller",
                       "predictor"])
    theta = rng.choice([0.0, 0.6, 0.8, 0.99, round(rng.uniform(0.0, 0.99), 3)])
    tuned = rng.choice(["", "ycsb_hc|theta=0.99", "ycsb_small|theta=0.6"])
    if kind == "ycsb":
        mode = rng.choice(["graph", "graph", "fused", "persistent", "plain"])
        scan = rng.choice([0, 0, 0, rng.randint(2, 16)])
        most = (1 << 16) if scan or mode == "plain" else (1 << 19)
        return dict(kind=kind, n_records=_log(rng, 100_000, 10_000_000), n_txn=_log(rng, 1000, most),
                    ops=rng.randint(2, 16), update_pct=rng.choice([5, 10, 50, rng.randint(0, 100)]), theta=theta,
                    scan_len=scan, rotate_every=rng.choice([0, 8]), batches=rng.randint(1, 4), mode=mode, shape=tuned)
    if kind == "tpcc":
        mode = rng.choice(["graph", "graph", "fused", "persistent", "plain"])
        return dict(kind=kind, warehouses=_log(rng, 1, 64), n_txn=_log(rng, 1000, 1 << 18 if mode == "plain" else 1 << 20),
                    mix=rng.choice([False, True]), batches=rng.randint(1, 2), mode=mode, shape=rng.choice(["", "tpcc"]))
    if kind == "host":
        work = rng.choice(["ycsb", "tpcc"])
        if work == "ycsb":
            return dict(kind=kind, work=work, n_records=_log(rng, 100_000, 1_000_000), n_txn=_log(rng, 100, 100_000),
                        ops=rng.randint(2, 16), update_pct=rng.choice([5, 50, rng.randint(0, 100)]), theta=theta,
                        scan_len=0, mode=rng.choice(["fused", "plain"]), shape=rng.choice(["", "ycsb_small|theta=0.6"]))
        return dict(kind=kind, work=work, warehouses=_log(rng, 1, 16), n_txn=_log(rng, 100, 100_000),
                    mix=rng.choice([False, True]), mode=rng.choice(["fused", "plain"]), shape="tpcc")
    if kind == "pipeline":
        if rng.choice([False, True]):
            return dict(kind=kind, work="ycsb", n_records=_log(rng, 1_000_000, 10_000_000),
                        n_txn=_log(rng, 50_000, 600_000), ops=rng.randint(4, 16), update_pct=rng.choice([5, 10, 50]),
                        theta=theta, scan_len=0, batches=3, mode="fused", shape=tuned)
        return dict(kind=kind, work="tpcc", warehouses=_log(rng, 8, 64), n_txn=_log(rng, 50_000, 600_000),
                    mix=rng.choice([False, True]), batches=3, mode="fused", shape="tpcc")
    if kind == "generate":
        if rng.choice([False, True]):
            return dict(kind=kind, work="ycsb", n_records=_log(rng, 100_000, 10_000_000),
                        n_txn=_log(rng, 10_000, 1 << 19), ops=rng.randint(2, 16), update_pct=rng.choice([5, 50]),
                        theta=theta, scan_len=0, rotate_every=rng.choice([0, 8]), batches=2, mode="fused", shape=tuned)
        return dict(kind=kind, work="tpcc", warehouses=_log(rng, 2, 64), n_txn=_log(rng, 10_000, 1 << 19),
                    mix=rng.choice([False, True]), batches=2, mode="fused", shape="tpcc")
    if kind == "serve":
        return dict(kind=kind, warehouses=_log(rng, 2, 64), n_records=_log(rng, 100_000, 1_000_000),
                    n_req=_log(rng, 300, 10_000), tpcc_pct=rng.choice([30, 70]), theta=theta, mode="fused",
                    shape="ycsb_small|theta=0.6", tpcc_shape="tpcc")
    if kind == "caller":
        return dict(kind=kind, n_records=_log(rng, 20_000, 1_000_000), n_txn=_log(rng, 1000, 50_000),
                    ops=rng.randint(2, 16), update_pct=rng.choice([5, 50, rng.randint(0, 100)]), theta=theta)
    return dict(kind="predictor", n_records=_log(rng, 1_000_000, 10_000_000), n_txn=_log(rng, 65_536, 1 << 18),
                ops=rng.choice([10, 16]), update_pct=rng.choice([5, 50]), theta=rng.choice([0.9, 0.99]),
                rotate_every=8, batches=rng.randint(2, 4), mode="fused")


# ---- what a program holds ------------------------------------------------------


def _pinned(n, dtype):
    """n elements of pinned host memory as an array."""
    nbytes = max(1, int(n)) * np.dtype(dtype).itemsize
    return torch.empty(nbytes, dtype=torch.uint8, pin_memory=True).numpy().view(dtype)[:int(n)]


def _pinned_copy(a):
    out = _pinned(a.size, a.dtype)
    out[:] = a
    return out


def _ptr(a):
    return C.c_void_p(a.ctypes.data)


def _ok(code, what):
    if code != abi.OK:
        raise RuntimeError("%s: status %d" % (what, code))


class _DeviceWords:
    """Device memory the engine owns, in the form torch takes without a copy;
    a tensor made of it keeps this object, and so the engine, alive."""

    def __init__(self, engine, ptr, n):
        self.engine = engine
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<i4", data=(ptr, False), version=3)


def _device_bitmap(engine, slot, n_txn):
    p = C.c_void_p()
    _ok(L.lib().ltpg_commit_bitmap_device(engine._h, slot, C.byref(p)), "commit bitmap")
    return torch.as_tensor(_DeviceWords(engine, p.value, (n_txn + 31) // 32), device="cuda")


def _shape(engine, workload, key):
    """The launch shape shipped for a tuned workload; "" keeps the engine's own."""
    cfg = tune.load_cached(key) if key else None
    if cfg:
        engine.set_launch(workload, **{k: v for k, v in cfg.items() if k in dict(abi.LaunchC._fields_)})


def _ycsb_gen(case, seed):
    return L.YcsbGenerator(seed, case["n_records"], case["n_txn"], case["ops"], case["update_pct"], case["theta"],
                           case.get("rotate_every", 0), case.get("scan_len", 0))


def _tpcc_gen(case, seed, n_txn=None):
    return L.TpccGenerator(seed, case["warehouses"], n_txn or case["n_txn"], **(MIX if case.get("mix") else {}))


class _Outputs:
    """Pinned host buffers for one slot's flags and results."""

    def __init__(self, engine, n_txn):
        self.e, self.n = engine, n_txn
        self.flags, self.results = _pinned(n_txn, np.uint8), _pinned(n_txn, np.int64)
        self.fp, self.rp = _ptr(self.flags), _ptr(self.results)

    def fetch(self, slot):
        _ok(L.lib().ltpg_txn_flags(self.e._h, slot, self.fp, self.n), "flags")
        _ok(L.lib().ltpg_txn_results(self.e._h, slot, self.rp, self.n), "results")
        return dict(flags=self.flags, results=self.results)


class _Engine:
    """An engine with its tables, a launch shape and a generator."""

    def __init__(self, case, seed, work, slots):
        n = case["n_txn"]
        if work == "ycsb":
            self.e = L.Engine(device=0, n_slots=slots, max_txn=n, max_ops_per_txn=case["ops"])
            self.e.load_ycsb(seed, case["n_records"])
            self.g = _ycsb_gen(case, seed)
        else:
            self.e = L.Engine(device=0, n_slots=slots, max_txn=n, max_ops_per_txn=4, max_lines=15 * n)
            self.e.load_tpcc(seed, case["warehouses"])
            self.g = _tpcc_gen(case, seed)
        _shape(self.e, work, case.get("shape", ""))

    def host_batch(self, i):
        """Batch i as a program with pinned host buffers holds it."""
        self.e.generate(0, self.g, i)
        b = self.e.download_batch(0)
        if isinstance(b, L.YcsbBatch):
            return L.YcsbBatch(_pinned_copy(b.ops), _pinned_copy(b.val_off), _pinned_copy(b.vals), b.n_txn,
                               b.ops_per_txn)
        return L.TpccBatch(_pinned_copy(b.txns.view(np.uint32)).view(L.TpccBatch.TXN_DTYPE),
                           _pinned_copy(b.lines.view(np.uint32)).view(L.TpccBatch.LINE_DTYPE), b.txn_base)


class _Resident(_Engine):
    def __init__(self, case, seed, work):
        super().__init__(case, seed, work, case["batches"])
        self.n, self.mode, n = case["batches"], case["mode"], case["n_txn"]
        for i in range(self.n):
            self.e.generate(i, self.g, i)
        self.e.sync()
        self.bitmaps = [_device_bitmap(self.e, i, n) for i in range(self.n)]
        self.out = _Outputs(self.e, n)

    def run(self):
        self.e.run_batches(0, self.n, self.mode)
        return dict(self.out.fetch(self.n - 1), bitmaps=self.bitmaps)


class _Predicted(_Resident):
    def __init__(self, case, seed):
        super().__init__(case, seed, "ycsb")
        self.e.set_launch("ycsb", ops_per_thread=1, filter=1, dedupe=1, stage_ways=1, blocks_per_sm=0)
        self.e.predictor(enable=True, train=True, stage=True, seed=7)

    def run(self):
        out = super().run()
        out["params"] = self.e.predictor_params()
        return out


class _Host(_Engine):
    def __init__(self, case, seed):
        super().__init__(case, seed, case["work"], 1)
        self.mode, n = case["mode"], case["n_txn"]
        self.batch = self.host_batch(0)
        self.bitmap = _pinned((n + 31) // 32, np.uint32)

    def run(self):
        return self.e.run_host(0, self.batch, self.mode, self.bitmap).view(np.int32)


class _Pipeline(_Engine):
    def __init__(self, case, seed):
        super().__init__(case, seed, case["work"], case["batches"])
        self.n, self.mode, n = case["batches"], case["mode"], case["n_txn"]
        self.batches = [self.host_batch(i) for i in range(self.n)]
        self.bitmaps = [_pinned((n + 31) // 32, np.uint32) for _ in range(self.n)]
        self.out = _Outputs(self.e, n)

    def run(self):
        for i in range(self.n):
            self.e.submit_host(i, self.batches[i], self.mode, self.bitmaps[i])
        for i in range(self.n):
            self.e.host_wait(i)
        return dict(self.out.fetch(self.n - 1), bitmaps=[b.view(np.int32) for b in self.bitmaps])


class _Generated(_Engine):
    def __init__(self, case, seed):
        super().__init__(case, seed, case["work"], case["batches"])
        self.n, self.mode, n = case["batches"], case["mode"], case["n_txn"]
        self.bitmaps = [_pinned((n + 31) // 32, np.uint32) for _ in range(self.n)]
        self.out = _Outputs(self.e, n)

    def run(self):
        for i in range(self.n):
            self.e.submit_generated(i, self.g, self.mode, self.bitmaps[i], batch_id=i)
        for i in range(self.n):
            self.e.host_wait(i)
        return dict(self.out.fetch(self.n - 1), bitmaps=[b.view(np.int32) for b in self.bitmaps])


class _Caller:
    def __init__(self, case, seed):
        n, b, k, dev = case["n_records"], case["n_txn"], case["ops"], torch.device("cuda", 0)
        e = L.Engine(device=0, n_slots=1, max_txn=b, max_ops_per_txn=k)
        e.load_ycsb(seed, n)
        e.generate(0, _ycsb_gen(case, seed), 0)
        batch = e.download_batch(0)
        self.rows = torch.from_numpy(e.download_table(abi.TABLE_YCSB).view(np.int64)).to(dev)
        e.close()
        self.ops = torch.from_numpy(batch.ops.view(np.int32)).to(dev)
        self.val_off = torch.from_numpy(batch.val_off.view(np.int32)).to(dev)
        self.vals = torch.from_numpy(np.append(batch.vals, np.uint64(0)).view(np.int64)).to(dev)
        self.flags = torch.empty(b, dtype=torch.uint8, device=dev)
        self.bitmap = torch.empty((b + 31) // 32, dtype=torch.int32, device=dev)
        self.results = torch.empty(b, dtype=torch.int64, device=dev)
        self.args = [0, C.c_void_p(self.rows.data_ptr()), n, C.c_void_p(self.ops.data_ptr()),
                     C.c_void_p(self.val_off.data_ptr()), C.c_void_p(self.vals.data_ptr()), b, k,
                     C.c_void_p(self.flags.data_ptr()), C.c_void_p(self.bitmap.data_ptr()),
                     C.c_void_p(self.results.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)]

    def run(self):
        _ok(L.lib().ltpg_ycsb_batch_noalloc(*self.args), "batch on the caller's buffers")
        return dict(rows=self.rows, flags=self.flags, bitmap=self.bitmap, results=self.results)


class _Serve:
    OPS = 10

    def __init__(self, case, seed):
        n, most = case["n_req"], 16_384
        self.n = n
        self.c = L.Engine(device=0, n_slots=2, max_txn=most, max_ops_per_txn=4, max_lines=15 * most)
        self.y = L.Engine(device=0, n_slots=2, max_txn=most, max_ops_per_txn=self.OPS)
        self.c.load_tpcc(seed, case["warehouses"])
        self.y.load_ycsb(seed, case["n_records"])
        _shape(self.c, "tpcc", case["tpcc_shape"])
        _shape(self.y, "ycsb", case["shape"])
        is_c = np.random.RandomState(seed % (1 << 32)).randint(0, 100, n) < case["tpcc_pct"]
        n_c = int(is_c.sum())
        self.tb = _tpcc_gen(case, seed, max(1, n_c)).next()
        self.yb = L.YcsbGenerator(seed, case["n_records"], max(1, n - n_c), self.OPS, 50, case["theta"]).batch(0)
        req = np.zeros(n, dtype=[("workload", "<i4"), ("n", "<u4"), ("txn", "<u8"), ("lines", "<u8"), ("ops", "<u8"),
                                 ("vals", "<u8")])
        x = self.tb.txns[:n_c]
        lines = np.where((x["kind_info"] & 0xFF) == abi.TPCC_NEWORDER, (x["kind_info"] >> 8) & 0xFF, 0)
        req["workload"] = np.where(is_c, abi.WORKLOAD_TPCC, abi.WORKLOAD_YCSB)
        req["n"][is_c] = lines
        req["txn"][is_c] = self.tb.txns.ctypes.data + 32 * np.arange(n_c, dtype=np.uint64)
        req["lines"][is_c] = self.tb.lines.ctypes.data + 8 * x["line_off"].astype(np.uint64)
        req["n"][~is_c] = self.OPS
        k = np.arange(n - n_c, dtype=np.uint64)
        req["ops"][~is_c] = self.yb.ops.ctypes.data + 4 * self.yb.op_stride * k
        req["vals"][~is_c] = self.yb.vals.ctypes.data + 8 * self.yb.val_off[:n - n_c].astype(np.uint64)
        self.req = req
        self.s = L.Server(self.c, self.y, max_batch=most, deadline_ms=1000.0, mode=case["mode"], slots=2,
                          ycsb_ops=self.OPS)

    def run(self):
        first = C.c_uint64()
        _ok(L.lib().ltpg_serve_submit(self.s._h, _ptr(self.req), self.n, C.byref(first)), "submit")
        self.s.flush()
        flags, results = self.s.poll(first.value, self.n)
        return dict(flags=flags, results=results)

    def __del__(self):
        if getattr(self, "s", None) is not None and self.s._h:
            self.s.close()  # before the engines it drives


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("ycsb", "tpcc"):
        return _Resident(case, seed, kind)
    return {"host": _Host, "pipeline": _Pipeline, "generate": _Generated, "serve": _Serve, "caller": _Caller,
            "predictor": _Predicted}[kind](case, seed)


def run(state):
    return state.run()


# ---- what a pass cannot do without ---------------------------------------------


def _distinct(n, theta, draws):
    """Expected distinct keys among `draws` Zipf draws of n keys."""
    if draws <= 0:
        return 0.0
    if theta == 0.0:
        return n * -math.expm1(-draws / n)
    edges = np.unique(np.floor(np.logspace(0, math.log10(n + 1), 400)))
    mid, width = np.sqrt(edges[:-1] * (edges[1:] - 1).clip(1)), np.diff(edges)
    p = mid ** -theta
    p /= (p * width).sum()
    return float((width * -np.expm1(-draws * p)).sum())


def _ycsb_bytes(case, n_txn, made=False):
    """Op words, values and offsets read (written when the batch is made here),
    every row that a read covers read once, updates written, outputs written."""
    k, u = case.get("ops", _Serve.OPS), case.get("update_pct", 50) / 100.0
    reads, updates = n_txn * k * (1 - u), n_txn * k * u
    rows = min(case["n_records"], _distinct(case["n_records"], case["theta"], reads) * max(1, case.get("scan_len", 0)))
    batch = 4 * n_txn * k + 4 * n_txn + 8 * updates
    return (2 if made else 1) * batch + 80 * rows + 8 * _distinct(case["n_records"], case["theta"], updates) + 9.125 * n_txn


def _tpcc_bytes(case, n_txn, made=False):
    """Records and order lines, the columns read for the results, outputs; and
    for the 30 % that commits at these batch sizes the columns written."""
    no, pay = (0.45, 0.43) if case.get("mix") else (0.5, 0.5)
    batch = 32 * n_txn + 8 * 10 * no * n_txn
    reads = (8 * 13 * no + 8 * (1 - no)) * n_txn
    writes = 0.3 * n_txn * (no * (64 + 24 + 10 * (24 + 80)) + pay * (24 + 64))
    return (2 if made else 1) * batch + reads + writes + 9.125 * n_txn


def work(case):
    kind, times = case["kind"], case.get("batches", 1)
    if kind == "serve":
        n_c = case["n_req"] * case["tpcc_pct"] / 100.0
        return dict(bytes=_tpcc_bytes(case, n_c) + _ycsb_bytes(case, case["n_req"] - n_c), flops=0)
    ycsb = kind in ("ycsb", "caller", "predictor") or case.get("work") == "ycsb"
    one = (_ycsb_bytes if ycsb else _tpcc_bytes)(case, case["n_txn"], kind == "generate")
    if kind == "predictor":  # 65,536 buckets forward, 4,096 forward and backward
        return dict(bytes=times * (one + 65_536 * 4 * 6), flops=times * 2 * 4416 * (65_536 + 3 * 4096))
    return dict(bytes=times * one, flops=0)


def exact(case, seed):
    """Whole numbers everywhere but the predictor's weights, whose inputs are
    counts that the staged kernels sample: no value of their own in 64 bits."""
    return None
