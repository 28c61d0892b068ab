// gen_dev.cu — the deterministic batch generators on the GPU: the batches of
// gen.cpp, byte for byte, made directly in a slot's device buffers (no host
// generation, no host-to-device copy).
//
// Compiled with -fmad=false: the Zipf sampler's double arithmetic (gen.h) must
// round exactly like the host's.
//
// YCSB: a block draws the keys of a tile of transactions one operation per
// thread, redraws the repeated ones until none is left (ycsb_gen_ops), an
// inclusive scan of the update counts gives val_off, and one lane per operation
// writes its update's value.
//
// TPC-C: the host generator is a loop whose per-warehouse counters (O_ID,
// NO_ID, OL_ID, H_ID) and order memory (for OrderStatus and Delivery) carry
// from one transaction to the next.  Each value a transaction reads is its
// warehouse's value at batch start plus a count over the batch's earlier
// transactions of the same warehouse, so the loop becomes:
//   1. head: kind, warehouse, district and line count of every transaction
//      (its first draws), counted per chunk of transactions and warehouse;
//   2. line offsets: an inclusive scan of the line counts;
//   3. the chunk counts scanned over chunks, and per-warehouse list starts;
//   4. ranks: per transaction the batch's earlier NewOrders (and their lines,
//      Payments, Deliveries) of its warehouse; each warehouse's NewOrders and
//      Deliveries listed in batch order;
//   5. NewOrder, Payment and StockLevel records;
//   6. Delivery's oldest-undelivered counter, the only true recurrence: a scan
//      of its steps, which compose, per warehouse;
//   7. OrderStatus and Delivery records, each remembered order read from the
//      batch's NewOrder that made it or from the order memory at batch start;
//   8. state: counters, order memory (last writer of each O_ID), slot header.
#include <algorithm>
#include <new>

#include "engine.h"
#include "gen_state.h"

using namespace ltpg;
using namespace ltpg::gen;

namespace {

constexpr uint32_t TB = 256;          // threads per block of the per-transaction kernels
constexpr uint32_t SCAN_T = 1024;     // threads per block of the scan
constexpr uint32_t SCAN_V = 4;        // values per scan thread
constexpr uint32_t SCAN_BLOCK = SCAN_T * SCAN_V;
constexpr uint32_t SCAN_DIRECT = 1024;  // up to this many block totals are summed by their users
constexpr uint32_t DL_TRACKED = 0x80000000u;
constexpr uint64_t MAX_CHUNK_COUNTERS = 8ull << 20;  // per class, chunks x warehouses

__device__ __forceinline__ uint32_t warp_scan_incl(uint32_t v) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// Inclusive scan over the threads of a block of SCAN_T threads.
__device__ __forceinline__ uint32_t block_scan_incl(uint32_t v, uint32_t *sh) {
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    uint32_t x = warp_scan_incl(v);
    if (lane == 31u) sh[wid] = x;
    __syncthreads();
    if (wid == 0) sh[lane] = warp_scan_incl(sh[lane]);
    __syncthreads();
    if (wid > 0) x += sh[wid - 1];
    __syncthreads();
    return x;
}

// In-place inclusive scan, pass 1: each block scans SCAN_BLOCK values and
// records its total.
__global__ void __launch_bounds__(SCAN_T) scan_blocks(uint32_t *a, uint32_t n, uint32_t *blk) {
    __shared__ uint32_t sh[32];
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_BLOCK + (uint64_t)threadIdx.x * SCAN_V;
    uint32_t v[SCAN_V], s = 0;
#pragma unroll
    for (uint32_t j = 0; j < SCAN_V; ++j) {
        v[j] = base + j < n ? a[base + j] : 0u;
        s += v[j];
        v[j] = s;
    }
    const uint32_t excl = block_scan_incl(s, sh) - s;
#pragma unroll
    for (uint32_t j = 0; j < SCAN_V; ++j)
        if (base + j < n) a[base + j] = v[j] + excl;
    if (threadIdx.x == SCAN_T - 1) blk[blockIdx.x] = excl + s;
}
// Pass 2: one block scans the block totals, SCAN_BLOCK at a time.
__global__ void __launch_bounds__(SCAN_T) scan_totals(uint32_t *blk, uint32_t nb) {
    __shared__ uint32_t sh[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint32_t b0 = 0; b0 < nb; b0 += SCAN_BLOCK) {
        const uint32_t base = b0 + threadIdx.x * SCAN_V;
        uint32_t v[SCAN_V], s = 0;
#pragma unroll
        for (uint32_t j = 0; j < SCAN_V; ++j) {
            v[j] = base + j < nb ? blk[base + j] : 0u;
            s += v[j];
            v[j] = s;
        }
        const uint32_t c0 = carry;
        const uint32_t incl = block_scan_incl(s, sh);
        const uint32_t excl = incl - s + c0;
#pragma unroll
        for (uint32_t j = 0; j < SCAN_V; ++j)
            if (base + j < nb) blk[base + j] = v[j] + excl;
        __syncthreads();
        if (threadIdx.x == SCAN_T - 1) carry = c0 + incl;
        __syncthreads();
    }
}
// Pass 3: block b adds the totals of blocks 0 .. b-1: the inclusive sum that
// pass 2 left, or (up to SCAN_DIRECT blocks, with no pass 2) summed here.
__global__ void __launch_bounds__(SCAN_T) scan_add(uint32_t *a, uint32_t n, const uint32_t *blk, bool scanned) {
    if (blockIdx.x == 0) return;
    __shared__ uint32_t sh[32];
    uint32_t add = 0;
    if (scanned) {
        add = blk[blockIdx.x - 1];
    } else {
        const uint32_t lane = threadIdx.x & 31u;
        for (uint32_t i = threadIdx.x; i < blockIdx.x; i += SCAN_T) add += blk[i];
        add = __reduce_add_sync(0xFFFFFFFFu, add);
        if (lane == 0u) sh[threadIdx.x >> 5] = add;
        __syncthreads();
        add = __reduce_add_sync(0xFFFFFFFFu, sh[lane]);
    }
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_BLOCK + (uint64_t)threadIdx.x * SCAN_V;
#pragma unroll
    for (uint32_t j = 0; j < SCAN_V; ++j)
        if (base + j < n) a[base + j] += add;
}

cudaError_t inclusive_scan(uint32_t *a, uint32_t n, uint32_t *blk, cudaStream_t st, uint64_t &launches) {
    if (n == 0) return cudaSuccess;
    const uint32_t nb = (n + SCAN_BLOCK - 1) / SCAN_BLOCK;
    const bool scanned = nb > SCAN_DIRECT;
    scan_blocks<<<nb, SCAN_T, 0, st>>>(a, n, blk);
    ++launches;
    if (scanned) {
        scan_totals<<<1, SCAN_T, 0, st>>>(blk, nb);
        ++launches;
    }
    if (nb > 1) {
        scan_add<<<nb, SCAN_T, 0, st>>>(a, n, blk, scanned);
        ++launches;
    }
    return cudaGetLastError();
}
uint32_t scan_scratch(uint32_t n) { return (n + SCAN_BLOCK - 1) / SCAN_BLOCK + 1; }

// ---- YCSB ----------------------------------------------------------------------
struct YcsbGenArgs {
    ltpg_ycsb_params p;
    FastZipf zipf;
    const FixTables *tab;
    const PolyCell *cells;
    Perm perm;
    bool rotate;
    uint64_t batch_id;
    uint32_t *ops, *val_off;
    uint64_t *vals;
    uint32_t tile;         // slots of a warp
    bool perm_table;       // the permutation's rounds tabulated by each block
    uint32_t k_inv, s_inv; // ceil(2^16 / k), ceil(2^16 / stride): i / k = i k_inv >> 16 for a tile's indices
};

// Draw number d (0-based) of the stream that starts at state s.
__device__ __forceinline__ uint64_t draw_at(uint64_t s, uint32_t d) {
    Rng r(s + (uint64_t)d * 0x9E3779B97F4A7C15ull);
    return r.next();
}

// Op words of a batch, the bytes of ycsb_txn.  A transaction's draws are a
// counter-based stream: operation j takes three (key, update?, field) from draw
// 3j + (redraws so far), a redraw one more.  A warp holds up to 32 transactions
// (256 words) in slots and repeats:
//   1. free slots take the block's next transactions;
//   2. every key not yet settled is drawn, one operation per lane, from a list:
//      all of a new transaction's, as if none repeated, and of an old one's
//      those from its first repeated key on, one draw up;
//   3. each drawn key is compared with its transaction's earlier ones; a
//      transaction without a repeat gets its update and field bits, its words
//      are stored (coalesced), and its slot is free.
// At theta = 0.99 over 10 M keys 45 % of the 16-op transactions repeat a key and
// the redrawn operations are 20 % of all; refilling the slots keeps the lists
// long (a thread per transaction ran as long as the warp's unluckiest lane; a
// tile finished before the next was begun ran half-empty passes for its last
// repeats, 146 us per 2^18 transactions against 120).  A transaction still
// repeating after GEN_ROUNDS rounds (tiny tables, whose walk to a free key
// starts at the 65th draw of an operation) is made by ycsb_txn, alone.  The hot
// set's permutation, four rounds of a hash of at most 12 bits for up to 2^24
// keys, is tabulated by the block (4 x 2^half entries of 16 bits).  2^20 x 16
// ops, theta 0.99: 1006 us one thread per transaction, 350 us now; bound by the
// integer pipes.
constexpr uint32_t GEN_T = 512, GEN_WORDS = 256, GEN_ROUNDS = 16, PERM_HALF = 12;
constexpr uint32_t PERM_BYTES = (4u << PERM_HALF) * sizeof(uint16_t);

struct __align__(16) GenSlots {
    uint64_t seed[32];            // stream state of each slot's transaction
    uint32_t first[32];           // its first repeated key (k: none)
    uint32_t redraws[32];
    uint32_t cnt[32];             // updates
    uint32_t key[GEN_WORDS];      // by word: slot * stride + j
    uint8_t shift[GEN_WORDS];     // by word: redraws up to and with the operation
    uint8_t list[GEN_WORDS];      // operations to draw, slot * k + j
    uint8_t settled[32];          // slots to store
    uint64_t pad[2];
};
constexpr uint32_t GEN_BYTES = POLY_CELLS * sizeof(PolyCell) + GEN_T / 32 * sizeof(GenSlots);  // + the permutation

__global__ void __launch_bounds__(GEN_T, 2) ycsb_gen_ops(YcsbGenArgs a) {
    extern __shared__ __align__(16) char gen_smem[];
    PolyCell *cells = reinterpret_cast<PolyCell *>(gen_smem);
    GenSlots *slots = reinterpret_cast<GenSlots *>(cells + POLY_CELLS);
    uint16_t *perm_tab = reinterpret_cast<uint16_t *>(slots + GEN_T / 32);  // [4][2^half] when tabulated
    __shared__ uint32_t next;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, k = a.p.ops_per_txn, stride = ycsb_stride(k), B = a.p.n_txn;
    const uint32_t half = a.perm.half, mask = (1u << half) - 1u, span = a.p.scan_len >= 2u ? a.p.scan_len - 1u : 0u;
    const bool tabulated = a.perm_table;
    if (a.zipf.fast)
        for (uint32_t i = tid; i < POLY_CELLS * sizeof(PolyCell) / 16u; i += GEN_T)
            reinterpret_cast<uint4 *>(cells)[i] = reinterpret_cast<const uint4 *>(a.cells)[i];
    if (tabulated)
        for (uint32_t i = tid; i < (4u << half); i += GEN_T)
            perm_tab[i] = (uint16_t)a.perm.round_fn(i & mask, i >> half);
    if (blockIdx.x == 0 && tid == 0) a.val_off[0] = 0;
    // the block's transactions: [begin, end)
    const uint32_t end = (uint32_t)((uint64_t)B * (blockIdx.x + 1u) / gridDim.x);
    if (tid == 0) next = (uint32_t)((uint64_t)B * blockIdx.x / gridDim.x);
    __syncthreads();

    GenSlots &g = slots[tid >> 5];
    bool active = false;  // this lane's slot holds a transaction
    uint32_t t = 0, from = 0;
    for (;;) {
        // 1. refill
        const unsigned free = __ballot_sync(0xFFFFFFFFu, lane < a.tile && !active);
        uint32_t base = 0;
        if (lane == 0u) base = atomicAdd(&next, __popc(free));
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if ((free >> lane) & 1u) {
            t = base + __popc(free & ((1u << lane) - 1u));
            active = base < end && t < end;
            from = 0;
            if (active) {
                g.seed[lane] = hash3(a.p.seed ^ DOM_YCSB_OPS, a.batch_id, t);
                g.redraws[lane] = 0u;
                g.cnt[lane] = 0u;
            }
        }
        if (!__any_sync(0xFFFFFFFFu, active)) break;
        // 2. the keys to draw, then the draws
        const uint32_t m = active ? k - from : 0u, incl = warp_scan_incl(m);
        const uint32_t n = __shfl_sync(0xFFFFFFFFu, incl, 31);
        if (active) {
            for (uint32_t j = from; j < k; ++j) g.list[incl - k + j] = (uint8_t)(lane * k + j);
            g.first[lane] = k;
        }
        __syncwarp();
        for (uint32_t e = lane; e < n; e += 32u) {
            const uint32_t i = g.list[e], lt = i * a.k_inv >> 16, j = i - lt * k, s = g.redraws[lt];
            uint64_t y = fast_sample(a.zipf, cells, *a.tab, draw_at(g.seed[lt], 3u * j + s));
            if (tabulated) {
                uint32_t l = (uint32_t)(y >> half), r = (uint32_t)y & mask;
                do {
#pragma unroll
                    for (uint32_t f = 0; f < 4; ++f) {
                        const uint32_t x = l ^ perm_tab[(f << half) + r];
                        l = r;
                        r = x;
                    }
                } while (((l << half) | r) >= (uint32_t)a.perm.n);
                y = (l << half) | r;
            } else if (a.rotate) {
                y = a.perm(y);
            }
            g.key[lt * stride + j] = (uint32_t)y;
            g.shift[lt * stride + j] = (uint8_t)s;
        }
        __syncwarp();
        // 3. repeats
        for (uint32_t e = lane; e < n; e += 32u) {
            const uint32_t i = g.list[e], lt = i * a.k_inv >> 16, j = i - lt * k;
            const uint32_t *row = g.key + lt * stride, key = row[j];
            bool dup = false;
            uint32_t q = 0;
            for (; q + 3u < j; q += 4u) {
                const uint4 w = *reinterpret_cast<const uint4 *>(row + q);
                dup |= w.x == key | w.y == key | w.z == key | w.w == key;
            }
            for (; q < j; ++q) dup |= row[q] == key;
            if (dup) atomicMin(&g.first[lt], j);
        }
        __syncwarp();
        bool settled = false;
        if (active) {
            from = g.first[lane];
            settled = from == k;
            if (!settled && ++g.redraws[lane] > GEN_ROUNDS) {
                uint32_t w[LTPG_YCSB_MAX_OPS];
                const uint32_t nu = ycsb_txn(a.p, a.zipf.z, *a.tab, a.rotate ? &a.perm : nullptr, a.batch_id, t, w);
                for (uint32_t j = 0; j < stride; ++j) a.ops[(uint64_t)t * stride + j] = w[j];
                a.val_off[t + 1u] = nu;
                active = false;
            }
        }
        const unsigned done = __ballot_sync(0xFFFFFFFFu, settled);
        if (settled) g.settled[__popc(done & ((1u << lane) - 1u))] = (uint8_t)lane;
        __syncwarp();
        const uint32_t words = __popc(done) * stride;
        for (uint32_t v0 = 0; v0 < words; v0 += 32u) {  // whole warps: the shuffle below
            const uint32_t v = v0 + lane, at = v < words ? v * a.s_inv >> 16 : 0u, j = v - at * stride;
            const uint32_t lt = g.settled[at], tt = __shfl_sync(0xFFFFFFFFu, t, lt);
            if (v >= words) continue;
            uint32_t w = LTPG_YCSB_OP_PAD;
            if (j < k) {
                const uint32_t d = 3u * j + g.shift[lt * stride + j];
                const bool upd = mulhi64(draw_at(g.seed[lt], d + 1u), 100u) < a.p.update_pct;
                uint32_t field = span;
                if (upd) {
                    field = (uint32_t)mulhi64(draw_at(g.seed[lt], d + 2u), LTPG_YCSB_FIELDS);
                    atomicAdd(&g.cnt[lt], 1u);
                }
                w = ycsb_word(g.key[lt * stride + j], upd, field);
            }
            a.ops[(uint64_t)tt * stride + j] = w;
        }
        __syncwarp();
        if (settled) {
            a.val_off[t + 1u] = g.cnt[lane];
            active = false;
        }
        __syncwarp();
    }
}

// One thread per transaction: batches whose transactions repeat most of their
// keys (each repeat draws the rest of the transaction again above), and the
// smallest ones (gen_ycsb has the rule).
__global__ void __launch_bounds__(TB) ycsb_gen_ops_txn(YcsbGenArgs a) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) a.val_off[0] = 0;
    if (t >= a.p.n_txn) return;
    a.val_off[t + 1] = ycsb_txn(a.p, a.zipf.z, *a.tab, a.rotate ? &a.perm : nullptr, a.batch_id, t,
                                a.ops + (uint64_t)t * ycsb_stride(a.p.ops_per_txn));
}

// Update values, and the value offsets completed: val_off[t + 1] holds the
// update count of transaction t's SCAN_BLOCK so far, blk[c] the total of block
// c.  A block of threads stays inside one SCAN_BLOCK and sums the totals before
// it; a warp takes 32 / (stride / 4) whole transactions at a time, four words
// per lane, and a lane's first value index is the count of its transaction's
// updates in the earlier lanes.
__global__ void __launch_bounds__(TB) ycsb_gen_vals(YcsbGenArgs a, const uint32_t *blk, bool scanned) {
    __shared__ uint32_t part[TB / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t B = a.p.n_txn, vpt = ycsb_stride(a.p.ops_per_txn) / 4u, tpw = 32u / vpt;
    const uint32_t t_begin = blockIdx.x * TB, t_end = min(B, t_begin + TB), c = t_begin / SCAN_BLOCK;
    uint32_t before = 0;
    if (scanned) {  // blk holds inclusive sums
        before = c ? blk[c - 1u] : 0u;
    } else {
        for (uint32_t i = threadIdx.x; i < c; i += TB) before += blk[i];
        before = __reduce_add_sync(0xFFFFFFFFu, before);
        if (lane == 0u) part[warp] = before;
        __syncthreads();
        before = 0;
        for (uint32_t i = 0; i < TB / 32; ++i) before += part[i];
    }
    const uint32_t lt = lane / vpt, seg = lane - lt * vpt;
    const uint4 *vp = reinterpret_cast<const uint4 *>(a.ops);
    for (uint32_t t0 = t_begin + warp * tpw; t0 < t_end; t0 += (TB / 32) * tpw) {
        const uint32_t t = t0 + lt;
        const bool act = lt < tpw && t < t_end;
        const uint4 w4 = act ? vp[(uint64_t)t * vpt + seg]
                             : make_uint4(LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD);
        const uint32_t end = act ? a.val_off[t + 1] + before : 0u;
        const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
        uint32_t n = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) n += !ycsb_is_pad(w[q]) && ycsb_is_update(w[q]);
        uint32_t incl = n;  // over the transaction's lanes so far
        for (uint32_t o = 1; o < vpt; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (seg >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, (lt * vpt + vpt - 1u) & 31u);
        uint32_t v = end - total + incl - n;
        if (n) {  // ycsb_value, its part that the transaction's operations share made once
            const uint64_t h = splitmix64(splitmix64(a.p.seed ^ DOM_YCSB_VAL) ^ (a.batch_id * (uint64_t)B + t));
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                if (!ycsb_is_pad(w[q]) && ycsb_is_update(w[q])) a.vals[v++] = splitmix64(h ^ (4u * seg + q));
        }
        __syncwarp();  // every lane of the transaction has read its count (a shuffle orders no memory access)
        if (act && seg == 0u) a.val_off[t + 1] = end;
    }
}

// ---- TPC-C ---------------------------------------------------------------------
enum { CL_NO = 0, CL_OL = 1, CL_PAY = 2, CL_DL = 3 };

struct TpccGenArgs {
    ltpg_tpcc_params p;
    uint64_t batch_id, txn_base;
    uint32_t B, W, G, C;  // transactions, warehouses, chunks, transactions per chunk
    uint32_t tracking;
    // generator state
    uint32_t *o_id, *no_id, *ol_id, *h_id;
    uint64_t *made, *delivered;
    uint16_t *o_cust;
    uint8_t *o_dist, *o_cnt;
    uint32_t *o_ol;
    const uint16_t *cust_name;
    const uint8_t *cust_rank;
    // per-batch scratch
    uint32_t *incl;     // B: inclusive scan of line counts
    uint32_t *nob;      // B: the batch's earlier NewOrders of the same warehouse
    uint32_t *aux;      // B: per kind (see tpcc_gen_rank, tpcc_gen_dl_walk)
    uint32_t *cc;       // 4 W G chunk counters [class][w][chunk]
    uint32_t *tot;      // 4 W batch totals [class][w]
    uint32_t *no_start, *dl_start;  // W + 1 list starts
    uint32_t *no_list;  // NewOrders by (warehouse, rank)
    uint64_t *dl_list;  // Deliveries by (warehouse, rank): nob << 32 | TID
    // slot
    ltpg_tpcc_txn *txns;
    ltpg_tpcc_line *lines;
    uint64_t *hdr;
};

__device__ __forceinline__ Rng tpcc_rng(const TpccGenArgs &a, uint32_t t) {
    return Rng(hash3(a.p.seed ^ DOM_TPCC, a.batch_id, t));
}
__device__ __forceinline__ uint32_t *ccp(const TpccGenArgs &a, uint32_t cl, uint32_t w, uint32_t g) {
    return a.cc + ((uint64_t)cl * a.W + w) * a.G + g;
}
__device__ __forceinline__ void store_txn(ltpg_tpcc_txn *dst, const ltpg_tpcc_txn &x) {
    uint4 *p = reinterpret_cast<uint4 *>(dst);
    p[0] = make_uint4(x.kind_info, x.w, x.c_w, x.c_id);
    p[1] = make_uint4(x.a, x.b, x.c, x.line_off);
}

// 1. Heads, line counts, chunk counters.
__global__ void __launch_bounds__(TB) tpcc_gen_head(TpccGenArgs a) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.B) return;
    Rng r = tpcc_rng(a, t);
    const TpccHead h = tpcc_head(a.p, r);
    a.incl[t] = h.cnt;
    const uint32_t g = t / a.C;
    if (h.kind == LTPG_TPCC_NEWORDER) {
        atomicAdd(ccp(a, CL_NO, h.w, g), 1u);
        atomicAdd(ccp(a, CL_OL, h.w, g), h.cnt);
    } else if (h.kind == LTPG_TPCC_PAYMENT) {
        atomicAdd(ccp(a, CL_PAY, h.w, g), 1u);
    } else if (h.kind == LTPG_TPCC_DELIVERY) {
        atomicAdd(ccp(a, CL_DL, h.w, g), 1u);
    }
}

// 3a. One block per (class, warehouse): exclusive scan of its chunk counters.
__global__ void __launch_bounds__(TB) tpcc_gen_chunk_scan(TpccGenArgs a) {
    __shared__ uint32_t part[TB / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t *c = a.cc + (uint64_t)blockIdx.x * a.G;
    uint32_t carry = 0;
    for (uint32_t g0 = 0; g0 < a.G; g0 += TB * 4u) {
        const uint32_t g = g0 + threadIdx.x * 4u;
        uint32_t v[4], sum = 0;
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) sum += v[i] = g + i < a.G ? c[g + i] : 0u;
        const uint32_t incl = warp_scan_incl(sum);
        if (lane == 31u) part[warp] = incl;
        __syncthreads();
        uint32_t before = carry + incl - sum;
        for (uint32_t i = 0; i < TB / 32; ++i) {
            before += i < warp ? part[i] : 0u;
            carry += part[i];
        }
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            if (g + i < a.G) c[g + i] = before;
            before += v[i];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) a.tot[blockIdx.x] = carry;
}

// 3b. One block: list starts of each warehouse's NewOrders and Deliveries.
__global__ void __launch_bounds__(SCAN_T) tpcc_gen_starts(TpccGenArgs a) {
    __shared__ uint32_t sh[32];
    __shared__ uint32_t carry[2];
    if (threadIdx.x < 2) carry[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t w0 = 0; w0 < a.W; w0 += SCAN_T) {
        const uint32_t w = w0 + threadIdx.x;
        const uint32_t vn = w < a.W ? a.tot[CL_NO * a.W + w] : 0u;
        const uint32_t vd = w < a.W ? a.tot[CL_DL * a.W + w] : 0u;
        const uint32_t cn = carry[0], cd = carry[1];
        const uint32_t in = block_scan_incl(vn, sh);
        const uint32_t id = block_scan_incl(vd, sh);
        if (w < a.W) {
            a.no_start[w] = cn + in - vn;
            a.dl_start[w] = cd + id - vd;
        }
        __syncthreads();
        if (threadIdx.x == SCAN_T - 1) {
            carry[0] = cn + in;
            carry[1] = cd + id;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        a.no_start[a.W] = carry[0];
        a.dl_start[a.W] = carry[1];
    }
}

// 4. One warp per chunk, 32 transactions per step in batch order.  A lane
// counts the step's earlier lanes of its warehouse by ballots (its peers by one
// match; line counts bit by bit); the warehouse's running counters of the chunk
// (the chunk counters, now prefixes) are advanced by the step's last lane of
// that warehouse.  Steps follow one another through those counters, so chunks
// are short: 128 transactions (W = 64, 2^18: 102 us with 1,024 and a shuffle
// per earlier lane, 16 us now).
//   nob[t]  NewOrders of w before t in the batch (every kind)
//   aux[t]  NewOrder: lines of w's earlier NewOrders; Payment: earlier
//           Payments of w; Delivery: earlier Deliveries of w
__global__ void __launch_bounds__(TB) tpcc_gen_rank(TpccGenArgs a) {
    const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (g >= a.G) return;
    const uint32_t t_end = min(a.B, (g + 1) * a.C);
    for (uint32_t base = g * a.C; base < t_end; base += 32) {
        const uint32_t t = base + lane;
        const bool valid = t < t_end;
        TpccHead h{0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u};
        if (valid) {
            Rng r = tpcc_rng(a, t);
            h = tpcc_head(a.p, r);
        }
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, h.w), earlier = peers & ((1u << lane) - 1u);
        const bool last = valid && (peers >> lane) == 1u;
        const uint32_t pno = __popc(__ballot_sync(0xFFFFFFFFu, h.kind == LTPG_TPCC_NEWORDER) & earlier);
        const uint32_t ppay = __popc(__ballot_sync(0xFFFFFFFFu, h.kind == LTPG_TPCC_PAYMENT) & earlier);
        const uint32_t pdl = __popc(__ballot_sync(0xFFFFFFFFu, h.kind == LTPG_TPCC_DELIVERY) & earlier);
        uint32_t pol = 0;  // h.cnt: lines of a NewOrder (at most 15), else 0
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) pol += __popc(__ballot_sync(0xFFFFFFFFu, (h.cnt >> i) & 1u) & earlier) << i;
        uint32_t bno = 0, bol = 0, bpay = 0, bdl = 0;
        if (valid) {
            bno = *ccp(a, CL_NO, h.w, g);
            bol = *ccp(a, CL_OL, h.w, g);
            bpay = *ccp(a, CL_PAY, h.w, g);
            bdl = *ccp(a, CL_DL, h.w, g);
            const uint32_t nb = bno + pno;
            a.nob[t] = nb;
            uint32_t aux = 0;
            if (h.kind == LTPG_TPCC_NEWORDER) {
                aux = bol + pol;
                a.no_list[a.no_start[h.w] + nb] = t;
            } else if (h.kind == LTPG_TPCC_PAYMENT) {
                aux = bpay + ppay;
            } else if (h.kind == LTPG_TPCC_DELIVERY) {
                aux = bdl + pdl;
                a.dl_list[a.dl_start[h.w] + aux] = ((uint64_t)nb << 32) | t;
            }
            a.aux[t] = aux;
        }
        __syncwarp();
        if (last) {
            const bool no = h.kind == LTPG_TPCC_NEWORDER;
            *ccp(a, CL_NO, h.w, g) = bno + pno + (no ? 1u : 0u);
            *ccp(a, CL_OL, h.w, g) = bol + pol + (no ? h.cnt : 0u);
            *ccp(a, CL_PAY, h.w, g) = bpay + ppay + (h.kind == LTPG_TPCC_PAYMENT ? 1u : 0u);
            *ccp(a, CL_DL, h.w, g) = bdl + pdl + (h.kind == LTPG_TPCC_DELIVERY ? 1u : 0u);
        }
        __syncwarp();
    }
}

// 5. NewOrder, Payment, StockLevel records.  A block takes TB transactions,
// NewOrders first, then the others, so that a warp draws one kind (a NewOrder
// with its 5 to 15 lines takes ten times a Payment's draws); the items drawn so
// far stand in shared memory for the check of a new one.  2^18 of the
// five-transaction mix: 47 us in batch order, 34 us now.
__global__ void __launch_bounds__(TB) tpcc_gen_main(TpccGenArgs a) {
    __shared__ uint32_t items[LTPG_TPCC_MAX_LINES][TB];
    __shared__ uint16_t order[TB];
    __shared__ uint32_t n_no[TB / 32], n_pay[TB / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, t0 = blockIdx.x * TB;
    {
        uint32_t kind = 0xFFFFFFFFu;
        if (t0 + tid < a.B) {
            Rng r = tpcc_rng(a, t0 + tid);
            kind = tpcc_head(a.p, r).kind;
        }
        const bool no = kind == LTPG_TPCC_NEWORDER;
        const bool pay = kind == LTPG_TPCC_PAYMENT || kind == LTPG_TPCC_STOCKLEVEL;
        const unsigned bn = __ballot_sync(0xFFFFFFFFu, no), bp = __ballot_sync(0xFFFFFFFFu, pay);
        if (lane == 0u) {
            n_no[warp] = __popc(bn);
            n_pay[warp] = __popc(bp);
        }
        order[tid] = 0xFFFFu;
        __syncthreads();
        uint32_t at = no ? __popc(bn & ((1u << lane) - 1u)) : __popc(bp & ((1u << lane) - 1u));
        for (uint32_t i = 0; i < TB / 32; ++i) {
            at += no ? (i < warp ? n_no[i] : 0u) : n_no[i];
            if (pay && i < warp) at += n_pay[i];
        }
        if (no || pay) order[at] = (uint16_t)tid;
        __syncthreads();
    }
    if (order[tid] == 0xFFFFu) return;
    const uint32_t t = t0 + order[tid];
    Rng r = tpcc_rng(a, t);
    const TpccHead h = tpcc_head(a.p, r);
    ltpg_tpcc_txn x{};
    x.line_off = a.incl[t] - h.cnt;
    x.w = h.w;
    if (h.kind == LTPG_TPCC_NEWORDER) {
        const uint32_t s = a.nob[t];
        x.a = (uint32_t)(((uint64_t)a.o_id[h.w] + s) % 30000u);
        x.b = (uint32_t)(((uint64_t)a.no_id[h.w] + s) % 30000u);
        x.c = (uint32_t)(((uint64_t)a.ol_id[h.w] + a.aux[t]) % 450000u);
        ltpg_tpcc_line *lines = a.lines + x.line_off;
        tpcc_neworder(
            a.p, r, h, x,
            [&](uint32_t i, const ltpg_tpcc_line &ln) {
                items[i][tid] = ln.i_id;
                reinterpret_cast<uint2 *>(lines)[i] = make_uint2(ln.i_id, ln.supply_w | ((uint32_t)ln.qty << 16));
            },
            [&](uint32_t i) { return items[i][tid]; });
    } else if (h.kind == LTPG_TPCC_PAYMENT) {
        x.a = (uint32_t)(((uint64_t)a.h_id[h.w] + a.aux[t]) % 30000u);
        tpcc_payment(a.p, r, h, x, a.cust_name, a.cust_rank);
    } else {
        tpcc_stocklevel(r, h, x);
    }
    store_txn(a.txns + t, x);
}

// 6. Oldest undelivered order D, per warehouse in batch order: a Delivery that
// follows M orders takes max(D, M - 30000) when D < M and leaves that + 1, which
// with D <= M is min(max(D + 1, M - 29999), M).  Such steps compose to another
// min(max(D + add, lo), hi), so a warp scans its warehouse's Deliveries 32 at a
// time (one thread stepping through them: 40 us at W = 64 and 2^18 of the mix).
// aux[t] of a Delivery becomes DL_TRACKED | O_ID, or 0 when w had no
// undelivered order.
__global__ void __launch_bounds__(TB) tpcc_gen_dl_walk(TpccGenArgs a) {
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (w >= a.W) return;
    long long D = (long long)a.delivered[w];
    const long long M0 = (long long)a.made[w];
    const uint32_t i1 = a.dl_start[w + 1];
    for (uint32_t i0 = a.dl_start[w]; i0 < i1; i0 += 32) {
        const bool act = i0 + lane < i1;
        const uint64_t e = act ? a.dl_list[i0 + lane] : 0ull;
        const long long M = M0 + (long long)(e >> 32);
        // this lane's step, then the steps of lanes 0 .. lane composed; a lane
        // past the end adds nothing
        long long add = act ? 1 : 0, lo = act ? M - 29999 : -(1ll << 60), hi = act ? M : 1ll << 60;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const long long add0 = __shfl_up_sync(0xFFFFFFFFu, add, o), lo0 = __shfl_up_sync(0xFFFFFFFFu, lo, o),
                            hi0 = __shfl_up_sync(0xFFFFFFFFu, hi, o);
            if (lane >= o) {
                const long long l = min(max(lo0 + add, lo), hi), u = min(max(hi0 + add, lo), hi);
                add += add0;
                lo = l;
                hi = u;
            }
        }
        const long long after = min(max(D + add, lo), hi);
        long long before = __shfl_up_sync(0xFFFFFFFFu, after, 1);
        if (lane == 0u) before = D;
        if (act)
            a.aux[(uint32_t)e] = before < M ? DL_TRACKED | (uint32_t)((uint64_t)max(before, M - 30000) % 30000u) : 0u;
        D = __shfl_sync(0xFFFFFFFFu, after, 31);
    }
    if (lane == 0u) a.delivered[w] = (uint64_t)D;
}

// 7. OrderStatus and Delivery records.
__global__ void __launch_bounds__(TB) tpcc_gen_osdl(TpccGenArgs a) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.B) return;
    Rng r = tpcc_rng(a, t);
    const TpccHead h = tpcc_head(a.p, r);
    if (h.kind != LTPG_TPCC_ORDERSTATUS && h.kind != LTPG_TPCC_DELIVERY) return;
    const uint32_t w = h.w, nb = a.nob[t];
    const uint32_t o_id_t = (uint32_t)(((uint64_t)a.o_id[w] + nb) % 30000u);
    // The order with O_ID o as the host loop sees it at t: made by the batch's
    // NewOrder of rank nb - 1 - delta when that is >= 0, else remembered.
    auto order = [&](uint32_t o) {
        const uint32_t delta = (o_id_t + 30000u - 1u - o) % 30000u;
        if (delta < nb) {
            const ltpg_tpcc_txn y = a.txns[a.no_list[a.no_start[w] + nb - 1u - delta]];
            return TpccOrder{y.c_id, tpcc_d(y.kind_info), y.c, tpcc_ol_cnt(y.kind_info)};
        }
        const size_t k = 30000ull * w + o;
        return TpccOrder{a.o_cust[k], a.o_dist[k], a.o_ol[k], a.o_cnt[k]};
    };
    ltpg_tpcc_txn x{};
    x.line_off = a.incl[t];
    x.w = w;
    if (h.kind == LTPG_TPCC_ORDERSTATUS) {
        const uint64_t made = a.tracking ? a.made[w] + nb : 0u;
        tpcc_orderstatus(a.p, r, h, x, made, o_id_t, order, a.cust_name, a.cust_rank);
    } else {
        const uint32_t v = a.tracking ? a.aux[t] : 0u;
        tpcc_delivery(r, h, x, (v & DL_TRACKED) != 0u, v & ~DL_TRACKED, order);
    }
    store_txn(a.txns + t, x);
}

// 8. Order memory (the batch's last NewOrder of each O_ID), counters, header.
__global__ void __launch_bounds__(TB) tpcc_gen_state(TpccGenArgs a) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < a.B && a.tracking) {
        const ltpg_tpcc_txn x = a.txns[t];
        if (tpcc_kind(x.kind_info) == LTPG_TPCC_NEWORDER && a.nob[t] + 30000u >= a.tot[CL_NO * a.W + x.w]) {
            const size_t k = 30000ull * x.w + x.a;
            a.o_cust[k] = (uint16_t)x.c_id;
            a.o_dist[k] = (uint8_t)tpcc_d(x.kind_info);
            a.o_ol[k] = x.c;
            a.o_cnt[k] = (uint8_t)tpcc_ol_cnt(x.kind_info);
        }
    }
    if (t < a.W) {
        const uint32_t n_no = a.tot[CL_NO * a.W + t];
        a.o_id[t] = (uint32_t)(((uint64_t)a.o_id[t] + n_no) % 30000u);
        a.no_id[t] = (uint32_t)(((uint64_t)a.no_id[t] + n_no) % 30000u);
        a.ol_id[t] = (uint32_t)(((uint64_t)a.ol_id[t] + a.tot[CL_OL * a.W + t]) % 450000u);
        a.h_id[t] = (uint32_t)(((uint64_t)a.h_id[t] + a.tot[CL_PAY * a.W + t]) % 30000u);
        if (a.tracking) a.made[t] += n_no;
    }
    if (t == 0) {
        a.hdr[0] = a.incl[a.B - 1];
        a.hdr[1] = a.txn_base;
    }
}

uint32_t blocks(uint64_t n, uint32_t per) { return (uint32_t)((n + per - 1) / per); }

}  // namespace

// Device side of a generator: YCSB, the sampler's power tables; TPC-C, the
// generator's state and the scratch of one batch.
struct ltpg_gen_dev {
    int device = -1;
    FixTables *tab = nullptr;
    PolyCell *cells = nullptr;
    FastZipf zipf;
    bool repeats = false;     // six redraws a transaction or more
    uint32_t gen_blocks = 0;  // resident blocks of ycsb_gen_ops on the device
    uint32_t G = 0, C = 0;
    uint32_t *o_id = nullptr, *no_id = nullptr, *ol_id = nullptr, *h_id = nullptr;
    uint64_t *made = nullptr, *delivered = nullptr;
    uint16_t *o_cust = nullptr;
    uint8_t *o_dist = nullptr, *o_cnt = nullptr;
    uint32_t *o_ol = nullptr;
    uint16_t *cust_name = nullptr;
    uint8_t *cust_rank = nullptr;
    uint32_t *incl = nullptr, *nob = nullptr, *aux = nullptr, *cc = nullptr, *tot = nullptr;
    uint32_t *no_start = nullptr, *dl_start = nullptr, *no_list = nullptr, *blk = nullptr;
    uint64_t *dl_list = nullptr;
    std::vector<void *> owned;
};

namespace {

template <class T>
cudaError_t dalloc(ltpg_gen_dev *d, T **p, uint64_t n) {
    *p = nullptr;
    if (n == 0) return cudaSuccess;
    cudaError_t e = cudaMalloc((void **)p, n * sizeof(T));
    if (e == cudaSuccess) d->owned.push_back(*p);
    return e;
}
template <class T>
cudaError_t dput(ltpg_gen_dev *d, T **p, const std::vector<T> &h) {
    cudaError_t e = dalloc(d, p, h.size());
    if (e == cudaSuccess && !h.empty()) e = cudaMemcpy(*p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
    return e;
}

void free_dev(ltpg_gen_dev *d) {
    if (!d) return;
    int cur = -1;
    cudaGetDevice(&cur);
    if (d->device >= 0 && d->device != cur) cudaSetDevice(d->device);
    for (void *p : d->owned) cudaFree(p);
    if (d->device >= 0 && d->device != cur && cur >= 0) cudaSetDevice(cur);
    delete d;
}

// Copies the host state of a TPC-C generator to the device (first device batch).
cudaError_t bind_tpcc(ltpg_gen *g, int device) {
    ltpg_gen_dev *d = new (std::nothrow) ltpg_gen_dev();
    if (!d) return cudaErrorMemoryAllocation;
    d->device = device;
    const uint32_t B = g->c.n_txn, W = g->c.warehouses;
    d->C = 128;
    if ((uint64_t)((B + d->C - 1) / d->C) * W > MAX_CHUNK_COUNTERS) {
        const uint64_t g_max = std::max<uint64_t>(1, MAX_CHUNK_COUNTERS / W);
        d->C = (uint32_t)(((B + g_max - 1) / g_max + 31) / 32 * 32);
    }
    d->G = (B + d->C - 1) / d->C;
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t x) {
        if (e == cudaSuccess) e = x;
    };
    ok(dput(d, &d->o_id, g->o_id));
    ok(dput(d, &d->no_id, g->no_id));
    ok(dput(d, &d->ol_id, g->ol_id));
    ok(dput(d, &d->h_id, g->h_id));
    if (!g->made.empty()) {
        ok(dput(d, &d->made, g->made));
        ok(dput(d, &d->delivered, g->delivered));
        ok(dput(d, &d->o_cust, g->o_cust));
        ok(dput(d, &d->o_dist, g->o_dist));
        ok(dput(d, &d->o_cnt, g->o_cnt));
        ok(dput(d, &d->o_ol, g->o_ol));
    }
    if (!g->cust_name.empty()) {
        ok(dput(d, &d->cust_name, g->cust_name));
        ok(dput(d, &d->cust_rank, g->cust_rank));
    }
    ok(dalloc(d, &d->incl, B));
    ok(dalloc(d, &d->nob, B));
    ok(dalloc(d, &d->aux, B));
    ok(dalloc(d, &d->cc, 4ull * W * d->G));
    ok(dalloc(d, &d->tot, 4ull * W));
    ok(dalloc(d, &d->no_start, (uint64_t)W + 1));
    ok(dalloc(d, &d->dl_start, (uint64_t)W + 1));
    ok(dalloc(d, &d->no_list, B));
    ok(dalloc(d, &d->dl_list, B));
    ok(dalloc(d, &d->blk, scan_scratch(B)));
    if (e != cudaSuccess) {
        free_dev(d);
        return e;
    }
    g->dev = d;
    g->dev_bound = true;
    return cudaSuccess;
}

// Whether a transaction of k distinct ranks takes six redraws or more, from 32 of them.
bool many_redraws(const Zipf &z, uint32_t k) {
    Rng r(1);
    uint32_t redraws = 0;
    for (uint32_t t = 0; t < 32; ++t) {
        uint64_t keys[LTPG_YCSB_MAX_OPS];
        for (uint32_t j = 0; j < k; ++j)
            for (uint32_t attempt = 0; attempt < 64; ++attempt) {
                keys[j] = z.sample(r, host_fix_tables());
                if (std::find(keys, keys + j, keys[j]) == keys + j) break;
                if (++redraws >= 6 * 32) return true;
            }
    }
    return false;
}

// The YCSB generator's power tables on the device (first device batch).
cudaError_t bind_ycsb(ltpg_gen *g, int device) {
    ltpg_gen_dev *d = new (std::nothrow) ltpg_gen_dev();
    if (!d) return cudaErrorMemoryAllocation;
    d->device = device;
    std::vector<PolyCell> cells(POLY_CELLS);
    d->zipf = fast_zipf(g->zipf, cells.data());
    d->repeats = many_redraws(g->zipf, g->y.ops_per_txn);
    cudaError_t e = dalloc(d, &d->tab, 1);
    if (e == cudaSuccess) e = cudaMemcpy(d->tab, &host_fix_tables(), sizeof(FixTables), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = dput(d, &d->cells, cells);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(ycsb_gen_ops, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(GEN_BYTES + PERM_BYTES));
    int per_sm = 0, sms = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ycsb_gen_ops, GEN_T, GEN_BYTES + PERM_BYTES);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    d->gen_blocks = (uint32_t)(std::max(per_sm, 1) * std::max(sms, 1));
    if (e != cudaSuccess) {
        free_dev(d);
        return e;
    }
    g->dev = d;
    return cudaSuccess;
}

}  // namespace

void gen_dev_free(ltpg_gen *g) {
    free_dev(g->dev);
    g->dev = nullptr;
}

extern "C" {

}  // extern "C"

namespace {

int gen_ycsb(ltpg_ctx *c, ltpg_gen *g, uint64_t batch_id, uint32_t slot, cudaStream_t st) {
    const ltpg_ycsb_params &p = g->y;
    if (cudaSetDevice(c->device) != cudaSuccess) return ctx_fail(c, LTPG_ERR_CUDA, "set device");
    if (p.n_records > c->ycsb.n) return ctx_fail(c, LTPG_ERR_INVALID, "generator keys exceed the loaded table");
    if (g->dev && g->dev->device != c->device)
        return ctx_fail(c, LTPG_ERR_INVALID, "generator tables live on another device");
    Slot *s = nullptr;
    int r = slot_prepare_ycsb(c, slot, p.n_txn, p.ops_per_txn, 0, &s);
    if (r) return r;
    cudaError_t e0 = cudaSuccess;
    if (!g->dev && (e0 = bind_ycsb(g, c->device)) != cudaSuccess) return ctx_cuda_fail(c, e0, "generator tables");
    YcsbGenArgs a;
    a.p = p;
    a.zipf = g->dev->zipf;
    a.tab = g->dev->tab;
    a.cells = g->dev->cells;
    a.rotate = p.rotate_every != 0;
    if (a.rotate) a.perm.init(p.n_records, hash3(p.seed ^ DOM_YCSB_PERM, batch_id / p.rotate_every, 0));
    a.batch_id = batch_id;
    a.ops = s->ops;
    a.val_off = s->val_off;
    a.vals = s->vals;
    const uint32_t stride = ycsb_stride(p.ops_per_txn), warps = g->dev->gen_blocks * (GEN_T / 32);
    // slots as the shared arrays take them, fewer while some warps would get no transaction
    a.tile = std::min(std::min<uint32_t>(32, GEN_WORDS / stride), std::max<uint32_t>(2, blocks(p.n_txn, warps)));
    a.k_inv = (65536u + p.ops_per_txn - 1) / p.ops_per_txn;
    a.s_inv = (65536u + stride - 1) / stride;
    const uint32_t grid = std::min(blocks(blocks(p.n_txn, a.tile), GEN_T / 32), g->dev->gen_blocks);
    // a table of 4 x 2^half rounds pays from as many draws a block as its side is long
    a.perm_table = a.rotate && a.perm.half <= PERM_HALF &&
                   (uint64_t)p.n_txn * p.ops_per_txn / grid >= (1u << a.perm.half);
    // One thread per transaction where that is the faster one (us, threads against
    // slots): cheap draws, i.e. uniform keys in rank order (440,861 x 10: 48 against
    // 73; not in small batches, 8,029 x 32: 33 against 23); transactions that
    // redraw most of their keys (292,566 x 32 of 302 keys at theta 0.999: 1,040
    // against 5,900; not in small batches either); and one or two keys in a small
    // batch (12 against 14).
    const bool small = p.n_txn <= 8192u, uniform = p.theta == 0.0 && !a.rotate;
    const bool threads = (uniform && !small) || (g->dev->repeats && (uniform || !small)) ||
                         (p.n_txn <= 4096u && (p.ops_per_txn == 1u || (p.ops_per_txn == 2u && !a.rotate)));
    if (threads)
        ycsb_gen_ops_txn<<<blocks(p.n_txn, TB), TB, 0, st>>>(a);
    else
        ycsb_gen_ops<<<grid, GEN_T, GEN_BYTES + (a.perm_table ? (4u << a.perm.half) * sizeof(uint16_t) : 0u), st>>>(a);
    count_launch(c);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) {
        const uint32_t nb = blocks(p.n_txn, SCAN_BLOCK);
        uint32_t *blk = s->off_blocks;
        const bool scanned = nb > SCAN_DIRECT;
        scan_blocks<<<nb, SCAN_T, 0, st>>>(s->val_off + 1, p.n_txn, blk);
        if (scanned) scan_totals<<<1, SCAN_T, 0, st>>>(blk, nb);
        ycsb_gen_vals<<<blocks(p.n_txn, TB), TB, 0, st>>>(a, blk, scanned);
        count_launch(c, scanned ? 3 : 2);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? LTPG_OK : ctx_cuda_fail(c, e, "device YCSB generation");
}

int gen_tpcc(ltpg_ctx *c, ltpg_gen *g, uint64_t batch_id, uint32_t slot, cudaStream_t st) {
    if (batch_id != g->next_batch) return ctx_fail(c, LTPG_ERR_STATE, "TPC-C batches are drawn in order");
    const ltpg_tpcc_params &p = g->c;
    if (cudaSetDevice(c->device) != cudaSuccess) return ctx_fail(c, LTPG_ERR_CUDA, "set device");
    if (p.warehouses > c->tpcc.W) return ctx_fail(c, LTPG_ERR_INVALID, "generator warehouses exceed the loaded tables");
    if (g->dev && g->dev->device != c->device)
        return ctx_fail(c, LTPG_ERR_INVALID, "generator state lives on another device");
    const uint64_t max_lines = (uint64_t)p.n_txn * LTPG_TPCC_MAX_LINES;
    if (max_lines > c->cfg.max_lines)
        return ctx_fail(c, LTPG_ERR_INVALID, "device generation needs max_lines >= 15 n_txn");
    Slot *s = nullptr;
    int r = slot_prepare_tpcc(c, slot, p.n_txn, max_lines, g->txn_base, &s);
    if (r) return r;
    slot_pick_registration(c, *s, p.orderstatus_pct || p.delivery_pct);
    cudaError_t e = cudaSuccess;
    if (!g->dev && (e = bind_tpcc(g, c->device)) != cudaSuccess) return ctx_cuda_fail(c, e, "generator state to device");
    ltpg_gen_dev *d = g->dev;
    TpccGenArgs a;
    a.p = p;
    a.batch_id = batch_id;
    a.txn_base = g->txn_base;
    a.B = p.n_txn;
    a.W = p.warehouses;
    a.G = d->G;
    a.C = d->C;
    a.tracking = d->made != nullptr;
    a.o_id = d->o_id;
    a.no_id = d->no_id;
    a.ol_id = d->ol_id;
    a.h_id = d->h_id;
    a.made = d->made;
    a.delivered = d->delivered;
    a.o_cust = d->o_cust;
    a.o_dist = d->o_dist;
    a.o_cnt = d->o_cnt;
    a.o_ol = d->o_ol;
    a.cust_name = d->cust_name;
    a.cust_rank = d->cust_rank;
    a.incl = d->incl;
    a.nob = d->nob;
    a.aux = d->aux;
    a.cc = d->cc;
    a.tot = d->tot;
    a.no_start = d->no_start;
    a.dl_start = d->dl_start;
    a.no_list = d->no_list;
    a.dl_list = d->dl_list;
    a.txns = s->txns;
    a.lines = s->lines;
    a.hdr = s->dev_hdr;
    const uint32_t nb = blocks(a.B, TB);
    uint64_t launches = 0;
    e = cudaMemsetAsync(a.cc, 0, 4ull * a.W * a.G * sizeof(uint32_t), st);
    if (e == cudaSuccess) {
        tpcc_gen_head<<<nb, TB, 0, st>>>(a);
        ++launches;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = inclusive_scan(a.incl, a.B, d->blk, st, launches);
    if (e == cudaSuccess) {
        tpcc_gen_chunk_scan<<<4u * a.W, TB, 0, st>>>(a);
        tpcc_gen_starts<<<1, SCAN_T, 0, st>>>(a);
        tpcc_gen_rank<<<blocks((uint64_t)a.G * 32, TB), TB, 0, st>>>(a);
        tpcc_gen_main<<<nb, TB, 0, st>>>(a);
        launches += 4;
        if (a.tracking) {
            tpcc_gen_dl_walk<<<blocks(32ull * a.W, TB), TB, 0, st>>>(a);
            ++launches;
        }
        tpcc_gen_osdl<<<nb, TB, 0, st>>>(a);
        tpcc_gen_state<<<blocks(std::max(a.B, a.W), TB), TB, 0, st>>>(a);
        launches += 2;
        e = cudaGetLastError();
    }
    count_launch(c, launches);
    if (e != cudaSuccess) return ctx_cuda_fail(c, e, "device TPC-C generation");
    g->txn_base += p.n_txn;
    g->next_batch++;
    return LTPG_OK;
}

}  // namespace

namespace ltpg {
int gen_device_batch(ltpg_ctx *c, ltpg_gen *g, uint64_t batch_id, uint32_t slot, cudaStream_t st) {
    if (!c || !g) return c ? ctx_fail(c, LTPG_ERR_INVALID, "null generator") : LTPG_ERR_INVALID;
    if (g->kind == LTPG_WORKLOAD_YCSB) return gen_ycsb(c, g, batch_id, slot, st);
    if (g->kind == LTPG_WORKLOAD_TPCC) return gen_tpcc(c, g, batch_id, slot, st);
    return ctx_fail(c, LTPG_ERR_INVALID, "unknown generator");
}
}  // namespace ltpg

extern "C" {

int ltpg_gen_ycsb_batch_device(ltpg_ctx *c, ltpg_gen *g, uint64_t batch_id, uint32_t slot) {
    if (!c || !g || g->kind != LTPG_WORKLOAD_YCSB)
        return c ? ctx_fail(c, LTPG_ERR_INVALID, "not a YCSB generator") : LTPG_ERR_INVALID;
    return gen_ycsb(c, g, batch_id, slot, c->stream);
}

int ltpg_gen_tpcc_batch_device(ltpg_ctx *c, ltpg_gen *g, uint64_t batch_id, uint32_t slot) {
    if (!c || !g || g->kind != LTPG_WORKLOAD_TPCC)
        return c ? ctx_fail(c, LTPG_ERR_INVALID, "not a TPC-C generator") : LTPG_ERR_INVALID;
    return gen_tpcc(c, g, batch_id, slot, c->stream);
}

}  // extern "C"
