// ycsb_tuned.cu — tuned YCSB path: fused kernels, CUDA-graph and persistent modes.
//
// Same protocol and outputs as the plain path (ycsb.cu); only the schedule
// changes:
//   * execute+register takes one op per lane, the rows read five lanes to a row
//     (or two or four ops per thread);
//   * a registration goes (a) to a shared-memory staging entry when the
//     predictor marked its key's bucket hot, else (b) through a dedupe (only
//     the smallest TID of each key in the block or the warp issues: batches of
//     a few waves, or a launch setting), then (c) an L1 read of the slot skips
//     the atomic when the slot already holds a smaller value.  Slot values only
//     decrease (newer batch tags are smaller, and within a batch atomicMin only
//     lowers), so any value observed, stale or not, is >= the current one: the
//     skip is exact;
//   * check and write-back run in one kernel: the commit decision of a tile is
//     made in shared memory, then the threads that hold a committed
//     transaction's op vectors store its updates, in op order;
//   * late reads (a launch setting): execute only registers, the check kernel
//     reads the rows of the committed transactions after the tile's commit
//     decision, and a third kernel stores the updates, so that no aborted
//     transaction's rows are read;
//   * write-first registration (late reads 3): the updates register first,
//     then each read touches its key's slot only when an update writes the
//     key; the read registration also lists the updates by value index, and
//     the check and the write-back walk that list instead of the op words.
#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "stage.cuh"

namespace ltpg {

struct YcsbTunedArgs {
    const uint32_t *ops;
    const uint32_t *val_off;
    const uint64_t *vals;
    uint32_t B, k, stride, tile;  // tile = transactions per block tile (multiple of 32)
    uint64_t *rows;
    uint64_t n;
    RegSlot *reg;
    int64_t *results;
    uint8_t *flags;
    uint32_t *bitmap;
    DevStats *st;
    DevCtl *ctl;
    const uint16_t *stage_map;
    const uint32_t *stage_bits;
    const uint32_t *stage_rank;
    uint32_t *bucket_counts;
    uint32_t ways, stage_entries;
    uint32_t filter;
    uint32_t grp;  // transactions of a warp's step in the cooperative execute kernel: 32 / k
    uint32_t lpt;  // lanes per transaction of the late reads: stride (at most 32) rounded up to a power of two
    uint32_t late; // late reads: 0 off, 1 in the check kernel's tiles, 2 in a kernel of their own,
                   // 3 write-first registration
    uint32_t *wbits;  // write-first: one bit per key, set for keys an update of the batch writes
    uint2 *upd;        // write-first update list: entry u = {TID, op word} of the u-th update (0 entries: none)
    uint64_t upd_cap;  // entries of the update list
    uint64_t vals_cap; // values the slot holds (bound of every value index)
};

__device__ __forceinline__ uint64_t ld_ca_u64(const unsigned long long *p) {
    uint64_t v;
    asm volatile("ld.global.ca.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ld_ca_u32(const unsigned *p) {
    uint32_t v;
    asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// kCoh (the persistent kernel, where the phases share one launch): every
// load of a word that an earlier phase of the launch wrote, or that this
// phase writes (slots, writer bits, flag bytes), is a GPU-scope relaxed load
// served by L2 (ld_gpu_*), never an L1 or read-only-path load, which could
// return a line cached before the grid barrier.  Op words, values and rows
// (read before the write-back) are written by no phase and keep the
// read-only path.  In the separate kernels L1 starts empty at every kernel.
// One exception: checkwb_tiles loads the slots through L1 in the persistent
// kernel too.  No thread loads a slot between its block's arrival at the grid
// barrier and the barrier's fence (thread 0's __threadfence behind the wait,
// then __syncthreads), after which a load does not see what L1 held before.
template <bool kCoh>
__device__ __forceinline__ uint64_t ld_filter_u64(const unsigned long long *p) {
    return kCoh ? ld_gpu_u64(p) : ld_ca_u64(p);
}
template <bool kCoh>
__device__ __forceinline__ uint32_t ld_wbits(const uint32_t *p) {
    return kCoh ? ld_gpu_u32(p) : __ldg(p);
}
template <bool kCoh>
__device__ __forceinline__ uint32_t ld_flag(const uint8_t *p) {
    return kCoh ? ld_gpu_u8(p) : (uint32_t)*p;
}

// Stores the updates of committed transaction t in op order: a transaction
// that updates a field twice leaves its later value (as a sequential replay
// does), and no two committed transactions write one row (WAW).
__device__ __forceinline__ void write_txn_updates(const YcsbTunedArgs &a, uint32_t t) {
    uint32_t v = a.val_off[t];
    if (v == a.val_off[t + 1]) return;
    // value indices stay below the batch's value count and the slot's
    // capacity: offsets that disagree with the op words are reported
    const uint64_t nv = min((uint64_t)__ldg(a.val_off + a.B), a.vals_cap);
    const uint4 *tw = reinterpret_cast<const uint4 *>(a.ops + (uint64_t)t * a.stride);
    for (uint32_t q4 = 0; q4 < a.stride / 4u; ++q4) {
        const uint4 w4 = ld_nc_u4(tw + q4);
        const uint32_t words[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t x = words[q];
            if (ycsb_is_pad(x) || !ycsb_is_update(x)) continue;
            const uint32_t key = ycsb_key(x), fld = ycsb_field(x);
            if (v >= nv) {
                report_error(a.ctl, DERR_BOUNDS, t);
                return;
            }
            if (key < a.n && fld < LTPG_YCSB_FIELDS) a.rows[(uint64_t)key * LTPG_YCSB_FIELDS + fld] = a.vals[v];
            ++v;
        }
    }
}

// Row gather of a warp: the rows of up to 32 keys, five lanes to a row (one
// 16-byte chunk each, six rows per round on lanes 0..29), so a row costs one or
// two cache-line requests.  `need` (a ballot) names the lanes that want a row;
// a lane's rank among them is its row's number.  Per-warp shared scratch: the
// keys by rank, and each chunk's xor at 5 * rank + chunk = 30 * round + lane,
// from where a row's owner folds its five (stride 40 bytes: no bank conflict).
// Folding through shared memory takes one store per round and five loads per
// warp, where shuffles took six per round: the late-read kernel was issue-bound
// (2^20 x 16 at theta 0.99: 190 -> 172 us, 100 G random sectors/s of DRAM; a
// 10,000 x 10 persistent batch with reads at execute 27.6 -> 25.2 us).
// Three rounds (18 rows) are folded at a time, which keeps the scratch of a
// 256-thread block below 7 KB (what shared memory takes, L1 loses).
struct RowScratch {
    uint32_t key[32];
    unsigned long long part[90];
};

// This warp's scratch; one array per kernel, whichever row-reading loops it
// runs, sized by the kernel's launch bounds.
template <int BS>
__device__ __forceinline__ RowScratch *row_scratch() {
    __shared__ RowScratch scratch[BS / 32];
    return scratch + (threadIdx.x >> 5);
}

// Puts the keys in place and issues every chunk load of the gather.
__device__ __forceinline__ void rows_issue(const uint64_t *rows, RowScratch *ws, uint32_t key, unsigned need,
                                           ulonglong2 *ch) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n5 = lane < 30u ? 5u * __popc(need) : 0u;
    if ((need >> lane) & 1u) ws->key[__popc(need & ((1u << lane) - 1u))] = key;
    __syncwarp();
    const char *base = reinterpret_cast<const char *>(rows) + 16u * (lane % 5u);
    const uint32_t grp = lane / 5u;
#pragma unroll
    for (uint32_t r = 0; r < 6; ++r) {
        ch[r] = make_ulonglong2(0ull, 0ull);
        if (30u * r + lane < n5)
            ch[r] = ld_nc16_issue(base + (uint64_t)ws->key[6u * r + grp] * (8u * LTPG_YCSB_FIELDS));
    }
}

// The xor of the row of each lane in `need` (0 for the other lanes).
__device__ __forceinline__ unsigned long long rows_fold(RowScratch *ws, unsigned need, const ulonglong2 *ch) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n = __popc(need), n5 = lane < 30u ? 5u * n : 0u;
    const uint32_t rank = __popc(need & ((1u << lane) - 1u));
    unsigned long long x = 0;
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        if (h) {
            if (n <= 18u) break;  // warp-uniform
            __syncwarp();
        }
#pragma unroll
        for (uint32_t r = 0; r < 3; ++r)
            if (90u * h + 30u * r + lane < n5) ws->part[30u * r + lane] = ch[3u * h + r].x ^ ch[3u * h + r].y;
        __syncwarp();
        if (((need >> lane) & 1u) && rank - 18u * h < 18u) {
            const unsigned long long *p = ws->part + 5u * (rank - 18u * h);
            x = p[0] ^ p[1] ^ p[2] ^ p[3] ^ p[4];
        }
    }
    // the next gather writes `part` after its own barrier, and `key` before it:
    // every key was read before this fold's first barrier
    return x;
}

// The same gather with no shared memory: round r searches the ballot for the
// (6r + g)-th row of group g, and shuffles fold the chunks and hand the row's
// xor to its owner.  The staged kernels use it: their table takes 48 KB a
// block, and its shared-memory atomics queue behind the other form's stores and
// loads (2^18 x 16 at theta 0.99, 42 % of the ops staged: 228 us against 304).
__device__ __forceinline__ void rows_issue_shfl(const uint64_t *rows, uint32_t key, unsigned need, ulonglong2 *ch) {
    const uint32_t lane = threadIdx.x & 31, grp = lane / 5u, n = __popc(need);
#pragma unroll
    for (uint32_t r = 0; r < 6; ++r) {
        const uint32_t idx = r * 6u + grp;
        const bool go = grp < 6u && idx < n;
        const uint32_t src = go ? __fns(need, 0, (int)idx + 1) : 0u;
        const uint32_t k_src = __shfl_sync(FULL, key, src & 31u);
        ch[r] = go ? ld_nc16_issue(reinterpret_cast<const char *>(rows + (uint64_t)k_src * LTPG_YCSB_FIELDS) +
                                   16u * (lane % 5u))
                   : make_ulonglong2(0ull, 0ull);
    }
}
__device__ __forceinline__ unsigned long long rows_fold_shfl(unsigned need, const ulonglong2 *ch) {
    const uint32_t lane = threadIdx.x & 31, n = __popc(need), rank = __popc(need & ((1u << lane) - 1u));
    unsigned long long x = 0;
#pragma unroll
    for (uint32_t r = 0; r < 6; ++r) {
        if (r * 6u >= n) break;  // warp-uniform
        // lane 5g: chunks 0 and 1, then 0..3, then chunk 4
        const unsigned long long c0 = ch[r].x ^ ch[r].y;
        unsigned long long c = c0 ^ __shfl_down_sync(FULL, c0, 1);
        c ^= __shfl_down_sync(FULL, c, 2);
        const unsigned long long rowx = c ^ __shfl_down_sync(FULL, c0, 4);
        const unsigned long long got = __shfl_sync(FULL, rowx, ((rank - r * 6u) * 5u) & 31u);
        if (((need >> lane) & 1u) && rank - r * 6u < 6u) x = got;
    }
    return x;
}

// The xor of the rows of each lane's scan in `scans` (the other lanes keep x):
// eight lanes to a scan, four scans at a time, each lane loading the 16-byte
// chunks of its place in the 128-byte lines that the scan's rows cover, four
// lines in flight.  Instructions bound it: a whole warp to a scan folded five
// levels of shuffles for two loads, and waited for them before the next scan's
// (2^18 x 10 scans of 10 keys at theta 0.99: 291 -> 153 us).
__device__ __forceinline__ unsigned long long scans_fold(const YcsbTunedArgs &a, RowScratch *ws, uint32_t w,
                                                         unsigned scans, unsigned long long x) {
    const uint32_t lane = threadIdx.x & 31, l = lane & 7u, n = __popc(scans);
    const uint32_t rank = __popc(scans & ((1u << lane) - 1u));
    const bool own = (scans >> lane) & 1u;
    const uint32_t key = ycsb_key(w);
    __syncwarp();  // the point reads' fold is over
    if (own) ws->key[rank] = key | ((uint32_t)scan_last(w, a.n) - key) << LTPG_YCSB_KEY_BITS;
    __syncwarp();
    for (uint32_t base = 0; base < n; base += 4u) {
        const uint32_t i = base + (lane >> 3);
        unsigned long long c = 0;
        if (i < n) {
            const uint32_t e = ws->key[i];
            const uint64_t first = (uint64_t)(e & ((1u << LTPG_YCSB_KEY_BITS) - 1u)) * 5u;  // in chunks of the table
            const uint32_t off = (uint32_t)first & 7u, end = off + ((e >> LTPG_YCSB_KEY_BITS) + 1u) * 5u;
            const ulonglong2 *p = reinterpret_cast<const ulonglong2 *>(a.rows) + (first - off);
            for (uint32_t q = l; q < end; q += 32u) {
                ulonglong2 v[4];
#pragma unroll
                for (uint32_t r = 0; r < 4; ++r) {
                    const uint32_t at = q + 8u * r;
                    v[r] = at >= off && at < end ? ld_nc16_issue(p + at) : make_ulonglong2(0ull, 0ull);
                }
#pragma unroll
                for (uint32_t r = 0; r < 4; ++r) c ^= v[r].x ^ v[r].y;
            }
        }
#pragma unroll
        for (uint32_t o = 4; o >= 1u; o >>= 1) c ^= __shfl_xor_sync(FULL, c, o);
        if (l == 0u && i < n) ws->part[i] = c;
    }
    __syncwarp();
    return own ? ws->part[rank] : x;
}

// Late reads of one tile whose commit flags are in fl: the lpt lanes of a
// transaction (a power of two, aligned in the warp) take one op each; the
// point reads of committed transactions are gathered five lanes to a row (one
// 16-byte chunk each, six rows per round), range scans eight
// lanes to a scan.  results[t] = sum over reads of xor(row) * (2j + 1), as
// at execute; 0 for an aborted transaction.  No row is written before the
// next kernel, so every read sees the batch-start image.
//
// One step of the lanes of a warp (all 32 call it): lane j of transaction t
// (own: the lane holds an op slot of a transaction; com: t committed).
__device__ __forceinline__ void late_read_step(const YcsbTunedArgs &a, RowScratch *ws, uint32_t t, uint32_t j,
                                               bool own, bool com) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lpt = a.lpt;
    {
        const uint32_t w = com && j < a.stride ? __ldg(a.ops + (uint64_t)t * a.stride + j) : LTPG_YCSB_OP_PAD;
        const uint32_t key = ycsb_key(w);
        const bool rd = !ycsb_is_pad(w) && !ycsb_is_update(w) && key < a.n;
        const bool scan = rd && ycsb_span(w) != 0u;
        const unsigned need = __ballot_sync(FULL, rd && !scan);
        unsigned long long x = 0;
        if (need) {  // warp-uniform
            ulonglong2 ch[6];
            rows_issue(a.rows, ws, key, need, ch);
            x = rows_fold(ws, need, ch);
        }
        const unsigned scans = __ballot_sync(FULL, scan);
        if (scans) x = scans_fold(a, ws, w, scans, x);  // warp-uniform
        unsigned long long part = rd ? x * (2ull * j + 1ull) : 0ull;
        for (uint32_t o = lpt >> 1; o >= 1; o >>= 1) part += __shfl_xor_sync(FULL, part, o);
        if (own && j == 0u) a.results[t] = (int64_t)part;
    }
}

__device__ __forceinline__ void late_read_tile(const YcsbTunedArgs &a, RowScratch *ws, const uint32_t *fl, uint32_t t0,
                                               uint32_t nt) {
    const uint32_t lsh = (uint32_t)__ffs(a.lpt) - 1u;
    const uint32_t nl = a.tile << lsh;
    for (uint32_t base = 0; base < nl; base += blockDim.x) {
        const uint32_t v = base + threadIdx.x;
        const uint32_t lt = v >> lsh, j = v & (a.lpt - 1u);
        const bool own = v < nl && lt < nt;
        late_read_step(a, ws, t0 + lt, j, own, own && (fl[lt] & LTPG_FLAG_COMMIT) != 0u);
    }
}

// Late reads as a kernel of their own (late_reads = 2), after the check: the
// lanes of the whole batch, lpt per transaction, commit flags from global memory.
template <bool kCoh>
__device__ __forceinline__ void late_read_loop(const YcsbTunedArgs &a, RowScratch *ws) {
    const uint32_t lsh = (uint32_t)__ffs(a.lpt) - 1u;
    const uint64_t nw = (uint64_t)a.B << lsh;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < nw; base += step) {
        const uint64_t v = base + threadIdx.x;
        const bool own = v < nw;
        const uint32_t t = (uint32_t)(v >> lsh), j = (uint32_t)v & (a.lpt - 1u);
        // the commit decision from the conflict bits (the check kernel of late
        // reads 2 also set COMMIT; write-first leaves it to the write-back)
        late_read_step(a, ws, t, j, own,
                       own && commits(ld_flag<kCoh>(a.flags + t) & (LTPG_FLAG_RAW | LTPG_FLAG_WAR | LTPG_FLAG_WAW)));
    }
}

// The grid-stride kernels below are instantiated per block size (BS = 128,
// 256, 512: launch setting block_threads), each with launch bounds of its own
// block: bounds above the block change the compiler's register choice.  The
// read kernel is held to 1,280 threads an SM (48 registers): left alone it took
// 32 and waited for each pair of rows (2^20 x 16 at theta 0.99 172 us against
// 169, scans 170 against 153); for 1,536 threads (40) 179 and 145.
template <int BS>
__global__ void __launch_bounds__(BS, 1280 / BS) ycsb_read_late(YcsbTunedArgs a) {
    late_read_loop<false>(a, row_scratch<BS>());
}

// ---- write-first registration (late_reads = 3) ---------------------------------
// The same RAW / WAR / WAW outcome with at most one random slot access per op
// instead of two.  (1) The updates register (write word) and set their key's
// bit in a writer bitmap.  (2) A read whose key has no writer in the batch has
// no RAW and no WAR to cause, and touches no slot; any other read loads its
// key's slot once: the write word is final, so RAW = (smallest writer < t),
// and the read registers in the read word.  A key with a writer thus gets
// every one of its reads registered, as in the protocol.  (3) The updates load
// their slot for WAR and WAW.  The flag bytes collect the conflict bits of (2)
// and (3).  (4) The committed reads gather their rows (late_read_loop; commit
// from the conflict bits); (5) the write-back decides the commits, writes the
// final flags, bitmap and counters, and stores.  Checking the updates in a
// kernel of their own keeps their slot loads out of the path of the row
// reads: 81 % of the warps of a 16-op, 5 %-update batch hold an update.

// 16-byte slot load through L1: the write words are final after (1), and L1
// is invalidated between dependent kernels; a read word seen stale is never
// below the current one, so skipping a red.min on it stays exact.
__device__ __forceinline__ ulonglong2 ld_slot_ca(const RegSlot *p) {
    ulonglong2 v;
    asm volatile("ld.global.ca.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}

constexpr uint32_t WF_FEW = 16;  // of a warp's 128 ops
// (1) the updates' registrations and writer bits: four op words per thread
// (transactions are 4-word aligned); every op's key is bounds-checked here.
// Also zeroes the flag bytes, which (2) and (3) OR the conflict bits into.
template <bool kCoh>
__device__ __forceinline__ void wf_register_writes(const YcsbTunedArgs &a, uint64_t tag) {
    // at most 2^26 transactions of 8 vectors: 32-bit indices (and divisions)
    const uint32_t vpt = a.stride / 4u, nvec = a.B * vpt;
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (a.B + 3u) / 4u; i += step)
        reinterpret_cast<unsigned *>(a.flags)[i] = 0u;
    const uint4 *vp = reinterpret_cast<const uint4 *>(a.ops);
    // a block-uniform loop, so that whole warps reach the warp-wide sum below
    for (uint32_t base = blockIdx.x * blockDim.x; base < nvec; base += step) {
        const uint32_t v = base + threadIdx.x;
        const uint4 w4 = v < nvec ? ld_nc_u4(vp + v)
                                  : make_uint4(LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD);
        const uint32_t t = v / vpt;
        const uint32_t words[4] = {w4.x, w4.y, w4.z, w4.w};
        const unsigned long long mine = tag | t;
        bool upd[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t w = words[q];
            upd[q] = !ycsb_is_pad(w) && ycsb_is_update(w) && ycsb_key(w) < a.n;
            if (!ycsb_is_pad(w) && ycsb_key(w) >= a.n) report_error(a.ctl, DERR_BOUNDS, t);
        }
        auto slot_of = [&](int q) { return &a.reg[ycsb_key(words[q])].w; };
        auto look_slot = [&](int q) { return upd[q] && a.filter ? ld_filter_u64<kCoh>(slot_of(q)) : ~0ull; };
        auto look_bit = [&](int q) {
            unsigned *bw = a.wbits + (ycsb_key(words[q]) >> 5);
            return !upd[q] ? ~0u : kCoh ? ld_gpu_u32(bw) : ld_ca_u32(bw);
        };
        // bits are only set within a batch: a bit seen set needs no atomic
        // (hot keys' updates would otherwise all hit one word)
        auto set_bit = [&](int q, uint32_t seen) {
            const uint32_t key = ycsb_key(words[q]);
            if (!((seen >> (key & 31u)) & 1u)) atomicOr(a.wbits + (key >> 5), 1u << (key & 31u));
        };
        // Few updates in the warp: the looks of a vector are in flight together, as
        // one after another they were this pass (2^20 x 16, 5 % updates: 36 -> 27
        // us; 50 -> 34 at theta 0).  Many: one op after another, as a look that
        // comes after the sends before it finds the hot keys registered; together
        // every update of a hot key was sent and queued at its slot (65,536 x 16 at
        // theta 0.99, two batches, half updates: 163 us together, 78 so; all
        // updates 288 and 134).
        if (__reduce_add_sync(FULL, (uint32_t)upd[0] + upd[1] + upd[2] + upd[3]) <= WF_FEW) {
            uint64_t cur[4];
            uint32_t seen[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                cur[q] = look_slot(q);
                seen[q] = look_bit(q);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (upd[q] && cur[q] > mine) red_min(slot_of(q), mine);
                set_bit(q, seen[q]);
            }
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (!upd[q]) continue;
                if (look_slot(q) > mine) red_min(slot_of(q), mine);
                set_bit(q, look_bit(q));
            }
        }
    }
}

// One key of a read that has a writer: RAW against the final write word, and
// the read's registration.  Returns the RAW bit.
__device__ __forceinline__ bool wf_read_key(const YcsbTunedArgs &a, uint32_t key, uint32_t t,
                                            uint32_t epoch, const ulonglong2 &s) {
    const unsigned long long mine = slot_tag(epoch) | t;
    const uint32_t wmin = slot_min(s.y, epoch);
    if (wmin != 0xFFFFFFFFu && s.x > mine) red_min(&a.reg[key].r, mine);
    return wmin < t;
}
template <bool kCoh>
__device__ __forceinline__ ulonglong2 ld_reg(const RegSlot *p) {
    return kCoh ? ld_gpu_slot(p) : ld_slot_ca(p);
}

// The keys of a range scan after its first (at most 15): their writer bits are
// in one or two bitmap words, and only the keys with a writer are looked at
// (2^18 x 10 scans of 10 keys: registration 73 -> 54 us; one dependent bitmap
// load per key before).
template <bool kCoh>
__device__ __forceinline__ bool wf_read_rest(const YcsbTunedArgs &a, uint32_t w, uint32_t t,
                                             uint32_t epoch) {
    const uint32_t k1 = ycsb_key(w) + 1u, last = (uint32_t)scan_last(w, a.n);
    if (last < k1) return false;  // a scan of the table's last key
    const uint32_t lo = k1 >> 5, hi = last >> 5;
    uint64_t win = ld_wbits<kCoh>(a.wbits + lo);
    if (hi != lo) win |= (uint64_t)ld_wbits<kCoh>(a.wbits + hi) << 32;
    uint32_t m = (uint32_t)(win >> (k1 & 31u)) & ((2u << (last - k1)) - 1u);
    bool raw = false;
    for (; m; m &= m - 1u) {
        const uint32_t key = k1 + (uint32_t)__ffs(m) - 1u;
        raw |= wf_read_key(a, key, t, epoch, ld_reg<kCoh>(a.reg + key));
    }
    return raw;
}

// The update list: the batch's u-th update (u = its value index, val_off[t]
// + its rank among transaction t's updates) is stored as {t, op word}, so that
// the check and the write-back walk the updates alone instead of every op word.
// A lane holds op vector seg of its transaction (vpt = stride / 4 vectors, at
// most 8).  With vpt a power of two the transaction's vectors are consecutive
// lanes of one warp and a segmented scan gives each lane the updates of the
// earlier vectors; otherwise the lane counts them in those vectors itself
// (loads that its neighbours made a moment before).  The transaction's last
// lane checks its update count against its value range: the list positions are
// only as good as val_off, so a batch whose offsets disagree with its op words
// is reported (LTPG_ERR_BOUNDS) and its positions are never used past the
// list.  Called by whole warps.
__device__ __forceinline__ uint32_t vec_updates(const uint32_t *w) {
    uint32_t n = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) n += (!ycsb_is_pad(w[q]) && ycsb_is_update(w[q])) ? 1u : 0u;
    return n;
}
__device__ __forceinline__ void wf_list_updates(const YcsbTunedArgs &a, bool act, uint32_t v, uint32_t t,
                                                const uint32_t *words) {
    const uint32_t vpt = a.stride / 4u, seg = act ? v - t * vpt : v % vpt;
    const bool pow2 = (vpt & (vpt - 1u)) == 0u;
    const uint32_t off = act ? __ldg(a.val_off + t) : 0u;
    const uint32_t end = act && seg == vpt - 1u ? __ldg(a.val_off + t + 1) : 0u;
    const uint32_t n_upd = vec_updates(words);
    uint32_t incl = n_upd;
    if (pow2) {
        for (uint32_t o = 1; o < vpt; o <<= 1) {
            const uint32_t x = __shfl_up_sync(FULL, incl, o);
            if (seg >= o) incl += x;
        }
    } else if (act) {
        const uint4 *vp = reinterpret_cast<const uint4 *>(a.ops) + (v - seg);
        for (uint32_t q = 0; q < seg; ++q) {
            const uint4 w4 = ld_nc_u4(vp + q);
            const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
            incl += vec_updates(w);
        }
    }
    if (act && seg == vpt - 1u && end - off != incl) report_error(a.ctl, DERR_BOUNDS, t);
    uint64_t u = (uint64_t)off + (incl - n_upd);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (!act || ycsb_is_pad(words[q]) || !ycsb_is_update(words[q])) continue;
        if (u < a.upd_cap) a.upd[u] = make_uint2(t, words[q]);
        else report_error(a.ctl, DERR_BOUNDS, t);
        ++u;
    }
}

// (2) reads: four op words per thread (one 16-byte load); the writer-bitmap
// words of the thread's reads are loaded together, then the slots of those
// with a writer; the RAW bit is OR-ed into the transaction's flag byte
// (zeroed by (1)) with a 32-bit atomic.
// kList: the pass also writes the update list (wf_list_updates); its stores
// wait behind the slot loads this pass is bound by.  Transactions t0 .. t1 - 1.
template <bool kCoh, bool kList = false>
__device__ __forceinline__ void wf_register_reads(const YcsbTunedArgs &a, uint32_t epoch, uint32_t t0, uint32_t t1) {
    const uint32_t vpt = a.stride / 4u, nvec = t1 * vpt;
    const uint32_t step = gridDim.x * blockDim.x;
    const uint4 *vp = reinterpret_cast<const uint4 *>(a.ops);
    // a block-uniform loop, so that whole warps reach the warp-wide calls below
    for (uint32_t base = t0 * vpt + blockIdx.x * blockDim.x; base < nvec; base += step) {
        const uint32_t v = base + threadIdx.x;
        const bool act = v < nvec;
        const uint4 w4 = act ? ld_nc_u4(vp + v)
                             : make_uint4(LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD);
        const uint32_t t = act ? v / vpt : 0xFFFFFFFFu;
        const uint32_t words[4] = {w4.x, w4.y, w4.z, w4.w};
        if (kList) wf_list_updates(a, act, v, t, words);
        bool rd[4];
        uint32_t bits[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t w = words[q], key = ycsb_key(w);
            rd[q] = !ycsb_is_pad(w) && !ycsb_is_update(w) && key < a.n;
            bits[q] = rd[q] ? ld_wbits<kCoh>(a.wbits + (key >> 5)) : 0u;
        }
        ulonglong2 s[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t key = ycsb_key(words[q]);
            s[q] = (bits[q] >> (key & 31u)) & 1u ? ld_reg<kCoh>(a.reg + key) : make_ulonglong2(~0ull, ~0ull);
        }
        bool raw = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            raw |= wf_read_key(a, ycsb_key(words[q]), t, epoch, s[q]);
            if (rd[q] && ycsb_span(words[q])) raw |= wf_read_rest<kCoh>(a, words[q], t, epoch);
        }
        // one atomic per transaction: the lowest of its threads in the warp
        // ORs the bit when any of them saw RAW
        const unsigned peers = __match_any_sync(FULL, t);
        const bool any = (__ballot_sync(FULL, raw) & peers) != 0u;
        if (act && any && (threadIdx.x & 31u) == (uint32_t)__ffs(peers) - 1u)
            atomicOr(reinterpret_cast<unsigned *>(a.flags) + (t >> 2), LTPG_FLAG_RAW << (8u * (t & 3u)));
    }
}


template <int BS>
__global__ void __launch_bounds__(BS) ycsb_wf_writes(YcsbTunedArgs a) {
    clear_stats(a.st);
    wf_register_writes<false>(a, slot_tag(a.ctl->epoch));
}

// ---- write-first with the update list (stride / 4 a power of two <= 8) --------
template <int BS>
__global__ void __launch_bounds__(BS) ycsb_wf_reads_list(YcsbTunedArgs a, uint32_t t0, uint32_t t1) {
    let_next_start();
    wait_for_previous();
    wf_register_reads<false, true>(a, a.ctl->epoch, t0, t1);
}

// Entries of the batch's update list: val_off[B], bounded by the list.
__device__ __forceinline__ uint64_t upd_count(const YcsbTunedArgs &a) {
    const uint64_t n = __ldg(a.val_off + a.B);
    return n < a.upd_cap ? n : a.upd_cap;
}

// (3) over the update list: each update's WAR / WAW, OR-ed into its
// transaction's flag byte.  Four entries per thread and step, their entry and
// slot loads issued together.
// An entry of the update list; kCoh: written earlier in the same launch (the
// persistent kernel), so loaded coherently at L2.
template <bool kCoh>
__device__ __forceinline__ uint2 ld_upd(const uint2 *p) {
    return kCoh ? ld_gpu_u2(p) : __ldg(p);
}

template <bool kCoh>
__device__ __forceinline__ void wf_check_list(const YcsbTunedArgs &a, uint32_t epoch) {
    const uint64_t nu = upd_count(a);
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t u0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u0 < nu; u0 += 4 * step) {
        uint2 e[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t u = u0 + (uint64_t)q * step;
            e[q] = u < nu ? ld_upd<kCoh>(a.upd + u) : make_uint2(0xFFFFFFFFu, 0u);
        }
        bool ok[4];
        ulonglong2 sl[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            ok[q] = e[q].x < a.B && ycsb_key(e[q].y) < a.n;
            sl[q] = ok[q] ? (kCoh ? ld_gpu_slot(a.reg + ycsb_key(e[q].y)) : ld_slot(a.reg + ycsb_key(e[q].y)))
                          : make_ulonglong2(~0ull, ~0ull);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t f = 0;
            if (slot_min(sl[q].x, epoch) < e[q].x) f |= LTPG_FLAG_WAR;
            if (slot_min(sl[q].y, epoch) < e[q].x) f |= LTPG_FLAG_WAW;
            if (ok[q] && f)
                atomicOr(reinterpret_cast<unsigned *>(a.flags) + (e[q].x >> 2), f << (8u * (e[q].x & 3u)));
        }
    }
}
template <int BS>
__global__ void __launch_bounds__(BS) ycsb_wf_check_list(YcsbTunedArgs a) { wf_check_list<false>(a, a.ctl->epoch); }

// Shared memory layout: [off: tile + 1 u32][fl: tile u32][upd: tile * stride / 4
// bytes, the updates of each op vector][stage table]; a tile is a multiple of 32.
__host__ __device__ __forceinline__ size_t ycsb_smem_bytes(uint32_t tile, uint32_t stride, uint32_t stage_entries) {
    return (size_t)tile * 8 + 16 + (size_t)tile * (stride / 4u) + (size_t)stage_entries * sizeof(StageEnt);
}

struct SmemPtrs {
    uint32_t *off, *fl;
    uint8_t *upd;
    StageEnt *tab;
};
__device__ __forceinline__ SmemPtrs carve(char *base, uint32_t tile, uint32_t stride) {
    SmemPtrs p;
    p.off = reinterpret_cast<uint32_t *>(base);
    p.fl = reinterpret_cast<uint32_t *>(base + (size_t)tile * 4 + 16);
    p.upd = reinterpret_cast<uint8_t *>(p.fl + tile);
    p.tab = reinterpret_cast<StageEnt *>(base + ycsb_smem_bytes(tile, stride, 0));
    return p;
}

// ---- check + write-back over all tiles assigned to this block ------------------
// fl: tile flags; off: the tile's value offsets.  kLate = 0: the third pass
// stores the committed updates; 1: it reads the committed transactions' rows
// (late_read_tile); 2: there is no third pass (the reads have a kernel of their
// own).  With late reads the updates are stored by a later kernel.
// Each pass is a chain of dependent loads, which bounds a batch of one wave, so
// a thread issues two slot loads together, the value offsets are on their way
// during the check, and an update is stored by the thread that holds its op
// word (one thread per transaction took its vectors in turn).  Slots come
// through L1: a hot key's is loaded by every warp, and its L2 slice was the
// bound at high skew.  In the persistent kernel the grid barrier's fences order
// these loads behind the registrations.  (65,536 x 10, half updates: theta 0.6
// 17 -> 12.4 us, 0.99 25 -> 11 us; 2^18 x 10 of 10 M at 0.99: 79 -> 33 us;
// 2,000 x 10: 10 -> 8.3 us.)
__device__ __forceinline__ ulonglong2 ld_slot_if(bool on, const RegSlot *p) {
    ulonglong2 v = make_ulonglong2(~0ull, ~0ull);  // nobody's
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %3, 0; @q ld.global.ca.v2.u64 {%0, %1}, [%2]; }"
                 : "+l"(v.x), "+l"(v.y) : "l"(p), "r"((uint32_t)on));
    return v;
}

template <int kLate>
__device__ __forceinline__ void checkwb_tiles(const YcsbTunedArgs &a, const SmemPtrs &sm, RowScratch *ws,
                                              uint32_t epoch) {
    uint32_t *fl = sm.fl, *off = sm.off;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t vpt = a.stride / 4;  // vectors of a transaction
    const uint32_t n_tiles = (a.B + a.tile - 1) / a.tile;
    const uint64_t nv = kLate ? 0ull : min((uint64_t)__ldg(a.val_off + a.B), a.vals_cap);
    TxnCounts cnt;
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t t0 = tile * a.tile;
        const uint32_t nt = min(a.tile, a.B - t0);
        const uint32_t nvec = nt * vpt;
        const uint4 *vp = reinterpret_cast<const uint4 *>(a.ops + (uint64_t)t0 * a.stride);
        uint4 w4 = make_uint4(0u, 0u, 0u, 0u);
        if (threadIdx.x < nvec) w4 = ld_nc_u4(vp + threadIdx.x);
        for (uint32_t i = threadIdx.x; i < a.tile; i += blockDim.x) fl[i] = 0u;
        if (!kLate)
            for (uint32_t i = threadIdx.x; i <= nt; i += blockDim.x) off[i] = __ldg(a.val_off + t0 + i);
        __syncthreads();
        // pass 1: conflict flags per transaction
        for (uint32_t v = threadIdx.x; v < nvec; v += blockDim.x) {
            const uint32_t lt = v / vpt, t = t0 + lt;
            if (v >= blockDim.x) w4 = ld_nc_u4(vp + v);
            const uint32_t words[4] = {w4.x, w4.y, w4.z, w4.w};
            uint32_t f = 0, scans = 0;
            ulonglong2 s[2];  // two slots in flight: four take the registers of a block
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q % 2 == 0)
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        s[r] = ld_slot_if(!ycsb_is_pad(words[q + r]) && ycsb_key(words[q + r]) < a.n,
                                          a.reg + ycsb_key(words[q + r]));
                const uint32_t w = words[q];
                const uint32_t rmin = slot_min(s[q % 2].x, epoch), wmin = slot_min(s[q % 2].y, epoch);
                if (ycsb_is_update(w)) {
                    if (rmin < t) f |= LTPG_FLAG_WAR;
                    if (wmin < t) f |= LTPG_FLAG_WAW;
                } else {
                    if (wmin < t) f |= LTPG_FLAG_RAW;
                    if (ycsb_span(w) && !ycsb_is_pad(w) && ycsb_key(w) < a.n) {
                        if (kLate != 1) scans |= 1u << q;
                        else if (!(f & LTPG_FLAG_RAW) && scan_rest_raw(a.reg, a.n, w, t, epoch)) f |= LTPG_FLAG_RAW;
                    }
                }
            }
            // range scans' other keys, out of the loop above: inside it they left
            // one slot load in flight at 40 registers.  Not with late reads 1, which
            // has more and whose row reads lost some of theirs to it (60,942 x 32
            // persistent 84 -> 88 us).
            for (; scans && !(f & LTPG_FLAG_RAW); scans &= scans - 1u) {
                const uint32_t q = (uint32_t)__ffs(scans) - 1u;
                const uint32_t w = q & 2u ? (q & 1u ? w4.w : w4.z) : q & 1u ? w4.y : w4.x;
                if (scan_rest_raw(a.reg, a.n, w, t, epoch)) f |= LTPG_FLAG_RAW;
            }
            if (f) atomicOr(&fl[lt], f);
            if (!kLate) sm.upd[v] = (uint8_t)vec_updates(words);
        }
        __syncthreads();
        // pass 2: commit decision, flags, bitmap words (tile is a multiple of 32)
        for (uint32_t i = threadIdx.x; i < a.tile; i += blockDim.x) {
            uint32_t f = i < nt ? fl[i] : 0u;
            const bool com = i < nt && commits(f);
            if (com) f |= LTPG_FLAG_COMMIT;
            if (i < nt) {
                a.flags[t0 + i] = (uint8_t)f;
                fl[i] = f;
            }
            const unsigned bal = __ballot_sync(FULL, com);
            const unsigned braw = __ballot_sync(FULL, (f & LTPG_FLAG_RAW) != 0u);
            const unsigned bwar = __ballot_sync(FULL, (f & LTPG_FLAG_WAR) != 0u);
            const unsigned bwaw = __ballot_sync(FULL, (f & LTPG_FLAG_WAW) != 0u);
            if (lane == 0 && i < nt) {
                a.bitmap[(t0 + i) >> 5] = bal;
                cnt.com += __popc(bal);
                cnt.raw += __popc(braw);
                cnt.war += __popc(bwar);
                cnt.waw += __popc(bwaw);
            }
        }
        __syncthreads();
        // pass 3: committed updates (or, with late reads, the committed
        // transactions' row reads)
        if (kLate == 1) {
            late_read_tile(a, ws, fl, t0, nt);
        } else if (kLate == 0) {
            // A transaction that updates a field twice leaves its later value, as
            // a sequential replay does: its vectors store one after another,
            // a barrier apart.  No two committed transactions write one row (WAW).
            for (uint32_t base = 0; base < nvec; base += blockDim.x) {
                const uint32_t v = base + threadIdx.x, lt = v / vpt, at = v - lt * vpt;
                uint64_t *to[4];
                uint64_t val[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) to[q] = nullptr;
                if (v < nvec && sm.upd[v] && (fl[lt] & LTPG_FLAG_COMMIT) && off[lt] != off[lt + 1]) {
                    uint64_t idx = off[lt];
                    for (uint32_t u = 1; u <= at; ++u) idx += sm.upd[v - u];
                    w4 = ld_nc_u4(vp + v);
                    const uint32_t words[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t w = words[q], key = ycsb_key(w), fld = ycsb_field(w);
                        if (ycsb_is_pad(w) || !ycsb_is_update(w)) continue;
                        if (idx >= nv) {  // offsets that disagree with the op words
                            report_error(a.ctl, DERR_BOUNDS, t0 + lt);
                        } else if (key < a.n && fld < LTPG_YCSB_FIELDS) {
                            to[q] = a.rows + (uint64_t)key * LTPG_YCSB_FIELDS + fld;
                            val[q] = __ldg(a.vals + idx);
                        }
                        ++idx;
                    }
                }
                for (uint32_t s = 0; s < vpt; ++s) {
                    if (s) __syncthreads();
                    if (s == at)
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (to[q]) *to[q] = val[q];
                }
            }
        }
        __syncthreads();
    }
    add_counters(a.st, a.ctl, cnt);
}

// ---- fast execute+register: transactions of 2^m words, no block barriers -----
// Each thread takes OPS consecutive op words of one transaction (one 4-, 8- or
// 16-byte load); the lpt = stride / OPS lanes of a transaction are adjacent and
// aligned inside a warp, so the per-transaction read checksum is a segmented
// shuffle reduction and the kernel needs no shared memory outside staging.
// All row loads and slot reads of a thread's ops are issued before any of them
// is consumed, to keep many requests in flight per SM.
template <int OPS>
struct OpVec;
template <>
struct OpVec<1> {
    static __device__ __forceinline__ void load(const uint32_t *p, uint32_t *w) { w[0] = __ldg(p); }
};
template <>
struct OpVec<2> {
    static __device__ __forceinline__ void load(const uint32_t *p, uint32_t *w) {
        uint2 v;
        asm("ld.global.nc.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
        w[0] = v.x;
        w[1] = v.y;
    }
};
template <>
struct OpVec<4> {
    static __device__ __forceinline__ void load(const uint32_t *p, uint32_t *w) {
        const uint4 v = ld_nc_u4(p);
        w[0] = v.x;
        w[1] = v.y;
        w[2] = v.z;
        w[3] = v.w;
    }
};

template <int OPS, bool kStage, bool kFilter, bool kDedupe, int BS>
__global__ void __launch_bounds__(BS) ycsb_exec_fast(YcsbTunedArgs a, uint32_t lpt) {
    extern __shared__ __align__(16) char smem[];
    StageEnt *tab = reinterpret_cast<StageEnt *>(smem);
    const uint64_t tag = slot_tag(a.ctl->epoch);
    const uint32_t lane = threadIdx.x & 31;
    let_next_start();
    if (!kStage) clear_stats(a.st);
    if (kStage) {
        stage_init(tab, a.stage_entries);
        __syncthreads();
    }
    const uint32_t nv = a.B * lpt;  // op vectors in the batch
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < nv; base += step) {
        const uint32_t v = base + threadIdx.x;
        const bool act = v < nv;
        uint32_t w[OPS];
        if (act) OpVec<OPS>::load(a.ops + (uint64_t)v * OPS, w);
        else
#pragma unroll
            for (int q = 0; q < OPS; ++q) w[q] = LTPG_YCSB_OP_PAD;
        const uint32_t t = v / lpt;
        const uint32_t j0 = (v % lpt) * OPS;
        bool rd[OPS], need[OPS];
        uint32_t key[OPS];
#pragma unroll
        for (int q = 0; q < OPS; ++q) {
            bool valid = act && !ycsb_is_pad(w[q]);
            key[q] = ycsb_key(w[q]);
            if (valid && key[q] >= a.n) {
                report_error(a.ctl, DERR_BOUNDS, t);
                valid = false;
            }
            rd[q] = valid && !ycsb_is_update(w[q]);
            need[q] = valid;
            if (kStage && valid) {
                const uint32_t b = key_bucket(key[q]);
                const uint32_t g = __ldg(a.stage_map + b);
                if (g != STAGE_NONE && (g + 1) * a.ways <= a.stage_entries) {
                    StageEnt *e = stage_find(tab, g, a.ways, key[q]);
                    if (e) {
                        atomicMin(ycsb_is_update(w[q]) ? &e->wmin : &e->rmin, t);
                        atomicAdd(&e->cnt, 1u);
                        need[q] = false;
                    }
                }
                if (need[q] && (t % COUNT_SAMPLE) == 0u) atomicAdd(a.bucket_counts + b, COUNT_SAMPLE);
            }
        }
        // issue every load of this thread's ops
        ulonglong2 r[OPS][5];
        uint64_t cur[OPS];
#pragma unroll
        for (int q = 0; q < OPS; ++q) {
            const char *p = reinterpret_cast<const char *>(a.rows + (uint64_t)key[q] * LTPG_YCSB_FIELDS);
#pragma unroll
            for (int i = 0; i < 5; ++i) r[q][i] = rd[q] ? ld_nc16_issue(p + 16 * i) : make_ulonglong2(0ull, 0ull);
            unsigned long long *slot = ycsb_is_update(w[q]) ? &a.reg[key[q]].w : &a.reg[key[q]].r;
            cur[q] = (kFilter && need[q]) ? ld_ca_u64(slot) : ~0ull;
        }
        // registration: optionally one atomic per distinct (key, kind) of the
        // warp, optionally skipped when the slot already holds a smaller value
#pragma unroll
        for (int q = 0; q < OPS; ++q) {
            bool leader = need[q];
            if (kDedupe) {
                const uint32_t mkey = need[q] ? (key[q] | (ycsb_is_update(w[q]) ? 0x80000000u : 0u)) : 0xFFFFFFFFu;
                const unsigned peers = __match_any_sync(FULL, mkey);
                // lanes are in transaction order, so the lowest peer holds the smallest TID
                leader = need[q] && (__ffs(peers) - 1) == (int)lane;
            }
            const unsigned long long mine = tag | t;
            if (leader && cur[q] > mine)
                red_min(ycsb_is_update(w[q]) ? &a.reg[key[q]].w : &a.reg[key[q]].r, mine);
        }
        unsigned long long part = 0;
#pragma unroll
        for (int q = 0; q < OPS; ++q) {
            unsigned long long x = r[q][0].x ^ r[q][0].y ^ r[q][1].x ^ r[q][1].y ^ r[q][2].x ^ r[q][2].y ^
                                   r[q][3].x ^ r[q][3].y ^ r[q][4].x ^ r[q][4].y;
            if (rd[q]) x ^= scan_rest(a.reg, a.rows, a.n, w[q], tag | t, kFilter);
            part += rd[q] ? x * (2ull * (j0 + q) + 1ull) : 0ull;
        }
        for (uint32_t o = lpt >> 1; o >= 1; o >>= 1) part += __shfl_xor_sync(FULL, part, o);
        if (act && (v % lpt) == 0u) a.results[t] = (int64_t)part;
    }
    if (kStage) {
        __syncthreads();
        const uint32_t ops = stage_flush(tab, a.stage_entries, a.reg, tag, a.bucket_counts);
        if (ops) red_add_u64(&a.st->staged_ops, ops);
    }
}

// ---- cooperative execute+register: one op per lane, rows read by 5 lanes ----
// A warp takes whole transactions (warp_lanes).  Each lane registers its own op; then the rows of the
// warp's reads are fetched six at a time, five lanes per row, each lane one
// contiguous 16-byte chunk, so a row costs one or two cache-line requests
// instead of five.  The five chunks are xor-folded within their lane group and
// handed back to the lane that owns the op.
// kReads = false (late reads): registration only; the rows are read after the
// check, by the committed transactions alone (late_read_tile).
// A warp's step takes grp = 32 / k consecutive transactions, k lanes each (10
// operations: three transactions on 30 lanes, where lanes rounded up to a power
// of two held two; 65,536 x 10: 19.7 -> 17.1 us.  The late reads keep the power
// of two: this layout cost them 16 % at 16 operations).  Step s of the batch's
// grp-transaction steps; this lane's transaction is s * grp + g, its op j; lanes
// past the last transaction (g >= grp) hold none.
struct WarpLanes {
    uint32_t g, j;
};
__device__ __forceinline__ WarpLanes warp_lanes(const YcsbTunedArgs &a) {
    const uint32_t lane = threadIdx.x & 31u;
    return WarpLanes{lane / a.k, lane % a.k};
}
// Sum over a transaction's lanes, valid in its lane j = 0.
__device__ __forceinline__ unsigned long long txn_sum(unsigned long long part, uint32_t j, uint32_t k) {
    for (uint32_t o = 1; o < k; o <<= 1) {
        const unsigned long long x = __shfl_down_sync(FULL, part, o);
        if (j + o < k) part += x;
    }
    return part;
}

// kDedupe: one registration per distinct (key, kind), of a warp by match_any
// (DEDUPE_WARP) or of the block (DEDUPE_BLOCK), by the first thread with it,
// which holds the smallest TID.  For a block: a bucket of a table in shared
// memory ends up with the step's smallest entry: step number (counting down, so
// that nothing is cleared between steps), the rest of the mixed key, thread.  A
// thread that finds a smaller thread of its own key there leaves the
// registration to it; one that finds anything else (another key, a later
// step's entry: the barrier is once a step) sends.  And all but the first
// eighth of the lanes send after their row reads, past a look at the slot,
// which by then holds the TIDs of that eighth if the key is hot.
// Reductions on neighbouring hot slots queue at one slice of L2, and in a batch
// of one wave no slot has been written when it is first looked at (10,000 x 10,
// theta 0.99: 18 us with one lane's registration per warp, 13.4 with the table,
// 8.4 with the late look).
enum : int { DEDUPE_NONE, DEDUPE_WARP, DEDUPE_BLOCK };
constexpr uint32_t OP_KEY_BITS = LTPG_YCSB_KEY_BITS + 1;  // key and kind
template <int BS>
__device__ __forceinline__ uint32_t *op_table() {
    __shared__ uint32_t t[4 * BS];
    return t;
}

template <bool kStage, bool kFilter, int kDedupe, bool kReads, int BS>
__device__ __forceinline__ void coop_exec_loop(const YcsbTunedArgs &a, StageEnt *tab, const uint32_t *sbits,
                                               const uint32_t *srank, RowScratch *ws,
                                               uint64_t tag) {
    constexpr bool kTable = kDedupe == DEDUPE_BLOCK, kPeers = kDedupe == DEDUPE_WARP || kStage;
    constexpr uint32_t kBits = BS == 128 ? 9 : BS == 256 ? 10 : 11, kRest = OP_KEY_BITS - kBits;  // 4 BS buckets
    constexpr uint32_t kSteps = 1u << (32 - 9 - kRest);
    static_assert(BS <= 512 && kRest + 9 < 32, "an entry is step | rest | thread");
    uint32_t *ops_tab = nullptr;
    uint32_t steps = 0;  // left before the table is cleared
    if (kTable) ops_tab = op_table<BS>();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t groups = a.ways ? a.stage_entries / a.ways : 0u;
    const WarpLanes l = warp_lanes(a);
    const uint32_t j = l.j, wpb = blockDim.x >> 5, warp = threadIdx.x >> 5;
    const uint32_t n_steps = (a.B + a.grp - 1u) / a.grp, step = gridDim.x * wpb;  // warps' steps
    // steps that register before their row reads: all where no filter is asked
    // for and a warp takes more than two
    const uint32_t early = kFilter || n_steps <= 2u * step ? step / 8u : ~0u;
    bool scans = false;  // some read of this thread's was a range scan
    auto txn_at = [&](uint32_t s) { return s < n_steps && l.g < a.grp ? s * a.grp + l.g : ~0u; };
    auto op_at = [&](uint32_t t) {
        return t < a.B ? __ldg(a.ops + (uint64_t)t * a.stride + j) : LTPG_YCSB_OP_PAD;
    };
    uint32_t next = op_at(txn_at(blockIdx.x * wpb + warp));  // one step ahead of its use
    for (uint32_t base = blockIdx.x * wpb; base < n_steps; base += step) {
        const uint32_t t = txn_at(base + warp);
        const bool act = t < a.B;
        const uint32_t w = next;
        next = op_at(txn_at(base + step + warp));
        bool valid = act && !ycsb_is_pad(w);
        const uint32_t key = ycsb_key(w);
        if (valid && key >= a.n) {
            report_error(a.ctl, DERR_BOUNDS, t);
            valid = false;
        }
        const bool upd = ycsb_is_update(w);
        const bool rd = valid && !upd;
        StageEnt *e = nullptr;
        bool have_dig = false;
        unsigned long long x = 0;
        if (kStage && valid) {
            const uint32_t b = key_bucket(key);
            const uint32_t g = stage_group(sbits, srank, b);
            if (g < groups) e = stage_find(tab, g, a.ways, key);
            if (!e && (t % COUNT_SAMPLE) == 0u) atomicAdd(a.bucket_counts + b, COUNT_SAMPLE);
            if (kReads && e && rd && *reinterpret_cast<volatile uint32_t *>(&e->dig_ok)) {
                __threadfence_block();
                x = *reinterpret_cast<volatile unsigned long long *>(&e->dig);
                have_dig = true;
            }
        }
        uint32_t entry = 0, bucket = 0;
        if (kTable) {
            if (steps == 0u) {
                __syncthreads();
                for (uint32_t i = threadIdx.x; i < 4u * BS; i += blockDim.x) ops_tab[i] = ~0u;
                __syncthreads();
                steps = kSteps - 1u;  // the largest stays for the cleared state
            }
            --steps;
            const uint32_t h = ((key | (upd ? 1u << LTPG_YCSB_KEY_BITS : 0u)) * 0x9E3779B1u) & ((1u << OP_KEY_BITS) - 1u);
            bucket = h >> kRest;
            entry = (((steps << kRest) | (h & ((1u << kRest) - 1u))) << 9) | threadIdx.x;
            if (valid) atomicMin(ops_tab + bucket, entry);
        }
        // one row read per distinct key of the warp: peers share the leader's
        unsigned peers = 1u << lane;
        if (kPeers) peers = __match_any_sync(FULL, valid ? (key | (upd ? 0x80000000u : 0u)) : 0xFFFFFFFFu);
        const uint32_t leader_lane = (uint32_t)__ffs(peers) - 1u;
        const bool leader = valid && leader_lane == lane;
        // rows still to read
        const unsigned need = kReads ? __ballot_sync(FULL, rd && !have_dig && leader) : 0u;
        ulonglong2 ch[6];
        if (kReads && kStage) rows_issue_shfl(a.rows, key, need, ch);
        else if (kReads && need) rows_issue(a.rows, ws, key, need, ch);  // warp-uniform
        // registration: staged rows in shared memory, the rest through the
        // warp dedupe and the slot filter
        const bool need_global = valid && !e;
        uint64_t cur = ~0ull;
        unsigned long long *slot = upd ? &a.reg[key].w : &a.reg[key].r;
        if (kFilter && !kTable && need_global) cur = ld_ca_u64(slot);
        if (kStage && e && leader) {
            atomicMin(upd ? &e->wmin : &e->rmin, t);
            atomicAdd(&e->cnt, (uint32_t)__popc(peers));
        }
        const unsigned long long mine = tag | t;
        bool send = need_global && (leader || kDedupe == DEDUPE_NONE);
        if (kTable) {
            __syncthreads();
            const uint32_t best = ops_tab[bucket];
            send = need_global && (best == entry || ((best ^ entry) >> 9) != 0u);
        }
        const bool late = kTable && base >= early;
        if (send && !late && cur > mine) red_min_exec(slot, mine);
        scans |= rd && ycsb_span(w) != 0u;
        if (kReads && need) {
            const unsigned long long rowx = kStage ? rows_fold_shfl(need, ch) : rows_fold(ws, need, ch);
            if ((need >> lane) & 1u) x = rowx;
        }
        if (send && late && ld_ca_u64(slot) > mine) red_min_exec(slot, mine);
        if (!kReads) continue;
        if (kPeers) {
            const unsigned long long from_leader = __shfl_sync(FULL, x, leader_lane);
            if (!have_dig) x = from_leader;
        }
        if (kStage && e && rd && !have_dig && leader) {  // publish the checksum for later reads in this block
            e->dig = x;
            __threadfence_block();
            *reinterpret_cast<volatile uint32_t *>(&e->dig_ok) = 1u;
        }
        unsigned long long part = rd ? x * (2ull * j + 1ull) : 0ull;
        part = txn_sum(part, j, a.k);
        if (act && j == 0u) a.results[t] = (int64_t)part;
    }
    // Range scans: the keys after each scan's first, in a second pass over the
    // block's ops (kept out of the loop above, whose code is the point-read
    // path: with the scan code inside, that loop ran 6 % slower on point-read
    // batches).  The same thread leads a transaction in both passes, so its
    // result is completed in program order.
    if (__syncthreads_or(scans)) {
        for (uint32_t base = blockIdx.x * wpb; base < n_steps; base += step) {
            const uint32_t t = txn_at(base + warp);
            const bool act = t < a.B;
            const uint32_t w = op_at(t);
            const bool rd = act && !ycsb_is_pad(w) && ycsb_key(w) < a.n && ycsb_span(w) != 0u;
            const uint32_t key = ycsb_key(w);
            const uint32_t last = rd ? (uint32_t)scan_last(w, a.n) : 0u;
            // eight lanes to a scan, four scans of the warp at a time: its rows
            // by the 128-byte lines they cover, two lines in flight, and its
            // keys after the first, one per lane
            unsigned long long xf = 0, xa = 0;  // this lane's scan: first row, all rows
            for (unsigned m = __ballot_sync(FULL, rd); m;) {
                uint32_t own[4], src = lane;
                bool have = false;
#pragma unroll
                for (uint32_t g = 0; g < 4; ++g) {
                    own[g] = m ? (uint32_t)__ffs(m) - 1u : 32u;
                    if (lane >> 3 == g && m) {
                        src = own[g];
                        have = true;
                    }
                    m &= m - 1u;
                }
                const uint32_t k0 = __shfl_sync(FULL, key, src), rest = __shfl_sync(FULL, last - key, src);
                const unsigned long long mine = tag | __shfl_sync(FULL, t, src);
                const uint32_t l = lane & 7u;
                unsigned long long c_all = 0, c_first = 0;
                if (kReads && have) {
                    const uint64_t first = (uint64_t)k0 * 5u;  // in chunks of the table
                    const uint32_t off = (uint32_t)first & 7u, end = off + (rest + 1u) * 5u;
                    const ulonglong2 *p = reinterpret_cast<const ulonglong2 *>(a.rows) + (first - off);
                    for (uint32_t q = l; q < end; q += 16u) {
                        ulonglong2 v[2];
#pragma unroll
                        for (uint32_t r = 0; r < 2; ++r) {
                            const uint32_t at = q + 8u * r;
                            v[r] = at >= off && at < end ? ld_nc16_issue(p + at) : make_ulonglong2(0ull, 0ull);
                        }
#pragma unroll
                        for (uint32_t r = 0; r < 2; ++r) {
                            c_all ^= v[r].x ^ v[r].y;
                            if (q + 8u * r < off + 5u) c_first ^= v[r].x ^ v[r].y;
                        }
                    }
                }
                for (uint32_t i = l; have && i < rest; i += 8u) {
                    unsigned long long *slot = &a.reg[(uint64_t)k0 + 1u + i].r;
                    if (!kFilter || ld_ca_u64(slot) > mine) red_min(slot, mine);
                }
                if (!kReads) continue;
#pragma unroll
                for (uint32_t o = 4; o >= 1u; o >>= 1) {
                    c_all ^= __shfl_xor_sync(FULL, c_all, o);
                    c_first ^= __shfl_xor_sync(FULL, c_first, o);
                }
#pragma unroll
                for (uint32_t g = 0; g < 4; ++g) {
                    const unsigned long long ga = __shfl_sync(FULL, c_all, 8u * g), gf = __shfl_sync(FULL, c_first, 8u * g);
                    if (lane == own[g]) {
                        xa = ga;
                        xf = gf;
                    }
                }
            }
            if (!kReads) continue;
            // the first pass added x_first * (2j + 1); the read's term is
            // x_all * (2j + 1): add the difference (mod 2^64)
            unsigned long long part = rd ? (xa - xf) * (2ull * j + 1ull) : 0ull;
            part = txn_sum(part, j, a.k);
            if (act && j == 0u && part) a.results[t] = (int64_t)((unsigned long long)a.results[t] + part);
        }
    }
}

template <bool kStage, bool kFilter, int kDedupe, bool kReads, int BS>
__global__ void __launch_bounds__(BS) ycsb_exec_coop(YcsbTunedArgs a) {
    extern __shared__ __align__(16) char smem[];
    uint32_t *sbits = reinterpret_cast<uint32_t *>(smem);
    uint32_t *srank = sbits + STAGE_WORDS;
    StageEnt *tab = reinterpret_cast<StageEnt *>(srank + STAGE_WORDS);
    const uint64_t tag = slot_tag(a.ctl->epoch);
    let_next_start();
    if (!kStage) clear_stats(a.st);
    if (kStage) {
        for (uint32_t i = threadIdx.x; i < STAGE_WORDS; i += blockDim.x) {
            sbits[i] = __ldg(a.stage_bits + i);
            srank[i] = __ldg(a.stage_rank + i);
        }
        stage_init(tab, a.stage_entries);
        __syncthreads();
    }
    coop_exec_loop<kStage, kFilter, kDedupe, kReads, BS>(a, tab, sbits, srank, kReads && !kStage ? row_scratch<BS>() : nullptr, tag);
    if (kStage) {
        __syncthreads();
        const uint32_t ops = stage_flush(tab, a.stage_entries, a.reg, tag, a.bucket_counts);
        if (ops) red_add_u64(&a.st->staged_ops, ops);
    }
}

// ---- execute + register by block tiles (ops_per_thread = 8) --------------------
// Four op words per thread in one load, the rows one thread each, the registrations
// through a warp dedupe; a tile's digests in shared memory.  Staging and batches
// beyond a few waves take it when 8 is asked for: there it beats the cooperative
// kernel on short scans and on staged updates (us for two batches: 488,324 x 3
// scans of 2 keys 326 against 448, 112,203 x 8 staged updates 130 against 191);
// on batches of a few waves the cooperative kernel is the faster one.
template <bool kStage>
__device__ __forceinline__ void exec_tiles(const YcsbTunedArgs &a, unsigned long long *dig, StageEnt *tab,
                                           uint64_t tag) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nvec_tile = a.tile * a.stride / 4;
    const uint32_t n_tiles = (a.B + a.tile - 1) / a.tile;
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t t0 = tile * a.tile;
        const uint32_t nt = min(a.tile, a.B - t0);
        const uint32_t nvec = nt * a.stride / 4;
        for (uint32_t i = threadIdx.x; i < a.tile; i += blockDim.x) dig[i] = 0ull;
        __syncthreads();
        const uint4 *vp = reinterpret_cast<const uint4 *>(a.ops + (uint64_t)t0 * a.stride);
        for (uint32_t base = 0; base < nvec_tile; base += blockDim.x) {
            const uint32_t v = base + threadIdx.x;
            const bool act = v < nvec;
            const uint4 w4 = act ? ld_nc_u4(vp + v) : make_uint4(LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD,
                                                                  LTPG_YCSB_OP_PAD, LTPG_YCSB_OP_PAD);
            const uint32_t lt = act ? (v * 4) / a.stride : 0;
            const uint32_t j0 = v * 4 - lt * a.stride;
            const uint32_t t = t0 + lt;
            const uint32_t words[4] = {w4.x, w4.y, w4.z, w4.w};
            unsigned long long part = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t w = words[q];
                bool valid = act && !ycsb_is_pad(w);
                const uint32_t key = ycsb_key(w);
                const bool upd = ycsb_is_update(w);
                if (valid && key >= a.n) {
                    report_error(a.ctl, DERR_BOUNDS, t);
                    valid = false;
                }
                bool staged = false;
                if (kStage && valid) {
                    const uint32_t b = key_bucket(key);
                    const uint32_t g = __ldg(a.stage_map + b);
                    if (g != STAGE_NONE && (g + 1) * a.ways <= a.stage_entries) {
                        StageEnt *e = stage_find(tab, g, a.ways, key);
                        if (e) {
                            atomicMin(upd ? &e->wmin : &e->rmin, t);
                            atomicAdd(&e->cnt, 1u);
                            staged = true;
                        }
                    }
                    if (!staged && (t % COUNT_SAMPLE) == 0u) atomicAdd(a.bucket_counts + b, COUNT_SAMPLE);
                }
                const bool need = valid && !staged;
                const uint32_t mkey = need ? (key | (upd ? 0x80000000u : 0u)) : 0xFFFFFFFFu;
                const unsigned peers = __match_any_sync(FULL, mkey);
                // lanes are in transaction order, so the lowest peer holds the smallest TID
                if (need && (__ffs(peers) - 1) == (int)lane) {
                    unsigned long long *slot = upd ? &a.reg[key].w : &a.reg[key].r;
                    const unsigned long long mine = tag | t;
                    if (!a.filter || ld_ca_u64(slot) > mine) red_min(slot, mine);
                }
                if (valid && !upd) {
                    const char *p = reinterpret_cast<const char *>(a.rows + (uint64_t)key * LTPG_YCSB_FIELDS);
                    const ulonglong2 r0 = ld_nc16(p), r1 = ld_nc16(p + 16), r2 = ld_nc16(p + 32),
                                     r3 = ld_nc16(p + 48), r4 = ld_nc16(p + 64);
                    const unsigned long long x = r0.x ^ r0.y ^ r1.x ^ r1.y ^ r2.x ^ r2.y ^ r3.x ^ r3.y ^ r4.x ^ r4.y ^
                                                 scan_rest(a.reg, a.rows, a.n, w, tag | t, a.filter != 0u);
                    part += x * (2ull * (j0 + q) + 1ull);
                }
            }
            if (part) atomicAdd(&dig[lt], part);
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) a.results[t0 + i] = (int64_t)dig[i];
    }
}

// Shared memory: [dig: tile u64][stage table]; a tile is a multiple of 32.
template <bool kStage>
__global__ void __launch_bounds__(512) ycsb_exec_tiles(YcsbTunedArgs a) {
    extern __shared__ __align__(16) char smem[];
    unsigned long long *dig = reinterpret_cast<unsigned long long *>(smem);
    StageEnt *tab = reinterpret_cast<StageEnt *>(dig + a.tile);
    const uint64_t tag = slot_tag(a.ctl->epoch);
    if (!kStage) clear_stats(a.st);
    if (kStage) {
        stage_init(tab, a.stage_entries);
        __syncthreads();
    }
    exec_tiles<kStage>(a, dig, tab, tag);
    if (kStage) {
        __syncthreads();
        const uint32_t ops = stage_flush(tab, a.stage_entries, a.reg, tag, a.bucket_counts);
        if (ops) red_add_u64(&a.st->staged_ops, ops);
    }
}

// Registers for three blocks of 512 an SM (two when rows are gathered here).
template <int kLate>
__global__ void __launch_bounds__(512, kLate == 1 ? 2 : 3) ycsb_checkwb_tuned(YcsbTunedArgs a) {
    extern __shared__ __align__(16) char smem[];
    const SmemPtrs p = carve(smem, a.tile, a.stride);
    wait_for_previous();
    checkwb_tiles<kLate>(a, p, kLate == 1 ? row_scratch<512>() : nullptr, a.ctl->epoch);
    if (!kLate) finish_batch<false>(a.ctl);
}

// Write-back after late reads: one thread per transaction; a committed one
// stores its updates.  kDecide (write-first registration): the flags hold the
// conflict bits only, and this pass makes the commit decision and writes the
// final flags, the bitmap (a warp's ballot over 32 consecutive transactions is
// one bitmap word) and the counters.  kStore = false: the decision only (the
// update-list write-back stores from the list).
template <bool kDecide, bool kCoh, bool kStore = true>
__device__ __forceinline__ TxnCounts writeback_late_loop(const YcsbTunedArgs &a) {
    const uint32_t step = gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31;
    TxnCounts cnt;
    for (uint32_t base = blockIdx.x * blockDim.x; base < a.B; base += step) {
        const uint32_t t = base + threadIdx.x;
        const bool act = t < a.B;
        const uint32_t f = act ? ld_flag<kCoh>(a.flags + t) : 0u;
        bool com;
        if (kDecide) {
            com = act && commits(f);
            if (act) a.flags[t] = (uint8_t)(f | (com ? LTPG_FLAG_COMMIT : 0u));
            const unsigned bc = __ballot_sync(FULL, com);
            const unsigned br = __ballot_sync(FULL, (f & LTPG_FLAG_RAW) != 0u);
            const unsigned bwr = __ballot_sync(FULL, (f & LTPG_FLAG_WAR) != 0u);
            const unsigned bww = __ballot_sync(FULL, (f & LTPG_FLAG_WAW) != 0u);
            if (lane == 0u && act) {
                a.bitmap[t >> 5] = bc;
                cnt.com += __popc(bc);
                cnt.raw += __popc(br);
                cnt.war += __popc(bwr);
                cnt.waw += __popc(bww);
            }
        } else {
            com = (f & LTPG_FLAG_COMMIT) != 0u;
        }
        if (kStore && com) write_txn_updates(a, t);
    }
    return cnt;
}

// Late reads 2: the check kernel made the decisions; this one stores.
template <int BS>
__global__ void __launch_bounds__(BS) ycsb_writeback_late(YcsbTunedArgs a) {
    writeback_late_loop<false, false>(a);
    finish_batch(a.ctl);
}

// Write-back over the update list: the decision per transaction (flags,
// bitmap, counters: writeback_late_loop with no stores), then one update per
// thread.  An update of a committing transaction stores its value unless a
// later op of the same transaction writes the same field: op order decides, as
// in a sequential replay (the transaction's entries are consecutive).  The
// decision is a function of the conflict bits, which nothing changes here, so
// an update that reads its transaction's flag byte before or after the first
// loop adds COMMIT to it decides the same.
template <bool kCoh>
__device__ __forceinline__ void writeback_list(const YcsbTunedArgs &a) {
    const TxnCounts cnt = writeback_late_loop<true, kCoh, false>(a);
    // a batch whose registration reported an error (a key past the table, or
    // offsets that disagree with the op words, which leave list positions
    // unwritten) stores nothing
    const uint64_t nu = ld_gpu_u32(&a.ctl->error) ? 0ull : upd_count(a);
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < nu; u += step) {
        const uint2 e = ld_upd<kCoh>(a.upd + u);
        const uint32_t key = ycsb_key(e.y), fld = ycsb_field(e.y);
        if (e.x >= a.B || key >= a.n || fld >= LTPG_YCSB_FIELDS) continue;
        if (!commits(ld_gpu_u8(a.flags + e.x) & (LTPG_FLAG_RAW | LTPG_FLAG_WAR | LTPG_FLAG_WAW))) continue;
        bool last = true;
        for (uint64_t u2 = u + 1; u2 < nu; ++u2) {
            const uint2 e2 = ld_upd<kCoh>(a.upd + u2);
            if (e2.x != e.x) break;
            if (ycsb_key(e2.y) == key && ycsb_field(e2.y) == fld) last = false;
        }
        if (last && u < a.vals_cap) a.rows[(uint64_t)key * LTPG_YCSB_FIELDS + fld] = __ldg(a.vals + u);
    }
    add_counters(a.st, a.ctl, cnt);
}
template <int BS>
__global__ void __launch_bounds__(BS) ycsb_writeback_list(YcsbTunedArgs a) {
    writeback_list<false>(a);
    finish_batch<false>(a.ctl);
}

// One cooperative kernel per batch: execute+register, grid barrier, check +
// write-back.  The barrier wait is bounded (grid_barrier); once a wait has
// run out, a block runs no further phase and calls no further barrier.
// With late reads (kLate): execute registers only,
// then check + reads, a second grid barrier, and the write-back.  Phases
// after the first load what earlier phases wrote with coherent loads
// (kCoh = true above), but for the slots in checkwb_tiles.
template <bool kStage, bool kLate, int BS>
__device__ __forceinline__ void ycsb_persistent_body(const YcsbTunedArgs &a) {
    extern __shared__ __align__(16) char smem[];
    const SmemPtrs p = carve(smem, a.tile, a.stride);
    RowScratch *ws = row_scratch<BS>();
    const uint32_t epoch = a.ctl->epoch;
    const uint64_t tag = slot_tag(epoch);
    if (!kStage) clear_stats(a.st);
    if (kLate && !kStage && a.late == 3u) {  // write-first: five phases, four grid barriers
        wf_register_writes<true>(a, tag);
        bool ok = grid_barrier(a.ctl);
        if (ok) wf_register_reads<true, true>(a, epoch, 0u, a.B);
        ok = ok && grid_barrier(a.ctl);
        if (ok) wf_check_list<true>(a, epoch);
        ok = ok && grid_barrier(a.ctl);
        if (ok) late_read_loop<true>(a, ws);
        ok = ok && grid_barrier(a.ctl);
        if (ok) writeback_list<true>(a);
        if (ok) finish_batch<false>(a.ctl);
        else finish_batch(a.ctl);
        return;
    }
    if (kStage) {
        stage_init(p.tab, a.stage_entries);
        __syncthreads();
    }
    constexpr int kDedupe = kStage ? DEDUPE_WARP : DEDUPE_BLOCK;
    if (a.filter) coop_exec_loop<kStage, true, kDedupe, !kLate, BS>(a, p.tab, a.stage_bits, a.stage_rank, ws, tag);
    else coop_exec_loop<kStage, false, kDedupe, !kLate, BS>(a, p.tab, a.stage_bits, a.stage_rank, ws, tag);
    if (kStage) {
        __syncthreads();
        const uint32_t ops = stage_flush(p.tab, a.stage_entries, a.reg, tag, a.bucket_counts);
        if (ops) red_add_u64(&a.st->staged_ops, ops);
    }
    bool ok = grid_barrier(a.ctl);
    if (ok) {
        if (!kLate) checkwb_tiles<0>(a, p, ws, epoch);
        else if (a.late == 2u) checkwb_tiles<2>(a, p, ws, epoch);
        else checkwb_tiles<1>(a, p, ws, epoch);
    }
    if (kLate) {
        if (a.late == 2u) {
            ok = ok && grid_barrier(a.ctl);
            if (ok) late_read_loop<true>(a, ws);
        }
        ok = ok && grid_barrier(a.ctl);
        if (ok) writeback_late_loop<false, true>(a);
    }
    if (!kLate && ok) finish_batch<false>(a.ctl);
    else finish_batch(a.ctl);
}
template <bool kStage, bool kLate>
__global__ void __launch_bounds__(512) ycsb_persistent(YcsbTunedArgs a) {
    ycsb_persistent_body<kStage, kLate, 512>(a);
}
// Late reads on blocks of at most 256 threads with registers budgeted for six
// resident blocks per SM (40, with a few spills, against 59 and four): the row
// gathers of the late-read phase want the warps more than the other phases
// want the registers.
__global__ void __launch_bounds__(256, 6) ycsb_persistent_late_x6(YcsbTunedArgs a) {
    ycsb_persistent_body<false, true, 256>(a);
}

// Static shared memory of a kernel, queried once per kernel.
static size_t static_smem(const void *k) {
    static std::mutex mu;
    static std::unordered_map<const void *, size_t> cache;
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(k);
    if (it != cache.end()) return it->second;
    cudaFuncAttributes fa{};
    const size_t v = cudaFuncGetAttributes(&fa, k) == cudaSuccess ? fa.sharedSizeBytes : 48 * 1024;
    cache.emplace(k, v);
    return v;
}

// Calls f with std::integral_constant<int, BS> for the launch's block size
// (128, 256 or 512; ltpg_set_launch admits no other).
template <class F>
static auto with_block(uint32_t block, F f) {
    switch (block) {
    case 128: return f(std::integral_constant<int, 128>());
    case 512: return f(std::integral_constant<int, 512>());
    default: return f(std::integral_constant<int, 256>());
    }
}

// Transactions per tile: as many whole transactions as the block reads with
// `per_thread` 16-byte vectors per thread, rounded down to a multiple of 32.
static uint32_t tuned_tile(uint32_t stride, uint32_t threads, uint32_t per_thread) {
    uint32_t t = threads * 4u * per_thread / stride;
    t = t / 32u * 32u;
    return t < 32u ? 32u : t;
}

// Launches the barrier-free execute kernel when stride / ops-per-thread is a
// power of two <= 32; returns false (nothing launched) otherwise.
template <int OPS, int BS>
static void launch_fast_t(ltpg_ctx *c, const YcsbTunedArgs &a, bool stage, uint32_t lpt) {
    const LaunchCfg &L = c->launch_y;
    const size_t smem = stage ? (size_t)a.stage_entries * sizeof(StageEnt) : 0;
    void (*k)(YcsbTunedArgs, uint32_t);
    const int sel = (stage ? 4 : 0) | (L.filter ? 2 : 0) | (L.dedupe ? 1 : 0);
    switch (sel) {
    case 0: k = ycsb_exec_fast<OPS, false, false, false, BS>; break;
    case 1: k = ycsb_exec_fast<OPS, false, false, true, BS>; break;
    case 2: k = ycsb_exec_fast<OPS, false, true, false, BS>; break;
    case 3: k = ycsb_exec_fast<OPS, false, true, true, BS>; break;
    case 4: k = ycsb_exec_fast<OPS, true, false, false, BS>; break;
    case 5: k = ycsb_exec_fast<OPS, true, false, true, BS>; break;
    case 6: k = ycsb_exec_fast<OPS, true, true, false, BS>; break;
    default: k = ycsb_exec_fast<OPS, true, true, true, BS>; break;
    }
    if (smem + static_smem((const void *)k) > 48 * 1024)
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const uint32_t threads = BS;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, (int)threads, smem);
    if (per_sm < 1) per_sm = 1;
    if (L.blocks_per_sm && (int)L.blocks_per_sm < per_sm) per_sm = (int)L.blocks_per_sm;
    const uint64_t nv = (uint64_t)a.B * lpt;
    const uint32_t grid = (uint32_t)std::min<uint64_t>((nv + threads - 1) / threads, (uint64_t)per_sm * c->sm_count);
    k<<<grid, threads, smem, c->stream>>>(a, lpt);
}

template <bool kReads, int BS>
static void (*coop_kernel(int sel))(YcsbTunedArgs) {
    switch (sel) {
    case 0: return ycsb_exec_coop<false, false, DEDUPE_NONE, kReads, BS>;
    case 1: return ycsb_exec_coop<false, false, DEDUPE_WARP, kReads, BS>;
    case 2: return ycsb_exec_coop<false, true, DEDUPE_NONE, kReads, BS>;
    case 3: return ycsb_exec_coop<false, true, DEDUPE_WARP, kReads, BS>;
    case 4: return ycsb_exec_coop<true, false, DEDUPE_NONE, kReads, BS>;
    case 5: return ycsb_exec_coop<true, false, DEDUPE_WARP, kReads, BS>;
    case 6: return ycsb_exec_coop<true, true, DEDUPE_NONE, kReads, BS>;
    case 7: return ycsb_exec_coop<true, true, DEDUPE_WARP, kReads, BS>;
    case 8: return ycsb_exec_coop<false, false, DEDUPE_BLOCK, kReads, BS>;
    default: return ycsb_exec_coop<false, true, DEDUPE_BLOCK, kReads, BS>;
    }
}

// Lanes of the cooperative execute kernel over the whole batch.
static uint64_t lanes_of(const YcsbTunedArgs &a) { return 32ull * ((a.B + a.grp - 1u) / a.grp); }

// A batch of up to about eight waves of lanes.  In one, a block registers a key
// once whatever is asked for (65,536 x 10: theta 0.99 29 -> 21 us, 0 and 0.6
// within 1 us; the launch setting dedupe has no say then, and up to two steps a
// warp most lanes look at the slot with filter off too); beyond, the barrier per
// step costs more than it saves (2^18 x 10 at theta 0.6: 48 -> 53 us).  And the
// check's launch overlaps the execute kernel (65,536 x 10: 29.5 -> 27 us a
// batch); beyond, its early blocks are in the way (2^20 x 10: 240 -> 242 us;
// with staging 414 -> 427).
static bool few_waves(const ltpg_ctx *c, const YcsbTunedArgs &a) {
    return lanes_of(a) <= 8192ull * c->sm_count;
}

// reads = false: registration only (late reads)
static void launch_coop(ltpg_ctx *c, const YcsbTunedArgs &a, bool stage, bool reads) {
    const LaunchCfg &L = c->launch_y;
    const size_t smem = stage ? 2 * STAGE_WORDS * sizeof(uint32_t) + (size_t)a.stage_entries * sizeof(StageEnt) : 0;
    const uint64_t nw = lanes_of(a);
    const int sel = !stage && few_waves(c, a) ? (L.filter ? 9 : 8) : (stage ? 4 : 0) | (L.filter ? 2 : 0) | (L.dedupe ? 1 : 0);
    void (*k)(YcsbTunedArgs) = with_block(L.block, [&](auto bs) {
        constexpr int BS = decltype(bs)::value;
        return reads ? coop_kernel<true, BS>(sel) : coop_kernel<false, BS>(sel);
    });
    if (smem + static_smem((const void *)k) > 48 * 1024)
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const uint32_t threads = L.block;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, (int)threads, smem);
    if (per_sm < 1) per_sm = 1;
    if (L.blocks_per_sm && (int)L.blocks_per_sm < per_sm) per_sm = (int)L.blocks_per_sm;
    const uint32_t grid = (uint32_t)std::min<uint64_t>((nw + threads - 1) / threads, (uint64_t)per_sm * c->sm_count);
    k<<<grid, threads, smem, c->stream>>>(a);
}

// Grid of a grid-stride kernel of block_threads threads over `items` lanes:
// at most the blocks that fit on the GPU at once (blocks_per_sm caps them
// when set).
static uint32_t stride_grid(ltpg_ctx *c, const void *k, uint64_t items) {
    const uint32_t threads = c->launch_y.block;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, (int)threads, 0) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    if (c->launch_y.blocks_per_sm && (int)c->launch_y.blocks_per_sm < per_sm) per_sm = (int)c->launch_y.blocks_per_sm;
    const uint64_t g = std::min<uint64_t>((items + threads - 1) / threads, (uint64_t)per_sm * c->sm_count);
    return (uint32_t)std::max<uint64_t>(g, 1);
}

// Write-first registration (late_reads = 3): write registration, read
// registration + RAW, WAR / WAW, committed reads, commit decision +
// write-back.  Profiled as [registration (both), check, reads, write-back].
// The read registration also lists the updates (the list is allocated with
// the slots' batch arrays, so it exists for every YCSB batch), and the check
// and the write-back walk that list.
template <int BS>
static cudaError_t launch_write_first_t(ltpg_ctx *c, const YcsbTunedArgs &a) {
    const uint64_t lanes = (uint64_t)a.B * a.lpt, nvec = (uint64_t)a.B * a.stride / 4;
    prof_mark(c, 0);
    count_launch(c, 2);
    ycsb_wf_writes<BS><<<stride_grid(c, (const void *)ycsb_wf_writes<BS>, nvec), BS, 0, c->stream>>>(a);
    // The smallest TIDs register first, in a launch of their own: a wave finds
    // every slot empty, so all reads of a hot key were sent and queued at its
    // slot, where now the filter knows the least TID of every key read in the
    // head (theta 0.99: 2^20 x 16 145 -> 123 us, 65,536 x 16 41 -> 22; a head of
    // 4,096 or 16,384 no better).  With the filter only, which says that keys
    // are hot, and from 8,192 transactions on: else the launch costs more (theta
    // 0: 2^20 x 16 125 -> 129 us, 65,536 x 16 16 -> 20).  The rest comes up beside
    // the head and waits for it (two batches of 9,000 x 13, half updates: 91 ->
    // 83 us).
    const uint32_t head = a.filter && a.B >= 8192u ? 1024u : 0u;
    if (head) {
        count_launch(c);
        ycsb_wf_reads_list<BS><<<stride_grid(c, (const void *)ycsb_wf_reads_list<BS>, (uint64_t)head * a.stride / 4),
                                 BS, 0, c->stream>>>(a, 0u, head);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = launch_next(ycsb_wf_reads_list<BS>, head != 0u && !c->profiling,
                    stride_grid(c, (const void *)ycsb_wf_reads_list<BS>, nvec), BS, 0, c->stream, a, head, a.B);
    if (e != cudaSuccess) return e;
    prof_mark(c, 1);
    count_launch(c, 2);
    ycsb_wf_check_list<BS><<<stride_grid(c, (const void *)ycsb_wf_check_list<BS>, nvec), BS, 0, c->stream>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    prof_mark(c, 2);
    ycsb_read_late<BS><<<stride_grid(c, (const void *)ycsb_read_late<BS>, lanes), BS, 0, c->stream>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    prof_mark(c, 3);
    count_launch(c);
    ycsb_writeback_list<BS><<<stride_grid(c, (const void *)ycsb_writeback_list<BS>, std::max<uint64_t>(a.B, nvec)),
                              BS, 0, c->stream>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    prof_mark(c, 4);
    return predictor_after_batch(c);
}

static cudaError_t launch_write_first(ltpg_ctx *c, const YcsbTunedArgs &a) {
    return with_block(c->launch_y.block, [&](auto bs) { return launch_write_first_t<decltype(bs)::value>(c, a); });
}

static void launch_tiles(ltpg_ctx *c, const YcsbTunedArgs &a, uint32_t tile, bool stage) {
    const LaunchCfg &L = c->launch_y;
    YcsbTunedArgs t = a;
    t.tile = tile;
    const size_t smem = (size_t)tile * 8 + (stage ? (size_t)a.stage_entries * sizeof(StageEnt) : 0);
    void (*k)(YcsbTunedArgs) = stage ? ycsb_exec_tiles<true> : ycsb_exec_tiles<false>;
    if (smem + static_smem((const void *)k) > 48 * 1024)
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, (int)L.block, smem);
    if (per_sm < 1) per_sm = 1;
    if (L.blocks_per_sm && (int)L.blocks_per_sm < per_sm) per_sm = (int)L.blocks_per_sm;
    k<<<std::min((a.B + tile - 1) / tile, (uint32_t)(per_sm * c->sm_count)), L.block, smem, c->stream>>>(t);
}

// Launch shapes of the execute phase, by ops_per_thread: 2 / 4 = per-thread row
// reads (ycsb_exec_fast) where stride / ops is a power of two; 8 = block tiles of
// `tile` transactions (ycsb_exec_tiles) with staging and beyond a few waves;
// otherwise cooperative row reads (ycsb_exec_coop).
static void launch_exec(ltpg_ctx *c, const YcsbTunedArgs &a, uint32_t tile, bool stage) {
    const uint32_t ops = c->launch_y.per_thread ? c->launch_y.per_thread : 4u;
    const uint32_t lpt = a.stride / ops;
    if (ops == 8u && (stage || !few_waves(c, a))) {
        launch_tiles(c, a, tile, stage);
        return;
    }
    if ((ops != 2u && ops != 4u) || (lpt & (lpt - 1))) {
        launch_coop(c, a, stage, true);
        return;
    }
    with_block(c->launch_y.block, [&](auto bs) {
        constexpr int BS = decltype(bs)::value;
        if (ops == 2) launch_fast_t<2, BS>(c, a, stage, lpt);
        else launch_fast_t<4, BS>(c, a, stage, lpt);
        return 0;
    });
}

cudaError_t ycsb_run_tuned(ltpg_ctx *c, Slot &s, int mode) {
    if (s.n_txn == 0) return cudaSuccess;
    const LaunchCfg &L = c->launch_y;
    const uint32_t threads = L.block;
    const uint32_t per_thread = std::max<uint32_t>(1u, (L.per_thread ? L.per_thread : 4u) / 4u);
    YcsbTunedArgs a;
    a.ops = s.ops;
    a.val_off = s.val_off;
    a.vals = s.vals;
    a.B = s.n_txn;
    a.k = s.k;
    a.stride = s.stride;
    a.grp = 32u / s.k;
    a.lpt = 4;
    while (a.lpt < s.stride) a.lpt <<= 1;
    a.tile = tuned_tile(s.stride, threads, per_thread);  // at most; small batches take less, below
    a.rows = c->ycsb.rows;
    a.n = c->ycsb.n;
    a.reg = c->ycsb.reg;
    a.results = s.results;
    a.flags = s.flags;
    a.bitmap = s.bitmap;
    a.st = s.stats;
    a.ctl = c->ctl;
    const bool stage = (c->stage_on || c->pred_on) && c->stage_map && c->bucket_counts;
    a.stage_map = c->stage_map;
    a.stage_bits = c->stage_bits;
    a.stage_rank = c->stage_rank;
    a.bucket_counts = c->bucket_counts;
    a.ways = L.ways ? L.ways : 4u;
    // with the predictor counting but staging off, the staging table is empty
    a.stage_entries = (stage && c->stage_on) ? STAGE_MAX_ENTRIES / a.ways * a.ways : 0u;
    // write-first registration has no staging path (with staging it reads late
    // in a kernel of their own)
    uint32_t late_mode = L.late_reads;
    if (late_mode == 3u && stage) late_mode = 2u;
    const bool late = late_mode != 0u;
    a.filter = L.filter;
    a.late = late_mode;
    a.wbits = c->ycsb.wbits;
    a.upd = c->ycsb.upd;
    a.upd_cap = c->ycsb.upd_cap;
    a.vals_cap = s.cap_vals;
    const size_t smem = ycsb_smem_bytes(a.tile, a.stride, a.stage_entries);
    const size_t smem_cwb = ycsb_smem_bytes(a.tile, a.stride, 0);  // check + write-back needs no staging table
    // a staging execute kernel adds to the counters; otherwise the first kernel clears them
    cudaError_t e = stage ? cudaMemsetAsync(s.stats, 0, sizeof(DevStats), c->stream) : cudaSuccess;
    if (e != cudaSuccess) return e;
    // write-first: the writer bitmap starts empty for every batch
    if (late_mode == 3u &&
        (e = cudaMemsetAsync(a.wbits, 0, (a.n + 31) / 32 * sizeof(uint32_t), c->stream)) != cudaSuccess)
        return e;
    auto pers_k = stage ? (late ? ycsb_persistent<true, true> : ycsb_persistent<true, false>)
                        : (late ? (threads <= 256 ? ycsb_persistent_late_x6 : ycsb_persistent<false, true>)
                                : ycsb_persistent<false, false>);
    auto cwb_k = !late ? ycsb_checkwb_tuned<0> : late_mode == 1u ? ycsb_checkwb_tuned<1> : ycsb_checkwb_tuned<2>;
    // above 48 KB of static + dynamic shared memory a kernel must opt in
    for (const void *k : {(const void *)cwb_k, (const void *)pers_k})
        if (smem + static_smem(k) > 48 * 1024)
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const bool persistent = mode == LTPG_MODE_PERSISTENT;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, persistent ? pers_k : cwb_k, (int)threads,
                                                      persistent ? smem : smem_cwb);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    if (persistent && L.blocks_per_sm && (int)L.blocks_per_sm < per_sm) per_sm = (int)L.blocks_per_sm;
    // A batch of less than one wave is spread over all resident blocks: the
    // kernels are chains of dependent accesses, which more threads shorten.
    const uint32_t resident = (uint32_t)(per_sm * c->sm_count);
    const uint32_t full_tile = a.tile;
    a.tile = std::min(a.tile, ((a.B + resident - 1) / resident + 31u) / 32u * 32u);
    const uint32_t n_tiles = (a.B + a.tile - 1) / a.tile;
    if (persistent) {
        // A lane per op in the first phase.  The write-first phases take a block to
        // a full tile where that fills half of the multiprocessors: more blocks only send
        // more of the hot keys' registrations at once (us for two batches, filter
        // off, theta 0.999: 30,273 x 16 285 with all resident blocks, 230 so;
        // 58,782 x 3 168 and 121; 158 x 32, which does not fill them, 59 and 84).
        // The other late reads meet at two or three barriers, and neighbouring blocks
        // share a multiprocessor (of 1,824 the first 17 sit on four), which then do
        // the later phases of a batch with fewer tiles than blocks: at most two
        // blocks to a tile, and four of 128 threads to a multiprocessor (twelve fit;
        // 12,630 x 32 updates 109 us with all of them, 63 so; of 256 threads all:
        // 132,766 x 3 77 us, with four 121).
        const uint32_t full = (a.B + full_tile - 1) / full_tile;
        const bool tiles = late_mode == 3u && full >= (uint32_t)c->sm_count / 2u;
        const uint64_t blocks = tiles ? full : std::max<uint64_t>(n_tiles, (lanes_of(a) + threads - 1) / threads);
        const uint32_t few = std::max<uint32_t>(2u * n_tiles, c->sm_count);
        const uint32_t most = late_mode == 1u || late_mode == 2u
                                  ? std::max(full, std::min(few, threads < 256u ? 4u * c->sm_count : resident))
                                  : resident;
        const uint32_t grid = (uint32_t)std::min<uint64_t>(std::min(most, resident), blocks);
        prof_mark(c, 0);
        void *args[] = {&a};
        count_launch(c);
        e = cudaLaunchCooperativeKernel((const void *)pers_k, dim3(grid), dim3(threads), args, smem, c->stream);
        if (e != cudaSuccess) return e;
        for (int m = 1; m < PROF_MARKS; ++m) prof_mark(c, m);
        return predictor_after_batch(c);
    }
    if (late_mode == 3u) return launch_write_first(c, a);
    prof_mark(c, 0);
    count_launch(c);
    if (late) launch_coop(c, a, stage, false);
    else launch_exec(c, a, full_tile, stage);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    prof_mark(c, 1);
    count_launch(c);
    const uint32_t grid_cwb = std::min(n_tiles, resident);
    e = launch_next(cwb_k, !stage && !c->profiling && few_waves(c, a), grid_cwb, threads, smem_cwb, c->stream, a);
    if (e != cudaSuccess) return e;
    prof_mark(c, 2);
    if (late_mode == 2u) {
        count_launch(c);
        with_block(threads, [&](auto bs) {
            constexpr int BS = decltype(bs)::value;
            ycsb_read_late<BS><<<stride_grid(c, (const void *)ycsb_read_late<BS>, (uint64_t)a.B * a.lpt), BS, 0,
                                 c->stream>>>(a);
            return 0;
        });
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    prof_mark(c, 3);
    if (late) {  // the write-back waits for every read of the batch
        count_launch(c);
        with_block(threads, [&](auto bs) {
            constexpr int BS = decltype(bs)::value;
            ycsb_writeback_late<BS>
                <<<stride_grid(c, (const void *)ycsb_writeback_late<BS>, a.B), BS, 0, c->stream>>>(a);
            return 0;
        });
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    prof_mark(c, 4);
    return predictor_after_batch(c);
}

}  // namespace ltpg
