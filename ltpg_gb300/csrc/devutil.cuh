// devutil.cuh — small device helpers shared by the kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "engine.h"

namespace ltpg {

constexpr unsigned FULL = 0xFFFFFFFFu;

// 16-byte load of a registration slot that bypasses L1: slots are written by
// atomics at L2 in the previous phase.
__device__ __forceinline__ ulonglong2 ld_slot(const RegSlot *p) {
    ulonglong2 v;
    asm volatile("ld.global.cg.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}
// Read-only 16-byte load through the non-coherent path (table rows, batches).
__device__ __forceinline__ ulonglong2 ld_nc16(const void *p) {
    ulonglong2 v;
    asm("ld.global.nc.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}
// Same load, kept in program order with the other volatile loads so that a
// thread's independent row reads are all issued before the first is consumed.
__device__ __forceinline__ ulonglong2 ld_nc16_issue(const void *p) {
    ulonglong2 v;
    asm volatile("ld.global.nc.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ld_nc_u4(const void *p) {
    uint4 v;
    asm("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p));
    return v;
}
// Loads of words that other blocks of the same launch wrote before a grid
// barrier (the persistent kernels' later phases): relaxed at GPU scope, so
// they are served coherently by L2 and never by a stale L1 line or the
// read-only path, and the "memory" clobber keeps them after the barrier.
__device__ __forceinline__ uint32_t ld_gpu_u32(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t ld_gpu_u64(const unsigned long long *p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_gpu_u8(const uint8_t *p) {
    uint16_t v;
    asm volatile("ld.relaxed.gpu.global.u8 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint2 ld_gpu_u2(const uint2 *p) {
    uint2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ ulonglong2 ld_gpu_slot(const RegSlot *p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
// Fire-and-forget atomic minimum (no return value, so it issues as a
// reduction at L2).
__device__ __forceinline__ void red_min(unsigned long long *p, unsigned long long v) {
    asm volatile("red.global.min.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// The same reduction without the compiler memory barrier, for the execute
// phases: it stays ordered with other volatile asm (the slot filter's load)
// and with barriers, but the compiler may move independent loads (rows, order
// lines, prices) across it, so they are in flight together.  Nothing in the
// execute phase reads back a slot it reduces into.
__device__ __forceinline__ void red_min_exec(unsigned long long *p, unsigned long long v) {
    asm volatile("red.global.min.u64 [%0], %1;" ::"l"(p), "l"(v));
}
__device__ __forceinline__ void red_add_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("red.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Xor of the 10 fields of a YCSB row (five 16-byte loads).
__device__ __forceinline__ unsigned long long row_xor(const uint64_t *__restrict__ rows, uint64_t key) {
    const char *p = reinterpret_cast<const char *>(rows + key * LTPG_YCSB_FIELDS);
    const ulonglong2 a = ld_nc16(p), b = ld_nc16(p + 16), c = ld_nc16(p + 32), d = ld_nc16(p + 48), e = ld_nc16(p + 64);
    return a.x ^ a.y ^ b.x ^ b.y ^ c.x ^ c.y ^ d.x ^ d.y ^ e.x ^ e.y;
}
// Last key a YCSB read covers (key + scan span, within the table).
__device__ __forceinline__ uint64_t scan_last(uint32_t w, uint64_t n) {
    const uint64_t last = (uint64_t)ycsb_key(w) + ycsb_span(w);
    return last < n ? last : n - 1;
}
// The keys of a range-scan read after its first (key + 1 .. last): each
// registered in its read slot (with `filter`, skipped when the slot already
// holds a smaller tag) and their rows xor-ed.  Point reads return 0.
__device__ __forceinline__ unsigned long long scan_rest(RegSlot *reg, const uint64_t *__restrict__ rows, uint64_t n,
                                                        uint32_t w, unsigned long long mine, bool filter) {
    unsigned long long x = 0;
    if (!ycsb_span(w)) return x;
    const uint64_t last = scan_last(w, n);
    for (uint64_t q = (uint64_t)ycsb_key(w) + 1; q <= last; ++q) {
        unsigned long long *p = &reg[q].r;
        bool go = true;
        if (filter) {
            unsigned long long cur;
            asm volatile("ld.global.ca.u64 %0, [%1];" : "=l"(cur) : "l"(p));
            go = cur > mine;
        }
        if (go) red_min(p, mine);
        x ^= row_xor(rows, q);
    }
    return x;
}
// Write word of a slot, nobody's when off.
__device__ __forceinline__ uint64_t ld_writer_if(bool on, const RegSlot *p) {
    uint64_t v = ~0ull;
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.cg.u64 %0, [%1]; }"
                 : "+l"(v) : "l"(&p->w), "r"((uint32_t)on));
    return v;
}
// RAW on the keys of a range-scan read after its first, four looks in flight.
__device__ __forceinline__ bool scan_rest_raw(const RegSlot *reg, uint64_t n, uint32_t w, uint32_t t, uint32_t epoch) {
    if (!ycsb_span(w)) return false;
    const uint64_t last = scan_last(w, n);
    bool raw = false;
    for (uint64_t q = (uint64_t)ycsb_key(w) + 1; q <= last; q += 4) {
        uint64_t v[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) v[i] = ld_writer_if(q + i <= last, reg + q + i);
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) raw |= slot_min(v[i], epoch) < t;
    }
    return raw;
}

__device__ __forceinline__ void report_error(DevCtl *ctl, uint32_t code, uint32_t index) {
    if (atomicOr(&ctl->error, code) == 0u) ctl->err_index = index;
}

// Transaction counters of a batch; a warp's lane 0 collects its warp's.
struct TxnCounts {
    uint32_t com = 0, raw = 0, war = 0, waw = 0;
};

// Adds a block's counters (lane 0 of each warp holds its warp's) to the
// batch's, and its commits to the context's total.  Every thread calls it.
// The four counters share one 32-byte sector, whose reductions retire one
// after another (1.56 G/s measured): one set per warp kept the write-back of a
// 2^20-transaction YCSB batch waiting (9,728 warps: 36 us, of which 25 were
// these), so a block sends one set.  Its last warp does, while the first thread
// goes on to finish_batch.
__device__ __forceinline__ void add_counters(DevStats *st, DevCtl *ctl, const TxnCounts &c) {
    __shared__ uint32_t cnt[4][32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (lane == 0u) {
        cnt[0][warp] = c.com;
        cnt[1][warp] = c.raw;
        cnt[2][warp] = c.war;
        cnt[3][warp] = c.waw;
    }
    __syncthreads();
    const uint32_t nw = blockDim.x >> 5;
    if (warp != nw - 1u) return;
    unsigned long long *const to[4] = {&st->commits, &st->raw, &st->war, &st->waw};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint32_t sum = __reduce_add_sync(FULL, lane < nw ? cnt[q][lane] : 0u);
        if (lane == 0u && sum) {
            red_add_u64(to[q], sum);
            if (q == 0) red_add_u64(&ctl->total_commits, sum);
        }
    }
}

// Called by every block at the very end of a batch's final kernel: the last
// block to finish advances the batch epoch.  kSync = false: right after
// add_counters, whose barrier the block's work has already met.  Nothing is
// published but that every block has read the epoch, so nothing is fenced: the
// end of the kernel makes the block's stores visible (waiting for them here
// cost a small batch 0.7 us).
template <bool kSync = true>
__device__ __forceinline__ void finish_batch(DevCtl *ctl) {
    if (kSync) __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned prev = atomicAdd(&ctl->done, 1u);
        if (prev == gridDim.x - 1u) {
            ctl->done = 0u;
            atomicAdd(&ctl->epoch, 1u);
        }
    }
}

// First thing in a batch's first kernel (no counter is added before the next
// one, or before a grid barrier): a memset node of its own took 1.5 us a batch.
__device__ __forceinline__ void clear_stats(DevStats *st) {
    if (blockIdx.x == 0u && threadIdx.x < sizeof(DevStats) / sizeof(unsigned long long))
        reinterpret_cast<unsigned long long *>(st)[threadIdx.x] = 0ull;
}

// A kernel whose launch may overlap the end of the one before it (launch_next):
// its blocks come up where they find room and wait here, which hides the launch
// (about 1 us; not with profiling events, whose split is of kernels one after
// another).  What the other kernel wrote is read by plain loads only: the
// read-only path may hold lines from before the wait.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// In the kernel before it, whose blocks are all resident by then.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;"); }

template <class... P, class... A>
static cudaError_t launch_next(void (*k)(P...), bool overlap, uint32_t grid, uint32_t threads, size_t smem,
                               cudaStream_t st, const A &...args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k, P(args)...);
}

__device__ __forceinline__ int warp_incl_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v += n;
    }
    return v;
}

}  // namespace ltpg
