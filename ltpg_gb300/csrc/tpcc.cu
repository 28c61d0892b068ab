// tpcc.cu — TPC-C NewOrder + Payment executors: table image and plain path.
//
// Concurrency-control ops per transaction follow NEWORDER_NAMESPACE and
// PAYMENT_NAMESPACE of the reference (TF/Execute_neworder.h:14-336,426-617,
// TF/Execute_payment.h:39-303,390-536); see tpcc_op() in proto.h.  The
// warehouse and district YTD updates of Payment are hot commutative adds that
// neither register nor check (the "isFrequent" path, TF/Execute_payment.h:86-99,
// 144-163); they are applied as exact int64 adds for committed Payments only.
//
// Transactions are ragged (5 + 3 * lines ops for NewOrder, 5 for Payment).  A
// block takes a tile of transactions, lays their ops out back to back by an
// in-tile prefix sum, and its threads walk that flat list, so short and long
// transactions cost the same per op (the reference leaves lanes idle per
// missing order line, TF/Execute_neworder.h:174-183).
#include <type_traits>

#include "devutil.cuh"

namespace ltpg {

struct TpccDev {
    uint64_t *tab[LTPG_TPCC_TABLES];
    uint64_t rows[LTPG_TPCC_TABLES];
    uint64_t base[LTPG_TPCC_TABLES];
    const uint64_t *name_idx;
    const uint16_t *name_dir;
    uint32_t W;
    uint32_t strict;
    uint32_t ref_names;
};

static TpccDev make_dev(ltpg_ctx *c) {
    TpccDev d{};
    for (int t = 0; t < LTPG_TPCC_TABLES; ++t) {
        d.tab[t] = c->tpcc.tab[t];
        d.rows[t] = c->tpcc.rows[t];
        d.base[t] = c->tpcc.base[t];
    }
    d.name_idx = c->tpcc.name_idx;
    d.name_dir = c->tpcc.name_dir;
    d.W = c->tpcc.W;
    d.strict = (c->cfg.flags & LTPG_CFG_STRICT_INSERT) ? 1u : 0u;
    d.ref_names = (c->cfg.flags & LTPG_CFG_REF_NAME_LOOKUP) ? 1u : 0u;
    return d;
}

__device__ __forceinline__ uint64_t *col_ptr(const TpccDev &db, uint32_t table, uint64_t row, uint32_t col) {
    return db.tab[table] + row * tpcc_cols(table) + col;
}
__device__ __forceinline__ uint64_t ld_col(const TpccDev &db, uint32_t table, uint64_t row, uint32_t col) {
    return __ldg(col_ptr(db, table, row, col));
}

// Field ranges of a transaction record (the keys the reference computes in
// op_k_0 would silently alias other rows if a field were out of range).
__device__ __forceinline__ bool txn_valid(const ltpg_tpcc_txn &x, uint32_t W, uint32_t n_lines) {
    const uint32_t kind = tpcc_kind(x.kind_info);
    if (x.w >= W || tpcc_d(x.kind_info) >= 10u || x.c_id >= 3000u) return false;
    switch (kind) {
    case LTPG_TPCC_NEWORDER: {
        const uint32_t cnt = tpcc_ol_cnt(x.kind_info);
        return cnt <= LTPG_TPCC_MAX_LINES && x.a < 30000u && x.b < 30000u && x.c < 450000u &&
               (uint64_t)x.line_off + cnt <= n_lines;
    }
    case LTPG_TPCC_PAYMENT: return x.c_w < W && tpcc_c_d(x.kind_info) < 10u && x.a < 30000u;
    case LTPG_TPCC_ORDERSTATUS:
        return x.c_w < W && tpcc_c_d(x.kind_info) < 10u && x.a < 30000u && x.b < 450000u;
    case LTPG_TPCC_DELIVERY: {
        const uint32_t carrier = tpcc_ol_cnt(x.kind_info);
        return x.a < 30000u && x.b < 30000u && x.c < 450000u && carrier >= 1u && carrier <= 10u;
    }
    case LTPG_TPCC_STOCKLEVEL: return x.a < 100000u;
    default: return false;
    }
}
__device__ __forceinline__ bool line_valid(const ltpg_tpcc_line &ln, uint32_t W) {
    return ln.i_id < 100000u && ln.supply_w < W;
}

// ---- table image (Database::initial_data, TF/Database.h:349-451) ------------
__global__ void tpcc_init_kernel(uint64_t *__restrict__ tab, uint64_t rows, uint32_t cols, uint32_t table,
                                 uint64_t seed) {
    const uint64_t total = rows * cols;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)gridDim.x * blockDim.x)
        tab[i] = tpcc_init_value(seed, table, i / cols, (uint32_t)(i % cols));
}

cudaError_t tpcc_init_tables(ltpg_ctx *c) {
    for (uint32_t t = 0; t < LTPG_TPCC_TABLES; ++t) {
        tpcc_init_kernel<<<c->sm_count * 8, 256, 0, c->stream>>>(c->tpcc.tab[t], c->tpcc.rows[t], tpcc_cols(t), t,
                                                                  c->tpcc_seed);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return tpcc_clear_slots(c);
}

cudaError_t tpcc_clear_slots(ltpg_ctx *c) {
    const cudaError_t e = cudaMemsetAsync(c->tpcc.reg, 0xFF, c->tpcc.n_slots * sizeof(RegSlot), c->stream);
    if (e != cudaSuccess || !c->tpcc.stock_w) return e;
    return cudaMemsetAsync(c->tpcc.stock_w, 0xFF, c->tpcc.rows[LTPG_T_STOCK] * sizeof(unsigned long long), c->stream);
}

// ---- customer last-name index (replaces INDEX.customer_name_index and its
// 3,000-entry warp scan, TF/Datastructure.h:131-134, TF/Genericfunction.h:29-77)
// One block per district sorts the district's keys (C_LAST << 32 | C_ID) in
// shared memory (bitonic, 4,096 slots).  A lookup takes the name's run from the
// district's directory of the 1,024 smallest names (all that the load makes;
// 2 KB) and the customer from the run: two dependent loads, where a binary
// search of the 24 KB run took twelve.  Larger names are searched for.
constexpr uint32_t NAME_SORT = 4096;

__global__ void __launch_bounds__(1024) tpcc_name_index_kernel(const uint64_t *__restrict__ cust,
                                                               uint64_t *__restrict__ idx,
                                                               uint16_t *__restrict__ dir) {
    __shared__ unsigned long long k[NAME_SORT];
    const uint64_t r0 = (uint64_t)blockIdx.x * 3000u;
    for (uint32_t i = threadIdx.x; i < NAME_SORT; i += blockDim.x) {
        unsigned long long v = ~0ull;
        if (i < 3000u) {
            const uint64_t name = cust[(r0 + i) * tpcc_cols(LTPG_T_CUSTOMER) + C_LAST];
            v = ((name < 0xFFFFFFFFull ? name : 0xFFFFFFFFull) << 32) | i;
        }
        k[i] = v;
    }
    __syncthreads();
    for (uint32_t size = 2; size <= NAME_SORT; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t i = threadIdx.x; i < NAME_SORT; i += blockDim.x) {
                const uint32_t j = i ^ stride;
                if (j > i) {
                    const bool up = (i & size) == 0u;
                    const unsigned long long a = k[i], b = k[j];
                    if ((a > b) == up) {
                        k[i] = b;
                        k[j] = a;
                    }
                }
            }
            __syncthreads();
        }
    for (uint32_t i = threadIdx.x; i < 3000u; i += blockDim.x) idx[r0 + i] = k[i];
    // directory: the first position of every name below NAME_DIR
    for (uint32_t name = threadIdx.x; name <= NAME_DIR; name += blockDim.x) {
        uint32_t lo = 0, hi = 3000u;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (k[mid] < (unsigned long long)name << 32) lo = mid + 1u;
            else hi = mid;
        }
        dir[(uint64_t)blockIdx.x * NAME_DIR_LEN + name] = (uint16_t)lo;
    }
}

cudaError_t tpcc_build_name_index(ltpg_ctx *c) {
    if (!c->tpcc.W || !c->tpcc.name_idx) return cudaSuccess;
    tpcc_name_index_kernel<<<c->tpcc.W * 10u, 1024, 0, c->stream>>>(c->tpcc.tab[LTPG_T_CUSTOMER], c->tpcc.name_idx,
                                                                    c->tpcc.name_dir);
    return cudaGetLastError();
}

// The nth (0-based) customer of district (w, d) whose C_LAST is name, in C_ID
// order: the first index key >= name << 32, then nth further.
__device__ __forceinline__ bool name_lookup(const TpccDev &db, uint32_t w, uint32_t d, uint32_t name, uint32_t nth,
                                            uint32_t &cid) {
    const uint64_t *k = db.name_idx + (10ull * w + d) * 3000u;
    uint32_t lo = 0, hi = 3000u;
    if (name < NAME_DIR) {
        const uint16_t *dir = db.name_dir + (10ull * w + d) * NAME_DIR_LEN + name;
        lo = __ldg(dir);
        hi = __ldg(dir + 1);
    } else {
        const uint64_t target = (uint64_t)name << 32;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(k + mid) < target) lo = mid + 1u;
            else hi = mid;
        }
        hi = 3000u;
    }
    const uint32_t p = lo + nth;
    if (p >= hi) return false;
    const uint64_t v = __ldg(k + p);
    if ((v >> 32) != name) return false;
    cid = (uint32_t)v;
    return true;
}

// The reference's __FIND_CID_INDEX (TF/Genericfunction.h:29-77) as its lane 0
// computes it: the lane's shuffle reads its own match flag 32 times, so it
// tests customers 0, 32, 64, ... and counts each match 32 times until the
// count reaches nth; it then walks back from the end of its last block of 32
// (down to position 1) over customers with that name, counting down to nth,
// and returns the C_ID column of the row it stops at; otherwise C_ID 0.
// Positions past the district read the next district's rows, as the
// reference's index does; past the table they match nothing.
__device__ __forceinline__ uint32_t ref_name_lookup(const TpccDev &db, uint32_t w, uint32_t d, uint32_t name,
                                                    uint32_t nth) {
    const uint64_t dist = 30000ull * w + 3000ull * d, rows = db.rows[LTPG_T_CUSTOMER];
    auto name_at = [&](uint64_t row) {
        return row < rows && ld_col(db, LTPG_T_CUSTOMER, row, C_LAST) == (uint64_t)name;
    };
    uint32_t cum = 0, flag = 0;
    for (uint32_t i = 0; i < 3000u; i += 32u) {
        cum += name_at(dist + i) ? 32u : 0u;
        flag += 32u;
        if (cum >= nth) break;
    }
    if (cum < nth) return 0u;
    uint64_t result = 0;
    for (uint32_t i = flag - 1u; i > 0u; --i) {
        if (!name_at(dist + i)) continue;
        if (cum == nth) {
            result = dist + i;
            break;
        }
        --cum;
    }
    return (uint32_t)ld_col(db, LTPG_T_CUSTOMER, result, C_ID);
}

// Marks a by-name Payment whose customer was not found (kept in the
// shared-memory copy of the record only; a Payment's bits 8..15 are flags,
// a NewOrder's its line count).
constexpr uint32_t KI_NOT_FOUND = 0x200u;
__device__ __forceinline__ bool txn_not_found(const ltpg_tpcc_txn &x) {
    const uint32_t kind = tpcc_kind(x.kind_info);
    return (kind == LTPG_TPCC_PAYMENT || kind == LTPG_TPCC_ORDERSTATUS) && (x.kind_info & KI_NOT_FOUND);
}

// Resolves a by-name Payment or OrderStatus in place: c_id becomes the
// customer's C_ID.  Returns false when the customer is not found;
// out-of-range fields are left for txn_valid to reject.
__device__ __forceinline__ bool resolve_by_name(const TpccDev &db, ltpg_tpcc_txn &x) {
    if (!tpcc_customer_by_name(x.kind_info)) return true;
    const uint32_t c_d = tpcc_c_d(x.kind_info);
    if (x.c_w >= db.W || c_d >= 10u) return true;
    const uint32_t name = x.c_id >> 8, nth = x.c_id & 0xFFu;
    if (db.ref_names) {
        x.c_id = ref_name_lookup(db, x.c_w, c_d, name, nth);
        return true;
    }
    uint32_t cid;
    if (!name_lookup(db, x.c_w, c_d, name, nth, cid)) return false;
    x.c_id = cid;
    return true;
}

constexpr uint32_t PT = 64;    // transactions per tile (plain path)
constexpr uint32_t PBS = 256;  // threads per block (plain path)
// Tuned path: blocks of 128 threads by default, 256 or 512 by the launch setting
// block_threads, on tiles of up to as many transactions.

template <uint32_t N>
struct TileHdrN {
    ltpg_tpcc_txn x[N];
    uint32_t off[N + 1];
    uint32_t ok[N];
};
using TileHdr = TileHdrN<PT>;

// Loads a tile and lays out its ops (n_ops_of = ops per transaction).
template <class H, class F>
__device__ __forceinline__ uint32_t load_tile(H &h, const ltpg_tpcc_txn *__restrict__ txns, uint32_t t0,
                                              uint32_t nt, const TpccDev &db, uint32_t n_lines, DevCtl *ctl,
                                              F n_ops_of) {
    if (threadIdx.x < nt) {
        const uint4 *p = reinterpret_cast<const uint4 *>(txns + t0 + threadIdx.x);
        const uint4 a = ld_nc_u4(p), b = ld_nc_u4(p + 1);
        ltpg_tpcc_txn x;
        x.kind_info = a.x; x.w = a.y; x.c_w = a.z; x.c_id = a.w;
        x.a = b.x; x.b = b.y; x.c = b.z; x.line_off = b.w;
        const bool found = resolve_by_name(db, x);
        if (!found) x.kind_info |= KI_NOT_FOUND;
        h.x[threadIdx.x] = x;
        const bool ok = found && txn_valid(x, db.W, n_lines);
        if (!ok && found) report_error(ctl, DERR_BOUNDS, t0 + threadIdx.x);
        h.ok[threadIdx.x] = ok;
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // warp 0: prefix sum of the tile's op counts
        uint32_t carry = 0;
        for (uint32_t base = 0; base < nt; base += 32) {
            const uint32_t i = base + threadIdx.x;
            const int n = i < nt ? (int)n_ops_of(i) : 0;
            const int incl = warp_incl_scan(n);
            if (i < nt) h.off[i] = carry + (uint32_t)(incl - n);
            carry += (uint32_t)__shfl_sync(FULL, incl, 31);
        }
        if (threadIdx.x == 0) h.off[nt] = carry;
    }
    __syncthreads();
    return h.off[nt];
}

// Transaction of flat op e: the last i with off[i] <= e.
template <class H>
__device__ __forceinline__ uint32_t tile_owner(const H &h, uint32_t nt, uint32_t e) {
    uint32_t lo = 0, hi = nt;  // off[lo] <= e < off[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (h.off[mid] <= e) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ ltpg_tpcc_line load_line(const ltpg_tpcc_line *__restrict__ lines, uint64_t idx) {
    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(lines) + idx);
    ltpg_tpcc_line ln;
    ln.i_id = v.x;
    ln.supply_w = (uint16_t)(v.y & 0xFFFFu);
    ln.qty = (uint16_t)(v.y >> 16);
    return ln;
}

// The execute-phase read that gives a non-NewOrder transaction its result, if
// op j is the op holding it: Payment j = 2 (C_BALANCE - amount), OrderStatus
// j = 0 (C_BALANCE), Delivery j = 2 (the line's OL_AMOUNT), StockLevel j = 0
// (S_QUANTITY).  Batch-start image.
__device__ __forceinline__ bool result_read(const TpccDev &db, const ltpg_tpcc_txn &x, uint32_t j, const TpccOp &op,
                                            long long &out) {
    switch (tpcc_kind(x.kind_info)) {
    case LTPG_TPCC_PAYMENT:
        if (j != 2u) return false;
        out = (long long)ld_col(db, LTPG_T_CUSTOMER, op.row, C_BALANCE) - tpcc_amount(x);
        return true;
    case LTPG_TPCC_ORDERSTATUS:
        if (j != 0u) return false;
        out = (long long)ld_col(db, LTPG_T_CUSTOMER, op.row, C_BALANCE);
        return true;
    case LTPG_TPCC_DELIVERY:
        if (j != 2u) return false;
        out = (long long)ld_col(db, LTPG_T_ORDERLINE, op.row, OL_AMOUNT);
        return true;
    case LTPG_TPCC_STOCKLEVEL:
        out = (long long)ld_col(db, LTPG_T_STOCK, op.row, S_QUANTITY);
        return true;
    default: return false;
    }
}

// In a tile's conflict flags, above the flag byte: some order line's supply
// warehouse is another one; some order line is out of range (its NewOrder does
// not commit: the write-back takes a committed order's lines as they are).
constexpr uint32_t FL_REMOTE = 0x100u, FL_BAD_LINE = 0x200u;

// ---- plain phase 1: execute + register (KERNEL_EXECUTE, TF/tp.cu:24-54) ----
__global__ void __launch_bounds__(PBS) tpcc_exec_plain(const ltpg_tpcc_txn *__restrict__ txns, uint32_t B,
                                                       const ltpg_tpcc_line *__restrict__ lines,
                                                       const uint64_t *__restrict__ hdr, TpccDev db,
                                                       RegSlot *__restrict__ reg, int64_t *__restrict__ results,
                                                       DevCtl *ctl) {
    const uint32_t n_lines = (uint32_t)hdr[0];
    __shared__ TileHdr h;
    __shared__ unsigned long long sum[PT];
    __shared__ uint32_t wtax[PT], dtax[PT], disc[PT];
    __shared__ long long res[PT];
    const uint64_t tag = slot_tag(ctl->epoch);
    const uint32_t t0 = blockIdx.x * PT, nt = min(PT, B - t0);
    if (threadIdx.x < PT) sum[threadIdx.x] = 0ull;
    const uint32_t total = load_tile(h, txns, t0, nt, db, n_lines, ctl,
                                     [&](uint32_t i) { return h.ok[i] ? tpcc_n_ops(h.x[i].kind_info) : 0u; });
    for (uint32_t e = threadIdx.x; e < total; e += PBS) {
        const uint32_t i = tile_owner(h, nt, e), j = e - h.off[i];
        const ltpg_tpcc_txn &x = h.x[i];
        const bool no = tpcc_kind(x.kind_info) == LTPG_TPCC_NEWORDER;
        ltpg_tpcc_line ln{0, 0, 0};
        if (no && j >= 5) {
            ln = load_line(lines, (uint64_t)x.line_off + (j - 5) / 3);
            if (!line_valid(ln, db.W)) {
                report_error(ctl, DERR_BOUNDS, t0 + i);
                continue;
            }
        }
        const TpccOp op = tpcc_op(x, j, ln, db.strict);
        RegSlot *s = reg + db.base[op.table] + op.row;
        const unsigned long long v = tag | (t0 + i);
        if (op.flags & OPF_REG_R) red_min(&s->r, v);
        if (op.flags & OPF_REG_W) red_min(&s->w, v);
        // Reads of the execute phase (batch-start snapshot).
        if (no) {
            if (j == 0) wtax[i] = (uint32_t)ld_col(db, LTPG_T_WAREHOUSE, op.row, W_TAX);
            else if (j == 1) dtax[i] = (uint32_t)ld_col(db, LTPG_T_DISTRICT, op.row, D_TAX);
            else if (j == 2) disc[i] = (uint32_t)ld_col(db, LTPG_T_CUSTOMER, op.row, C_DISCOUNT);
            else if (op.table == LTPG_T_ITEM)
                atomicAdd(&sum[i], (unsigned long long)ln.qty * ld_col(db, LTPG_T_ITEM, op.row, I_PRICE));
        } else {
            long long r;
            if (result_read(db, x, j, op, r)) res[i] = r;
        }
    }
    __syncthreads();
    if (threadIdx.x < nt) {
        const uint32_t i = threadIdx.x;
        int64_t r = 0;
        if (h.ok[i])
            r = tpcc_kind(h.x[i].kind_info) == LTPG_TPCC_NEWORDER
                    ? neworder_total((int64_t)sum[i], disc[i], wtax[i], dtax[i])
                    : (int64_t)res[i];
        results[t0 + i] = r;
    }
}

// ---- plain phase 2: check (KERNEL_CHECK, TF/tp.cu:55-85) ---------------------
__global__ void __launch_bounds__(PBS) tpcc_check_plain(const ltpg_tpcc_txn *__restrict__ txns, uint32_t B,
                                                        const ltpg_tpcc_line *__restrict__ lines,
                                                        const uint64_t *__restrict__ hdr, TpccDev db,
                                                        const RegSlot *__restrict__ reg,
                                                        uint8_t *__restrict__ flags, DevCtl *ctl) {
    const uint32_t n_lines = (uint32_t)hdr[0];
    __shared__ TileHdr h;
    __shared__ uint32_t fl[PT];
    const uint32_t epoch = ctl->epoch;
    const uint32_t t0 = blockIdx.x * PT, nt = min(PT, B - t0);
    if (threadIdx.x < PT) fl[threadIdx.x] = 0u;
    const uint32_t total = load_tile(h, txns, t0, nt, db, n_lines, ctl,
                                     [&](uint32_t i) { return h.ok[i] ? tpcc_n_ops(h.x[i].kind_info) : 0u; });
    for (uint32_t e = threadIdx.x; e < total; e += PBS) {
        const uint32_t i = tile_owner(h, nt, e), j = e - h.off[i];
        const ltpg_tpcc_txn &x = h.x[i];
        ltpg_tpcc_line ln{0, 0, 0};
        if (tpcc_kind(x.kind_info) == LTPG_TPCC_NEWORDER && j >= 5) {
            ln = load_line(lines, (uint64_t)x.line_off + (j - 5) / 3);
            if (!line_valid(ln, db.W)) {
                atomicOr(&fl[i], FL_BAD_LINE);
                continue;
            }
        }
        const TpccOp op = tpcc_op(x, j, ln, db.strict);
        const ulonglong2 s = ld_slot(reg + db.base[op.table] + op.row);
        const uint32_t rmin = slot_min(s.x, epoch), wmin = slot_min(s.y, epoch), t = t0 + i;
        uint32_t f = 0;
        if ((op.flags & OPF_CHK_RAW) && wmin < t) f |= LTPG_FLAG_RAW;
        if ((op.flags & OPF_CHK_WAR) && rmin < t) f |= LTPG_FLAG_WAR;
        if ((op.flags & OPF_CHK_WAW) && wmin < t) f |= LTPG_FLAG_WAW;
        if (f) atomicOr(&fl[i], f);
    }
    __syncthreads();
    if (threadIdx.x < nt) {
        uint32_t f = fl[threadIdx.x];
        if (h.ok[threadIdx.x] && !(f & FL_BAD_LINE) && commits(f)) f |= LTPG_FLAG_COMMIT;
        if (txn_not_found(h.x[threadIdx.x])) f |= LTPG_FLAG_NOT_FOUND;
        flags[t0 + threadIdx.x] = (uint8_t)f;
    }
}

// Write op q of a committed transaction (its order lines are in range: one that
// is not keeps its NewOrder from committing).  NewOrder: 0 ORDER insert, 1
// NEW-ORDER insert, 2+2i stock update of line i, 3+2i ORDER-LINE insert of
// line i.  Payment: 0 W_YTD add, 1 D_YTD add, 2 customer update, 3 HISTORY
// insert.  Delivery: 0 NEW-ORDER delete, 1 ORDER carrier, 2 ORDER-LINE delivery
// date, 3 customer credit (`result` = the line's OL_AMOUNT read by the execute
// phase).  Rows written here have exactly one committed writer in the batch
// (a second one would have seen WAW), so plain read-modify-writes are safe;
// the YTD adds are commutative and use atomics.
__device__ __forceinline__ uint32_t tpcc_n_writes(uint32_t kind_info) {
    switch (tpcc_kind(kind_info)) {
    case LTPG_TPCC_NEWORDER: return 2u + 2u * tpcc_ol_cnt(kind_info);
    case LTPG_TPCC_PAYMENT: return 4u;
    case LTPG_TPCC_DELIVERY: return 4u;
    default: return 0u;  // OrderStatus, StockLevel: read-only
    }
}

__device__ __forceinline__ void tpcc_apply_write(const TpccDev &db, const ltpg_tpcc_txn &x, uint32_t q,
                                                 const ltpg_tpcc_line *__restrict__ lines, uint64_t date,
                                                 int64_t result) {
    const uint32_t d = tpcc_d(x.kind_info);
    if (tpcc_kind(x.kind_info) == LTPG_TPCC_DELIVERY) {
        if (q == 0) {
            uint64_t *o = col_ptr(db, LTPG_T_NEWORDER, 30000ull * x.w + x.b, 0);
            o[NO_O_ID] = o[NO_D_ID] = o[NO_W_ID] = ~0ull;  // deleted
        } else if (q == 1) {
            *col_ptr(db, LTPG_T_ORDER, 30000ull * x.w + x.a, O_CARRIER_ID) = tpcc_ol_cnt(x.kind_info);
        } else if (q == 2) {
            *col_ptr(db, LTPG_T_ORDERLINE, 450000ull * x.w + x.c, OL_DELIVERY_D) = date;
        } else {
            uint64_t *cst = col_ptr(db, LTPG_T_CUSTOMER, tpcc_cust_row(x.w, d, x.c_id), 0);
            cst[C_BALANCE] = (uint64_t)((int64_t)cst[C_BALANCE] + result);
            cst[C_DELIVERY_CNT] += 1u;
        }
        return;
    }
    if (tpcc_kind(x.kind_info) == LTPG_TPCC_NEWORDER) {
        const uint32_t cnt = tpcc_ol_cnt(x.kind_info);
        if (q == 0) {
            uint64_t *o = col_ptr(db, LTPG_T_ORDER, 30000ull * x.w + x.a, 0);
            bool all_local = true;
            for (uint32_t i = 0; i < cnt; ++i) all_local &= load_line(lines, (uint64_t)x.line_off + i).supply_w == x.w;
            o[O_ID] = x.a; o[O_D_ID] = d; o[O_W_ID] = x.w; o[O_C_ID] = x.c_id;
            o[O_ENTRY_D] = date; o[O_CARRIER_ID] = 0; o[O_OL_CNT] = cnt; o[O_ALL_LOCAL] = all_local;
            return;
        }
        if (q == 1) {
            uint64_t *o = col_ptr(db, LTPG_T_NEWORDER, 30000ull * x.w + x.b, 0);
            o[NO_O_ID] = x.a; o[NO_D_ID] = d; o[NO_W_ID] = x.w;
            return;
        }
        const uint32_t i = (q - 2) / 2;
        const ltpg_tpcc_line ln = load_line(lines, (uint64_t)x.line_off + i);
        const uint64_t srow = 100000ull * ln.supply_w + ln.i_id;
        if ((q & 1u) == 0u) {
            // Atomic, so that an order listing one stock row twice (the
            // reference's generator draws distinct items, a caller's batch
            // need not) updates it once per line.  Order does not matter: for
            // S_QUANTITY in [10, 100] and quantities <= 91 the rule keeps the
            // value in [10, 100], so after any set of lines it is
            // 10 + ((q - sum - 10) mod 91) whatever their order; the counters
            // add.  No other committed transaction writes the row (WAW).
            uint64_t *s = col_ptr(db, LTPG_T_STOCK, srow, 0);
            unsigned long long *qp = reinterpret_cast<unsigned long long *>(s + S_QUANTITY);
            unsigned long long cur = *qp;
            for (uint32_t tries = 0; tries < 64u; ++tries) {  // contenders: the order's own lines
                const unsigned long long prev = atomicCAS(qp, cur, (unsigned long long)stock_after(cur, ln.qty));
                if (prev == cur) break;
                cur = prev;
            }
            red_add_u64(reinterpret_cast<unsigned long long *>(s + S_YTD), ln.qty);
            red_add_u64(reinterpret_cast<unsigned long long *>(s + S_ORDER_CNT), 1ull);
            if (ln.supply_w != x.w) red_add_u64(reinterpret_cast<unsigned long long *>(s + S_REMOTE_CNT), 1ull);
        } else {
            uint64_t *o = col_ptr(db, LTPG_T_ORDERLINE, tpcc_ol_row(x.w, x.c, i), 0);
            o[OL_O_ID] = x.a; o[OL_D_ID] = d; o[OL_W_ID] = x.w; o[OL_NUMBER] = i + 1u;
            o[OL_I_ID] = ln.i_id; o[OL_SUPPLY_W_ID] = ln.supply_w; o[OL_DELIVERY_D] = 0u;
            o[OL_QUANTITY] = ln.qty;
            o[OL_AMOUNT] = (uint64_t)ln.qty * ld_col(db, LTPG_T_ITEM, ln.i_id, I_PRICE);
            o[OL_DIST_INFO] = ld_col(db, LTPG_T_STOCK, srow, S_DIST_01 + d);
        }
        return;
    }
    const int64_t amt = tpcc_amount(x);
    const uint32_t c_d = tpcc_c_d(x.kind_info);
    if (q == 0) {
        red_add_u64(reinterpret_cast<unsigned long long *>(col_ptr(db, LTPG_T_WAREHOUSE, x.w, W_YTD)),
                    (unsigned long long)amt);
    } else if (q == 1) {
        red_add_u64(reinterpret_cast<unsigned long long *>(col_ptr(db, LTPG_T_DISTRICT, 10ull * x.w + d, D_YTD)),
                    (unsigned long long)amt);
    } else if (q == 2) {
        uint64_t *cst = col_ptr(db, LTPG_T_CUSTOMER, tpcc_cust_row(x.c_w, c_d, x.c_id), 0);
        cst[C_BALANCE] = (uint64_t)((int64_t)cst[C_BALANCE] - amt);
        cst[C_YTD_PAYMENT] = (uint64_t)((int64_t)cst[C_YTD_PAYMENT] + amt);
        cst[C_PAYMENT_CNT] += 1u;
    } else {
        uint64_t *hh = col_ptr(db, LTPG_T_HISTORY, 30000ull * x.w + x.a, 0);
        hh[H_C_ID] = x.c_id; hh[H_C_D_ID] = c_d; hh[H_C_W_ID] = x.c_w; hh[H_D_ID] = d;
        hh[H_W_ID] = x.w; hh[H_AMOUNT] = (uint64_t)amt; hh[H_DATE] = date; hh[H_DATA] = 0u;
    }
}

// ---- plain phase 3: write-back (KERNEL_WRITEBACK, TF/tp.cu:86-117) ----------
__global__ void __launch_bounds__(PBS) tpcc_writeback_plain(const ltpg_tpcc_txn *__restrict__ txns, uint32_t B,
                                                            const ltpg_tpcc_line *__restrict__ lines,
                                                            const uint64_t *__restrict__ hdr, TpccDev db,
                                                            const int64_t *__restrict__ results,
                                                            const uint8_t *__restrict__ flags,
                                                            uint32_t *__restrict__ bitmap, DevStats *st,
                                                            DevCtl *ctl) {
    const uint32_t n_lines = (uint32_t)hdr[0];
    const uint64_t txn_base = hdr[1];
    __shared__ TileHdr h;
    __shared__ uint8_t fl[PT];
    const uint32_t t0 = blockIdx.x * PT, nt = min(PT, B - t0);
    TxnCounts cnt;
    if (threadIdx.x < PT) {
        const uint32_t f = threadIdx.x < nt ? flags[t0 + threadIdx.x] : 0u;
        fl[threadIdx.x] = (uint8_t)f;
        const unsigned bal = __ballot_sync(FULL, (f & LTPG_FLAG_COMMIT) != 0u);
        const unsigned braw = __ballot_sync(FULL, (f & LTPG_FLAG_RAW) != 0u);
        const unsigned bwar = __ballot_sync(FULL, (f & LTPG_FLAG_WAR) != 0u);
        const unsigned bwaw = __ballot_sync(FULL, (f & LTPG_FLAG_WAW) != 0u);
        if ((threadIdx.x & 31) == 0 && threadIdx.x < nt) {
            bitmap[(t0 + threadIdx.x) >> 5] = bal;
            cnt.com = __popc(bal);
            cnt.raw = __popc(braw);
            cnt.war = __popc(bwar);
            cnt.waw = __popc(bwaw);
        }
    }
    __syncthreads();
    const uint32_t total = load_tile(h, txns, t0, nt, db, n_lines, ctl, [&](uint32_t i) {
        return (h.ok[i] && (fl[i] & LTPG_FLAG_COMMIT)) ? tpcc_n_writes(h.x[i].kind_info) : 0u;
    });
    for (uint32_t e = threadIdx.x; e < total; e += PBS) {
        const uint32_t i = tile_owner(h, nt, e), q = e - h.off[i];
        tpcc_apply_write(db, h.x[i], q, lines, txn_base + t0 + i, results[t0 + i]);
    }
    add_counters(st, ctl, cnt);
    finish_batch<false>(ctl);
}

cudaError_t tpcc_phase(ltpg_ctx *c, Slot &s, int phase) {
    const uint32_t B = s.n_txn;
    if (B == 0) return cudaSuccess;
    const TpccDev db = make_dev(c);
    const uint32_t grid = (B + PT - 1) / PT;
    if (phase == 0) {
        cudaError_t e = cudaMemsetAsync(s.stats, 0, sizeof(DevStats), c->stream);
        if (e != cudaSuccess) return e;
        tpcc_exec_plain<<<grid, PBS, 0, c->stream>>>(s.txns, B, s.lines, s.dev_hdr, db, c->tpcc.reg, s.results,
                                                     c->ctl);
    } else if (phase == 1) {
        tpcc_check_plain<<<grid, PBS, 0, c->stream>>>(s.txns, B, s.lines, s.dev_hdr, db, c->tpcc.reg, s.flags,
                                                      c->ctl);
    } else {
        tpcc_writeback_plain<<<grid, PBS, 0, c->stream>>>(s.txns, B, s.lines, s.dev_hdr, db, s.results, s.flags,
                                                          s.bitmap, s.stats, c->ctl);
    }
    return cudaGetLastError();
}

}  // namespace ltpg


// ============================================================================
// Tuned path: the same tiles, with deduplicated + filtered registration, check
// and write-back fused, and the hot W_YTD / D_YTD adds of a block summed in
// shared memory and flushed once per block (one atomic per warehouse and per
// district instead of one per Payment).
// ============================================================================
#include "stage.cuh"

namespace ltpg {

constexpr uint32_t HOT_SMEM_MAX_W = 256;  // shared-memory YTD sums up to 256 warehouses

struct TpccTunedArgs {
    const ltpg_tpcc_txn *txns;
    const ltpg_tpcc_line *lines;
    const uint64_t *hdr;  // {n_lines, txn_base} of the slot
    uint32_t B;
    TpccDev db;
    RegSlot *reg;
    int64_t *results;
    uint8_t *flags;
    uint32_t *bitmap;
    DevStats *st;
    DevCtl *ctl;
    uint32_t filter;
    uint32_t dedupe;  // one registration per distinct slot of a warp (header ops)
    // claims (see below): claimed rows' bits and rows claimed twice, claim_words(W)
    // words each; whether there are any of the latter, and any StockLevel; the
    // STOCK rows that StockLevels read; the STOCK rows' smallest writers
    uint32_t *claim, *multi, *any, *sl_bits;
    unsigned long long *stock_w;
};
enum : uint32_t { ANY_MULTI = 0, ANY_STOCKLEVEL = 1 };

__device__ __forceinline__ uint64_t ld_cg_u64(const unsigned long long *p) {
    uint64_t v;
    asm volatile("ld.global.cg.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint64_t ld_ca_u64t(const unsigned long long *p) {
    uint64_t v;
    asm volatile("ld.global.ca.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}

// Tables that no NewOrder or Payment registers a write on: WAREHOUSE and
// DISTRICT (their YTD updates are unregistered hot adds, D_NEXT_O_ID is
// host-assigned, TF/Query.h:54-88) and ITEM (read-only).  A read of such a row
// never sees RAW, and its registration can never give a writer WAR, so the
// tuned kernels neither register nor check those reads; the outcome is the
// plain path's, which keeps the reference's full op list.
//
// A block of T threads takes tiles of P <= T transactions.  Thread i < P owns
// transaction i: it registers (checks) the transaction's header ops; then all
// threads take the tile's order lines, laid out back to back with a map of
// their owners.  (One lane per header op and a search for every line's owner
// took three times the instructions.)
//
// Claims (kClaim).  The rows of HISTORY, NEW-ORDER, ORDER and ORDER-LINE are
// mostly inserted by one transaction and touched by no other of the batch, and
// such a row can give no conflict.  So a transaction only sets its rows' bits in
// a claim bitmap (one word or two for its order lines); a row whose bit was set
// already gets its bit in a second bitmap, `multi`.  tpcc_register_multi then
// registers the ops on multi rows in their slots, as all ops were registered
// before, and the check looks at those slots alone.  Half of the NewOrder and
// Payment registrations and slot loads go (7 M of 13.6 M per 2^20 transactions
// 50/50), each a random access at L2; the price is clearing the bitmaps (147 KB
// per warehouse) and a kernel that ends at once when no row is multi.
//
// A claiming batch also keeps the STOCK rows' smallest writers in an array of
// their own, 8 bytes a row: order lines write STOCK rows all over the table, and
// random reductions run at 200 G/s on 51 MB (W = 64), which stay in L2, against
// 152 G/s on the 102 MB of whole slots and 54 G/s beyond L2 (measured alone).
// Only a StockLevel reads STOCK rows: it registers in the row's slot and sets
// the row's bit, and a line looks at the slot when that bit is set.
// tpcc_claims() says from which batch size all this pays.

// Rows of the claimed tables (HISTORY, NEW-ORDER, ORDER, ORDER-LINE) are one
// range of slots; bit = slot - base[HISTORY].
__device__ __forceinline__ uint32_t claim_bit(const TpccDev &db, uint32_t table, uint64_t row) {
    return (uint32_t)(db.base[table] - db.base[LTPG_T_HISTORY] + row);
}
// True when a row was claimed before.
__device__ __forceinline__ bool claim_seen(const TpccTunedArgs &a, uint32_t word, uint32_t before, uint32_t mask) {
    if (before & mask) atomicOr(a.multi + word, before & mask);
    return (before & mask) != 0u;
}
// Up to 32 rows from bit `bit` on: their words and masks.
struct ClaimRun {
    uint32_t word, m0, m1;
};
__device__ __forceinline__ ClaimRun claim_run(uint32_t bit, uint32_t len) {
    const uint64_t m = ((1ull << len) - 1u) << (bit & 31u);
    return ClaimRun{bit >> 5, (uint32_t)m, (uint32_t)(m >> 32)};
}
// A NewOrder's order-line rows, which wrap inside its warehouse's range: the
// run up to the wrap and the one after it (usually empty).
__device__ __forceinline__ void line_runs(const TpccDev &db, const ltpg_tpcc_txn &x, uint32_t cnt, ClaimRun *run) {
    const uint32_t first = min(cnt, 450000u - x.c);
    run[0] = claim_run(claim_bit(db, LTPG_T_ORDERLINE, 450000ull * x.w + x.c), first);
    run[1] = claim_run(claim_bit(db, LTPG_T_ORDERLINE, 450000ull * x.w), cnt - first);
}

// Header ops of a transaction.  `main`: the op on a row that transactions share
// (CUSTOMER; StockLevel's STOCK row); the others are on claimed tables.
struct HeadOps {
    uint64_t main_slot;
    uint32_t main_flags;   // OPF_* (0: no transaction here)
    uint32_t n;            // ops on claimed tables
    uint32_t table[3];
    uint32_t row[3];
    uint32_t flags[3];
};
__device__ __forceinline__ HeadOps head_ops(const TpccDev &db, const ltpg_tpcc_txn &x, bool ok) {
    HeadOps o;
    o.main_flags = 0;
    o.main_slot = 0;
    o.n = 0;
    if (!ok) return o;
    const uint32_t d = tpcc_d(x.kind_info), c_d = tpcc_c_d(x.kind_info);
    const uint64_t cust = db.base[LTPG_T_CUSTOMER], w3 = 30000ull * x.w;
    auto add = [&](uint32_t table, uint64_t row, uint32_t flags) {
        o.table[o.n] = table;
        o.row[o.n] = (uint32_t)row;
        o.flags[o.n] = flags;
        ++o.n;
    };
    switch (tpcc_kind(x.kind_info)) {
    case LTPG_TPCC_NEWORDER:
        o.main_slot = cust + tpcc_cust_row(x.w, d, x.c_id);
        o.main_flags = OPF_READ;
        add(LTPG_T_NEWORDER, w3 + x.b, db.strict ? OPF_WRITE : OPF_NO_INSERT_COMPAT);
        add(LTPG_T_ORDER, w3 + x.a, OPF_WRITE);
        break;
    case LTPG_TPCC_PAYMENT:  // the customer's read op and write op are on one row
        o.main_slot = cust + tpcc_cust_row(x.c_w, c_d, x.c_id);
        o.main_flags = OPF_RW;
        add(LTPG_T_HISTORY, w3 + x.a, OPF_WRITE);
        break;
    case LTPG_TPCC_ORDERSTATUS:
        o.main_slot = cust + tpcc_cust_row(x.c_w, c_d, x.c_id);
        o.main_flags = OPF_READ;
        add(LTPG_T_ORDER, w3 + x.a, OPF_READ);
        add(LTPG_T_ORDERLINE, 450000ull * x.w + x.b, OPF_READ);
        break;
    case LTPG_TPCC_DELIVERY:
        o.main_slot = cust + tpcc_cust_row(x.w, d, x.c_id);
        o.main_flags = OPF_WRITE;
        add(LTPG_T_NEWORDER, w3 + x.b, OPF_WRITE);
        add(LTPG_T_ORDER, w3 + x.a, OPF_RW);
        add(LTPG_T_ORDERLINE, 450000ull * x.w + x.c, OPF_RW);
        break;
    default:
        o.main_slot = db.base[LTPG_T_STOCK] + 100000ull * x.w + x.a;
        o.main_flags = OPF_READ;
        break;
    }
    return o;
}

// One registration; `dedupe`: one atomic per distinct slot of the warp (lanes
// are in TID order, so the lowest lane of a same-slot group holds the smallest
// TID), `filter`: skipped when the slot already holds a smaller tag.
// Warp-uniform.
__device__ __forceinline__ void tuned_register(const TpccTunedArgs &a, bool valid, uint64_t slot_idx, bool is_w,
                                               unsigned long long mine, bool dedupe, bool filter) {
    bool leader = valid;
    if (dedupe) {
        const unsigned long long mkey = valid ? (slot_idx << 1) | (is_w ? 1ull : 0ull) : ~0ull;
        const unsigned peers = __match_any_sync(FULL, mkey);
        leader = valid && (__ffs(peers) - 1) == (int)(threadIdx.x & 31);
    }
    if (!leader) return;
    RegSlot *s = a.reg + slot_idx;
    unsigned long long *p = is_w ? &s->w : &s->r;
    if (!filter || ld_ca_u64t(p) > mine) red_min_exec(p, mine);
}

__device__ __forceinline__ uint32_t conflicts_of(const ulonglong2 &s, uint32_t flags, uint32_t t, uint32_t epoch) {
    const uint32_t rmin = slot_min(s.x, epoch), wmin = slot_min(s.y, epoch);
    uint32_t f = 0;
    if ((flags & OPF_CHK_RAW) && wmin < t) f |= LTPG_FLAG_RAW;
    if ((flags & OPF_CHK_WAR) && rmin < t) f |= LTPG_FLAG_WAR;
    if ((flags & OPF_CHK_WAW) && wmin < t) f |= LTPG_FLAG_WAW;
    return f;
}

// Exact 64-bit sum in shared memory (lo, hi): 32-bit atomics with the carry
// passed on.  A 64-bit shared add is a compare-and-swap loop, and the lines of
// an order are neighbouring lanes: 15 of them took 15 rounds.
__device__ __forceinline__ void smem_add64(uint32_t *p, unsigned long long v) {
    const uint32_t lo = (uint32_t)v, before = atomicAdd(p, lo);
    const uint32_t hi = (uint32_t)(v >> 32) + (before + lo < lo ? 1u : 0u);
    if (hi) atomicAdd(p + 1, hi);
}

template <uint32_t P>
struct TpccTile {
    ltpg_tpcc_txn x[P];
    uint32_t off[P + 1];                     // first line of each transaction in the tile's list
    uint32_t part[P / 32];                   // lines of each owner warp
    uint32_t acc[2 * P];                     // exec: order totals, 64 bits each; check: conflict flags, multi lines
    typename std::conditional<P <= 256, uint8_t, uint16_t>::type own[P * LTPG_TPCC_MAX_LINES];  // owner of each line
};

// The record of transaction t0 + i with its customer resolved; ok: it is valid.
__device__ __forceinline__ ltpg_tpcc_txn load_txn(const TpccTunedArgs &a, uint32_t t, uint32_t n_lines, bool report,
                                                  bool &ok) {
    const uint4 *p = reinterpret_cast<const uint4 *>(a.txns + t);
    const uint4 u = ld_nc_u4(p), v = ld_nc_u4(p + 1);
    ltpg_tpcc_txn x;
    x.kind_info = u.x; x.w = u.y; x.c_w = u.z; x.c_id = u.w;
    x.a = v.x; x.b = v.y; x.c = v.z; x.line_off = v.w;
    const bool found = resolve_by_name(a.db, x);
    if (!found) x.kind_info |= KI_NOT_FOUND;
    ok = found && txn_valid(x, a.db.W, n_lines);
    if (!ok && found && report) report_error(a.ctl, DERR_BOUNDS, t);
    return x;
}

// Lays out `n` lines of this thread's transaction (threads >= P: 0) in the
// tile's list; returns the list's length.  Two barriers.
template <uint32_t P>
__device__ __forceinline__ uint32_t layout_lines(TpccTile<P> &h, uint32_t n) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = 0;
    if (threadIdx.x < P) {  // whole warps
        incl = (uint32_t)warp_incl_scan((int)n);
        if (lane == 31u) h.part[warp] = incl;
    }
    __syncthreads();
    uint32_t off = incl - n, total = 0;
#pragma unroll
    for (uint32_t i = 0; i < P / 32; ++i) {
        off += i < warp ? h.part[i] : 0u;
        total += h.part[i];
    }
    if (threadIdx.x < P) {
        h.off[threadIdx.x] = off;
        for (uint32_t i = 0; i < n; ++i) h.own[off + i] = threadIdx.x;
    }
    __syncthreads();
    return total;
}

template <uint32_t P, uint32_t T, bool kClaim>
__device__ __forceinline__ void tpcc_exec_tiles(const TpccTunedArgs &a, TpccTile<P> &h, uint64_t tag) {
    const uint32_t n_lines = (uint32_t)a.hdr[0];
    const bool filt = a.filter != 0u, dedupe = a.dedupe != 0u;
    uint32_t *sum = h.acc;
    bool multi = false, stocklevel = false;  // this thread met one
    const uint32_t n_tiles = (a.B + P - 1) / P;
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t t0 = tile * P, nt = min(P, a.B - t0), i = threadIdx.x;
        uint32_t cnt = 0, disc = 0, wtax = 0, dtax = 0, kind = 0;
        long long res = 0;
        bool ok = false;
        if (i < P) {  // whole warps
            ltpg_tpcc_txn x{};
            if (i < nt) x = load_txn(a, t0 + i, n_lines, true, ok);
            h.x[i] = x;
            sum[2u * i] = sum[2u * i + 1u] = 0u;
            kind = tpcc_kind(x.kind_info);
            const unsigned long long mine = tag | (t0 + i);
            const HeadOps o = head_ops(a.db, x, ok);
            tuned_register(a, o.main_flags & OPF_REG_R, o.main_slot, false, mine, dedupe, filt);
            tuned_register(a, o.main_flags & OPF_REG_W, o.main_slot, true, mine, dedupe, filt);
            const bool no = ok && kind == LTPG_TPCC_NEWORDER;
            cnt = no ? tpcc_ol_cnt(x.kind_info) : 0u;
            if (kClaim && ok && kind == LTPG_TPCC_STOCKLEVEL) {
                const uint32_t row = 100000u * x.w + x.a;
                atomicOr(a.sl_bits + (row >> 5), 1u << (row & 31u));
                stocklevel = true;
            }
            if (kClaim) {
                ClaimRun run[2];
                uint32_t b[3], before[3], line_before[4] = {0, 0, 0, 0};
#pragma unroll
                for (uint32_t q = 0; q < 3; ++q) {
                    b[q] = q < o.n ? claim_bit(a.db, o.table[q], o.row[q]) : 0u;
                    before[q] = q < o.n ? atomicOr(a.claim + (b[q] >> 5), 1u << (b[q] & 31u)) : 0u;
                }
                if (cnt) {
                    line_runs(a.db, x, cnt, run);
                    line_before[0] = atomicOr(a.claim + run[0].word, run[0].m0);
                    if (run[0].m1) line_before[1] = atomicOr(a.claim + run[0].word + 1, run[0].m1);
                    if (run[1].m0) line_before[2] = atomicOr(a.claim + run[1].word, run[1].m0);
                    if (run[1].m1) line_before[3] = atomicOr(a.claim + run[1].word + 1, run[1].m1);
                }
#pragma unroll
                for (uint32_t q = 0; q < 3; ++q)
                    if (q < o.n) multi |= claim_seen(a, b[q] >> 5, before[q], 1u << (b[q] & 31u));
                if (cnt) {
                    multi |= claim_seen(a, run[0].word, line_before[0], run[0].m0);
                    multi |= claim_seen(a, run[0].word + 1, line_before[1], run[0].m1);
                    multi |= claim_seen(a, run[1].word, line_before[2], run[1].m0);
                    multi |= claim_seen(a, run[1].word + 1, line_before[3], run[1].m1);
                }
            } else {
#pragma unroll
                for (uint32_t q = 0; q < 3; ++q) {
                    if (q >= o.n) continue;
                    RegSlot *s = a.reg + a.db.base[o.table[q]] + o.row[q];
                    if (o.flags[q] & OPF_REG_R) red_min_exec(&s->r, mine);
                    if (o.flags[q] & OPF_REG_W) red_min_exec(&s->w, mine);
                }
            }
            // the reads behind the result (batch-start image)
            if (no) {
                const uint32_t d = tpcc_d(x.kind_info);
                wtax = (uint32_t)ld_col(a.db, LTPG_T_WAREHOUSE, x.w, W_TAX);
                dtax = (uint32_t)ld_col(a.db, LTPG_T_DISTRICT, 10ull * x.w + d, D_TAX);
                disc = (uint32_t)ld_col(a.db, LTPG_T_CUSTOMER, o.main_slot - a.db.base[LTPG_T_CUSTOMER], C_DISCOUNT);
            } else if (ok) {
                const uint64_t main_row = o.main_slot - a.db.base[LTPG_T_CUSTOMER];
                if (kind == LTPG_TPCC_PAYMENT)
                    res = (long long)ld_col(a.db, LTPG_T_CUSTOMER, main_row, C_BALANCE) - tpcc_amount(x);
                else if (kind == LTPG_TPCC_ORDERSTATUS)
                    res = (long long)ld_col(a.db, LTPG_T_CUSTOMER, main_row, C_BALANCE);
                else if (kind == LTPG_TPCC_DELIVERY)
                    res = (long long)ld_col(a.db, LTPG_T_ORDERLINE, 450000ull * x.w + x.c, OL_AMOUNT);
                else
                    res = (long long)ld_col(a.db, LTPG_T_STOCK, 100000ull * x.w + x.a, S_QUANTITY);
            }
        }
        const uint32_t lines_n = layout_lines<P>(h, cnt);
        for (uint32_t e = i; e < lines_n; e += T) {
            const uint32_t q = h.own[e], li = e - h.off[q];
            const ltpg_tpcc_txn &x = h.x[q];
            const ltpg_tpcc_line ln = load_line(a.lines, (uint64_t)x.line_off + li);
            if (!line_valid(ln, a.db.W)) {
                report_error(a.ctl, DERR_BOUNDS, t0 + q);
                continue;
            }
            const unsigned long long mine = tag | (t0 + q);
            const uint64_t srow = 100000ull * ln.supply_w + ln.i_id;
            unsigned long long *p = kClaim ? a.stock_w + srow : &a.reg[a.db.base[LTPG_T_STOCK] + srow].w;
            if (!filt || ld_ca_u64t(p) > mine) red_min_exec(p, mine);
            if (!kClaim) red_min_exec(&a.reg[a.db.base[LTPG_T_ORDERLINE] + tpcc_ol_row(x.w, x.c, li)].w, mine);
            smem_add64(sum + 2u * q, (unsigned long long)ln.qty * ld_col(a.db, LTPG_T_ITEM, ln.i_id, I_PRICE));
        }
        __syncthreads();
        if (i < nt) {
            int64_t r = res;
            if (ok && kind == LTPG_TPCC_NEWORDER)
                r = neworder_total((int64_t)(((uint64_t)sum[2u * i + 1u] << 32) | sum[2u * i]), disc, wtax, dtax);
            a.results[t0 + i] = r;
        }
        // the next tile writes x and sum by the same threads, the rest after its barriers
    }
    // one store per block: same-address stores queue
    if (kClaim && __syncthreads_or(multi) && threadIdx.x == 0) a.any[ANY_MULTI] = 1u;
    if (kClaim && __syncthreads_or(stocklevel) && threadIdx.x == 0) a.any[ANY_STOCKLEVEL] = 1u;
}

// The ops of a transaction on multi rows, registered in their slots.
__device__ __forceinline__ bool multi_row(const TpccTunedArgs &a, uint32_t bit) {
    return (__ldg(a.multi + (bit >> 5)) >> (bit & 31u)) & 1u;
}
// Mask over the lines of a NewOrder: its ORDER-LINE row is multi.
__device__ __forceinline__ uint32_t multi_lines(const TpccTunedArgs &a, const ltpg_tpcc_txn &x, uint32_t cnt) {
    ClaimRun run[2];
    line_runs(a.db, x, cnt, run);
    const uint32_t first = min(cnt, 450000u - x.c);
    uint32_t out = 0;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (!(run[r].m0 | run[r].m1)) continue;
        uint64_t w = run[r].m0 ? __ldg(a.multi + run[r].word) & run[r].m0 : 0u;
        if (run[r].m1) w |= (uint64_t)(__ldg(a.multi + run[r].word + 1) & run[r].m1) << 32;
        if (!w) continue;
        const uint32_t sh = (uint32_t)(claim_bit(a.db, LTPG_T_ORDERLINE, 450000ull * x.w + (r ? 0u : x.c)) & 31u);
        out |= (uint32_t)(w >> sh) << (r ? first : 0u);
    }
    return out;
}

__global__ void __launch_bounds__(256, 8) tpcc_register_multi(TpccTunedArgs a) {
    if (!a.any[ANY_MULTI]) return;
    const uint64_t tag = slot_tag(a.ctl->epoch);
    const uint32_t n_lines = (uint32_t)a.hdr[0];
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < a.B; t += gridDim.x * blockDim.x) {
        const uint4 *p = reinterpret_cast<const uint4 *>(a.txns + t);
        const uint4 u = ld_nc_u4(p), v = ld_nc_u4(p + 1);
        ltpg_tpcc_txn x;
        x.kind_info = u.x; x.w = u.y; x.c_w = u.z; x.c_id = 0u;  // the customer has no part in claimed rows
        x.a = v.x; x.b = v.y; x.c = v.z; x.line_off = v.w;
        if (!txn_valid(x, a.db.W, n_lines)) continue;
        const HeadOps o = head_ops(a.db, x, true);
        const uint32_t cnt = tpcc_kind(x.kind_info) == LTPG_TPCC_NEWORDER ? tpcc_ol_cnt(x.kind_info) : 0u;
        uint32_t head = 0;
#pragma unroll
        for (uint32_t q = 0; q < 3; ++q)
            if (q < o.n && multi_row(a, claim_bit(a.db, o.table[q], o.row[q]))) head |= 1u << q;
        uint32_t lines = cnt ? multi_lines(a, x, cnt) : 0u;
        if (!head && !lines) continue;
        bool ok;  // a customer that is not found, or out of range, registers nothing
        (void)load_txn(a, t, n_lines, false, ok);
        if (!ok) continue;
        const unsigned long long mine = tag | t;
#pragma unroll
        for (uint32_t q = 0; q < 3; ++q) {
            if (!((head >> q) & 1u)) continue;
            RegSlot *s = a.reg + a.db.base[o.table[q]] + o.row[q];
            if (o.flags[q] & OPF_REG_R) red_min(&s->r, mine);
            if (o.flags[q] & OPF_REG_W) red_min(&s->w, mine);
        }
        for (; lines; lines &= lines - 1u) {
            const uint32_t li = (uint32_t)__ffs(lines) - 1u;
            if (line_valid(load_line(a.lines, (uint64_t)x.line_off + li), a.db.W))
                red_min(&a.reg[a.db.base[LTPG_T_ORDERLINE] + tpcc_ol_row(x.w, x.c, li)].w, mine);
        }
    }
}

// Two columns of a row in one 16-byte store (rows of an even number of columns).
__device__ __forceinline__ void st_cols2(uint64_t *p, uint64_t a, uint64_t b) {
    *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(a, b);
}
__device__ __forceinline__ void hot_add(uint32_t *hot, uint64_t *direct, int64_t amt) {
    if (hot) smem_add64(hot, (unsigned long long)amt);
    else red_add_u64(reinterpret_cast<unsigned long long *>(direct), (unsigned long long)amt);
}

// Writes of a committed transaction apart from its order lines, by its owner
// thread (the same values as tpcc_apply_write).
__device__ __forceinline__ void write_head(const TpccDev &db, const ltpg_tpcc_txn &x, bool all_local, uint64_t date,
                                           int64_t result, uint32_t *hot) {
    const uint32_t d = tpcc_d(x.kind_info), c_d = tpcc_c_d(x.kind_info);
    switch (tpcc_kind(x.kind_info)) {
    case LTPG_TPCC_NEWORDER: {
        uint64_t *o = col_ptr(db, LTPG_T_ORDER, 30000ull * x.w + x.a, 0);
        st_cols2(o + O_ID, x.a, d);
        st_cols2(o + O_W_ID, x.w, x.c_id);
        st_cols2(o + O_ENTRY_D, date, 0u);
        st_cols2(o + O_OL_CNT, tpcc_ol_cnt(x.kind_info), all_local);
        uint64_t *n = col_ptr(db, LTPG_T_NEWORDER, 30000ull * x.w + x.b, 0);
        n[NO_O_ID] = x.a; n[NO_D_ID] = d; n[NO_W_ID] = x.w;
        return;
    }
    case LTPG_TPCC_PAYMENT: {
        const int64_t amt = tpcc_amount(x);
        uint64_t *cst = col_ptr(db, LTPG_T_CUSTOMER, tpcc_cust_row(x.c_w, c_d, x.c_id), 0);
        const uint64_t bal = cst[C_BALANCE], ytd = cst[C_YTD_PAYMENT], pc = cst[C_PAYMENT_CNT];
        hot_add(hot ? hot + 2u * x.w : nullptr, col_ptr(db, LTPG_T_WAREHOUSE, x.w, W_YTD), amt);
        hot_add(hot ? hot + 2u * (db.W + 10u * x.w + d) : nullptr, col_ptr(db, LTPG_T_DISTRICT, 10ull * x.w + d, D_YTD),
                amt);
        cst[C_BALANCE] = (uint64_t)((int64_t)bal - amt);
        cst[C_YTD_PAYMENT] = (uint64_t)((int64_t)ytd + amt);
        cst[C_PAYMENT_CNT] = pc + 1u;
        uint64_t *hh = col_ptr(db, LTPG_T_HISTORY, 30000ull * x.w + x.a, 0);
        st_cols2(hh + H_C_ID, x.c_id, c_d);
        st_cols2(hh + H_C_W_ID, x.c_w, d);
        st_cols2(hh + H_W_ID, x.w, (uint64_t)amt);
        st_cols2(hh + H_DATE, date, 0u);
        return;
    }
    case LTPG_TPCC_DELIVERY: {
        uint64_t *n = col_ptr(db, LTPG_T_NEWORDER, 30000ull * x.w + x.b, 0);
        uint64_t *cst = col_ptr(db, LTPG_T_CUSTOMER, tpcc_cust_row(x.w, d, x.c_id), 0);
        const uint64_t bal = cst[C_BALANCE], dc = cst[C_DELIVERY_CNT];
        n[NO_O_ID] = n[NO_D_ID] = n[NO_W_ID] = ~0ull;  // deleted
        *col_ptr(db, LTPG_T_ORDER, 30000ull * x.w + x.a, O_CARRIER_ID) = tpcc_ol_cnt(x.kind_info);
        *col_ptr(db, LTPG_T_ORDERLINE, 450000ull * x.w + x.c, OL_DELIVERY_D) = date;
        cst[C_BALANCE] = (uint64_t)((int64_t)bal + result);
        cst[C_DELIVERY_CNT] = dc + 1u;
        return;
    }
    default: return;
    }
}

// Line li of a committed NewOrder, which is in range: the stock update (atomic: an order may list
// a row twice, see tpcc_apply_write) and the ORDER-LINE insert.
__device__ __forceinline__ void write_line(const TpccDev &db, const ltpg_tpcc_txn &x, uint32_t li,
                                           const ltpg_tpcc_line &ln) {
    const uint32_t d = tpcc_d(x.kind_info);
    uint64_t *s = col_ptr(db, LTPG_T_STOCK, 100000ull * ln.supply_w + ln.i_id, 0);
    unsigned long long *qp = reinterpret_cast<unsigned long long *>(s + S_QUANTITY);
    unsigned long long cur = *qp;
    const uint64_t price = ld_col(db, LTPG_T_ITEM, ln.i_id, I_PRICE), info = s[S_DIST_01 + d];
    for (uint32_t tries = 0; tries < 64u; ++tries) {  // contenders: the order's own lines
        const unsigned long long prev = atomicCAS(qp, cur, (unsigned long long)stock_after(cur, ln.qty));
        if (prev == cur) break;
        cur = prev;
    }
    red_add_u64(reinterpret_cast<unsigned long long *>(s + S_YTD), ln.qty);
    red_add_u64(reinterpret_cast<unsigned long long *>(s + S_ORDER_CNT), 1ull);
    if (ln.supply_w != x.w) red_add_u64(reinterpret_cast<unsigned long long *>(s + S_REMOTE_CNT), 1ull);
    uint64_t *o = col_ptr(db, LTPG_T_ORDERLINE, tpcc_ol_row(x.w, x.c, li), 0);
    st_cols2(o + OL_O_ID, x.a, d);
    st_cols2(o + OL_W_ID, x.w, li + 1u);
    st_cols2(o + OL_I_ID, ln.i_id, ln.supply_w);
    st_cols2(o + OL_DELIVERY_D, 0u, ln.qty);
    st_cols2(o + OL_AMOUNT, (uint64_t)ln.qty * price, info);
}

// hot: 11 W 64-bit sums in shared memory (W <= HOT_SMEM_MAX_W), or null.
template <uint32_t P, uint32_t T, bool kClaim>
__device__ __forceinline__ TxnCounts tpcc_checkwb_tiles(const TpccTunedArgs &a, TpccTile<P> &h, uint32_t epoch,
                                                        uint32_t *hot) {
    const uint32_t n_lines = (uint32_t)a.hdr[0];
    const uint64_t txn_base = a.hdr[1];
    const uint32_t lane = threadIdx.x & 31, i = threadIdx.x;
    const bool any_multi = kClaim && a.any[ANY_MULTI] != 0u, any_sl = kClaim && a.any[ANY_STOCKLEVEL] != 0u;
    const uint32_t n_tiles = (a.B + P - 1) / P;
    uint32_t *fl = h.acc, *ml = h.acc + P;  // conflict flags; lines whose ORDER-LINE row is multi
    TxnCounts cnt;
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t t0 = tile * P, nt = min(P, a.B - t0), t = t0 + i;
        uint32_t f = 0, n = 0;
        bool ok = false, com = false;
        ltpg_tpcc_txn x{};
        if (i < P) {
            if (i < nt) x = load_txn(a, t, n_lines, false, ok);
            h.x[i] = x;
            const HeadOps o = head_ops(a.db, x, ok);
            n = ok && tpcc_kind(x.kind_info) == LTPG_TPCC_NEWORDER ? tpcc_ol_cnt(x.kind_info) : 0u;
            if (ok) {
                ulonglong2 s = ld_slot(a.reg + o.main_slot);
                if (kClaim && tpcc_kind(x.kind_info) == LTPG_TPCC_STOCKLEVEL)
                    s.y = ld_cg_u64(a.stock_w + 100000ull * x.w + x.a);
                f = conflicts_of(s, o.main_flags, t, epoch);
            }
            uint32_t lines = 0;
            if (!kClaim || any_multi) {
#pragma unroll
                for (uint32_t q = 0; q < 3; ++q) {
                    if (q >= o.n || (kClaim && !multi_row(a, claim_bit(a.db, o.table[q], o.row[q])))) continue;
                    f |= conflicts_of(ld_slot(a.reg + a.db.base[o.table[q]] + o.row[q]), o.flags[q], t, epoch);
                }
                if (kClaim && n) lines = multi_lines(a, x, n);
            }
            fl[i] = f;
            if (kClaim) ml[i] = lines;
        }
        const uint32_t lines_n = layout_lines<P>(h, n);
        for (uint32_t e = i; e < lines_n; e += T) {
            const uint32_t q = h.own[e], li = e - h.off[q];
            const ltpg_tpcc_txn &y = h.x[q];
            const ltpg_tpcc_line ln = load_line(a.lines, (uint64_t)y.line_off + li);
            uint32_t g = ln.supply_w != y.w ? FL_REMOTE : 0u;
            if (line_valid(ln, a.db.W)) {
                // stock write and ORDER-LINE insert: WAR and WAW each
                const uint64_t srow = 100000ull * ln.supply_w + ln.i_id;
                ulonglong2 s = make_ulonglong2(~0ull, 0ull);
                if (kClaim) {
                    s.y = ld_cg_u64(a.stock_w + srow);
                    if (any_sl && ((__ldg(a.sl_bits + (srow >> 5)) >> (srow & 31u)) & 1u))
                        s.x = ld_slot(a.reg + a.db.base[LTPG_T_STOCK] + srow).x;
                } else {
                    s = ld_slot(a.reg + a.db.base[LTPG_T_STOCK] + srow);
                }
                g |= conflicts_of(s, OPF_WRITE, t0 + q, epoch);
                if (!kClaim || (any_multi && ((ml[q] >> li) & 1u)))
                    g |= conflicts_of(ld_slot(a.reg + a.db.base[LTPG_T_ORDERLINE] + tpcc_ol_row(y.w, y.c, li)),
                                      OPF_WRITE, t0 + q, epoch);
            } else {
                g |= FL_BAD_LINE;
            }
            if (g & ~fl[q]) atomicOr(&fl[q], g);
        }
        __syncthreads();
        if (i < P) {  // whole warps
            const uint32_t all = fl[i];
            f = all & (LTPG_FLAG_RAW | LTPG_FLAG_WAR | LTPG_FLAG_WAW);
            com = ok && !(all & FL_BAD_LINE) && commits(f);
            if (com) f |= LTPG_FLAG_COMMIT;
            if (i < nt) {
                if (txn_not_found(x)) f |= LTPG_FLAG_NOT_FOUND;
                a.flags[t] = (uint8_t)f;
            }
            const unsigned bal = __ballot_sync(FULL, com);
            const unsigned braw = __ballot_sync(FULL, (f & LTPG_FLAG_RAW) != 0u);
            const unsigned bwar = __ballot_sync(FULL, (f & LTPG_FLAG_WAR) != 0u);
            const unsigned bwaw = __ballot_sync(FULL, (f & LTPG_FLAG_WAW) != 0u);
            if (lane == 0 && i < nt) {
                a.bitmap[t >> 5] = bal;
                cnt.com += __popc(bal);
                cnt.raw += __popc(braw);
                cnt.war += __popc(bwar);
                cnt.waw += __popc(bwaw);
            }
            if (com)
                write_head(a.db, x, !(all & FL_REMOTE), txn_base + t,
                           tpcc_kind(x.kind_info) == LTPG_TPCC_DELIVERY ? a.results[t] : 0, hot);
        }
        // the committed orders' lines, laid out back to back
        const uint32_t wlines = layout_lines<P>(h, com ? n : 0u);
        for (uint32_t e = i; e < wlines; e += T) {
            const uint32_t q = h.own[e], li = e - h.off[q];
            const ltpg_tpcc_txn &y = h.x[q];
            write_line(a.db, y, li, load_line(a.lines, (uint64_t)y.line_off + li));
        }
        __syncthreads();
    }
    return cnt;
}

__device__ __forceinline__ void hot_init(uint32_t *hot, uint32_t n) {
    for (uint32_t i = threadIdx.x; i < 2u * n; i += blockDim.x) hot[i] = 0u;
    __syncthreads();
}
// After the last tile's barrier, or hot_init's.
__device__ __forceinline__ void hot_flush(const TpccDev &db, const uint32_t *hot) {
    for (uint32_t i = threadIdx.x; i < 11u * db.W; i += blockDim.x) {
        const unsigned long long v = ((unsigned long long)hot[2u * i + 1u] << 32) | hot[2u * i];
        if (!v) continue;
        uint64_t *p = i < db.W ? col_ptr(db, LTPG_T_WAREHOUSE, i, W_YTD) : col_ptr(db, LTPG_T_DISTRICT, i - db.W, D_YTD);
        red_add_u64(reinterpret_cast<unsigned long long *>(p), v);
    }
}

template <uint32_t P, uint32_t T, bool kClaim>
__global__ void __launch_bounds__(T, 1536 / T) tpcc_exec_tuned(TpccTunedArgs a) {
    __shared__ TpccTile<P> h;
    if (P < T) let_next_start();
    clear_stats(a.st);
    tpcc_exec_tiles<P, T, kClaim>(a, h, slot_tag(a.ctl->epoch));
}

template <uint32_t P, uint32_t T, bool kClaim>
__global__ void __launch_bounds__(T, 1536 / T) tpcc_checkwb_tuned(TpccTunedArgs a) {
    __shared__ TpccTile<P> h;
    extern __shared__ __align__(16) uint32_t hot_dyn[];
    uint32_t *hot = a.db.W <= HOT_SMEM_MAX_W ? hot_dyn : nullptr;
    if (hot) hot_init(hot, 11u * a.db.W);
    if (P < T) wait_for_previous();
    const TxnCounts cnt = tpcc_checkwb_tiles<P, T, kClaim>(a, h, a.ctl->epoch, hot);
    if (hot) hot_flush(a.db, hot);
    add_counters(a.st, a.ctl, cnt);
    finish_batch<false>(a.ctl);
}

// One cooperative kernel per batch: execute+register, a bounded grid barrier,
// check + write-back.  What the second phase loads that the first wrote:
// registration slots (ld_slot: ld.global.cg, served by L2) and the tile's
// results (written by the same block, ordered by __syncthreads).  Table rows
// are read through the read-only path only in the first phase, before any
// row is written, apart from ITEM's (no transaction writes them); the second
// phase's read-modify-writes (C_BALANCE, S_QUANTITY by atomicCAS) touch rows
// that one committed transaction writes (WAW), whose batch-start value is what
// they must see.
template <uint32_t P, uint32_t T>
__global__ void __launch_bounds__(T, 1536 / T) tpcc_persistent(TpccTunedArgs a) {
    __shared__ TpccTile<P> h;
    extern __shared__ __align__(16) uint32_t hot_dyn[];
    uint32_t *hot = a.db.W <= HOT_SMEM_MAX_W ? hot_dyn : nullptr;
    const uint32_t epoch = a.ctl->epoch;
    clear_stats(a.st);
    if (hot) hot_init(hot, 11u * a.db.W);
    tpcc_exec_tiles<P, T, false>(a, h, slot_tag(epoch));
    TxnCounts cnt;
    if (grid_barrier(a.ctl)) cnt = tpcc_checkwb_tiles<P, T, false>(a, h, epoch, hot);
    if (hot) hot_flush(a.db, hot);
    add_counters(a.st, a.ctl, cnt);
    finish_batch<false>(a.ctl);
}

template <uint32_t P, uint32_t T, bool kClaim>
static cudaError_t tpcc_launch_tuned(ltpg_ctx *c, const TpccTunedArgs &a_in, int mode) {
    TpccTunedArgs a = a_in;
    constexpr uint32_t threads = T;
    const size_t smem = a.db.W <= HOT_SMEM_MAX_W ? 11u * a.db.W * sizeof(long long) : 0u;
    const bool persistent = mode == LTPG_MODE_PERSISTENT;
    const void *k = persistent ? (const void *)tpcc_persistent<P, T> : (const void *)tpcc_checkwb_tuned<P, T, kClaim>;
    // above 48 KB of static (at most 38) + dynamic shared memory a kernel must opt in
    cudaError_t e = cudaSuccess;
    if (smem > 9 * 1024) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    if (c->launch_c.blocks_per_sm && (int)c->launch_c.blocks_per_sm < per_sm) per_sm = (int)c->launch_c.blocks_per_sm;
    const uint32_t n_tiles = (a.B + P - 1) / P;
    const uint32_t grid = std::min<uint32_t>(n_tiles, (uint32_t)(per_sm * c->sm_count));
    if (persistent) {
        prof_mark(c, 0);
        void *args[] = {&a};
        count_launch(c);
        e = cudaLaunchCooperativeKernel((const void *)tpcc_persistent<P, T>, dim3(grid), dim3(threads), args, smem,
                                        c->stream);
        if (e != cudaSuccess) return e;
        for (int m = 1; m < PROF_MARKS; ++m) prof_mark(c, m);
        return cudaSuccess;
    }
    prof_mark(c, 0);
    count_launch(c);
    if (kClaim) {
        e = cudaMemsetAsync(a.claim, 0, claim_total_words(a.db.W) * sizeof(uint32_t), c->stream);
        if (e != cudaSuccess) return e;
    }
    tpcc_exec_tuned<P, T, kClaim><<<grid, threads, 0, c->stream>>>(a);
    if (kClaim) {
        tpcc_register_multi<<<std::min<uint32_t>((a.B + 255) / 256, 8u * (uint32_t)c->sm_count), 256, 0, c->stream>>>(a);
        count_launch(c);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    prof_mark(c, 1);
    count_launch(c);
    // on small tiles only: the early blocks of a full wave are in the way (the
    // mix at 2^20: 283 -> 316 us; at 20,000: 21 -> 19)
    e = launch_next(tpcc_checkwb_tuned<P, T, kClaim>, P < T && !c->profiling, grid, threads, smem, c->stream, a);
    if (e != cudaSuccess) return e;
    for (int m = 2; m < PROF_MARKS; ++m) prof_mark(c, m);
    return cudaSuccess;
}

// Tile of a block of T threads: the smallest of T/8 (at least a warp), T/4, T/2
// and T transactions that still gives every tile a block of its own among those
// resident (1,536 threads an SM).  A small tile's threads fetch one order line
// or two in turn where a full tile's fetch five (W = 64, 2,000 transactions:
// 32 us on full tiles, 17 us on T/8).
template <uint32_t T>
static cudaError_t tpcc_launch_block(ltpg_ctx *c, const TpccTunedArgs &a, int mode, bool claim) {
    constexpr uint32_t S = T / 8 < 32u ? 32u : T / 8;
    const uint32_t blocks = (uint32_t)c->sm_count * (1536u / T);
    if (claim) return tpcc_launch_tuned<T, T, true>(c, a, mode);
    if (a.B <= (uint64_t)blocks * S) return tpcc_launch_tuned<S, T, false>(c, a, mode);
    if (T / 4 > S && a.B <= (uint64_t)blocks * (T / 4)) return tpcc_launch_tuned<(T / 4 > S ? T / 4 : S), T, false>(c, a, mode);
    if (a.B <= (uint64_t)blocks * (T / 2)) return tpcc_launch_tuned<T / 2, T, false>(c, a, mode);
    return tpcc_launch_tuned<T, T, false>(c, a, mode);
}

// Claims pay in large batches over large tables whose inserts meet no other op
// (us a batch, slots -> claims; NewOrder + Payment at W = 64: 160,000
// transactions 70 -> 67, 2^18 108 -> 97, 2^20 282 -> 210; W = 16, 2^18: 82 ->
// 78; W = 8, 2^19: 114 -> 116).  They do not where orders are read or delivered
// in the batch that makes them (the five-transaction mix at 2^18: 110 -> 118) or
// the ids of a warehouse wrap in it (W = 4, 2^20: 161 -> 244).
bool tpcc_claims(const Slot &s, const TpccDb &db) {
    return !db.no_claims && !s.reads_orders && db.W >= 16u && s.n_txn >= CLAIM_MIN_TXNS && s.n_txn <= 32768ull * db.W;
}

cudaError_t tpcc_run_tuned(ltpg_ctx *c, Slot &s, int mode) {
    if (s.n_txn == 0) return cudaSuccess;
    TpccTunedArgs a;
    a.txns = s.txns;
    a.lines = s.lines;
    a.hdr = s.dev_hdr;
    a.B = s.n_txn;
    a.db = make_dev(c);
    a.reg = c->tpcc.reg;
    a.results = s.results;
    a.flags = s.flags;
    a.bitmap = s.bitmap;
    a.st = s.stats;
    a.ctl = c->ctl;
    a.filter = c->launch_c.filter;
    a.dedupe = c->launch_c.dedupe;
    a.claim = c->tpcc.claim;
    a.multi = a.claim + claim_words(a.db.W);
    a.any = a.multi + claim_words(a.db.W);
    a.sl_bits = a.any + 2;
    a.stock_w = c->tpcc.stock_w;
    const bool claim = mode != LTPG_MODE_PERSISTENT && c->tpcc.claim && tpcc_claims(s, c->tpcc);
    switch (c->launch_c.block) {
    case 256: return tpcc_launch_block<256>(c, a, mode, claim);
    case 512: return tpcc_launch_block<512>(c, a, mode, claim);
    default: return tpcc_launch_block<128>(c, a, mode, claim);
    }
}

// Packed order lines (ltpg_tpcc_pack_lines) back to ltpg_tpcc_line: one
// 4-byte load and one 8-byte store per line.
__global__ void __launch_bounds__(256) tpcc_unpack_lines_kernel(const uint32_t *__restrict__ packed, uint64_t n,
                                                                 ltpg_tpcc_line *__restrict__ lines) {
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
        const uint32_t p = __ldg(packed + i);
        reinterpret_cast<uint2 *>(lines)[i] = make_uint2(p & 0x1FFFFu, ((p >> 17) & 0x7FFu) | ((p >> 28) << 16));
    }
}

cudaError_t tpcc_unpack_lines(Slot &s, cudaStream_t st) {
    const uint64_t n = s.n_lines;
    if (!n) return cudaSuccess;
    const uint32_t grid = (uint32_t)std::min<uint64_t>((n + 255) / 256, 4096);
    tpcc_unpack_lines_kernel<<<grid, 256, 0, st>>>(s.packed_lines, n, s.lines);
    return cudaGetLastError();
}

}  // namespace ltpg
