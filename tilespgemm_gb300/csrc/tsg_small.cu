// tsg_small.cu -- the small-product path of tsg_spgemm: C = A*B row by row,
// one warp per row of C, the row kept in a shared-memory hash table (or, for
// rows of at most 32 products, in the warp's registers).
//
// The tiled pipeline (conversion, two symbolic steps, binned numeric step)
// costs some 27 launches and three host waits per call, which is most of
// the time of a product of a few million intermediate products (a 2D
// Laplacian on a 256x256 grid: 1.6 M products).  Products whose every row of
// A meets at most SMALL_MAX_PRODUCTS entries of B take this path instead:
//   k_small_count  per row, the distinct columns among its products (hash
//                  insertions) -> rowcnt; rows over the limit are counted in
//                  stat[0] (the caller then takes the tiled path), the
//                  products in stat[1]
//   (the look-back scan of rowcnt gives C's row pointer)
//   k_small_fill   per row, the same walk accumulating values, then the row's
//                  entries written in column order.  With `kept` (C's row
//                  pointer kept from the last call of the same shape, no
//                  count pass before it) a row whose entries differ from the
//                  kept count, or that is over the limit, adds 1 to kept[0]
//                  (the caller then runs the count pass), the products go
//                  to kept[1].
//   k_small_fill_one  the same for a repeated shape whose rows of A have up to
//                  32 entries and bring up to 32 products: a warp takes four
//                  rows (one where there are few), whose loads share their
//                  latencies, and the last CTA writes the counts and flags to
//                  the host's memory, so that the call is one launch and one wait
// The row's products are dealt 32 at a time in A's order then B's (lane =
// position in the concatenation of the B rows of up to 32 A entries); lanes
// of one round that meet in one output apply in lane order, so every entry
// of C sees exactly the sequence fma(a_ik, b_kj, c) over k in A's row order,
// as in the tiled path and the oracle: the two paths give identical values.
// The reference has no such path; its per-call setup is the overhead
// (main_spgemm-col.cu:4529-4774) that this path removes for small products.
#include "tsg_internal.cuh"

namespace tsg {

namespace {

constexpr int SH_WARPS = 8;                    // rows per CTA (one warp each)
constexpr int SH_BITS = 8;
constexpr int SH_CAP = 1 << SH_BITS;           // hash slots per warp
static_assert(SMALL_MAX_PRODUCTS * 2 <= SH_CAP, "the table stays at most half full");

__device__ __forceinline__ int sh_hash(int col) { return (int)(((unsigned)col * 2654435761u) >> (32 - SH_BITS)); }

// slot of `col` in the warp's table, inserting it if absent (fresh: it was);
// -1 if the table is full (not reached: at most SMALL_MAX_PRODUCTS keys)
__device__ __forceinline__ int sh_insert(int *key, int col, bool &fresh)
{
    int h = sh_hash(col);
    fresh = false;
    for (int probe = 0; probe < SH_CAP; ++probe) {
        const int old = atomicCAS(key + h, -1, col);
        if (old == -1) { fresh = true; return h; }
        if (old == col) return h;
        h = (h + 1) & (SH_CAP - 1);
    }
    return -1;
}

// Up to 32 A entries of row r, lane q < na holding entry q's B row
// [bs, bs + len) (len clamped to SMALL_MAX_PRODUCTS + 1, empty for an
// out-of-range column of A; B's row pointers clamped into [0, nnzB], so
// that an unchecked row pointer reads nothing outside B).
struct Batch {
    long long bs = 0;
    int len = 0;
};

__device__ __forceinline__ Batch load_batch(const SmallOperands &o, long long p, int na, int lane, int *flags, int &k)
{
    Batch b;
    k = -1;
    if (lane < na) {
        k = o.colA[p + lane];
        if (o.check && (unsigned)k >= (unsigned)o.ka) set_flag(flags, FLAG_BAD_INPUT);
        if ((unsigned)k < (unsigned)o.ka) {
            const RowPtr rpB = o.rpB;
            const long long nnzB = o.nnzB;
            const long long s0 = rpB[k], s1 = rpB[k + 1];
            b.bs = s0 < 0 ? 0 : (s0 > nnzB ? nnzB : s0);
            const long long l = (s1 > nnzB ? nnzB : s1) - b.bs;
            b.len = (int)(l < 0 ? 0 : (l > SMALL_MAX_PRODUCTS + 1 ? SMALL_MAX_PRODUCTS + 1 : l));
        } else {
            k = -1;
        }
    }
    return b;
}

// Row r's entries [a0, a1) of A, clamped into [0, nnzA]; with `check` the
// row pointer is validated as the validation kernel does (bounds, order,
// first 0, last nnzA: lane 0 flags FLAG_BAD_INPUT).
__device__ __forceinline__ void row_span(RowPtr rp, int r, int m, long long nnz, bool check, int lane, int *flags,
                                         long long &a0, long long &a1)
{
    const long long v0 = rp[r], v1 = rp[r + 1];
    if (check && lane == 0) {
        const bool bad = v0 < 0 || v0 > nnz || v1 < v0 || v1 > nnz || (r == 0 && v0 != 0) || (r == m - 1 && v1 != nnz);
        if (bad) set_flag(flags, FLAG_BAD_INPUT);
    }
    a0 = v0 < 0 ? 0 : (v0 > nnz ? nnz : v0);
    a1 = v1 < a0 ? a0 : (v1 > nnz ? nnz : v1);
}

// the lane whose B row holds position f of the concatenation (last lane
// whose exclusive offset is at or before f)
__device__ __forceinline__ int owner_lane(int off, int f)
{
    int q = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const int oc = __shfl_sync(0xffffffffu, off, q + step);
        if (oc <= f) q += step;
    }
    return q;
}

// Rows whose products fit one round (at most 32, from at most 32 A
// entries) skip the table: the 32 lanes' keys are sorted across the warp
// (bitonic network on shuffles), equal columns then sit in adjacent lanes
// in product order, and the first lane of each run of equal columns starts
// an entry of C.
template <typename K>
__device__ __forceinline__ K warp_sort_up(K key, int lane)
{
    // the lanes that sort downwards in a phase hold their keys complemented,
    // so that a stage keeps the smaller or the larger by one bit of the lane
    K flip = 0;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
        const K down = (lane & k) && k < 32 ? ~(K)0 : (K)0;
        key ^= flip ^ down;
        flip = down;
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const K other = __shfl_xor_sync(0xffffffffu, key, j);
            key = (lane & j) ? max(key, other) : min(key, other);
        }
    }
    return key;
}

// One round's products sorted by (column, product index f = lane): lane
// i gets the i-th smallest, its column, and the A and B values of the lane
// that held it; live = false for the lanes past the products (c0 < 0).
template <typename K>
__device__ __forceinline__ void sort_products(int c0, double a, double bv, int lane, bool &live, int &col, double &sa,
                                              double &sb)
{
    K key = c0 >= 0 ? (((K)(unsigned)c0 << 5) | (K)(unsigned)lane) : ~(K)0;
    key = warp_sort_up(key, lane);
    live = key != ~(K)0;
    const int src = (int)(key & 31u);
    col = (int)(key >> 5);
    sa = __shfl_sync(0xffffffffu, a, src);
    sb = __shfl_sync(0xffffffffu, bv, src);
}

__global__ void __launch_bounds__(SH_WARPS * 32)
k_small_count(SmallOperands o, int *rowcnt, unsigned long long *stat)
{
    __shared__ int s_key[SH_WARPS][SH_CAP];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * SH_WARPS + warp;
    if (r >= o.m) return;
    const int *__restrict__ colB = o.colB;
    const int nb = o.nb;
    int *key = s_key[warp];
    bool table = false;      // the hash table is set up on the first batch that needs it
    long long a0, a1;
    row_span(o.rpA, r, o.m, o.nnzA, false, lane, nullptr, a0, a1);
    int cnt = 0, P = 0;
    bool over = false;
    for (long long pb = a0; pb < a1; pb += 32) {
        const int na = (int)min(32ll, a1 - pb);
        int k;
        const Batch b = load_batch(o, pb, na, lane, nullptr, k);
        const int incl = warp_incl_scan(b.len, lane);
        const int T = __shfl_sync(0xffffffffu, incl, 31);
        P += T;
        if (P > SMALL_MAX_PRODUCTS) { over = true; break; }
        const int off = incl - b.len;
        if (a1 - a0 <= 32 && T <= 32) {
            // one round: sort the columns, count the runs
            const int q = owner_lane(off, lane);
            const long long e = __shfl_sync(0xffffffffu, b.bs, q) + (lane - __shfl_sync(0xffffffffu, off, q));
            unsigned key = 0xffffffffu;
            if (lane < T) {
                const int col = colB[e];
                if ((unsigned)col < (unsigned)nb) key = (unsigned)col;
            }
            key = warp_sort_up(key, lane);
            const unsigned prev = __shfl_up_sync(0xffffffffu, key, 1);
            const bool head = key != 0xffffffffu && (lane == 0 || prev != key);
            const unsigned heads = __ballot_sync(0xffffffffu, head);   // every lane takes part
            cnt = lane == 0 ? __popc(heads) : 0;
            break;
        }
        if (!table) {
            for (int t = lane; t < SH_CAP; t += 32) key[t] = -1;
            __syncwarp();
            table = true;
        }
        for (int base = 0; base < T; base += 32) {
            const int f = base + lane;
            const int q = owner_lane(off, f);
            const long long e = __shfl_sync(0xffffffffu, b.bs, q) + (f - __shfl_sync(0xffffffffu, off, q));
            if (f < T) {
                const int col = colB[e];
                if ((unsigned)col < (unsigned)nb) {
                    bool fresh;
                    sh_insert(key, col, fresh);
                    cnt += fresh ? 1 : 0;
                }
            }
        }
    }
    cnt = warp_sum_int(cnt);
    if (lane == 0) {
        rowcnt[r] = over ? 0 : cnt;
        if (over) atomicAdd(stat, 1ull);
        else if (P) atomicAdd(stat + 1, (unsigned long long)P);
        // stat[2]: a row that does not fit one round (more than 32 products or A entries)
        if (!over && (P > 32 || a1 - a0 > 32) && stat[2] == 0) atomicMax(stat + 2, 1ull);
    }
}

// B's row pointer and columns, checked across the whole grid (A*B; with A*A
// the rows' own checks cover them)
__device__ __forceinline__ void check_b(const SmallOperands &o, int *flags)
{
    if (!o.check || o.b_is_a) return;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    bool bad = false;
    for (long long i = t0; i <= o.kb; i += stride) {
        const long long v = o.rpB[i];
        bad |= v < 0 || v > o.nnzB || (i == 0 && v != 0) || (i == o.kb && v != o.nnzB) || (i < o.kb && o.rpB[i + 1] < v);
    }
    for (long long q = t0; q < o.nnzB; q += stride) bad |= (unsigned)o.colB[q] >= (unsigned)o.nb;
    if (bad) set_flag(flags, FLAG_BAD_INPUT);
}

__global__ void __launch_bounds__(SH_WARPS * 32)
k_small_fill(SmallOperands o, const long long *__restrict__ rowptrC, long long cap, int *colC, double *valC,
             int *flags, unsigned long long *kept, void *rp_out, int rp_bits)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * SH_WARPS + warp;
    check_b(o, flags);
    const int m = o.m;
    if (r >= m) return;
    const int *__restrict__ colB = o.colB;
    const double *__restrict__ valA = o.valA;
    const double *__restrict__ valB = o.valB;
    const int nb = o.nb;
    const long long Rb = rowptrC[r], Re = rowptrC[r + 1];
    // C larger than the buffers: nothing is written (the caller sees nnzC
    // and runs this pass again into buffers of that size)
    if (rowptrC[m] > cap) return;
    if (rp_out && lane == 0) {   // the caller's row pointer, in its type
        if (rp_bits == 64) {
            static_cast<long long *>(rp_out)[r] = Rb;
            if (r == m - 1) static_cast<long long *>(rp_out)[m] = Re;
        } else {
            static_cast<int *>(rp_out)[r] = (int)Rb;
            if (r == m - 1) static_cast<int *>(rp_out)[m] = (int)Re;
        }
    }
    long long a0, a1;
    row_span(o.rpA, r, m, o.nnzA, o.check, lane, flags, a0, a1);
    if (a1 - a0 <= 32) {
        const int na = (int)(a1 - a0);
        int k;
        const Batch b = load_batch(o, a0, na, lane, flags, k);
        const int incl = warp_incl_scan(b.len, lane);
        const int T = __shfl_sync(0xffffffffu, incl, 31);
        if (T <= 32) {
            // one round: lane f holds product f (A's order, then B's); the
            // keys (column, f) sorted across the warp put each column's
            // products in adjacent lanes in product order, and the run's
            // first lane applies them in that order
            const double av = (lane < na && k >= 0) ? valA[a0 + lane] : 0.0;
            const int off = incl - b.len;
            const int q = owner_lane(off, lane);
            const long long e = __shfl_sync(0xffffffffu, b.bs, q) + (lane - __shfl_sync(0xffffffffu, off, q));
            const double a = __shfl_sync(0xffffffffu, av, q);
            int c0 = -1;
            double bv = 0.0;
            if (lane < T) {
                const int cb = colB[e];
                if ((unsigned)cb < (unsigned)nb) {
                    c0 = cb;
                    bv = valB[e];
                }
            }
            // 32-bit keys when B's columns leave room for the 5 bits of f
            bool live;
            int col;
            double sa, sb;
            if (nb <= (1 << 26)) sort_products<unsigned>(c0, a, bv, lane, live, col, sa, sb);
            else sort_products<unsigned long long>(c0, a, bv, lane, live, col, sa, sb);
            const int pcol = __shfl_up_sync(0xffffffffu, col, 1);
            const bool head = live && (lane == 0 || pcol != col);
            const unsigned heads = __ballot_sync(0xffffffffu, head);
            const int n = __popc(heads);
            if ((long long)n != Re - Rb) {
                if (lane == 0) {
                    if (kept) atomicAdd(kept, 1ull);
                    else set_flag(flags, FLAG_INTERNAL);
                }
                return;
            }
            if (kept && lane == 0 && T) atomicAdd(kept + 1, (unsigned long long)T);
            // run of lane i: lanes i, i+1, ... while the column stays col
            double acc = 0.0;
            bool more = head;
            for (int j = 0; __any_sync(0xffffffffu, more); ++j) {
                const int cj = __shfl_down_sync(0xffffffffu, col, j);
                const bool lj = __shfl_down_sync(0xffffffffu, live ? 1 : 0, j) != 0;
                const double aj = __shfl_down_sync(0xffffffffu, sa, j), bj = __shfl_down_sync(0xffffffffu, sb, j);
                more = more && lane + j < 32 && lj && cj == col;
                if (more) acc = fma(aj, bj, acc);
            }
            if (head) {
                const int rank = __popc(heads & lanemask_lt());
                colC[Rb + rank] = col;
                valC[Rb + rank] = acc;
            }
            return;
        }
    }
    __shared__ int s_key[SH_WARPS][SH_CAP];
    __shared__ double s_val[SH_WARPS][SH_CAP];
    __shared__ int s_ck[SH_WARPS][SMALL_MAX_PRODUCTS];
    __shared__ double s_cv[SH_WARPS][SMALL_MAX_PRODUCTS];
    int *key = s_key[warp];
    double *val = s_val[warp];
    for (int t = lane; t < SH_CAP; t += 32) { key[t] = -1; val[t] = 0.0; }
    __syncwarp();
    int P = 0;
    for (long long pb = a0; pb < a1; pb += 32) {
        const int na = (int)min(32ll, a1 - pb);
        int k;
        const Batch b = load_batch(o, pb, na, lane, flags, k);
        const double av = (lane < na && k >= 0) ? valA[pb + lane] : 0.0;
        const int incl = warp_incl_scan(b.len, lane);
        const int T = __shfl_sync(0xffffffffu, incl, 31);
        P += T;
        if (P > SMALL_MAX_PRODUCTS) {   // counted as over the limit: the row is empty here
            if (kept && lane == 0) atomicAdd(kept, 1ull);
            return;
        }
        const int off = incl - b.len;
        for (int base = 0; base < T; base += 32) {
            const int f = base + lane;
            const int q = owner_lane(off, f);
            const long long e = __shfl_sync(0xffffffffu, b.bs, q) + (f - __shfl_sync(0xffffffffu, off, q));
            const double a = __shfl_sync(0xffffffffu, av, q);
            int slot = -1;
            double bv = 0.0;
            if (f < T) {
                const int col = colB[e];
                if ((unsigned)col < (unsigned)nb) {
                    bool fresh;
                    slot = sh_insert(key, col, fresh);
                    bv = valB[e];
                }
            }
            // lanes on one output apply in lane order (A's order, then B's)
            const unsigned peers = __match_any_sync(0xffffffffu, slot >= 0 ? slot : -2 - lane);
            const int rank = __popc(peers & lanemask_lt());
            if (!__any_sync(0xffffffffu, rank > 0)) {
                if (slot >= 0) val[slot] = fma(a, bv, val[slot]);
            } else {
                const int rounds = __reduce_max_sync(0xffffffffu, (unsigned)__popc(peers));
                for (int q2 = 0; q2 < rounds; ++q2) {
                    if (q2 == rank && slot >= 0) val[slot] = fma(a, bv, val[slot]);
                    __syncwarp();
                }
            }
            __syncwarp();
        }
    }
    // the row's entries, compacted in slot order, then each to its rank by column
    int *ck = s_ck[warp];
    double *cv = s_cv[warp];
    int n = 0;
    for (int t0 = 0; t0 < SH_CAP; t0 += 32) {
        const int t = t0 + lane;
        const int kk = key[t];
        const unsigned bal = __ballot_sync(0xffffffffu, kk >= 0);
        if (kk >= 0) {
            const int p = n + __popc(bal & lanemask_lt());
            if (p < SMALL_MAX_PRODUCTS) { ck[p] = kk; cv[p] = val[t]; }
        }
        n += __popc(bal);
    }
    __syncwarp();
    if ((long long)n != Re - Rb || n > SMALL_MAX_PRODUCTS) {
        if (lane == 0) {
            if (kept) atomicAdd(kept, 1ull);
            else set_flag(flags, FLAG_INTERNAL);
        }
        return;
    }
    if (kept && lane == 0 && P) atomicAdd(kept + 1, (unsigned long long)P);
    for (int p = lane; p < n; p += 32) {
        const int c = ck[p];
        int rank = 0;
        for (int j = 0; j < n; ++j) rank += ck[j] < c ? 1 : 0;
        colC[Rb + rank] = c;
        valC[Rb + rank] = cv[p];
    }
}

// The fill at a kept row pointer for shapes whose rows all fit one round (at
// most 32 products from at most 32 A entries): a warp takes ONE_ROWS rows.
//   1. the rows' A entries side by side, one a lane (rows follow one another in
//      A), their B rows' places staged;
//   2. per row, lane f holds product f; the keys (column, f) sorted across
//      the warp put a column's products side by side in product order;
//   3. the rows' entries of C, one a lane: its products applied in order.
// A row that does not fit, or whose entries differ from the kept count, is
// reported through `kept`; its C is not used then.
// Bound by issue and by the FP64 pipe (a DFMA warp instruction holds it 20
// clocks whatever its lanes): a row of its own a warp issued one DFMA per
// product of its longest column, 5 on a 5-point Laplacian squared, 4 rows
// together 2.5 a row, and the sorted products needed 12 shuffles each.
// 256 x 256 Laplacian, A*A: 48 -> 33 us, 490 -> 315 instructions a row.
constexpr int ONE_WARPS = 4;

struct __align__(16) OneShare {   // an A entry's B row: entry f + delta for the group's product f
    int delta, pad;
    double a;
};

template <int ONE_ROWS>
struct OneWarp {
    double2 ab[ONE_ROWS * 32];         // products: A's and B's value
    OneShare share[32];
    uint2 out[ONE_ROWS * 32];          // entries of C: column, first sorted product | products << 8
    unsigned char src[ONE_ROWS * 32];  // sorted products' places in ab
};

template <int ONE_ROWS, typename K>
__global__ void __launch_bounds__(ONE_WARPS * 32)
k_small_fill_one(SmallOperands o, const long long *__restrict__ rowptrC, long long cap, int *__restrict__ colC,
                 double *__restrict__ valC, SmallReport *rep, long long *host, void *rp_out, int rp_bits)
{
    __shared__ OneWarp<ONE_ROWS> s_w[ONE_WARPS];
    int *flags = rep->flags;
    unsigned long long *kept = rep->kept;
    __shared__ unsigned s_prod[ONE_WARPS];
    constexpr unsigned FULL = 0xffffffffu;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    check_b(o, flags);
    OneWarp<ONE_ROWS> &w = s_w[warp];
    const int m = o.m, nb = o.nb;
    const int r0 = (blockIdx.x * ONE_WARPS + warp) * ONE_ROWS, nr = max(0, min(ONE_ROWS, m - r0));
    unsigned products = 0;
    if (nr > 0 && rowptrC[m] <= cap) {
        // lane i: row r0 + i's span in A and C, and the caller's row pointer
        int a0 = 0, a1 = 0, nc = 0;
        long long Rb = 0;
        if (lane < nr) {
            const int r = r0 + lane;
            long long s, e;
            row_span(o.rpA, r, m, o.nnzA, o.check, 0, flags, s, e);
            a0 = (int)s;
            a1 = (int)e;
            Rb = rowptrC[r];
            const long long Re = rowptrC[r + 1];
            nc = (int)(Re - Rb);
            if (rp_out) {
                if (rp_bits == 64) {
                    static_cast<long long *>(rp_out)[r] = Rb;
                    if (r == m - 1) static_cast<long long *>(rp_out)[m] = Re;
                } else {
                    static_cast<int *>(rp_out)[r] = (int)Rb;
                    if (r == m - 1) static_cast<int *>(rp_out)[m] = (int)Re;
                }
            }
        }
        Rb = __shfl_sync(FULL, Rb, 0);
        unsigned bad = 0;
        int nout = 0;
        for (int g0 = 0; g0 < nr;) {
            // rows [g0, g1): as many as bring at most 32 A entries together
            const int first = __shfl_sync(FULL, a0, g0);
            const unsigned fit = __ballot_sync(FULL, lane >= g0 && lane < nr && a1 - first <= 32 && a0 >= first);
            int g1 = g0 + __ffs(~(fit >> g0)) - 1;
            if (g1 == g0) {     // one row of more than 32 A entries
                ++bad;
                ++g0;
                continue;
            }
            const int last = __shfl_sync(FULL, a1, g1 - 1);
            int k;
            const Batch b = load_batch(o, first, last - first, lane, flags, k);
            const int incl = warp_incl_scan(b.len, lane);
            const int off = incl - b.len;
            const unsigned full = __ballot_sync(FULL, b.len > 0);
            __syncwarp();
            if (b.len > 0) {
                OneShare &x = w.share[__popc(full & lanemask_lt())];
                x.delta = (int)b.bs - off;
                x.a = o.valA[first + lane];
            }
            __syncwarp();
            int col[ONE_ROWS], cnt[ONE_ROWS];
#pragma unroll
            for (int u = 0; u < ONE_ROWS; ++u) {
                col[u] = -1;
                cnt[u] = 0;
                const int i = g0 + u;
                if (i < g1) {
                    const int e0 = __shfl_sync(FULL, a0, i) - first, e1 = __shfl_sync(FULL, a1, i) - first;
                    const int p0 = e0 > 0 ? __shfl_sync(FULL, incl, (e0 - 1) & 31) : 0;
                    const int p1 = e1 > 0 ? __shfl_sync(FULL, incl, (e1 - 1) & 31) : 0;
                    const int T = p1 - p0, d = off - p0;
                    cnt[u] = T;
                    if (T > 32) ++bad;
                    else {
                        // a share that starts at this row's product d sets bit d
                        const unsigned st = __reduce_or_sync(FULL, (b.len > 0 && d >= 0 && d < T) ? 1u << d : 0u);
                        if (lane < T) {
                            const int q = __popc(full & ((1u << (e0 & 31)) - 1u)) + __popc(st & (lanemask_lt() | (1u << lane))) - 1;
                            const OneShare x = w.share[q];
                            const int e = x.delta + p0 + lane;
                            const int c = o.colB[e];
                            if ((unsigned)c < (unsigned)nb) col[u] = c;
                            w.ab[u * 32 + lane] = make_double2(x.a, o.valB[e]);
                        }
                        products += (unsigned)T;
                    }
                }
            }
            // the sorts, and the entries of C in order
            const int base = nout;
#pragma unroll
            for (int u = 0; u < ONE_ROWS; ++u) {
                const int i = g0 + u;
                if (i < g1 && cnt[u] <= 32) {
                    K key = col[u] >= 0 ? (((K)(unsigned)col[u] << 5) | (K)(unsigned)lane) : ~(K)0;
                    key = warp_sort_up(key, lane);
                    const bool live = key != ~(K)0;
                    const int c = (int)(key >> 5);
                    const int pc = __shfl_up_sync(FULL, c, 1);
                    const bool head = live && (lane == 0 || pc != c);
                    const unsigned heads = __ballot_sync(FULL, head), lives = __ballot_sync(FULL, live);
                    const int n = __popc(heads);
                    if (n != __shfl_sync(FULL, nc, i)) {
                        ++bad;
                    } else {
                        w.src[u * 32 + lane] = (unsigned char)(key & 31u);
                        if (head) {
                            const unsigned later = lane < 31 ? heads >> (lane + 1) : 0u;
                            const int len = later ? __ffs(later) : __popc(lives) - lane;
                            w.out[nout - base + __popc(heads & lanemask_lt())] =
                                make_uint2((unsigned)c, (unsigned)(u * 32 + lane) | (unsigned)len << 8);
                        }
                        nout += n;
                    }
                }
            }
            __syncwarp();
            for (int t = lane; t < nout - base; t += 32) {
                const uint2 x = w.out[t];
                const int at = (int)(x.y & 0xffu), row = at & ~31;
                double acc = 0.0;
                for (int q = at; q < at + (int)(x.y >> 8); ++q) {
                    const double2 p = w.ab[row + w.src[q]];
                    acc = fma(p.x, p.y, acc);
                }
                colC[Rb + base + t] = (int)x.x;
                valC[Rb + base + t] = acc;
            }
            g0 = g1;
        }
        if (bad && lane == 0) atomicAdd(kept, (unsigned long long)bad);
    }
    if (lane == 0) s_prod[warp] = products;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long sum = 0;
        for (int q = 0; q < ONE_WARPS; ++q) sum += s_prod[q];
        if (sum) atomicAdd(kept + 1, sum);
        // the last CTA reports to the host and clears the counts for the next call
        __threadfence();
        if (atomicAdd(&rep->done, 1u) == gridDim.x - 1) {
            __threadfence();
            volatile SmallReport *v = rep;
            host[0] = (long long)v->kept[0];
            host[1] = (long long)v->kept[1];
            for (int f = 0; f < FLAG_COUNT; ++f) {
                host[2 + f] = v->flags[f];
                v->flags[f] = 0;
            }
            v->kept[0] = v->kept[1] = 0;
            v->done = 0;
            __threadfence_system();
        }
    }
}

}  // namespace

cudaError_t small_count(Pool &pool, const SmallOperands &o, int *rowcnt, unsigned long long *stat)
{
    if (o.m <= 0) return cudaSuccess;
    k_small_count<<<(unsigned)((o.m + SH_WARPS - 1) / SH_WARPS), SH_WARPS * 32, 0, pool.stream>>>(o, rowcnt, stat);
    ::tsg::count_launch();
    return cudaGetLastError();
}

cudaError_t small_fill(Pool &pool, const SmallOperands &o, const long long *rowptrC, long long cap, int *colC,
                       double *valC, int *flags, unsigned long long *kept, void *rp_out, int rp_bits)
{
    const int m = o.m;
    if (m <= 0) {   // C's row pointer is the single 0
        if (!rp_out) return cudaSuccess;
        return cudaMemsetAsync(rp_out, 0, rp_bits == 64 ? 8 : 4, pool.stream);
    }
    const unsigned grid = (unsigned)((m + SH_WARPS - 1) / SH_WARPS);
    k_small_fill<<<grid, SH_WARPS * 32, 0, pool.stream>>>(o, rowptrC, cap, colC, valC, flags, kept, rp_out, rp_bits);
    ::tsg::count_launch();
    return cudaGetLastError();
}

cudaError_t small_fill_one(Pool &pool, const SmallOperands &o, const long long *rowptrC, long long cap, int *colC,
                           double *valC, SmallReport *rep, long long *host, void *rp_out, int rp_bits)
{
    // one row a warp while the rows do not fill the SMs' warps (1,024 rows:
    // 8.7 us, 11.3 with four); 32-bit keys when B's columns leave room for
    // the 5 bits of f
    const int rows = o.m < 20000 ? 1 : 4;
    const unsigned grid = (unsigned)((o.m + ONE_WARPS * rows - 1) / (ONE_WARPS * rows));
    auto run = [&](auto kernel) {
        kernel<<<grid, ONE_WARPS * 32, 0, pool.stream>>>(o, rowptrC, cap, colC, valC, rep, host, rp_out, rp_bits);
    };
    const bool narrow = o.nb <= (1 << 26);
    if (rows == 1) narrow ? run(k_small_fill_one<1, unsigned>) : run(k_small_fill_one<1, unsigned long long>);
    else narrow ? run(k_small_fill_one<4, unsigned>) : run(k_small_fill_one<4, unsigned long long>);
    ::tsg::count_launch();
    return cudaGetLastError();
}

}  // namespace tsg
