// tsg_rows.cu -- the row path of tsg_spgemm: C = A*B row by row for products
// whose 16x16 tiles are nearly empty (graphs, unstructured matrices).
//
// A tile of such a matrix holds one to three entries, so tile masks move 16
// halfwords for each of them, a hub's tile-row is one CTA's work, and its
// wide rows accumulate in C itself.  Here a row of C is cut into *items* by
// its own entries, each one warp's or one CTA's work anywhere on the GPU:
//   k_row_sample    the products of every 16th row (the choice of the path)
//   k_row_extents / k_row_products   per row of C its products and the blocks
//                   of ROW_BLK columns it can reach; heavy rows listed by
//                   weight, so that the longest chains start first
//   k_row_cuts      per row of B the first entry at or past every block (the
//                   cut table), when a row of C has several items
//   k_row_symbolic  per row of C a bitmap of its columns in shared memory, its
//                   entries per block, and from them its items: one for a
//                   light row, else runs of blocks that close at ITEM_T
//                   entries or ITEM_BLKS blocks; dense enough bitmaps are kept
//   (the look-back scan of the row counts gives C's row pointer)
//   k_row_numeric   per item: the bitmap of its columns (kept, or marked again)
//                   and running counts (a column's position = count + popc),
//                   then its products in
//                   steps, one A entry's B entries each: one fma a product on
//                   its position's accumulator in shared memory
// The steps follow one another in A's row order and a step's columns differ,
// so every entry of C sees fma(a_ik, b_kj, c) over k in A's row order, from
// 0.0, as in the tiled kernels and the oracle: the values are the same bits.
// B's rows must be strictly increasing (checked on the device by
// k_count_descents; the tiled path takes the others).
//
// Short rows with wide spans are sorted instead (k_row_sort, below).
//
// Measured on GB300, before (tiled) and after, whole call on the device:
//   R-MAT 2^12 x 8 A*A^T 1,170 -> 373 us, 2^15 x 16 A*A^T 8.9 -> 1.5 ms,
//   2^16 x 12 A*A 12.9 -> 2.45 ms, 2^18 x 16 A*A^T 81 -> 33.5 ms;
//   uniform 120,007 x 80,021 x 100,003, 16 and 12 a row: 10.3 -> 0.59 ms;
//   512 mixed products of 64 to 16,384 rows: 41.9 -> 22.6 ms.
// What bounds it (2^16, counters): k_row_numeric, 2/3 of the time: FP64 pipe 46
// to 56 % busy (a step holds it as long with 3 lanes as with 32; 2^18: half of
// the 211 M steps bring 8 entries or fewer), issue 39 to 44 %, and between
// them the latency of a step's chain (B's entry, its word, its accumulator,
// the fma) over the 14 to 20 warps that an SM's shared memory holds: 28
// instructions a step and 7 to stage it; marking an item's columns again cost
// another 28 (2^18: 41.0 ms without kept bitmaps).  k_row_symbolic is bound by
// its bitmap's shared-memory accesses and, for short rows, by a row's fixed cost.
// Tried without gain: products flattened 32 at a time over an item's A
// entries, half the rounds, lanes that meet in a column ordered by match (2^18:
// 77 ms; a match costs 2 clocks a distinct value and SM), by atomicMin in a
// table of 512 slots (37.3 for 34.8 ms: its 2 KB cost two warps an SM), or one
// A entry after another (34.5 to 37.7; 512 mixed products 28 for 24.4); items
// of 6,144 entries as a CTA's, 128 entries a step (67 ms: idle warps and a
// barrier a step); groups of 2 or 8 steps in flight in place of 4 (50 / 58
// against 45 ms: loads exposed, code outgrows the instruction cache); 24
// warps an SM at 80 registers, or a finer list of classes (within 2 %).
// The reference bins C's rows by intermediate products for its tile-level
// symbolic step (spgemm_nsparse_kernel.h:32-311); it has no row path.
#include "tsg_internal.cuh"
#include "tsg_rows.cuh"

#include <algorithm>
#include <climits>

namespace tsg {

namespace {

constexpr unsigned FULL = 0xffffffffu;
// Rows sorted in place of a bitmap: the bitmap costs by the row's blocks, the
// sort by its products, but the line looks at the blocks alone, where R-MAT
// graphs' rows turn.  Call with bitmaps / sorted: 32 blocks (R-MAT 2^15 x 16
// A*A^T) 2,229 / 2,311 us, 64 (2^16 x 12 A*A) 3,008 / 3,155, 256 (2^18 x 16)
// 35,674 / 35,066.  Uniform rows would gain by the sort from further down:
// 120,000 of 192 products over 20 blocks 832 / 519 us, 59 1,290 / 520, 79 1,834 /
// 517, 98 1,986 / 513; of 484 products 1,132 / 1,274, 2,101 / 1,293, 2,238 / 1,297
// and 2,401 / 1,297.
__device__ __forceinline__ bool sorted_row(const RowArgs &g, long long p, int nb)
{
    return p > 0 && p <= g.sort_max && nb >= SORT_NB;
}

// The products of every step-th row of C, times step (one warp a row).
__global__ void __launch_bounds__(256)
k_row_sample(RowArgs g, int step, unsigned long long *out, const int *flags)
{
    if (flags[FLAG_BAD_INPUT]) return;
    const long long r = (blockIdx.x * 8ll + (threadIdx.x >> 5)) * step;
    if (r >= g.m) return;
    long long p = 0;
    for (long long e = g.rpA[r] + (threadIdx.x & 31); e < g.rpA[r + 1]; e += 32) {
        const int k = g.colA[e];
        if ((unsigned)k < (unsigned)g.k) p += g.rpB[k + 1] - g.rpB[k];
    }
    p = warp_sum_ll(p);
    if ((threadIdx.x & 31) == 0 && p) atomicAdd(out, (unsigned long long)(p * step));
}

// Per row of B its first and last block of columns and its entries (one thread each).
__global__ void k_row_extents(const long long *__restrict__ rpB, const int *__restrict__ colB, int kB, int4 *ext)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kB) return;
    const long long s = rpB[k], e = rpB[k + 1];
    ext[k] = e > s ? make_int4(colB[s] >> ROW_BLK_LOG, colB[e - 1] >> ROW_BLK_LOG, (int)(e - s), 0)
                   : make_int4(INT_MAX, -1, 0, 0);
}

// Per row of C its products, INT_MAX at most, and its blocks [x, y); rows of
// more than ROW_HEAVY products are listed by weight.  One warp a row, four
// gathers a lane in flight; a row of A longer than WIDE_A entries is left to
// the whole CTA, whose chain is eight times shorter.  Bound by the latency of
// a row's chain (row pointer, column, extent); what all rows add up goes
// through registers and one set of atomics a CTA, of which there are as many
// as the SMs hold: a flag tested per row is one L2 line for all of them.
// Measured on GB300 (cold, a launch): uniform, 16 entries a row, 120,007 rows
// 147 -> 40 us; R-MAT 2^12 x 8 40 -> 8, 2^15 x 16 98 -> 31, 2^18 x 16 406 -> 150.
constexpr int WIDE_A = 2048, WIDE_LIST = 32;

struct RowSum {
    long long p = 0;
    int lo = INT_MAX, hi = -1;
    bool out = false;
};

// Entries e, e + stride, ... of A's row up to e1, four in flight.
__device__ __forceinline__ RowSum sum_entries(const RowArgs &g, const int4 *__restrict__ ext, long long e, long long e1,
                                              int stride)
{
    RowSum s;
    for (; e < e1; e += 4 * stride) {
        int k[4];
        int4 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) k[u] = e + u * stride < e1 ? g.colA[e + u * stride] : -1;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            x[u] = (unsigned)k[u] < (unsigned)g.k ? ext[k[u]] : make_int4(INT_MAX, -1, 0, 0);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            s.lo = min(s.lo, x[u].x);
            s.hi = max(s.hi, x[u].y);
            s.p += x[u].z;
            s.out |= e + u * stride < e1 && (unsigned)k[u] >= (unsigned)g.k;
        }
    }
    s.p = warp_sum_ll(s.p);
    s.lo = __reduce_min_sync(FULL, s.lo);
    s.hi = __reduce_max_sync(FULL, s.hi);
    s.out = __any_sync(FULL, s.out);
    return s;
}

__global__ void __launch_bounds__(256)
k_row_products(RowArgs g, const int4 *__restrict__ ext, int *prod, int2 *rng, int *heavy, RowStat *stat,
               const int *flags)
{
    if (flags[FLAG_BAD_INPUT]) return;
    __shared__ unsigned long long s_p[8], s_i[8], s_b[8];
    __shared__ int s_w[8], s_lo[8], s_hi[8], s_long[WIDE_LIST], s_nlong;
    __shared__ long long s_sum[8];
    __shared__ unsigned s_seen;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) s_nlong = 0, s_seen = 0;
    __syncthreads();
    unsigned long long sp = 0, si = 0, sb = 0;
    unsigned seen = 0;
    int width = 0;
    auto finish = [&](int r, const RowSum &s) {      // one thread
        const long long p = s.p;
        const int nb = s.hi < s.lo ? 0 : s.hi - s.lo + 1;
        prod[r] = (int)min(p, (long long)INT_MAX);
        rng[r] = make_int2(nb ? s.lo : 0, nb ? s.hi + 1 : 0);
        sp += (unsigned long long)p;
        if (sorted_row(g, p, nb)) {          // no bitmap, no item
            seen |= p > 256 ? SEEN_SORT << 2 : p > 128 ? SEEN_SORT << 1 : SEEN_SORT;
        } else {
            width = max(width, nb);
            if (p >= KEEP_BITS * (long long)nb) sb += (unsigned long long)nb;
            si += (unsigned long long)item_bound(p, nb, g.n);
            if (p > LIGHT_ROW || nb > SYM_BLKS) seen |= SEEN_CUTS;
            if (p > LIGHT_MANY) seen |= SEEN_MANY;
        }
        if (s.out) seen |= SEEN_BAD;
        if (p > ROW_HEAVY) {
            const int c = heavy_class(p);
            heavy[(long long)c * g.m + atomicAdd(stat->heavy + c, 1u)] = r;
        }
    };
    for (long long r = blockIdx.x * 8ll + warp; r < g.m; r += gridDim.x * 8ll) {
        const long long e0 = g.rpA[r], e1 = g.rpA[r + 1];
        if (e1 - e0 > WIDE_A) {
            int at = WIDE_LIST;
            if (lane == 0) at = atomicAdd(&s_nlong, 1);
            at = __shfl_sync(FULL, at, 0);
            if (at < WIDE_LIST) {
                if (lane == 0) s_long[at] = (int)r;
                continue;
            }
        }
        const RowSum s = sum_entries(g, ext, e0 + lane, e1, 32);
        if (lane == 0) finish((int)r, s);
    }
    __syncthreads();
    const int nlong = min(s_nlong, WIDE_LIST);
    for (int t = 0; t < nlong; ++t) {
        const int r = s_long[t];
        RowSum s = sum_entries(g, ext, g.rpA[r] + tid, g.rpA[r + 1], 256);
        if (lane == 0) {
            s_sum[warp] = s.p;
            s_lo[warp] = s.lo;
            s_hi[warp] = s.out ? INT_MIN : s.hi;
        }
        __syncthreads();
        if (tid == 0) {
            for (int q = 1; q < 8; ++q) {
                s.p += s_sum[q];
                s.lo = min(s.lo, s_lo[q]);
                s.out |= s_hi[q] == INT_MIN;
                s.hi = max(s.hi, s_hi[q]);
            }
            finish(r, s);
        }
        __syncthreads();
    }
    if (lane == 0) {
        s_p[warp] = sp; s_i[warp] = si; s_b[warp] = sb; s_w[warp] = width;
        if (seen) atomicOr(&s_seen, seen);
    }
    __syncthreads();
    if (tid == 0) {
        unsigned long long a = 0, b = 0, c = 0;
        int w = 0;
        for (int q = 0; q < 8; ++q) { a += s_p[q]; b += s_i[q]; c += s_b[q]; w = max(w, s_w[q]); }
        atomicAdd(&stat->products, a);
        atomicAdd(&stat->items, b);
        if (c) atomicAdd(&stat->blocks, c);
        if (w) atomicMax(&stat->width, w);
        if (s_seen) atomicOr(&stat->seen, s_seen);
    }
}

// Row k of the cut table (one warp each): B's first entry of row k at or past
// each of width + 1 blocks from the row's base on.  Written coalesced, read
// back by k_row_numeric as two neighbouring ints per A entry and item.
__global__ void __launch_bounds__(256)
k_row_cuts(const long long *__restrict__ rpB, const int *__restrict__ colB, int kB, int width,
           const int *__restrict__ base, int *__restrict__ cut)
{
    const long long k = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (k >= kB) return;
    const int b0 = (int)rpB[k], b1 = (int)rpB[k + 1], j0 = base ? base[k >> 4] : 0;
    int *row = cut + k * (width + 1);
    for (int j = lane; j <= width; j += 32) {
        int a = b0, b = b1;
        const long long key = (long long)(j0 + j) << ROW_BLK_LOG;
        while (a < b) {
            const int md = (a + b) >> 1;
            if (colB[md] < key) a = md + 1; else b = md;
        }
        row[j] = a;
    }
}

// The heavy rows' lists (HEAVY_CLASSES of m), the heaviest class last.
struct HeavyRows {
    const int *list = nullptr;
    int n[HEAVY_CLASSES] = {};
    long long m = 0;
    __device__ int row(int i) const {
        int c = HEAVY_CLASSES - 1;
        while (c > 0 && i >= n[c]) i -= n[c--];
        return list[c * m + i];
    }
};

// One CTA per row of C with products in (p0, p1]: the row's columns as a
// bitmap of up to SYM_BLKS blocks at a time in shared memory, then its entry
// count and its items.  heavy.list: those rows, the heaviest first; without a
// list the grid is all rows (rows of no product belong to p0 = 0).
template <int NT>
__global__ void __launch_bounds__(NT)
k_row_symbolic(RowArgs g, const int *__restrict__ prod, int p0, int p1, HeavyRows heavy, int width, int *rowcnt,
               int4 *items, unsigned cap, RowStat *stat)
{
    __shared__ unsigned s_bit;
    constexpr int NW = NT / 32;
    extern __shared__ __align__(16) unsigned s_sym[];
    const int r = heavy.list ? heavy.row(blockIdx.x) : blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int p = prod[r];
    if (p <= p0 || p > p1) {
        if (p == 0 && p1 == ROW_TINY && tid == 0) rowcnt[r] = 0;
        return;
    }
    // the row's blocks: first, then counted from it
    const int2 rng = g.rng[r];
    const int first = rng.x, nblk = rng.y - rng.x;
    if (sorted_row(g, p, nblk)) return;
    unsigned *bits = s_sym;
    int *cnt = reinterpret_cast<int *>(s_sym + min(width, SYM_BLKS) * (ROW_BLK / 32));
    const long long a0 = g.rpA[r], a1 = g.rpA[r + 1];
    const bool keep = g.bits && p >= KEEP_BITS * (long long)nblk;
    if (g.bits && tid == 0) {      // the row's place among the kept bitmaps
        if (keep) s_bit = atomicAdd(&stat->bitblk, (unsigned)nblk);
        g.bitoff[r] = keep ? (int)s_bit : -1;
    }
    for (int wb = 0; wb < nblk; wb += SYM_BLKS) {
        const int nb = min(SYM_BLKS, nblk - wb);
        const int c0 = (first + wb) << ROW_BLK_LOG;
        {
            uint4 *z = reinterpret_cast<uint4 *>(bits);
            for (int t = tid; t < nb * (ROW_BLK / 128); t += NT) z[t] = make_uint4(0u, 0u, 0u, 0u);
        }
        __syncthreads();
        auto mark = [&](int c) {      // most columns of a long row are met before: the atomic is left out
            const int o = c - c0;
            const unsigned bit = 1u << (o & 31);
            volatile unsigned *w = bits + (o >> 5);
            if (!(*w & bit)) atomicOr(bits + (o >> 5), bit);
        };
        auto share = [&](long long a, int &s, int &e) {
            s = e = 0;
            if (a < a1) {
                const int k = g.colA[a];
                if (nblk <= SYM_BLKS) { s = (int)g.rpB[k]; e = (int)g.rpB[k + 1]; }
                else {
                    const int *row = g.cuts(k, first + wb);
                    s = row[0];
                    e = row[nb];
                }
            }
        };
        auto range = [&](int t, int e, int step) {   // entries t, t + step, ... below e, four on their way
            for (; t + 3 * step < e; t += 4 * step) {
                const int x0 = g.colB[t], x1 = g.colB[t + step], x2 = g.colB[t + 2 * step], x3 = g.colB[t + 3 * step];
                mark(x0); mark(x1); mark(x2); mark(x3);
            }
            for (; t < e; t += step) mark(g.colB[t]);
        };
        if (a1 - a0 > 4 * NW) {
            // many A entries: warp w takes those at w, w + NW, ... (the hubs'
            // long B rows lie side by side), four shares on their way
            for (long long a = a0 + warp; a < a1; a += 32 * NW) {
                int s, e;
                share(a + (long long)lane * NW, s, e);
                unsigned live = __ballot_sync(FULL, e > s);
                while (live) {
                    int sq[4], eq[4], c[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int q = live ? __ffs(live) - 1 : 0;
                        sq[u] = __shfl_sync(FULL, s, q);
                        eq[u] = live ? __shfl_sync(FULL, e, q) : sq[u];
                        live &= live - 1;
                        c[u] = sq[u] + lane < eq[u] ? g.colB[sq[u] + lane] : -1;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (c[u] >= 0) mark(c[u]);
                        range(sq[u] + 32 + lane, eq[u], 32);
                    }
                }
            }
        } else {
            for (long long a = a0; a < a1; a += 32) {
                int s, e;
                share(a + lane, s, e);
                // long B rows are the whole CTA's, the others a warp's each
                unsigned big = __ballot_sync(FULL, e - s > 64 * NW);
                unsigned small = __ballot_sync(FULL, e > s) & ~big;
                while (big) {
                    const int q = __ffs(big) - 1;
                    big &= big - 1;
                    range(__shfl_sync(FULL, s, q) + tid, __shfl_sync(FULL, e, q), NT);
                }
                for (int turn = 0; small; ++turn) {
                    const int q = __ffs(small) - 1;
                    small &= small - 1;
                    const int sq = __shfl_sync(FULL, s, q), eq = __shfl_sync(FULL, e, q);
                    if ((turn & (NW - 1)) == warp) range(sq + lane, eq, 32);
                }
            }
        }
        __syncthreads();
        if (keep) {
            uint4 *out = reinterpret_cast<uint4 *>(g.bits + ((long long)s_bit + wb) * (ROW_BLK / 32));
            for (int t = tid; t < nb * (ROW_BLK / 128); t += NT) out[t] = reinterpret_cast<const uint4 *>(bits)[t];
        }
        for (int j = warp; j < nb; j += NW) {
            const unsigned c = __reduce_add_sync(FULL, (unsigned)__popc(bits[j * (ROW_BLK / 32) + lane]));
            if (lane == 0) cnt[wb + j] = (int)c;
        }
        __syncthreads();
    }
    if (warp != 0) return;
    // the items: block j starts one when it is a multiple of ITEM_BLKS or the
    // entries before it have passed another multiple of ITEM_T (light rows:
    // every LIGHT_BLKS blocks only); a start closes the item before it.  Two passes: the items of each class counted, then
    // written where the row's share of the class's list begins.
    __shared__ unsigned s_cls[ITEM_CLASSES];
    const long long la = a1 - a0;
    const bool early = la > LONG_A;
    unsigned *nitems = early ? stat->front : stat->back;
    auto put = [&](int c, unsigned i, int4 it) {
        if (i < cap) items[(unsigned long long)c * cap + (early ? i : cap - 1 - i)] = it;
    };
    int tclose = ITEM_T, bmax = ITEM_BLKS;      // a row's items close at so many entries, or blocks
    auto close = [&](int j, int e, int pj, int pe, bool write) {   // blocks [pj, j), entries [pe, e) of the row
        const int z = e - pe, nb = j - pj;
        if (z <= 0) return;
        const int c = item_class(z, nb, tclose == ITEM_T || (float)p * (float)z <= g.each * (float)la * (float)cnt[nblk]);
        const unsigned i = atomicAdd(s_cls + c, 1u);
        if (write) put(c, i, make_int4(r, first + pj, pe, (nb << 16) | z));
    };
    auto pass = [&](bool write) -> int {
        int run = 0, pj = 0, pe = 0;
        for (int jb = 0; jb < nblk; jb += 32) {
            const int j = jb + lane;
            const int c = j < nblk ? cnt[j] : 0;
            const int incl = warp_incl_scan(c, lane);
            const int excl = run + incl - c;
            int before = __shfl_up_sync(FULL, excl, 1);
            if (lane == 0) before = run - (jb > 0 ? cnt[jb - 1] : 0);
            const bool st = j < nblk && j > 0 && (j % bmax == 0 || excl / tclose != before / tclose);
            const unsigned starts = __ballot_sync(FULL, st);
            const unsigned lower = starts & lanemask_lt();
            const int q = 31 - __clz(lower);
            const int qe = __shfl_sync(FULL, excl, q & 31);
            if (st) close(j, excl, lower ? jb + q : pj, lower ? qe : pe, write);
            if (starts) {
                const int last = 31 - __clz(starts);
                pj = jb + last;
                pe = __shfl_sync(FULL, excl, last);
            }
            run += __shfl_sync(FULL, incl, 31);
        }
        if (lane == 0) {
            close(nblk, run, pj, pe, write);
        }
        __syncwarp();
        return run;
    };
    {   // the row's entries, which the classes go by
        int t = 0;
        for (int j = lane; j < nblk; j += 32) t += cnt[j];
        t = warp_sum_int(t);
        if (lane == 0) { cnt[nblk] = t; rowcnt[r] = t; }
        if (t <= g.light) { tclose = LIGHT_ROW + 1; bmax = LIGHT_BLKS; }
        __syncwarp();
    }
    if (cnt[nblk] <= g.light && nblk <= LIGHT_BLKS) {      // one item
        const int z = cnt[nblk];
        if (lane == 0 && z > 0) {
            const int c = item_class(z, nblk, (float)p <= g.each * (float)la);
            const unsigned i = atomicAdd(nitems + c, 1u);
            put(c, i, make_int4(r, first, 0, (nblk << 16) | z));
        }
        return;
    }
    if (lane < ITEM_CLASSES) s_cls[lane] = 0;
    __syncwarp();
    pass(false);
    if (lane < ITEM_CLASSES) {
        const unsigned mine = s_cls[lane];
        s_cls[lane] = mine ? atomicAdd(nitems + lane, mine) : 0u;
    }
    __syncwarp();
    pass(true);
}

struct __align__(16) Step {  // up to NT of one A entry's products: B's entries at..last
    int at, last;
    double a;
};

// One item, one CTA.  Its products come in steps of up to NT entries of one
// A entry's B row: the threads' columns differ, so a step is one fma per
// position, and the steps follow one another in A's order, a barrier between
// them.  A step's idle lanes repeat its last entry and keep the result to
// themselves; warps without a product only meet the barrier.
template <int NT>
__global__ void __launch_bounds__(NT)
k_row_numeric(RowArgs g, const int4 *__restrict__ items, unsigned front, unsigned last, const long long *__restrict__ rowptrC,
              int *__restrict__ colC, double *__restrict__ valC, int *flags)
{
    constexpr int NW = NT / 32, STEPS = row_steps(NT);
    extern __shared__ __align__(16) unsigned char s_num[];
    __shared__ int s_sum[NW + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto sync = [] { if constexpr (NT > 32) __syncthreads(); else __syncwarp(); };
    const int4 it = items[blockIdx.x < front ? blockIdx.x : last - blockIdx.x];
    const int r = it.x, j0 = it.y, z = it.w & 0xffff, nb = it.w >> 16;
    const int c0 = j0 << ROW_BLK_LOG, nw = nb * (ROW_BLK / 32);
    const bool dense = item_dense(z, nb);
    Step *steps = reinterpret_cast<Step *>(s_num);
    uint2 *word = reinterpret_cast<uint2 *>(steps + STEPS);                     // column bits, entries before them
    unsigned char *tag = reinterpret_cast<unsigned char *>(steps + STEPS);     // dense items: the columns met
    double *acc = reinterpret_cast<double *>(tag + (dense ? nb * ROW_BLK : nw * 8));
    int *ccol = reinterpret_cast<int *>(acc + z);      // ranked items of many blocks: the positions' columns
    const bool wide = nb > ITEM_BLKS;
    const long long a0 = g.rpA[r], a1 = g.rpA[r + 1];
    const int2 rng = g.rng[r];
    const bool whole = nb == rng.y - rng.x;      // the row's only item: whole B rows
    // the symbolic pass's bitmap, when it is no longer than the item's values
    const int bit = !dense && g.bits && KEEP_BITS * nb <= z ? g.bitoff[r] : -1;
    if (bit < 0)
        for (int w = tid; w < (dense ? nb * (ROW_BLK / 16) : nw / 2); w += NT)
            reinterpret_cast<uint4 *>(tag)[w] = make_uint4(0u, 0u, 0u, 0u);
    for (int t = tid; t < (dense ? nb * ROW_BLK : z); t += NT) acc[t] = 0.0;
    int nk = -1, ns = 0, ne = 0;       // the next NT A entries' B rows and shares, loaded ahead
    double nav = 0.0;
    auto load_k = [&](long long a) { nk = a + tid < a1 ? g.colA[a + tid] : -1; };
    auto load_share = [&](long long a) {
        ns = ne = 0;
        if (nk >= 0) {
            nav = g.valA[a + tid];
            if (whole) { ns = (int)g.rpB[nk]; ne = (int)g.rpB[nk + 1]; }
            else {
                const int *row = g.cuts(nk, j0);
                ns = row[0];
                ne = row[nb];
            }
        }
    };
    // f(number of steps staged) over all of the item's steps; the list is
    // filled up to a multiple of ROW_GROUP with steps without entries
    auto walk = [&](auto f) {
        load_k(a0);
        load_share(a0);
        load_k(a0 + NT);
        for (long long a = a0; a < a1; a += NT) {
            const int s = ns, e = ne;
            const double av = nav;
            load_share(a + NT);
            load_k(a + 2 * NT);
            const int cnt = (e - s + NT - 1) / NT;
            int incl = warp_incl_scan(cnt, lane), total = __shfl_sync(FULL, incl, 31);
            if constexpr (NT > 32) {
                __syncthreads();
                if (lane == 0) s_sum[warp] = total;
                __syncthreads();
                total = 0;
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    if (w < warp) incl += s_sum[w];
                    total += s_sum[w];
                }
            }
            for (int base = 0; base < total; base += STEPS) {
                const int at = incl - cnt - base;            // of this thread's first step
                const int n = min(STEPS, total - base);
                sync();
                for (int q = max(0, -at); q < cnt && at + q < STEPS; ++q) {
                    const int last = min(s + NT * q + NT, e) - 1;
                    steps[at + q] = Step{s + NT * q, last, av};
                    if (at + q == n - 1)
                        for (int w = n; w & (ROW_GROUP - 1); ++w) steps[w] = Step{last + 1, last, 0.0};
                }
                sync();
                f(n);
            }
        }
        sync();
    };
    if (!dense) {
        // the columns: kept by the symbolic pass, or marked again: a warp takes
        // every NW-th group of steps, or, with steps wider than a warp, every
        // NW-th step
        if (bit < 0) walk([&](int n) {
            auto mark = [&](int c) { atomicOr(&word[(c - c0) >> 5].x, 1u << (c & 31)); };
            if constexpr (NT == 32) {
                for (int i = 0; i < n; i += ROW_GROUP) {
                    int c[ROW_GROUP];
                    bool live[ROW_GROUP];
#pragma unroll
                    for (int u = 0; u < ROW_GROUP; ++u) {
                        const int t = steps[i + u].at + lane;
                        live[u] = t <= steps[i + u].last;
                        c[u] = live[u] ? g.colB[t] : 0;
                    }
#pragma unroll
                    for (int u = 0; u < ROW_GROUP; ++u)
                        if (live[u]) mark(c[u]);
                }
            } else {
                for (int i = warp; i < n; i += NW) {
                    const int last = steps[i].last;
                    int c[NW];
#pragma unroll
                    for (int u = 0; u < NW; ++u) {
                        const int t = steps[i].at + 32 * u + lane;
                        c[u] = t <= last ? g.colB[t] : -1;
                    }
#pragma unroll
                    for (int u = 0; u < NW; ++u)
                        if (c[u] >= 0) mark(c[u]);
                }
            }
        });
        // the entries before each word: a warp takes a run of words, 64 a
        // round; then the warps' totals
        const int per = ((nw + NW - 1) / NW + 63) & ~63, w1 = min(nw, (warp + 1) * per);
        int run = 0;
        auto rank = [&](int w, uint4 x) {
            const int n0 = __popc(x.x), sum = n0 + __popc(x.z);
            const int incl = warp_incl_scan(sum, lane);
            x.y = (unsigned)(run + incl - sum);
            x.w = x.y + (unsigned)n0;
            run += __shfl_sync(FULL, incl, 31);
            if (w < w1) *reinterpret_cast<uint4 *>(word + w) = x;
        };
        if (bit < 0) {
            for (int w = warp * per + 2 * lane; w - 2 * lane < w1; w += 64)
                rank(w, w < w1 ? *reinterpret_cast<const uint4 *>(word + w) : make_uint4(0u, 0u, 0u, 0u));
        } else {
            const uint2 *kept = reinterpret_cast<const uint2 *>(g.bits + ((long long)bit + j0 - rng.x) * (ROW_BLK / 32));
            for (int w = warp * per + 2 * lane; w - 2 * lane < w1; w += 4 * 64) {
                uint2 x[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) x[u] = w + 64 * u < w1 ? kept[(w >> 1) + 32 * u] : make_uint2(0u, 0u);
#pragma unroll
                for (int u = 0; u < 4; ++u) rank(w + 64 * u, make_uint4(x[u].x, 0u, x[u].y, 0u));
            }
        }
        int total = run;
        if constexpr (NT > 32) {
            if (lane == 0) s_sum[warp] = run;
            __syncthreads();
            int base = 0;
            total = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                if (w < warp) base += s_sum[w];
                total += s_sum[w];
            }
            if (base)
                for (int w = warp * per + lane; w < w1; w += 32) word[w].y += (unsigned)base;
        }
        sync();
        if (total != z) {
            if (tid == 0) set_flag(flags, FLAG_INTERNAL);
            return;
        }
    }
    // the values: two groups of steps, one's entries loaded while the other's
    // are applied
    auto values = [&](auto position) {
        walk([&](int n) {
            struct Group {
                int col[ROW_GROUP];
                bool live[ROW_GROUP], on[ROW_GROUP];
                double b[ROW_GROUP], a[ROW_GROUP];
            } x, y;
            auto load = [&](int i, Group &v) {
                if (i >= n) return;
#pragma unroll
                for (int u = 0; u < ROW_GROUP; ++u) {
                    const Step q = steps[i + u];
                    const int t = q.at + tid;
                    v.live[u] = t <= q.last;
                    v.on[u] = NT == 32 || q.at + warp * 32 <= q.last;
                    if (v.on[u]) {
                        const int e = min(t, q.last);
                        v.col[u] = g.colB[e];
                        v.b[u] = g.valB[e];
                        v.a[u] = q.a;
                    }
                }
            };
            auto apply = [&](int i, const Group &v) {
                if (i >= n) return;
                int p[ROW_GROUP];
#pragma unroll
                for (int u = 0; u < ROW_GROUP; ++u)
                    if (v.on[u]) p[u] = position(v.col[u], v.live[u]);
#pragma unroll
                for (int u = 0; u < ROW_GROUP; ++u) {
                    if (v.on[u]) {
                        const double c = fma(v.a[u], v.b[u], acc[p[u]]);
                        if (v.live[u]) acc[p[u]] = c;
                    }
                    sync();
                }
            };
            load(0, x);
            load(ROW_GROUP, y);
            for (int i = 0; i < n; i += 2 * ROW_GROUP) {
                apply(i, x);
                load(i + 2 * ROW_GROUP, x);
                apply(i + ROW_GROUP, y);
                load(i + 3 * ROW_GROUP, y);
            }
        });
    };
    const long long Rb = rowptrC[r] + it.z;
    const int shift = g.coloff ? g.coloff[r >> 4] : 0;
    if (dense) {
        values([&](int c, bool live) {
            const int o = live ? c - c0 : 0;
            if (live) tag[o] = 1;
            return o;
        });
        // a word's columns a round; a warp takes a run of words, counted first
        const int per = (nw + NW - 1) / NW, w0 = warp * per, w1 = min(nw, w0 + per);
        int run = 0, total = 0;
        if constexpr (NT > 32) {
            int c = 0;
            for (int w = w0; w < w1; ++w) c += tag[w * 32 + lane];
            c = (int)__reduce_add_sync(FULL, (unsigned)c);
            if (lane == 0) s_sum[warp] = c;
            __syncthreads();
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                if (w < warp) run += s_sum[w];
                total += s_sum[w];
            }
            if (total != z) {
                if (tid == 0) set_flag(flags, FLAG_INTERNAL);
                return;
            }
        }
#pragma unroll 4
        for (int w = w0; w < w1; ++w) {
            const bool met = tag[w * 32 + lane] != 0;
            const unsigned m = __ballot_sync(FULL, met);
            const int t = run + __popc(m & lanemask_lt());
            if (met && t < z) {
                valC[Rb + t] = acc[w * 32 + lane];
                colC[Rb + t] = c0 - shift + w * 32 + lane;
            }
            run += __popc(m);
        }
        if (NT == 32 && run != z && lane == 0) set_flag(flags, FLAG_INTERNAL);
        return;
    }
    const uint2 *word0 = word - (c0 >> 5);
    auto rank = [&](int c) {
        const uint2 w = word0[c >> 5];
        return (int)w.y + __popc(w.x & ((1u << (c & 31)) - 1u));
    };
    if (wide) {
        values([&](int c, bool live) {
            const int pos = rank(c);
            if (live) ccol[pos] = c - shift;
            return pos;
        });
    } else {
        values([&](int c, bool) { return rank(c); });
    }
    for (int t = tid; t < z; t += NT) valC[Rb + t] = acc[t];
    if (!wide) {   // the columns from the bitmap, through the accumulators' memory so that they leave coalesced
        sync();
        ccol = reinterpret_cast<int *>(acc);
        for (int w = tid; w < nw; w += NT) {
            const uint2 x = word[w];
            unsigned m = x.x;
            int t = (int)x.y;
            const int cb = c0 - shift + (w << 5);
            while (m) {
                ccol[t++] = cb + __ffs(m) - 1;
                m &= m - 1;
            }
        }
        sync();
    }
    for (int t = tid; t < z; t += NT) colC[Rb + t] = ccol[t];
}

// ---- rows of few products: sorted in registers ---------------------------------
//
// A row of up to SORT_MAX products needs no bitmap of its span.  To count its
// columns one warp puts them in a hash table, half full at most; to fill C's
// row it sorts the keys (column, product) -- E a lane, a bitonic network,
// strides below E inside a lane -- and a column's products then lie side by
// side in product order, to be applied to its entry in that order.  The
// product number in the low bits leaves 23 bits for the column.
// Bound by issue (the network: 650 instructions for 256 keys); the bitmap of
// such a row took 3,000 over 98 blocks, and 27 KB of shared memory.
// Measured on GB300: uniform 120,007 x 80,021 x 100,003, 192 products a row over
// 98 blocks: 2,080 -> 600 us a call (k_row_sort 104 us to count, 140 when it
// sorted there too, and 227 to fill).
constexpr int SORT_WARPS = 4;

struct __align__(16) Share {     // one A entry's B row: entry f + delta for the row's product f
    int delta, pad;
    double a;
};

template <int E, bool FILL>
struct SortSmem {
    unsigned met[64 * E];           // the columns met: a hash table, half full at most
    Share share[32];
};
template <int E>
struct SortSmem<E, true> {
    unsigned key[32 * E];
    Share share[32];
    double2 ab[32 * E];             // product: A's and B's value
    unsigned short at[32 * E + 2];  // C entry: its first sorted product
};

template <int E>
__device__ __forceinline__ void sort_keys(unsigned (&x)[E], int lane)
{
#pragma unroll
    for (int k = 2; k < E; k <<= 1)          // inside a lane, both directions
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
            for (int e = 0; e < E; ++e)
                if ((e & j) == 0) {
                    const unsigned lo = min(x[e], x[e | j]), hi = max(x[e], x[e | j]);
                    x[e] = (e & k) ? hi : lo;
                    x[e | j] = (e & k) ? lo : hi;
                }
    unsigned flip = 0;
#pragma unroll
    for (int k = E; k <= 32 * E; k <<= 1) {
        // lanes that sort downwards hold their keys complemented
        const unsigned down = k < 32 * E && (lane & (k / E)) ? 0xffffffffu : 0u;
        const unsigned turn = flip ^ down;
        flip = down;
#pragma unroll
        for (int e = 0; e < E; ++e) x[e] ^= turn;
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= E) {
                const bool up = lane & (j / E);
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const unsigned y = __shfl_xor_sync(FULL, x[e], j / E);
                    x[e] = up ? max(x[e], y) : min(x[e], y);
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e)
                    if ((e & j) == 0) {
                        const unsigned lo = min(x[e], x[e | j]), hi = max(x[e], x[e | j]);
                        x[e] = lo;
                        x[e | j] = hi;
                    }
            }
        }
    }
}

// One warp per row of C with products in (lo, 32 E].
template <int E, bool FILL>
__global__ void __launch_bounds__(SORT_WARPS * 32)
k_row_sort(RowArgs g, const int *__restrict__ prod, int lo, int *rowcnt, const long long *__restrict__ rowptrC,
           int *__restrict__ colC, double *__restrict__ valC, int *flags)
{
    __shared__ SortSmem<E, FILL> s_w[SORT_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * SORT_WARPS + warp;
    if (r >= g.m) return;
    const int p = prod[r];
    if (p <= lo || p > 32 * E) return;
    const int2 rng = g.rng[r];
    if (!sorted_row(g, p, rng.y - rng.x)) return;
    SortSmem<E, FILL> &w = s_w[warp];
    if constexpr (FILL) {
        for (int t = p + lane; t < 32 * E; t += 32) w.key[t] = 0xffffffffu;
    } else {
        for (int t = lane; t < 16 * E; t += 32)
            reinterpret_cast<uint4 *>(w.met)[t] = make_uint4(~0u, ~0u, ~0u, ~0u);
    }
    int fresh = 0;
    const long long a1 = g.rpA[r + 1];
    int f0 = 0;                                     // products before this batch of A entries
    for (long long a = g.rpA[r]; a < a1; a += 32) {
        int s = 0, len = 0;
        double av = 0.0;
        if (a + lane < a1) {
            const int k = g.colA[a + lane];
            if (FILL) av = g.valA[a + lane];
            s = (int)g.rpB[k];
            len = (int)g.rpB[k + 1] - s;
        }
        const int incl = warp_incl_scan(len, lane), off = incl - len, T = __shfl_sync(FULL, incl, 31);
        const unsigned live = __ballot_sync(FULL, len > 0);
        __syncwarp();
        if (len > 0) {
            Share &x = w.share[__popc(live & lanemask_lt())];
            x.delta = s - off;
            x.a = av;
        }
        __syncwarp();
        int done = 0;
        for (int base = 0; base < T; base += 32) {
            // a share that starts in this round sets the bit of the lane it starts at
            const int d = off - base;
            const unsigned m = __reduce_or_sync(FULL, (len > 0 && (unsigned)d < 32u) ? 1u << d : 0u);
            const int q = done + __popc(m & (lanemask_lt() | (1u << lane))) - 1;
            done += __popc(m);
            const int f = base + lane;
            if (f < T) {
                const int e = w.share[q].delta + f;
                const unsigned c = (unsigned)g.colB[e];
                if constexpr (FILL) {
                    w.key[f0 + f] = c << SORT_BITS | (unsigned)(f0 + f);
                    w.ab[f0 + f] = make_double2(w.share[q].a, g.valB[e]);
                } else {
                    unsigned h = (c * 0x9e3779b1u) >> (32 - __ffs(64 * E) + 1);
                    unsigned was;
                    while ((was = atomicCAS(&w.met[h], ~0u, c)) != ~0u && was != c) h = (h + 1) & (64 * E - 1);
                    fresh += was == ~0u;
                }
            }
        }
        f0 += T;
    }
    if constexpr (!FILL) {
        const int z = (int)__reduce_add_sync(FULL, (unsigned)fresh);
        if (lane == 0) rowcnt[r] = z;
        return;
    } else {
        __syncwarp();
        unsigned x[E];
#pragma unroll
        for (int e = 0; e < E; ++e) x[e] = w.key[lane * E + e];
        sort_keys<E>(x, lane);
        // the first product of each column starts an entry of C
        unsigned before = __shfl_up_sync(FULL, x[E - 1], 1);
        unsigned heads = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const bool first = lane == 0 && e == 0;
            if (x[e] != 0xffffffffu && (first || (x[e] >> SORT_BITS) != (before >> SORT_BITS))) heads |= 1u << e;
            before = x[e];
        }
        const int n = __popc(heads);
        const int incl = warp_incl_scan(n, lane), z = __shfl_sync(FULL, incl, 31);
        int o = incl - n;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            w.key[lane * E + e] = x[e];
            if ((heads >> e) & 1u) w.at[o++] = (unsigned short)(lane * E + e);
        }
        if (lane == 0) w.at[z] = (unsigned short)p;
        __syncwarp();
        const long long Rb = rowptrC[r];
        if (rowptrC[r + 1] - Rb != z) {
            if (lane == 0) set_flag(flags, FLAG_INTERNAL);
            return;
        }
        const int shift = g.coloff ? g.coloff[r >> 4] : 0;
        for (int t = lane; t < z; t += 32) {
            const int q0 = w.at[t], q1 = w.at[t + 1];
            unsigned k = w.key[q0];
            colC[Rb + t] = (int)(k >> SORT_BITS) - shift;
            double acc = 0.0;
            for (int q = q0; q < q1; ++q) {
                const double2 v = w.ab[w.key[q] & (unsigned)(SORT_MAX - 1)];
                acc = fma(v.x, v.y, acc);
            }
            valC[Rb + t] = acc;
        }
    }
}

template <bool FILL>
cudaError_t sort_rows(cudaStream_t s, const RowArgs &g, const int *prod, const RowStat &h, int *rowcnt,
                      const long long *rowptrC, int *colC, double *valC, int *flags)
{
    const unsigned grid = (unsigned)((g.m + SORT_WARPS - 1) / SORT_WARPS);
    auto run = [&](auto kernel, int lo) {
        kernel<<<grid, SORT_WARPS * 32, 0, s>>>(g, prod, lo, rowcnt, rowptrC, colC, valC, flags);
        ::tsg::count_launch();
    };
    if (h.seen & SEEN_SORT << 2) run(k_row_sort<16, FILL>, 256);
    if (h.seen & SEEN_SORT << 1) run(k_row_sort<8, FILL>, 128);
    if (h.seen & SEEN_SORT) run(k_row_sort<4, FILL>, 0);
    return cudaGetLastError();
}

size_t sym_smem(int width) { return (size_t)std::min(width, SYM_BLKS) * (ROW_BLK / 8) + 4 * ((size_t)width + 1); }

unsigned warps_grid(long long rows) { return (unsigned)std::min<long long>(std::max<long long>((rows + 7) / 8, 1), 152 * 32); }

cudaError_t fork_lanes(cudaStream_t s, const RowLanes &l, int n)
{
    cudaError_t e = n > 0 ? cudaEventRecord(l.fork, s) : cudaSuccess;
    for (int t = 0; t < n && e == cudaSuccess; ++t) e = cudaStreamWaitEvent(l.lane[t], l.fork, 0);
    return e;
}

cudaError_t join_lanes(cudaStream_t s, const RowLanes &l, int n)
{
    cudaError_t e = cudaSuccess;
    for (int t = 0; t < n; ++t) {      // every lane, also after a failure
        cudaError_t j = cudaEventRecord(l.join[t], l.lane[t]);
        if (j == cudaSuccess) j = cudaStreamWaitEvent(s, l.join[t], 0);
        if (e == cudaSuccess) e = j;
    }
    return e;
}

template <int NT>
cudaError_t numeric_class(cudaStream_t s, const RowArgs &g, const int4 *items, unsigned cap, const RowStat &h,
                          int c, const long long *rowptrC, int *colC, double *valC, int *flags)
{
    const unsigned n = h.front[c] + h.back[c];
    k_row_numeric<NT><<<n, NT, class_smem(c) + row_steps(NT) * sizeof(Step), s>>>(
        g, items, h.front[c], cap - 1 + h.front[c], rowptrC, colC, valC, flags);
    ::tsg::count_launch();
    return cudaGetLastError();
}

}  // namespace

cudaError_t rows_init_attributes()
{
    const auto dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const int most = (int)sym_smem(ROW_MAX_BLKS);
    cudaError_t e = cudaFuncSetAttribute(k_row_symbolic<256>, dyn, most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_row_symbolic<64>, dyn, most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_row_symbolic<1024>, dyn, most);
    const int num = class_smem(ITEM_CLASSES - 1) + row_steps(NT_WIDE) * (int)sizeof(Step);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_row_numeric<32>, dyn, num);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_row_numeric<NT_WIDE>, dyn, num);
    return e;
}

cudaError_t row_sample(Pool &pool, const RowArgs &g, int step, unsigned long long *out, const int *flags)
{
    const long long rows = (g.m + step - 1) / step;
    k_row_sample<<<(unsigned)((rows + 7) / 8), 256, 0, pool.stream>>>(g, step, out, flags);
    ::tsg::count_launch();
    return cudaGetLastError();
}

cudaError_t row_products(Pool &pool, const RowArgs &g, int *prod, int2 *rng, int *heavy, RowStat *stat,
                         const int *flags)
{
    int4 *ext = pool.alloc_n<int4>(g.k);
    if (!ext) return pool.err;
    k_row_extents<<<(unsigned)((g.k + 255) / 256), 256, 0, pool.stream>>>(g.rpB, g.colB, g.k, ext);
    k_row_products<<<warps_grid(g.m), 256, 0, pool.stream>>>(g, ext, prod, rng, heavy, stat, flags);
    ::tsg::count_launch();
    ::tsg::count_launch();
    pool.free(ext);
    return cudaGetLastError();
}

cudaError_t row_cuts(Pool &pool, const RowArgs &g, int *cut)
{
    k_row_cuts<<<(unsigned)((g.k + 7) / 8), 256, 0, pool.stream>>>(g.rpB, g.colB, g.k, g.width, g.base, cut);
    ::tsg::count_launch();
    return cudaGetLastError();
}

cudaError_t row_symbolic(Pool &pool, const RowArgs &g, const int *prod, const int *heavy, const RowStat &hs,
                         int *rowcnt, int4 *items, unsigned cap, RowStat *stat, const RowLanes &l)
{
    cudaStream_t s = pool.stream;
    const int width = hs.width;
    const size_t sm = sym_smem(width);
    HeavyRows h;
    int total = 0;
    for (int c = 0; c < HEAVY_CLASSES; ++c) total += h.n[c] = (int)hs.heavy[c];
    cudaError_t e = cudaSuccess;
    if (width == 0)      // every row is sorted, or empty
        e = cudaMemsetAsync(rowcnt, 0, sizeof(int) * (size_t)g.m, s);
    const bool sorts = hs.seen & SEEN_SORT * 7;
    const int lanes = sorts ? 3 : 2;
    if (e == cudaSuccess) e = fork_lanes(s, l, lanes);
    if (e != cudaSuccess) return e;
    if (total > 0) {   // the heaviest first: the others run beside their tail
        HeavyRows hl = h;
        hl.list = heavy;
        hl.m = g.m;
        k_row_symbolic<1024><<<(unsigned)total, 1024, sm, l.lane[0]>>>(g, prod, ROW_HEAVY, INT_MAX, hl, width, rowcnt, items, cap, stat);
        ::tsg::count_launch();
    }
    if (width > 0) {
        k_row_symbolic<256><<<(unsigned)g.m, 256, sm, s>>>(g, prod, ROW_TINY, ROW_HEAVY, h, width, rowcnt, items, cap, stat);
        k_row_symbolic<64><<<(unsigned)g.m, 64, sm, l.lane[1]>>>(g, prod, 0, ROW_TINY, h, width, rowcnt, items, cap, stat);
        ::tsg::count_launch();
        ::tsg::count_launch();
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = sort_rows<false>(l.lane[2], g, prod, hs, rowcnt, nullptr, nullptr, nullptr, nullptr);
    const cudaError_t j = join_lanes(s, l, lanes);
    return e == cudaSuccess ? j : e;
}

cudaError_t row_numeric(Pool &pool, const RowArgs &g, const int *prod, const int4 *items, unsigned cap, const RowStat &h,
                        const long long *rowptrC, int *colC, double *valC, int *flags, const RowLanes &l)
{
    cudaStream_t s = pool.stream;
    // every class on a stream of its own, so that none waits for another's last
    // items, and in this order, the longest chains (large items, and a heavy
    // row's many small ones) first.  Two streams in place of these: R-MAT
    // 2^15 x 16 A*A^T 2,190 us a call for 1,692, 2^16 x 12 A*A 2,950 for 2,552
    constexpr int order[ITEM_CLASSES] = {3, 2, 0, 1, 6, 5, 4};
    static_assert(ROW_LANES == ITEM_CLASSES - 1, "a stream for each class");
    int list[ITEM_CLASSES], n = 0;
    for (int c : order)
        if (h.front[c] + h.back[c] > 0) list[n++] = c;
    cudaError_t e = fork_lanes(s, l, n - 1);
    for (int q = 0; q < n && e == cudaSuccess; ++q) {
        const int c = list[q];
        cudaStream_t on = q == n - 1 ? s : l.lane[q];
        const int4 *it = items + (long long)c * cap;
        e = c < CLASS_WARP ? numeric_class<32>(on, g, it, cap, h, c, rowptrC, colC, valC, flags)
                           : numeric_class<NT_WIDE>(on, g, it, cap, h, c, rowptrC, colC, valC, flags);
    }
    if (e == cudaSuccess) e = sort_rows<true>(s, g, prod, h, nullptr, rowptrC, colC, valC, flags);
    const cudaError_t j = join_lanes(s, l, n - 1);
    return e == cudaSuccess ? j : e;
}

}  // namespace tsg
