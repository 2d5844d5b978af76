// tsg_rows.cuh -- the row path's sizes and entry points (tsg_rows.cu).
#pragma once
#include "tsg_internal.cuh"

namespace tsg {

constexpr int ROW_BLK_LOG = 10, ROW_BLK = 1 << ROW_BLK_LOG;   // columns of a block: a warp of bitmap words
constexpr int ITEM_T = 1024;                  // an item closes once its row's entries pass a multiple of this
constexpr int ITEM_CAP = ITEM_T + ROW_BLK;    // entries of an item at most (a block adds at most ROW_BLK)
constexpr int ITEM_BLKS = 16;                 // blocks of an item at most
constexpr int LIGHT_ROW = 4096, LIGHT_BLKS = 256;   // rows of so few entries: one item per so many blocks
// ... of a product of more than MANY_PRODUCTS, which fills the GPU without the
// light rows' CTAs of 128 threads (R-MAT 2^18 x 16 A*A^T 34.3 ms a call with
// 4,096, 33.5 with 2,048; 512 mixed products, 2.1 G: 23.1 and 22.5, 23.4 with
// 1,024); below it those shorten the longest chains (R-MAT 2^12 x 8 379 us with
// 4,096, 392 with 2,048; 2^15 x 16 1,498 and 1,533)
constexpr int LIGHT_MANY = 2048;
constexpr long long MANY_PRODUCTS = 400000000;
constexpr int KEEP_BITS = 16;               // products a block from which a row's bitmap is kept for the numeric
                                              // pass (and entries a block from which an item reads it: 128 bytes a
                                              // block against 8 an entry; with none of its own, uniform rows of 192
                                              // products over 98 blocks: 2.0 ms marked again, 2.7 read back)
constexpr int SYM_BLKS = 256;                 // blocks of the symbolic bitmap at a time (32 KB)
constexpr int ROW_MAX_BLKS = 4096;            // blocks of a row's columns at most (4 M columns)
constexpr int ROW_HEAVY = 48 << 10;           // rows of more products take a CTA of 1,024 threads
constexpr int ROW_TINY = 4096;                // rows of so few products take a CTA of 64 threads
constexpr int HEAVY_CLASSES = 4;              // ... listed by weight: the longest chains start first
__host__ __device__ inline int heavy_class(long long p)
{
    return p > 32 * ROW_HEAVY ? 3 : p > 8 * ROW_HEAVY ? 2 : p > 3 * ROW_HEAVY ? 1 : 0;
}
constexpr int ROW_GROUP = 4;                  // steps whose entries are loaded together
constexpr int NT_WIDE = 128;                  // threads of the items whose A entries bring many products each
static_assert(ROW_BLK == 1024, "a block is 32 bitmap words");

__host__ __device__ constexpr int row_steps(int nt) { return nt > 32 ? 128 : 32; }   // steps staged at a time

// Classes of items: shared memory beside the staged steps, so that an SM holds
// 21, 14, 10 and 6 single-warp items (the first CLASS_WARP classes) or 5, 3
// and 2 items of NT_WIDE threads; the occupancy hides their loads (one class
// of 20 KB in place of the first two: R-MAT 2^18 A*A^T 52.3 against 45.3 ms).
constexpr int ITEM_CLASSES = 7, CLASS_WARP = 4;
// A row's items are chains over its A entries.  Those of rows with more than
// LONG_A start first, or they run on alone at the end (R-MAT 2^15 x 16 A*A^T
// 1,692 us a call in any order, 1,494 so, and 1,515 to 1,545 from 128 to 2,048;
// 2^12 x 8 414 and 395).
constexpr int LONG_A = 256;
__host__ __device__ constexpr int class_smem(int c)
{
    return c == 0 ? 9 << 10 : c == 1 ? 14 << 10 : c == 2 ? 20 << 10 : c == 3 ? 34 << 10 : c == 4 ? 40 << 10 : c == 5 ? 72 << 10 : 112 << 10;
}

// Items whose blocks are half full or more keep an accumulator per column:
// no bitmap pass over their products, no ranks.
__host__ __device__ inline bool item_dense(int z, int nb) { return nb * ROW_BLK <= 2 * z; }
__host__ __device__ inline int item_smem(int z, int nb)
{
    return item_dense(z, nb) ? nb * ROW_BLK * 9 : nb * (ROW_BLK / 4) + z * (nb > ITEM_BLKS ? 12 : 8);
}
// warp: the item is one warp's where it fits.  A heavy row's always is; a
// light row's while an A entry brings few products (RowArgs::each), for a
// step of NT_WIDE would idle most of its threads.
__host__ __device__ inline int item_class(int z, int nb, bool warp)
{
    const int b = item_smem(z, nb);
    if (warp && b <= class_smem(3)) return b <= class_smem(0) ? 0 : b <= class_smem(1) ? 1 : b <= class_smem(2) ? 2 : 3;
    return b <= class_smem(4) ? 4 : b <= class_smem(5) ? 5 : 6;
}
static_assert(LIGHT_BLKS * (ROW_BLK / 4) + LIGHT_ROW * 12 <= class_smem(6), "every light row's item fits the last class");
static_assert(LIGHT_ROW * 2 * 9 <= class_smem(6) && ITEM_CAP * 2 * 9 <= class_smem(6), "dense items fit");
static_assert(ITEM_BLKS * (ROW_BLK / 4) + ITEM_CAP * 12 <= class_smem(3), "every other item fits a warp's classes");

// The items of a row of p products over nb of n columns' blocks at most: its
// entries are no more than its products or its columns.  A row that is light
// whatever the product's size closes items at LIGHT_BLKS blocks alone.  The
// seven lists of items are as long as these bounds' sum, 112 bytes an item.
__host__ __device__ inline long long item_bound(long long p, int nb, int n)
{
    const long long span = (long long)nb * ROW_BLK, most = span < n ? span : n, z = p < most ? p : most;
    const long long k = z <= LIGHT_MANY ? (nb + LIGHT_BLKS - 1) / LIGHT_BLKS : (nb + ITEM_BLKS - 1) / ITEM_BLKS + z / ITEM_T;
    return p < k ? p : k;
}
static_assert(LIGHT_MANY <= LIGHT_ROW, "light in a large product is light in a small one");

constexpr int SORT_BITS = 9, SORT_MAX = 1 << SORT_BITS;   // products of a row that is sorted at most
constexpr int SORT_COLS = (1 << (32 - SORT_BITS)) - 1;    // C's columns up to which it is (32-bit keys)
constexpr int SORT_NB = 80;                                // blocks of its span from which it is

struct RowArgs {
    int m = 0, k = 0, n = 0;
    const long long *rpA = nullptr, *rpB = nullptr;
    const int *colA = nullptr, *colB = nullptr;
    const double *valA = nullptr, *valB = nullptr;
    int light = LIGHT_ROW;                    // rows of so many entries at most are light
    int sort_max = 0;                         // rows of so many products at most are sorted (0: none)
    float each = 32;                          // light rows: products of an A entry from which an item is a CTA's
    const int2 *rng = nullptr;                // each row of C: its blocks [x, y)
    // The cut table, k rows of width + 1 blocks; null when every row is one
    // item.  base (optional, batches): per 16 rows of B the block a table row
    // starts at, so that it is as wide as an instance and not as the batch.
    const int *cut = nullptr;
    const int *base = nullptr;
    int width = 0;
    const int *coloff = nullptr;              // batches: per 16 rows of C, subtracted from its columns
    // The rows' column bitmaps, kept by k_row_symbolic for k_row_numeric when
    // there is room: row r's 32 words a block from block bitoff[r] on (-1: not kept).
    unsigned *bits = nullptr;
    int *bitoff = nullptr;
    __device__ __forceinline__ const int *cuts(int k, int j) const {   // B row k's, from block j on
        return cut + (long long)k * (width + 1) + (j - (base ? base[k >> 4] : 0));
    }
};

// What row_products finds (zeroed before).
constexpr unsigned SEEN_BAD = 1;     // a column of A outside B's rows
constexpr unsigned SEEN_CUTS = 2;    // a row needs the cut table (more than one item or window)
constexpr unsigned SEEN_MANY = 32;   // the same were LIGHT_MANY the line
constexpr unsigned SEEN_SORT = 4;    // rows of up to 128 (<< 1: 256, << 2: SORT_MAX) products to sort

struct RowStat {
    unsigned long long products, items;       // intermediate products; an upper bound of the items
    unsigned heavy[HEAVY_CLASSES];
    int width;                                // blocks of the widest row
    unsigned seen;                            // SEEN_*
    unsigned bitblk;                          // row_symbolic: blocks of kept bitmaps handed out
    int pad;
    unsigned long long blocks;                // blocks of the rows that keep their bitmaps
    // row_symbolic: items of each class; those of rows with many A entries, the
    // long chains, fill its list from the front, the others from the back
    unsigned front[ITEM_CLASSES], back[ITEM_CLASSES];
};

// Streams beside the main one; fork and join tie them to it.
constexpr int ROW_LANES = ITEM_CLASSES - 1;
struct RowLanes {
    cudaStream_t lane[ROW_LANES];
    cudaEvent_t fork, join[ROW_LANES];
};

cudaError_t rows_init_attributes();
// Both may run on row pointers that the check has refused (flags), and do nothing then.
// adds step * the products of every step-th row
cudaError_t row_sample(Pool &pool, const RowArgs &g, int step, unsigned long long *out, const int *flags);
cudaError_t row_products(Pool &pool, const RowArgs &g, int *prod, int2 *rng, int *heavy, RowStat *stat, const int *flags);
cudaError_t row_cuts(Pool &pool, const RowArgs &g, int *cut);
// items: ITEM_CLASSES lists of cap
cudaError_t row_symbolic(Pool &pool, const RowArgs &g, const int *prod, const int *heavy, const RowStat &h,
                         int *rowcnt, int4 *items, unsigned cap, RowStat *stat, const RowLanes &l);
cudaError_t row_numeric(Pool &pool, const RowArgs &g, const int *prod, const int4 *items, unsigned cap, const RowStat &h,
                        const long long *rowptrC, int *colC, double *valC, int *flags, const RowLanes &l);

}  // namespace tsg
