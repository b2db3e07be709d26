// sort.cu — stable LSD radix sort of (u32 key, u32 payload).
//
// Replaces thrust::sort_by_key (include/FMkernel.cuh:190, a stable cub radix sort of int keys
// carrying 72-byte Cell values).
// Keys are the Morton code + 1 (0 for a cell outside the grid, so it orders first like the
// reference's -1), and only the bits a key of this grid can set are sorted.  Payloads are cell
// indices; the cell records themselves move once, in the gather that follows (mech.cu).
//
// One pass per digit of d <= 10 bits: k_hist (per-tile digit counts), k_digit_scan (a CTA per digit,
// exclusive scan of its row of the digit-major count table; left out for up to 32 tiles), k_scatter
// (stable rank inside the tile with warp match, then scatter).  A tile is 16 warps x 8 items; item k of
// lane l of warp w is tile element w*256 + k*32 + l, so processing k in order and lanes in order visits
// the tile in input order, which is what makes the ranks, and the sort, stable.  Up to 6,144 cells one
// CTA does it all (k_sort_one, with the keys; mech.cu).
#include "mech_body.cuh"

namespace gell {

namespace {
__global__ void __launch_bounds__(kSortThreads) k_hist(const uint32_t* __restrict__ keys, int n, int shift,
                                                   int R, uint32_t* __restrict__ hist, int nb) {
    grid_dep_wait();
    grid_dep_launch();
    hist_body(keys, n, shift, R, hist, nb, blockIdx.x);
}

__global__ void __launch_bounds__(kSortThreads) k_digit_scan(uint32_t* __restrict__ hist, int nb,
                                                         uint32_t* __restrict__ totals) {
    grid_dep_wait();
    grid_dep_launch();
    digit_scan_body(hist, nb, totals, blockIdx.x);
}

__global__ void __launch_bounds__(kSortThreads) k_scatter(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                      uint32_t* __restrict__ kout, uint32_t* __restrict__ vout, int n,
                                                      int shift, int R, const uint32_t* __restrict__ offs, int nb,
                                                      const uint32_t* __restrict__ totals, int iota) {
    grid_dep_wait();
    grid_dep_launch();
    scatter_body(kin, vin, kout, vout, n, shift, R, offs, nb, totals, iota, blockIdx.x);
}

}  // namespace

// digit-major count table, then the digit totals
size_t sort_hist_entries(int cap) { return (size_t)kSortDigits * ((cap + kSortTile - 1) / kSortTile) + kSortDigits + 64; }

gell_status radix_sort(gell_ctx* c, int n, int bits, bool vals_are_iota) {
    SortScratch& S = c->sort;
    int in = 0;
    if (n <= 0) {
        S.which = 0;
        return GELL_OK;
    }
    const int nb = (n + kSortTile - 1) / kSortTile;
    const SortPlan plan = sort_plan(bits);
    const int passes = plan.passes, d = plan.bits;
    const int R = 1 << d;
    bool iota = vals_are_iota;
    for (int p = 0; p < passes; ++p) {
        const int shift = p * d;
        GELL_KERNEL(c, "k_hist", launch_dependent(k_hist, nb, kSortThreads, 0, c->stream, S.keys[in], n, shift, R, S.hist, nb));
        uint32_t* totals = S.hist + (size_t)R * nb;
        if (nb > kSortScanTiles)
            GELL_KERNEL(c, "k_digit_scan", launch_dependent(k_digit_scan, R, kSortThreads, 0, c->stream, S.hist, nb, totals));
        GELL_KERNEL(c, "k_scatter", launch_dependent(k_scatter, nb, kSortThreads, 0, c->stream, S.keys[in], S.vals[in], S.keys[in ^ 1], S.vals[in ^ 1], n, shift,
                                                   R, S.hist, nb, totals, iota ? 1 : 0));
        iota = false;
        in ^= 1;
    }
    S.which = in;
    return GELL_OK;
}

}  // namespace gell
