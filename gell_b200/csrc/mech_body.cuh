// mech_body.cuh — the per-block bodies of the mechanics kernels (mech.cu: keys, gather, force and
// move; sort.cu: the radix sort's histogram, digit scan and scatter; lod.cu: the uptake map), shared
// by the one-context kernels and the ensemble's batched kernels (mech_batch.cu), which run the same
// body for block `blk` of one member.  Each body is the kernel it came from with blockIdx.x
// replaced by `blk`, so a batched launch computes what the member's own launches compute.
#pragma once

#include "async_copy.cuh"
#include "gell_internal.cuh"

namespace gell {

// ------------------------------------------------------------------ FM_update (mech.cu)

// Also advances the cell-list epoch, which lives in device memory so that a captured step reads
// the current one when it is replayed.
__device__ __forceinline__ void keys_body(const CellsSoA& c, int n, const Geom& g, uint32_t* __restrict__ keys,
                                          int* __restrict__ epoch, int blk) {
    const int i = blk * blockDim.x + threadIdx.x;
    if (i == 0) *epoch += 1;
    if (i >= n) return;
    const float4 pr = c.posr[i];
    const int3 b = find_bin(pr.x, pr.y, pr.z, g.len);
    if (!inside(b.x, b.y, b.z, g.N)) {
        c.sign[i] = 0;
        keys[i] = 0u;
        return;
    }
    keys[i] = morton3(b.x, b.y, b.z) + 1u;
    c.mesh[i] = b.x + b.y * g.N + b.z * g.N * g.N;
}

__device__ __forceinline__ void gather_body(const CellsSoA& s, const CellsSoA& d, const uint32_t* __restrict__ keys,
                                            const uint32_t* __restrict__ perm, int n, int4* __restrict__ bins,
                                            const int* __restrict__ epoch_p, int blk) {
    const int i = blk * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int epoch = *epoch_p;
    const int j = (int)perm[i];
    d.sign[i] = s.sign[j];
    const int m = s.mesh[j];
    d.mesh[i] = m;
    d.posr[i] = s.posr[j];
    d.force[i] = s.force[j];
    d.oldf[i] = s.oldf[j];
    d.V[i] = s.V[j];
    d.Vf[i] = s.Vf[j];
    d.Vcs[i] = s.Vcs[j];
    d.Vns[i] = s.Vns[j];
    d.clock[i] = s.clock[j];
    d.phase[i] = s.phase[j];
    const uint32_t k = keys[i];
    if (k == 0u) return;  // outside the grid: in no bin
    // a run of equal keys is one bin; its head writes the start and epoch, its tail the end
    if (i == 0 || keys[i - 1] != k) {
        bins[m].x = i;
        bins[m].z = epoch;
    }
    if (i == n - 1 || keys[i + 1] != k) bins[m].y = i;
}

struct MechArgs {
    CellsSoA cur, alt;
    const int4* bins;
    const int* epoch;
    int n;
    Geom g;
    float max_dist, cccr, ccca;
    double ra_ratio;
    float ra_f;  // the ratio as a float
    int ra_exact;  // which loses nothing
    float sure;  // scale of a cutoff's square below which a distance is surely under it (negative: never)
    float half_dt;
};

// forcekernel + movementkernel.  Per candidate j, in the order xi, yi, zi (bins), then ascending
// sorted index, with the cutoff `thres` carried from the previous accepted candidate:
//   d = sqrt(float(double(fma(dz,dz, fma(dx,dx, dy*dy))) + 0.0001)); skip if d >= thres;
//   R = max(r_j + r_i, 0.01); thres = float(double(R) * Ra_ratio); skip if d >= thres;
//   coefr = Cccr*((1-d/R)^2/d) if d <= R; coefa = Ccca*((1-d/thres)^2/d);
//   f = fma(p_i - p_j, coefr - coefa, f)
// then pos += dt/2 * (3f - f_old) as fma(dt/2, fma(3, f, -f_old), pos).
struct Pair {
    float dx, dy, dz, ss;
};
__device__ __forceinline__ Pair pair_of(const float4& p, const float4& q) {
    Pair v;
    v.dx = __fsub_rn(p.x, q.x);
    v.dy = __fsub_rn(p.y, q.y);
    v.dz = __fsub_rn(p.z, q.z);
    v.ss = __fmaf_rn(v.dz, v.dz, __fmaf_rn(v.dx, v.dx, __fmul_rn(v.dy, v.dy)));
    return v;
}
__device__ __forceinline__ float pair_dist(float ss) { return __fsqrt_rn(__double2float_rn(__dadd_rn((double)ss, 0.0001))); }
__device__ __forceinline__ float pair_reach(float rj, float ri) {
    const float rs = __fadd_rn(rj, ri);
    return rs > 0.01f ? rs : 0.01f;
}
// float(double(R) * Ra_ratio); where the ratio is a float the double product is exact, and one rounding to
// float is the float product
__device__ __forceinline__ float cutoff_of(const MechArgs& a, float R) {
    return a.ra_exact ? __fmul_rn(R, a.ra_f) : __double2float_rn(__dmul_rn((double)R, a.ra_ratio));
}
__device__ __forceinline__ float pair_coef(const MechArgs& a, float d, float R, float thres) {
    float cr = 0.f, ca = 0.f;
    if (d <= R) {
        const float t = __fsub_rn(1.f, __fdiv_rn(d, R));
        cr = __fmul_rn(a.cccr, __fdiv_rn(__fmul_rn(t, t), d));
    }
    if (d <= thres) {
        const float t = __fsub_rn(1.f, __fdiv_rn(d, thres));
        ca = __fmul_rn(a.ccca, __fdiv_rn(__fmul_rn(t, t), d));
    }
    return __fsub_rn(cr, ca);
}
// a dead cell: copied, not moved
__device__ __forceinline__ void dead_move(const MechArgs& a, int i, const float4& pr, const float4& of) {
    a.alt.sign[i] = 0;
    a.alt.posr[i] = pr;
    a.alt.oldf[i] = of;
    a.alt.force[i] = a.cur.force[i];
    a.alt.mesh[i] = a.cur.mesh[i];
}
__device__ __forceinline__ void live_move(const MechArgs& a, int i, const float4& pr, const float4& of, float fx, float fy, float fz) {
    const int N = a.g.N;
    const float h = a.half_dt;
    const float nx = __fmaf_rn(h, __fmaf_rn(3.f, fx, -of.x), pr.x);
    const float ny = __fmaf_rn(h, __fmaf_rn(3.f, fy, -of.y), pr.y);
    const float nz = __fmaf_rn(h, __fmaf_rn(3.f, fz, -of.z), pr.z);
    const int3 nb = find_bin(nx, ny, nz, a.g.len);
    if (!inside(nb.x, nb.y, nb.z, N)) {
        // leaves the grid: only the sign changes (the reference returns before writing)
        a.alt.sign[i] = 0;
        a.alt.posr[i] = pr;
        a.alt.oldf[i] = of;
        a.alt.force[i] = make_float4(fx, fy, fz, 0.f);
        a.alt.mesh[i] = a.cur.mesh[i];
        return;
    }
    a.alt.sign[i] = 1;
    a.alt.posr[i] = make_float4(nx, ny, nz, pr.w);
    a.alt.oldf[i] = make_float4(fx, fy, fz, 0.f);
    a.alt.force[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    a.alt.mesh[i] = nb.x + nb.y * N + nb.z * N * N;
}

// One thread per cell.  A warp's lanes sit in different bins: its ~60 rounds over candidates hold ~30 of each
// lane's and ~9 accepted ones, so that with the force computed in the walk the warp issued the force's code
// for a sixth of its lanes.  The walk therefore only decides which candidates are accepted, from |dp|^2 and
// bounds of the cutoff's square that leave the distance itself to a margin of 2^-18, and lists those that act;
// the lists are worked through afterwards, entry by entry.  What bounds it is the issue of instructions (5,770 a
// warp before, 4,800 now, 70% of the cycles); 1M cells 237 -> 207 us, 100,000 57 -> 43.
constexpr int kForceThreads = 256;
constexpr int kForceList = 16;  // entries; a full list is worked off before the walk goes on
// above hi, d >= t is certain; up to lo, d < t is: margins far above the roundings between |dp|^2 + 0.0001 and d
struct Cutoff {
    float t, hi, lo;
};
__device__ __forceinline__ Cutoff cutoff_bounds(float t, float sure) {
    const float m = __fmul_rn(t, t);
    return Cutoff{t, __fmul_rn(m, 1.f + 0x1p-18f), fminf(__fmaf_rn(m, sure, -0.00011f), 1e37f)};
}
__device__ __forceinline__ void force_move_body(const MechArgs& a, int blk) {
    __shared__ int list[kForceList][kForceThreads];
    const int i = blk * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const uint8_t sg = a.cur.sign[i];
    const float4 pr = a.cur.posr[i];
    const float4 of = a.cur.oldf[i];
    if (!sg) {
        dead_move(a, i, pr, of);
        return;
    }
    const int N = a.g.N;
    const long long NN = (long long)N * N;
    const int epoch = *a.epoch;
    const int3 b = find_bin(pr.x, pr.y, pr.z, a.g.len);
    float fx = 0.f, fy = 0.f, fz = 0.f;
    Cutoff c = cutoff_bounds(a.max_dist, a.max_dist > 0.f ? 1.f - 0x1p-18f : -1.f);
    int cnt = 0;
    auto work_off = [&] {
#pragma unroll 1
        for (int k = 0; k < cnt; ++k) {
            const float4 q = a.cur.posr[list[k][threadIdx.x]];
            const Pair v = pair_of(pr, q);
            const float d = pair_dist(v.ss);
            const float R = pair_reach(q.w, pr.w);
            const float own = cutoff_of(a, R);
            if (d >= own) continue;
            const float cf = pair_coef(a, d, R, own);
            fx = __fmaf_rn(v.dx, cf, fx);
            fy = __fmaf_rn(v.dy, cf, fy);
            fz = __fmaf_rn(v.dz, cf, fz);
        }
        cnt = 0;
    };
    // the 27 bins in the reference's order: xi outer, then yi, then zi; the three of a column requested at once
#pragma unroll 1
    for (int o = 0; o < 9; ++o) {
        const int xi = b.x - 1 + o / 3, yi = b.y - 1 + o % 3;
        if (xi < 0 || xi >= N || yi < 0 || yi >= N) continue;
        const int4* col = a.bins + xi + (long long)yi * N + b.z * NN;
        const int4 none = make_int4(0, -1, epoch, 0);
        int4 e = b.z >= 1 && b.z - 1 < N ? col[-NN] : none;
        int4 e1 = b.z >= 0 && b.z < N ? col[0] : none;
        int4 e2 = b.z >= -1 && b.z + 1 < N ? col[NN] : none;
#pragma unroll 1
        for (int z = 0; z < 3; ++z) {
            const int last = e.z == epoch ? e.y : -1;
#pragma unroll 1
            for (int j = e.x; j <= last; ++j) {
                const float4 q = a.cur.posr[j];
                const uint8_t sj = a.cur.sign[j];
                const Pair v = pair_of(pr, q);
                if (v.ss > c.hi || !sj) continue;
                if (!(v.ss <= c.lo) && pair_dist(v.ss) >= c.t) continue;
                c = cutoff_bounds(cutoff_of(a, pair_reach(q.w, pr.w)), a.sure);
                if (v.ss > c.hi) continue;
                list[cnt][threadIdx.x] = j;
                if (++cnt == kForceList) work_off();
            }
            e = e1;
            e1 = e2;
        }
    }
    work_off();
    live_move(a, i, pr, of, fx, fy, fz);
}

// One warp per cell, for n too small to fill the chip with a thread per cell, where that walk's chain of
// loads is all there is (2,000 cells: 43 -> 9 us, 10,000: 49 -> 14).  Lane o takes bin o; the bins' candidates, numbered in order,
// go to the lanes 32 at a time; each lane computes its pair as if accepted.  Which are accepted is the
// solution of "d < cutoff of the last accepted one before me", found by repeating that test from a guess
// until it stands (each repetition settles at least one more lane).  Lanes 0-2 then add the accepted
// terms of one component in order.
__device__ __forceinline__ void force_move_warp_body(const MechArgs& a, int blk) {
    __shared__ float4 terms[kForceThreads / 32][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = blk * (kForceThreads / 32) + w;
    if (i >= a.n) return;
    const uint8_t sg = a.cur.sign[i];
    const float4 pr = a.cur.posr[i];
    const float4 of = a.cur.oldf[i];
    if (!sg) {
        if (lane == 0) dead_move(a, i, pr, of);
        return;
    }
    const int N = a.g.N;
    const int epoch = *a.epoch;
    const int3 b = find_bin(pr.x, pr.y, pr.z, a.g.len);
    const int xi = b.x - 1 + lane / 9, yi = b.y - 1 + (lane / 3) % 3, zi = b.z - 1 + lane % 3;
    int first = 0, num = 0;
    if (lane < 27 && inside(xi, yi, zi, N)) {
        const int4 e = a.bins[xi + (long long)yi * N + (long long)zi * N * N];
        if (e.z == epoch && e.y >= e.x) {
            first = e.x;
            num = e.y - e.x + 1;
        }
    }
    int upto = num;  // candidates of the bins up to this lane's
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, upto, o);
        if (lane >= o) upto += y;
    }
    first -= upto - num;  // candidate number k of this bin is sorted index first + k
    const int total = __shfl_sync(FULL, upto, 31);
    float thres = a.max_dist, f = 0.f;
    const unsigned lt = (1u << lane) - 1u;
    for (int c0 = 0; c0 < total; c0 += 32) {
        const int k = c0 + lane;
        int o = 0;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
            if (__shfl_sync(FULL, upto, o + s - 1) <= k) o += s;
        const int j = __shfl_sync(FULL, first, o) + k;
        bool live = k < total;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (live) {
            q = a.cur.posr[j];
            live = a.cur.sign[j] != 0;
        }
        const Pair v = pair_of(pr, q);
        const float d = pair_dist(v.ss);
        const float R = pair_reach(q.w, pr.w);
        const float own = cutoff_of(a, R);
        unsigned acc = __ballot_sync(FULL, live && !(d >= own));
        for (int it = 0; it < 33; ++it) {
            const unsigned before = acc & lt;
            const float prev = __shfl_sync(FULL, own, before ? 31 - __clz(before) : 0);
            const unsigned next = __ballot_sync(FULL, live && !(d >= (before ? prev : thres)));
            if (next == acc) break;
            acc = next;
        }
        if (acc) thres = __shfl_sync(FULL, own, 31 - __clz(acc));
        const bool use = ((acc >> lane) & 1u) && !(d >= own);
        const unsigned used = __ballot_sync(FULL, use);
        if (use) terms[w][__popc(used & lt)] = make_float4(v.dx, v.dy, v.dz, pair_coef(a, d, R, own));
        __syncwarp();
        if (lane < 3) {
            const float* t = reinterpret_cast<const float*>(terms[w]);
            const int m = __popc(used);
            for (int e = 0; e < m; ++e) f = __fmaf_rn(t[4 * e + lane], t[4 * e + 3], f);
        }
        __syncwarp();
    }
    const float fx = __shfl_sync(FULL, f, 0), fy = __shfl_sync(FULL, f, 1), fz = __shfl_sync(FULL, f, 2);
    if (lane == 0) live_move(a, i, pr, of, fx, fy, fz);
}

// ------------------------------------------------------------------ radix sort (sort.cu)

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ void hist_body(const uint32_t* __restrict__ keys, int n, int shift, int R,
                                          uint32_t* __restrict__ hist, int nb, int blk) {
    __shared__ uint32_t h[256];
    for (int d = threadIdx.x; d < R; d += kSortThreads) h[d] = 0;
    __syncthreads();
    const long long base = (long long)blk * kSortTile;
    const uint32_t mask = (uint32_t)R - 1u;
#pragma unroll 4
    for (int k = 0; k < kSortItems; ++k) {
        long long i = base + k * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & mask], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < R; d += kSortThreads) hist[(long long)d * nb + blk] = h[d];
}

// Exclusive scan of one digit's per-tile counts (row d of the digit-major table), in place, by
// CTA d (`blk`); the digit's total goes to totals[d].  The scatter adds the prefix of the totals.
__device__ __forceinline__ void digit_scan_body(uint32_t* __restrict__ hist, int nb, uint32_t* __restrict__ totals,
                                                int blk) {
    __shared__ uint32_t ws[kSortThreads / 32];
    uint32_t* row = hist + (long long)blk * nb;
    const int per = (nb + kSortThreads - 1) / kSortThreads;
    const int lo = threadIdx.x * per, hi = lo + per < nb ? lo + per : nb;
    uint32_t s = 0;
    for (int i = lo; i < hi; ++i) s += row[i];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    uint32_t wpre = 0;
    for (int j = 0; j < w; ++j) wpre += ws[j];
    uint32_t run = wpre + x - s;
    for (int i = lo; i < hi; ++i) {
        const uint32_t v = row[i];
        row[i] = run;
        run += v;
    }
    if (threadIdx.x == kSortThreads - 1) totals[blk] = run;
}

__device__ __forceinline__ void scatter_body(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                             uint32_t* __restrict__ kout, uint32_t* __restrict__ vout, int n, int shift,
                                             int R, const uint32_t* __restrict__ offs, int nb,
                                             const uint32_t* __restrict__ totals, int iota, int blk) {
    __shared__ uint32_t wcnt[kSortThreads / 32][256];
    __shared__ uint32_t gbase[256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < (kSortThreads / 32) * 256; i += kSortThreads) (&wcnt[0][0])[i] = 0;
    if (w == 0) {
        // exclusive prefix of the digit totals: lane l sums digits 8l .. 8l+7 (R <= 256)
        uint32_t t[8], s = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int d = 8 * lane + k;
            t[k] = d < R ? totals[d] : 0u;
            s += t[k];
        }
        uint32_t x = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        uint32_t run = x - s;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int d = 8 * lane + k;
            if (d < R) gbase[d] = run;
            run += t[k];
        }
    }
    __syncthreads();
    for (int d = threadIdx.x; d < R; d += kSortThreads) gbase[d] += offs[(long long)d * nb + blk];
    __syncthreads();
    const uint32_t mask = (uint32_t)R - 1u;
    const long long base = (long long)blk * kSortTile + w * (kSortTile / (kSortThreads / 32));
    uint32_t key[kSortItems], loc[kSortItems];
    const unsigned lt = lanemask_lt();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const long long i = base + k * 32 + lane;
        const bool valid = i < n;
        key[k] = valid ? kin[i] : 0u;
        const uint32_t dig = (key[k] >> shift) & mask;
        const unsigned peers = __match_any_sync(FULL, valid ? dig : 0xffffffffu);
        const uint32_t before = wcnt[w][dig & 255];
        loc[k] = before + __popc(peers & lt);
        __syncwarp();
        if (valid && (peers & lt) == 0) wcnt[w][dig] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    for (int d = threadIdx.x; d < R; d += kSortThreads) {
        uint32_t run = 0;
#pragma unroll
        for (int ww = 0; ww < kSortThreads / 32; ++ww) {
            uint32_t c = wcnt[ww][d];
            wcnt[ww][d] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const long long i = base + k * 32 + lane;
        if (i < n) {
            const uint32_t dig = (key[k] >> shift) & mask;
            const uint32_t pos = gbase[dig] + wcnt[w][dig] + loc[k];
            kout[pos] = key[k];
            vout[pos] = iota ? (uint32_t)i : vin[i];
        }
    }
}

// ------------------------------------------------------------------ uptake map (lod.cu)

// Clear the lines flagged by the previous map (oxy_consumption_reset, include/LODkernel.cuh:183-190,
// restricted to the lines that can be nonzero).
// One warp per listed line: the row (P floats, P a multiple of 4) is cleared with 16-byte stores.
template <class A>
__device__ __forceinline__ void rate_reset_body(const A& a, int blk, int nblk) {
    const int P4 = a.g.P >> 2;
    const int lane = threadIdx.x & 31;
    const long long gw = ((long long)blk * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)nblk * blockDim.x) >> 5;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < a.nsub; ++s) {
        const int cnt = *a.count[s];
        for (long long li = gw; li < cnt; li += nw) {
            const int line = a.list[s][li];
            float4* row = reinterpret_cast<float4*>(a.rate[s] + (long long)line * a.g.P);
            for (int x4 = lane; x4 < P4; x4 += 32) row[x4] = z;
            if (lane == 0) a.flag[s][line] = 0;
        }
    }
}

// oxy_consumption_update (include/LODkernel.cuh:12-22) with Cell::O2_consume (include/Cells.cuh:74-89)
// at O2 = 1: rate[mesh_idx] += coef * (V/len/len/len) (times the dead factor for phase >= 3).
template <class A>
__device__ __forceinline__ void rate_accum_body(const CellsSoA& c, int n, const A& a, int blk) {
    const int i = blk * blockDim.x + threadIdx.x;
    if (i >= n || !c.sign[i]) return;
    const int ph = c.phase[i];
    if (ph < 0) return;
    const int N = a.g.N;
    const int m = c.mesh[i];
    if (m < 0 || (long long)m >= (long long)N * N * N) return;
    const int x = m % N, line = m / N;
    const float len = a.g.len;
    const float vf = __fdiv_rn(__fdiv_rn(__fdiv_rn(c.V[i], len), len), len);
    for (int s = 0; s < a.nsub; ++s) {
        float r = __fmul_rn(a.coef[s], vf);
        if (ph >= 3) r = __fmul_rn(r, a.dead);
        atomicAdd(a.rate[s] + (long long)line * a.g.P + x, r);
        uint32_t* f = a.flag[s] + line;
        if (*(volatile uint32_t*)f == 0 && atomicExch(f, 1u) == 0u) a.list[s][atomicAdd(a.count[s], 1)] = line;
    }
}

}  // namespace gell
