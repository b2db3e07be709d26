// mech_body.cuh — the per-block bodies of the mechanics kernels (mech.cu: keys, gather, force and
// move; sort.cu: the radix sort's histogram, digit scan and scatter; lod.cu: the uptake map), shared
// by the one-context kernels and the ensemble's batched kernels (mech.cu), which run the same
// body for block `blk` of one member.  Each body is the kernel it came from with blockIdx.x
// replaced by `blk`, so a batched launch computes what the member's own launches compute.
#pragma once

#include <type_traits>

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
// the lists are worked through afterwards, entry by entry.  What bounds it is the issue of instructions;
// 1M cells 237 us with the force in the walk, 204 so, 100,000 54 and 41.  Five blocks an SM (48 registers)
// rather than four (60): 204 against 211 us at 1M cells, 573 against 603 at 3M.
//
// Where many candidates are accepted the list is the detour: a warp whose bins promise more than a list holds
// (kForceCrowd accepted candidates, from the count of a bin near by and the cutoff's sphere) computes the
// forces in the walk, and a lane whose list fills up leaves the walk, waits until the warp has worked its
// lists off, and goes on from there in that way.  (Lists worked off by each lane by itself in the middle of
// its walk took the warp up to 32 lists' time: 1M cells at random, 3, 8 and 37 to a bin, 1,550, 4,300 and
// 18,400 us; all forces in the walk 580, 1,090 and 3,560; so 568, 1,078 and 3,490.)
constexpr int kForceThreads = 256;
constexpr int kForceList = 24;   // entries
constexpr int kForceCrowd = 24;  // accepted candidates, estimated
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
    const uint8_t sg = i < a.n ? a.cur.sign[i] : 0;
    const unsigned live = __ballot_sync(FULL, sg != 0);
    if (i >= a.n) return;
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
    auto add = [&](const Pair& v, float d, float R, float own) {
        const float cf = pair_coef(a, d, R, own);
        fx = __fmaf_rn(v.dx, cf, fx);
        fy = __fmaf_rn(v.dy, cf, fy);
        fz = __fmaf_rn(v.dz, cf, fz);
    };
    // The walk over the 27 bins in the reference's order: xi outer, then yi, then zi; the three of a column
    // requested at once.  It begins at candidate j0 of bin z0 of column o0, and leaves there where it stood
    // when the list was full (o0 = 9: at its end).
    int o0 = 0, z0 = 0, j0 = 0;
    auto walk = [&](auto listed) {
#pragma unroll 1
        for (int o = listed.value ? 0 : o0; o < 9; ++o) {
            const int xi = b.x - 1 + o / 3, yi = b.y - 1 + o % 3;
            if (xi < 0 || xi >= N || yi < 0 || yi >= N) continue;
            const int4* col = a.bins + xi + (long long)yi * N + b.z * NN;
            const int4 none = make_int4(0, -1, epoch, 0);
            int4 e = b.z >= 1 && b.z - 1 < N ? col[-NN] : none;
            int4 e1 = b.z >= 0 && b.z < N ? col[0] : none;
            int4 e2 = b.z >= -1 && b.z + 1 < N ? col[NN] : none;
#pragma unroll 1
            for (int z = 0; z < 3; ++z) {
                int last = e.z == epoch ? e.y : -1, j = e.x;
                if constexpr (!listed.value) {
                    if (o == o0 && z < z0) last = -1;
                    if (o == o0 && z == z0 && j < j0) j = j0;
                }
#pragma unroll 1
                for (; j <= last; ++j) {
                    const float4 q = a.cur.posr[j];
                    const uint8_t sj = a.cur.sign[j];
                    const Pair v = pair_of(pr, q);
                    if (v.ss > c.hi || !sj) continue;
                    if (!(v.ss <= c.lo) && pair_dist(v.ss) >= c.t) continue;
                    const float R = pair_reach(q.w, pr.w);
                    c = cutoff_bounds(cutoff_of(a, R), a.sure);
                    if (v.ss > c.hi) continue;
                    if constexpr (listed.value) {
                        list[cnt][threadIdx.x] = j;
                        if (++cnt == kForceList) {
                            o0 = o;
                            z0 = z;
                            j0 = j + 1;
                            return;
                        }
                    } else {
                        const float d = pair_dist(v.ss);
                        if (!(d >= c.t)) add(v, d, R, c.t);
                    }
                }
                e = e1;
                e1 = e2;
            }
        }
        o0 = 9;
    };
    const float cut = cutoff_of(a, pair_reach(pr.w, pr.w)) / a.g.len;
    const int xf = b.x > 0 ? b.x - 1 : 0, yf = b.y > 0 ? b.y - 1 : 0;
    const int4 near = inside(xf, yf, b.z, N) ? a.bins[xf + (long long)yf * N + b.z * NN] : make_int4(0, -1, epoch, 0);
    // (4.19: 4 pi / 3; the count is that of the bins the walk begins with)
    const bool crowded = near.z == epoch && 4.19f * cut * cut * cut * (float)(near.y - near.x + 1) > (float)kForceCrowd;
    if (2 * __popc(__ballot_sync(live, crowded)) <= __popc(live)) walk(std::true_type());
    __syncwarp(live);
#pragma unroll 1
    for (int k = 0; k < cnt; ++k) {
        const float4 q = a.cur.posr[list[k][threadIdx.x]];
        const Pair v = pair_of(pr, q);
        const float d = pair_dist(v.ss);
        const float R = pair_reach(q.w, pr.w);
        const float own = cutoff_of(a, R);
        if (!(d >= own)) add(v, d, R, own);
    }
    if (o0 < 9) walk(std::false_type());
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

constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096
constexpr int kSortBits = 10;                         // bits of a digit, at most
constexpr int kSortDigits = 1 << kSortBits;
// Up to this many tiles the scatter adds the other tiles' counts itself (a row of at most 32 words a digit).
constexpr int kSortScanTiles = 32;

struct SortPlan {
    int passes, bits;
};
// As few passes as digits of 10 bits allow, in equal digits (4 passes of 7 bits to 3 of 9 at 400^3).
__host__ __device__ __forceinline__ SortPlan sort_plan(int bits) {
    const int passes = bits <= kSortBits ? 1 : (bits + kSortBits - 1) / kSortBits;
    return SortPlan{passes, (bits + passes - 1) / passes};
}

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// The valid lanes whose digit (`bits` bits) is this lane's, by one vote a bit: the match instruction takes the
// lanes' values one after the other (k_scatter at 1M cells 20.8 -> 19.2 us).
__device__ __forceinline__ unsigned digit_peers(uint32_t dig, int bits, bool valid) {
    unsigned peers = __ballot_sync(FULL, valid);
#pragma unroll
    for (int b = 0; b < kSortBits; ++b) {
        if (b >= bits) break;
        const unsigned one = __ballot_sync(FULL, dig >> b & 1u);
        peers &= dig >> b & 1u ? one : ~one;
    }
    return peers;
}

// Every thread's keys are requested before the first is counted: with a request between two counts a tile
// waited for memory once per item (a launch at 1M cells, with its start: 10.6 -> 7.1 us).
__device__ __forceinline__ void hist_body(const uint32_t* __restrict__ keys, int n, int shift, int R,
                                          uint32_t* __restrict__ hist, int nb, int blk) {
    __shared__ uint32_t h[kSortDigits];
    const long long base = (long long)blk * kSortTile;
    uint32_t key[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const long long i = base + k * kSortThreads + threadIdx.x;
        key[k] = i < n ? keys[i] : 0u;
    }
    for (int d = threadIdx.x; d < R; d += kSortThreads) h[d] = 0;
    __syncthreads();
    const uint32_t mask = (uint32_t)R - 1u;
#pragma unroll
    for (int k = 0; k < kSortItems; ++k)
        if (base + k * kSortThreads + threadIdx.x < n) atomicAdd(&h[(key[k] >> shift) & mask], 1u);
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

// The tile's keys and payloads are requested at the start, for the same reason as in hist_body (a
// launch at 1M cells 23.2 -> 19.2 us; what bounds it is the 4-byte scatter).
__device__ __forceinline__ void scatter_body(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                             uint32_t* __restrict__ kout, uint32_t* __restrict__ vout, int n, int shift,
                                             int R, const uint32_t* __restrict__ offs, int nb,
                                             const uint32_t* __restrict__ totals, int iota, int blk) {
    __shared__ uint16_t wcnt[kSortWarps][kSortDigits];
    __shared__ uint32_t gbase[kSortDigits];
    __shared__ uint32_t ws[kSortWarps];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long base = (long long)blk * kSortTile + w * (kSortTile / kSortWarps);
    uint32_t key[kSortItems], val[kSortItems], loc[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const long long i = base + k * 32 + lane;
        key[k] = i < n ? kin[i] : 0u;
        val[k] = iota || i >= n ? (uint32_t)i : vin[i];
    }
    for (int i = lane; i < R / 2; i += 32) reinterpret_cast<uint32_t*>(wcnt[w])[i] = 0;
    {
        // this tile's first slot of each digit: thread t takes digits 2t and 2t + 1
        uint32_t tot[2], off[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int d = 2 * threadIdx.x + e;
            tot[e] = off[e] = 0;
            if (d >= R) continue;
            const uint32_t* row = offs + (long long)d * nb;
            if (nb <= kSortScanTiles) {
                for (int b = 0; b < nb; ++b) {
                    const uint32_t v = row[b];
                    tot[e] += v;
                    off[e] += b < blk ? v : 0u;
                }
            } else {
                tot[e] = totals[d];
                off[e] = row[blk];
            }
        }
        const uint32_t s = tot[0] + tot[1];
        uint32_t x = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[w] = x;
        __syncthreads();
        uint32_t run = x - s;
        for (int j = 0; j < w; ++j) run += ws[j];
        const int d = 2 * threadIdx.x;
        if (d < R) {
            gbase[d] = run + off[0];
            gbase[d + 1] = run + tot[0] + off[1];
        }
    }
    const uint32_t mask = (uint32_t)R - 1u;
    const unsigned lt = lanemask_lt();
    const int bits = __popc(mask);
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const bool valid = base + k * 32 + lane < n;
        const uint32_t dig = (key[k] >> shift) & mask;
        const unsigned peers = digit_peers(dig, bits, valid);
        const uint32_t before = wcnt[w][dig];
        loc[k] = before + __popc(peers & lt);
        __syncwarp();
        if (valid && (peers & lt) == 0) wcnt[w][dig] = (uint16_t)(before + __popc(peers));
        __syncwarp();
    }
    __syncthreads();
    for (int d = threadIdx.x; d < R; d += kSortThreads) {
        uint32_t run = 0;
#pragma unroll
        for (int ww = 0; ww < kSortWarps; ++ww) {
            const uint32_t c = wcnt[ww][d];
            wcnt[ww][d] = (uint16_t)run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        if (base + k * 32 + lane < n) {
            const uint32_t dig = (key[k] >> shift) & mask;
            const uint32_t pos = gbase[dig] + wcnt[w][dig] + loc[k];
            kout[pos] = key[k];
            vout[pos] = val[k];
        }
    }
}

// Keys and their sort for at most kOneCells cells, by one CTA that keeps keys and payloads in registers and
// passes them through shared memory: one launch where keys and passes of their own are 5 to 7, each of which
// takes longer to start than to sort this many.  What bounds it is the one SM's shared memory (~1,500 cycles
// per 1,024 cells and pass), hence the line: 2,000 cells 20 us against 42 (sums of launches with their
// starts, ~4.5 us each), 5,000 25 against 46, but 10,000 38 against 46, whose starts overlap.  The order of
// elements is that of the tiles: chunk w of warp w, round k, lane.
constexpr int kOneCells = 6144;
constexpr int kOneThreads = 1024;
constexpr int kOneRounds = kOneCells / kOneThreads;
constexpr int kOneBits = 8;
constexpr int kOneSmem = kOneCells * 6 + 32 * 256 * 2 + (4 * 256 + 8) * 4;
struct OneJob {
    CellsSoA c;
    Geom g;
    uint32_t *keys, *vals;
    int* epoch;
    int n, bits;
};
__device__ __forceinline__ void sort_one_body(const OneJob& a) {
    extern __shared__ __align__(16) uint8_t one_smem[];
    uint32_t* sk = reinterpret_cast<uint32_t*>(one_smem);
    uint32_t* part = sk + kOneCells;                                // [4][256]
    uint32_t* ws = part + 4 * 256;                                  // [8]
    uint16_t* sv = reinterpret_cast<uint16_t*>(ws + 8);             // [kOneCells]
    uint16_t* cnt = sv + kOneCells;                                 // [32][256]
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (t == 0) *a.epoch += 1;
    const int n = a.n, rounds = (n + kOneThreads - 1) / kOneThreads;
    const int first = w * rounds * 32 + lane;
    uint32_t key[kOneRounds], vl[kOneRounds];  // payload, and its rank within warp and digit in the upper half
#pragma unroll
    for (int k = 0; k < kOneRounds; ++k) {
        const int i = first + 32 * k;
        key[k] = 0u;
        vl[k] = (uint32_t)i;
        if (k >= rounds || i >= n) continue;
        const float4 pr = a.c.posr[i];
        const int3 b = find_bin(pr.x, pr.y, pr.z, a.g.len);
        if (!inside(b.x, b.y, b.z, a.g.N)) {
            a.c.sign[i] = 0;
        } else {
            key[k] = morton3(b.x, b.y, b.z) + 1u;
            a.c.mesh[i] = b.x + b.y * a.g.N + b.z * a.g.N * a.g.N;
        }
    }
    const int passes = a.bits <= kOneBits ? 1 : (a.bits + kOneBits - 1) / kOneBits;
    const int bits = (a.bits + passes - 1) / passes;
    const uint32_t mask = (1u << bits) - 1u;
    const unsigned lt = lanemask_lt();
    for (int p = 0; p < passes; ++p) {
        const int shift = p * bits;
        for (int i = t; i < 32 * 256 / 2; i += kOneThreads) reinterpret_cast<uint32_t*>(cnt)[i] = 0;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kOneRounds; ++k) {
            if (k >= rounds) break;
            const bool valid = first + 32 * k < n;
            const uint32_t dig = (key[k] >> shift) & mask;
            const unsigned peers = digit_peers(dig, bits, valid);
            const uint32_t before = cnt[w * 256 + dig];
            vl[k] = (vl[k] & 0xffffu) | (before + __popc(peers & lt)) << 16;
            __syncwarp();
            if (valid && (peers & lt) == 0) cnt[w * 256 + dig] = (uint16_t)(before + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        {
            // counts of 8 warps each, then of the quarters and digits
            const int d = t & 255, q = t >> 8;
            uint32_t run = 0;
#pragma unroll
            for (int ww = 8 * q; ww < 8 * q + 8; ++ww) {
                const uint32_t c = cnt[ww * 256 + d];
                cnt[ww * 256 + d] = (uint16_t)run;
                run += c;
            }
            part[t] = run;
        }
        __syncthreads();
        uint32_t s = 0, x = 0;
        if (t < 256) {
            s = part[t] + part[256 + t] + part[512 + t] + part[768 + t];
            x = s;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) ws[w] = x;
        }
        __syncthreads();
        if (t < 256) {
            uint32_t run = x - s;
            for (int j = 0; j < w; ++j) run += ws[j];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t c = part[256 * q + t];
                part[256 * q + t] = run;
                run += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kOneRounds; ++k) {
            if (k >= rounds || first + 32 * k >= n) continue;
            const uint32_t dig = (key[k] >> shift) & mask;
            const uint32_t pos = part[256 * (w >> 3) + dig] + cnt[w * 256 + dig] + (vl[k] >> 16);
            sk[pos] = key[k];
            sv[pos] = (uint16_t)vl[k];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kOneRounds; ++k) {
            const int i = first + 32 * k;
            if (k >= rounds || i >= n) continue;
            key[k] = sk[i];
            vl[k] = sv[i];
        }
    }
#pragma unroll
    for (int k = 0; k < kOneRounds; ++k) {
        const int i = first + 32 * k;
        if (k >= rounds || i >= n) continue;
        a.keys[i] = key[k];
        a.vals[i] = vl[k];
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
