// surrogate.cu — learned oxygen surrogate: a 3-D convolutional operator that replaces K LOD substeps
// of one substrate, judged after every use by one plain LOD substep and replaced by the plain solve
// when the judge rejects it.  No reference counterpart: the reference only has the plain solver
// (include/LODkernel.cuh:280-300), which is the fallback here and the source of the training pairs.
//
// Operator.  Input channels [p / b, rate * rate_scale, shell mask] (b = the substrate's boundary
// value, shell = the four boundary layers that Setboundary rewrites), a 3x3x3 convolution to 32
// channels with ReLU, four residual blocks h += conv(relu(conv(h))) (the inner one with ReLU), and a
// 3x3x3 convolution to one channel d; the output field is p + b * d inside and b on the shell.  All
// convolutions are zero-padded ("same"), weights and activations are bf16, sums are fp32.
//
// Activation layout in HBM ("8-channel planes").  A tensor of C channels over the N^3 voxels is
// C/8 planes; plane q holds channels 8q..8q+7 of voxel v = x + N*(y + N*z) as 16 contiguous bytes at
// byte 16*v.  An x-run of voxels of one plane is then exactly the canonical no-swizzle K-major
// operand layout of the tensor cores (8 rows of 16 bytes per core matrix, consecutive voxels 16
// bytes apart), so the operand of tap dx is the run staged for dx = 0 moved by 16*dx bytes; zero fill
// outside the grid gives the padding.
// Every wait is bounded (codes 21-27 in the context's error word).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "async_copy.cuh"
#include "gell_internal.cuh"

namespace gell {

struct SurrogateState;

namespace {

constexpr int kTileM = 128;               // voxels per tile
constexpr int kRunPlaneB = kTileM * 16;   // bytes of one plane of one staged run of voxels (2048)
constexpr int kLayers = 10;                  // conv_in, 4 x (conv_a, conv_b), conv_out
constexpr int kHidden = 32;
constexpr int kInCh = 3;

// Epilogues: forward (kRelu, kResidual, kField) and the data gradients of the backward pass
// (kLinear: the gradient of a linear layer's input; kMask: times [aux > 0], the ReLU's gradient
// with aux = the ReLU's stored output; kResMask: residual add, then times [aux > 0]).
enum ConvMode { kRelu = 0, kResidual = 1, kField = 2, kLinear = 3, kMask = 4, kResMask = 5 };

// Maps of a planes tensor (plane_map) over half voxels, planes in the last dimension: boxes of 128 voxels of
// one x-line of one plane, of 2 voxels of one plane, and of 128 voxels of all planes.
struct PlaneMaps {
    CUtensorMap run, tail, all;
};
struct ConvArgs {
    PlaneMaps in;
    const uint8_t* w;               // packed weights, the shared-memory image
    const float* bias;              // NOUT
    uint4* out;                     // planes (kRelu, kResidual)
    const uint4* res;               // residual planes (kResidual, kResMask; may equal out)
    const uint4* aux;               // mask planes (kMask, kResMask): a channel passes where aux > 0
    float* field_out;               // pitched field (kField)
    const float* field_in;          // pitched field (kField)
    int N, P;
    long long PN;
    long long nvox;                 // N^3: plane length in voxels
    int tiles_x, unit_z;
    float scale, bval;              // kField: out = in + scale * d inside, bval on the shell
    int* err;
};

// ---------------------------------------------------------------- tcgen05 / TMEM (inline PTX)

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// Shared-memory matrix descriptor, no swizzle: start, leading-dimension byte offset (between the
// two 8-element K chunks of an MMA), stride byte offset (between 8-row core-matrix groups), all in
// 16-byte units; bit 46 = descriptor version of sm_100.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// Instruction descriptor of kind::f16: fp32 accumulator, bf16 A and B, both K-major, M = 128.
__host__ __device__ constexpr uint32_t idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// One MMA, issued by the lanes with `on` set of a warp that runs the whole loop together: operands that
// are uniform over the warp then stay in uniform registers, where the instruction wants them.  (From
// inside a one-lane branch each operand is moved there again: 75 cycles an MMA.)
__device__ __forceinline__ void mma_bf16_on(uint32_t on, uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(on)
        : "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r;
}
// The mbarrier completes one phase when every MMA issued so far by this thread has finished.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 32 lanes x 32 columns of fp32: thread t gets lane (base lane + t).
__device__ __forceinline__ void tmem_ld32(uint32_t a, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(a));
}

__device__ __forceinline__ void tmem_ld16(uint32_t a, uint32_t (&v)[16]) {  // 16 columns
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(a));
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* tm, int c0, int c1, int c2, int c3, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(smem_u32(dst)),
        "l"(tm), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t u) {
    __nv_bfloat162 h = *reinterpret_cast<__nv_bfloat162*>(&u);
    return __bfloat1622float2(h);
}

// What the epilogue of one accumulator row (voxel x of line (y, z)) reads besides the accumulator.
template <int NOUT, int MODE>
struct TileIn {
    static constexpr bool kRes = MODE == kResidual || MODE == kResMask, kAux = MODE == kMask || MODE == kResMask;
    uint4 res[kRes ? NOUT / 8 : 1], aux[kAux ? NOUT / 8 : 1];
    float field;
    __device__ __forceinline__ void request(const ConvArgs& a, int x, int y, int z) {
        if (x >= a.N) return;
        const long long vox = (long long)x + (long long)a.N * (y + (long long)a.N * z);
#pragma unroll
        for (int pl = 0; pl < NOUT / 8; ++pl) {
            if constexpr (kRes) res[pl] = a.res[pl * a.nvox + vox];
            if constexpr (kAux) aux[pl] = a.aux[pl * a.nvox + vox];
        }
        if constexpr (MODE == kField) field = a.field_in[(long long)x + (long long)a.P * y + a.PN * z];
    }
};

// Epilogue of one accumulator row: bias, then ReLU, residual add or the field update, and the store.
template <int NOUT, int MODE>
__device__ __forceinline__ void store_tile(const ConvArgs& a, const uint32_t (&v)[NOUT], const float (&bias)[NOUT],
                                           const TileIn<NOUT, MODE>& in, int x, int y, int z) {
    if (x >= a.N) return;
    if constexpr (MODE == kField) {
        const long long pi = (long long)x + (long long)a.P * y + a.PN * z;
        const int N = a.N;
        const bool shell = x < 2 || x > N - 3 || y < 2 || y > N - 3 || z < 2 || z > N - 3;
        const float d = __uint_as_float(v[0]) + bias[0];
        a.field_out[pi] = shell ? a.bval : __fmaf_rn(a.scale, d, in.field);
    } else {
        const long long vox = (long long)x + (long long)a.N * (y + (long long)a.N * z);
        float f[NOUT];
#pragma unroll
        for (int n = 0; n < NOUT; ++n) f[n] = __uint_as_float(v[n]) + bias[n];
#pragma unroll
        for (int pl = 0; pl < NOUT / 8; ++pl) {
            if constexpr (MODE == kResidual || MODE == kResMask) {
                const uint32_t rr[4] = {in.res[pl].x, in.res[pl].y, in.res[pl].z, in.res[pl].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 u = unpack_bf16(rr[j]);
                    f[8 * pl + 2 * j] += u.x;
                    f[8 * pl + 2 * j + 1] += u.y;
                }
            }
            if constexpr (MODE == kMask || MODE == kResMask) {
                const uint32_t mm[4] = {in.aux[pl].x, in.aux[pl].y, in.aux[pl].z, in.aux[pl].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 u = unpack_bf16(mm[j]);
                    if (!(u.x > 0.f)) f[8 * pl + 2 * j] = 0.f;
                    if (!(u.y > 0.f)) f[8 * pl + 2 * j + 1] = 0.f;
                }
            }
            if constexpr (MODE == kRelu) {
#pragma unroll
                for (int j = 0; j < 8; ++j) f[8 * pl + j] = fmaxf(f[8 * pl + j], 0.f);
            }
            a.out[pl * a.nvox + vox] =
                make_uint4(pack_bf16(f[8 * pl], f[8 * pl + 1]), pack_bf16(f[8 * pl + 2], f[8 * pl + 3]),
                           pack_bf16(f[8 * pl + 4], f[8 * pl + 5]), pack_bf16(f[8 * pl + 6], f[8 * pl + 7]));
        }
    }
}

// ---------------------------------------------------------------- k_conv3
// The 3x3x3 convolution as an implicit GEMM on tcgen05.  A tile is 128 voxels of one x-line (M = 128) by
// the output channels; K is 27 taps x the input channels, 16 to an MMA.  An MMA's cost is the fetch of its
// 4 KB A operand from shared memory, whatever its width, so the three z taps of an input line are three
// column groups of one MMA (N = 3 NOUT): line z' adds to the accumulators of the output lines z'-1, z',
// z'+1, which lie side by side in tensor memory, and every input line is multiplied by 18 MMAs (32
// channels) instead of taking part in 54.  (27 separate taps of N = NOUT: 69 cycles an MMA, 3,700 of a
// tile's 5,200 cycles.)  Each output still is one accumulator's sum over the taps in the order dz, dy, dx.
//
// Work comes in units: up to kUnitZ consecutive output lines z0 .. z1-1 at one x tile and y; accumulator i
// is line z0 + i.  The input lines z0-1 .. z1 pass through a ring of kRing slots: the runs y-1, y, y+1 of
// 130 voxels, each plane at a multiple of 128 bytes, so that the taps dx = 0 read whole core matrices (the
// other two straddle them, which doubles the fetch).  A run's plane comes as one box of 128 voxels and one
// of the last two: rows of 2 KB, since boxes of 16-byte rows (8 channels of a voxel) cost the TMA unit two
// cycles a row.  Warp 0 issues the MMAs, warps 1-3 the loads (one dy each), and two groups of four
// epilogue warps take the lines of even and odd index.
//
// (256^3, 32 -> 32 channels: 2.52 -> 0.90 ms a launch; what bounds it now is shared memory: 77 cycles of
// operand fetch an MMA and the staging's writes, 1,600 of a line's 1,700 cycles.)
constexpr int kUnitZ = 16;    // accumulators: 16 x 32 columns are all of tensor memory
constexpr int kRing = 6;
constexpr int kPlaneB = 2176; // bytes from one plane of a staged run to the next: 130 voxels, rounded up to 128 bytes
constexpr int kConvThreads = 384;

template <int CIN8, int NOUT>
struct ConvSmem {
    static constexpr int kRunB = CIN8 * kPlaneB;
    static constexpr int kGroupB = 3 * kRunB;
    static constexpr int kHalves = CIN8 / 2;               // MMAs (16 input channels) per (dy, dx)
    static constexpr int kWBlk = 3 * NOUT * 32;            // one (dy, dx, half) weight block
    static constexpr int kWB = 9 * kHalves * kWBlk;
    static constexpr int kBars = kRing * kGroupB + kWB;
    static constexpr int kBytes = kBars + (2 * kRing + 2 * kUnitZ + 2) * 8 + 16;
};

struct Unit {
    int x0, y, z0, z1;
};
__device__ __forceinline__ Unit unit_of(int N, int tiles_x, int unit_z, long long u) {
    const long long r = u / tiles_x, s = r / N;
    Unit o;
    o.x0 = (int)(u - r * tiles_x) * kTileM;
    o.y = (int)(r - s * N);
    o.z0 = (int)s * unit_z;
    o.z1 = o.z0 + unit_z < N ? o.z0 + unit_z : N;
    return o;
}
__device__ __forceinline__ long long unit_count(int N, int tiles_x, int unit_z) {
    return (long long)tiles_x * ((N + unit_z - 1) / unit_z) * N;
}

template <int CIN8, int NOUT, int MODE>
__global__ void __launch_bounds__(kConvThreads, 1) k_conv3(const __grid_constant__ ConvArgs a) {
    using L = ConvSmem<CIN8, NOUT>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* wsm = smem + kRing * L::kGroupB;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
    uint64_t* full = bars;               // [kRing] input line loaded (three producers)
    uint64_t* empty = bars + kRing;      // [kRing] input line released by the MMAs
    uint64_t* accf = bars + 2 * kRing;   // [kUnitZ] accumulator complete
    uint64_t* acce = accf + kUnitZ;      // [kUnitZ] accumulator read (4 epilogue warps)
    uint64_t* wbar = acce + kUnitZ;
    uint64_t* done = wbar + 1;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kRing; ++i) {
            mbar_init(&full[i], 3);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < kUnitZ; ++i) {
            mbar_init(&accf[i], 1);
            mbar_init(&acce[i], 4);
        }
        mbar_init(wbar, 1);
        mbar_init(done, 1);
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(tslot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const long long U = unit_count(a.N, a.tiles_x, a.unit_z);

    if (warp == 0) {
        // the whole warp runs the loop, one lane issues (see mma_bf16_on)
        const uint32_t on = elect_one();
        bool ok = mbar_wait(wbar, 0, a.err, 22);
        const uint64_t b0 = sdesc(smem_u32(wsm), 3 * NOUT * 16, 128);
        const uint32_t rbase = smem_u32(smem);
        uint32_t used = 0, phase = 0;  // per accumulator: written before; parity of its last hand-over
        auto wait_acc = [&](int m, int nz) {  // an output line's accumulator has been read before line m starts it
            if (m >= nz) return true;
            const uint32_t bit = 1u << m;
            if (used & bit) {
                if (!mbar_wait(&acce[m], (phase & bit) != 0u, a.err, 24)) return false;
                phase ^= bit;
            }
            used |= bit;
            return true;
        };
        long long u = blockIdx.x;
        int m = 0, nz = 0, sl = 0;  // input line z0 - 1 + m of the unit, in ring slot sl
        uint32_t gph = 0;           // parity of the ring's current round
        // the hand-overs of the line before (its slot; the output line it completed): they are committed a
        // few MMAs into this line, because the warp cannot go on from a commit before the tensor pipe has
        // drained up to it, and the pipe then has these MMAs to run through the next commits and waits
        int csl = -1, cacc = -1;
        auto commit = [&] {
            if (on && csl >= 0) {
                mma_commit(&empty[csl]);
                if (cacc >= 0) mma_commit(&accf[cacc]);
            }
            __syncwarp();
        };
        if (u < U) {
            const Unit w = unit_of(a.N, a.tiles_x, a.unit_z, u);
            nz = w.z1 - w.z0;
        }
        while (ok && u < U) {
            ok = mbar_wait(&full[sl], gph, a.err, 23);
            if (ok) ok = wait_acc(m, nz);
            if (!ok) break;
            tc_fence_after();
            // output lines lo .. hi: m-2 (dz = 2), m-1 (dz = 1), m (dz = 0), as far as the unit has them
            const int lo = m > 2 ? m - 2 : 0, hi = m < nz ? m : nz - 1, n = hi - lo + 1;
            const bool first = hi == m;  // line m starts here
            const uint32_t d = tmem + (uint32_t)(lo * NOUT), dm = tmem + (uint32_t)(m * NOUT);
            const uint64_t bl = b0 + (uint64_t)((lo - m + 2) * NOUT);  // rows of 16 bytes
            const uint64_t ga = sdesc(rbase + (uint32_t)(sl * L::kGroupB), kPlaneB, 128);
            const uint32_t idn = idesc_bf16(NOUT * n);
            // descriptors differ only in the start address (low 14 bits, 16-byte units, no carry out:
            // shared memory is below 256 KB).  The line's first sum starts from zero, the others' go on.
            if (first) {
                if (n > 1) mma_bf16_on(on, d, ga, bl, idesc_bf16(NOUT * (n - 1)), 1u);
                mma_bf16_on(on, dm, ga, b0 + (uint64_t)(2 * NOUT), idesc_bf16(NOUT), 0u);
            } else {
                mma_bf16_on(on, d, ga, bl, idn, 1u);
            }
#pragma unroll
            for (int k = 1; k < 9 * L::kHalves; ++k) {
                const int r = k / L::kHalves, h = k % L::kHalves;  // (dy, dx) and the half
                const uint32_t ao = ((r / 3) * L::kRunB + (r % 3) * 16 + 2 * h * kPlaneB) >> 4;
                mma_bf16_on(on, d, ga + ao, bl + ((k * L::kWBlk) >> 4), idn, 1u);
                if (k == 3 * L::kHalves) commit();
            }
            csl = sl;
            cacc = m - 2;
            if (++m == nz + 2) {
                if (nz == 1) {
                    // the next unit's first line waits for this very accumulator
                    commit();
                    csl = -1;
                }
                m = 0;
                u += gridDim.x;
                if (u < U) {
                    const Unit w = unit_of(a.N, a.tiles_x, a.unit_z, u);
                    nz = w.z1 - w.z0;
                }
            }
            if (++sl == kRing) {
                sl = 0;
                gph ^= 1u;
            }
        }
        commit();
        if (on) mma_commit(done);
        __syncwarp();
        mbar_wait(done, 0, a.err, 25);
    } else if (warp < 4) {
        if (lane == 0) {
            const int dy = warp - 1;
            if (dy == 0) {
                mbar_arrive_expect(wbar, (uint32_t)L::kWB);
                for (int off = 0; off < L::kWB; off += 16384) {
                    const int nb = L::kWB - off < 16384 ? L::kWB - off : 16384;
                    bulk_load(wsm + off, a.w + off, (uint32_t)nb, wbar);
                }
            }
            bool ok = true;
            int g = 0;
            for (long long u = blockIdx.x; ok && u < U; u += gridDim.x) {
                const Unit w = unit_of(a.N, a.tiles_x, a.unit_z, u);
                for (int zz = w.z0 - 1; zz <= w.z1; ++zz, ++g) {
                    const int sl = g % kRing;
                    if (g >= kRing && !mbar_wait1(&empty[sl], ((g / kRing) - 1) & 1, a.err, 21)) {
                        ok = false;
                        break;
                    }
                    uint8_t* rb = smem + sl * L::kGroupB + dy * L::kRunB;
                    mbar_arrive_expect(&full[sl], (uint32_t)(CIN8 * (kTileM + 2) * 16));
                    // elements of the maps are half voxels (8 bytes); the run starts at x0 - 1
#pragma unroll
                    for (int pl = 0; pl < CIN8; ++pl) {
                        tma_load_4d(rb + pl * kPlaneB, &a.in.run, 2 * (w.x0 - 1), w.y + dy - 1, zz, pl, &full[sl]);
                        tma_load_4d(rb + pl * kPlaneB + kTileM * 16, &a.in.tail, 2 * (w.x0 + kTileM - 1), w.y + dy - 1, zz, pl, &full[sl]);
                    }
                }
            }
        }
    } else {
        const int q = warp & 3, grp = (warp - 4) >> 2;  // TMEM lanes 32q.. are this warp's
        float bias[NOUT];
#pragma unroll
        for (int n = 0; n < NOUT; ++n) bias[n] = a.bias[n];
        uint32_t phase = 0;
        bool ok = true;
        for (long long u = blockIdx.x; ok && u < U; u += gridDim.x) {
            const Unit w = unit_of(a.N, a.tiles_x, a.unit_z, u);
            const int x = w.x0 + 32 * q + lane;
            for (int i = grp; i < w.z1 - w.z0; i += 2) {
                TileIn<NOUT, MODE> in;
                in.request(a, x, w.y, w.z0 + i);  // residual and mask planes on their way during the wait
                if (!mbar_wait(&accf[i], (phase >> i) & 1u, a.err, 26)) {
                    ok = false;
                    break;
                }
                phase ^= 1u << i;
                tc_fence_after();
                uint32_t v[NOUT];
                const uint32_t ta = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(i * NOUT);
                tmem_ld32(ta, v);
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acce[i]);
                store_tile<NOUT, MODE>(a, v, bias, in, x, w.y, w.z0 + i);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// ---------------------------------------------------------------- weight gradients
// k_wgrad (tcgen05): S[t][b][a] = sum over voxels v of A[a, v] * B[b, v - t], t the 27 taps, A of 4 planes
// (32 channels), B of BP planes, zero outside the grid.  With A = the layer's input and B = the gradient of
// its output this is dW[b][a][t]; the first layer, whose input has 3 channels, takes A = the gradient and
// B = its input, which is dW[a][b][-t].  The voxels are the K dimension, so both operands are read MN-major
// from the 8-channel planes as staged (8 channels of one voxel = 16 contiguous bytes, consecutive voxels 16
// bytes apart: the canonical no-swizzle MN-major layout, channel groups SBO apart, voxel groups of 8 LBO =
// 128 bytes apart).  Per tile (128 voxels of one x-line): a row group of A (the runs y-1, y, y+1 at one z)
// as M = 128 rows (dy, a) (the rows past 96 are whatever lies behind the group and are discarded), one of
// the three groups dz; three copies of the B run moved by -1, 0, 1 voxels as N = 24 BP columns (dx, b).
// 3 dz x 8 blocks of 16 voxels = 24 MMAs per tile into 3 accumulators.  A's row groups go through a ring:
// units of up to kUnitZ lines, each group loaded once per unit.  At the end each CTA writes its sums.
//
// The tensor cores drop what lies below the accumulator's last bit, so the error grows with the number of
// MMAs in a chain: over all of a CTA's lines it came to 6e-5 of a 32 -> 32 layer's gradient at 128^3.  Three
// reader warps per dz therefore take the accumulators over into fp32 sums in registers: for B of 2 planes
// after every line (two sets in turn, 8 MMAs a chain: 2e-7 of the gradient, which sums on the CUDA cores had
// to 4e-7), for B of 4 planes (288 columns, one set fits tensor memory, so that the MMAs wait) two thirds
// through the CTA's units and at the end.
//
// (As 72 MMAs of N = 32 with A moved by dx voxels, off the 128-byte core matrices, all 9 runs of the input
// loaded per tile and partial sums written 108 bytes apart, a 32 -> 32 launch at 96^3 took 206 us, 106 now;
// the first and last layers took 670 us each on the CUDA cores, 106 now.)
constexpr int kWgPart = 27 * 32 * 32;  // floats of one CTA's partial sums, at most
constexpr int kWgCtas = 148;           // CTAs at most (room for their partial sums)
constexpr int kWgRing = 6;
constexpr int kWgThreads = 448;        // loads, MMAs, 3 x 4 reader warps
template <int BP>
struct WgradSmem {
    static constexpr int kGroupB = 12 * kRunPlaneB;  // one row group of A
    static constexpr int kCopyB = 3 * BP * kRunPlaneB;  // the three copies of the B run
    // the operand A spans 16 planes from a group's start: with the copies of B behind the ring, always inside
    static constexpr int kBars = kWgRing * kGroupB + 2 * kCopyB;
    static constexpr int kBytes = kBars + (2 * kWgRing + 9) * 8 + 16;
    static constexpr int kCols = 24 * BP;        // columns of one dz
    static constexpr int kSets = BP == 2 ? 2 : 1;  // sets of accumulators
};

__host__ __device__ constexpr uint32_t idesc_bf16_mn(int n) {
    return idesc_bf16(n) | (1u << 15) | (1u << 16);
}

struct WgradArgs {
    CUtensorMap a, b;  // plane_map of A and of B
    float* partial;    // [gridDim.x][27][8 BP][32]
    int N, tiles_x, unit_z;
    int* err;
};

template <int BP>
__global__ void __launch_bounds__(kWgThreads, 1) k_wgrad(const __grid_constant__ WgradArgs a) {
    using L = WgradSmem<BP>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* bsm = smem + kWgRing * L::kGroupB;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
    uint64_t* full = bars;                // [kWgRing] row group of A loaded
    uint64_t* empty = bars + kWgRing;     // [kWgRing]
    uint64_t* bfull = bars + 2 * kWgRing; // [2] copies of B loaded
    uint64_t* bempty = bfull + 2;         // [2]
    uint64_t* sfull = bempty + 2;         // [2] a set's chain is complete
    uint64_t* sread = sfull + 2;          // [2] ... and has been read (9 warps)
    uint64_t* done = sread + 2;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kWgRing; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bfull[i], 1);
            mbar_init(&bempty[i], 1);
            mbar_init(&sfull[i], 1);
            mbar_init(&sread[i], 9);
        }
        mbar_init(done, 1);
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc(tslot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const long long U = unit_count(a.N, a.tiles_x, a.unit_z);
    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int g = 0, k = 0;
            for (long long u = blockIdx.x; ok && u < U; u += gridDim.x) {
                const Unit w = unit_of(a.N, a.tiles_x, a.unit_z, u);
                for (int zz = w.z0 - 1; ok && zz <= w.z1; ++zz, ++g) {
                    const int sl = g % kWgRing;
                    if (g >= kWgRing && !mbar_wait1(&empty[sl], ((g / kWgRing) - 1) & 1, a.err, 31)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect(&full[sl], (uint32_t)L::kGroupB);
                    for (int dy = 0; dy < 3; ++dy)
                        tma_load_4d(smem + sl * L::kGroupB + dy * 4 * kRunPlaneB, &a.a, 2 * w.x0, w.y + dy - 1, zz, 0, &full[sl]);
                    if (zz < w.z0 || zz >= w.z1) continue;
                    const int s = k & 1;
                    if (k >= 2 && !mbar_wait1(&bempty[s], ((k >> 1) - 1) & 1, a.err, 34)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect(&bfull[s], (uint32_t)L::kCopyB);
                    // copy dx holds B[v + 1 - dx]
                    for (int dx = 0; dx < 3; ++dx)
                        tma_load_4d(bsm + s * L::kCopyB + dx * BP * kRunPlaneB, &a.b, 2 * (w.x0 + 1 - dx), w.y, zz, 0, &bfull[s]);
                    ++k;
                }
            }
        }
    } else if (warp == 1) {
        // the whole warp runs the loop, one lane issues; hand-overs are committed a few MMAs into the next
        // line (see k_conv3)
        constexpr uint32_t idesc = idesc_bf16_mn(L::kCols);
        const uint32_t on = elect_one();
        bool ok = true;
        int g = 0, k = 0, f = 0;                  // row groups, lines, chains begun
        const int nu = (int)((U - blockIdx.x + gridDim.x - 1) / gridDim.x), half = nu - (nu + 1) / 3;
        int n = 0;                               // units begun
        int crel = 0, cg = 0, cs = -1, cf = -1;  // the line before: groups to release from group cg on, its copies of B, the set it completes
        auto commit = [&] {
            if (on && cs >= 0) {
                mma_commit(&bempty[cs]);
                for (int j = 0; j < crel; ++j) mma_commit(&empty[(cg + j) % kWgRing]);
                if (cf >= 0) mma_commit(&sfull[cf]);
            }
            __syncwarp();
        };
        for (long long u = blockIdx.x; ok && u < U; u += gridDim.x) {
            const Unit w = unit_of(a.N, a.tiles_x, a.unit_z, u);
            const int nz = w.z1 - w.z0;
            for (int i = 0; i < nz; ++i, ++k) {
                const int s = k & 1;
                if (i == 0) {
                    // a unit's first line may wait for slots or sums that the last line still holds
                    commit();
                    cs = -1;
                }
                const bool begin = BP == 2 || (i == 0 && (n == 0 || n == half));
                const int set = f % L::kSets;
                for (int j = i == 0 ? 0 : 2; j < 3 && ok; ++j) {
                    const int gg = g + i + j;
                    ok = mbar_wait(&full[gg % kWgRing], (gg / kWgRing) & 1, a.err, 32);
                }
                if (ok) ok = mbar_wait(&bfull[s], (k >> 1) & 1, a.err, 35);
                if (ok && begin && f >= L::kSets) ok = mbar_wait(&sread[set], (f / L::kSets - 1) & 1, a.err, 37);
                if (!ok) break;
                tc_fence_after();
                const uint64_t b0 = sdesc(smem_u32(bsm + s * L::kCopyB), 128, kRunPlaneB);
                const uint32_t acc = begin ? 0u : 1u;
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const uint64_t a0 = sdesc(smem_u32(smem) + (uint32_t)(((g + i + j) % kWgRing) * L::kGroupB), 128, kRunPlaneB);
#pragma unroll
                    for (int kb = 0; kb < 8; ++kb) {
                        mma_bf16_on(on, tmem + (uint32_t)(128 * j + 64 * set), a0 + 16 * kb, b0 + 16 * kb, idesc, kb > 0 ? 1u : acc);
                        if (j == 0 && kb == 3) commit();
                    }
                }
                cs = s;
                cg = g + i;
                crel = i < nz - 1 ? 1 : 3;
                const bool end = BP == 2 || (i == nz - 1 && (n == half - 1 || n == nu - 1));
                cf = end ? set : -1;
                if (end) ++f;
            }
            g += nz + 2;
            ++n;
        }
        commit();
        if (on) mma_commit(done);
        __syncwarp();
        mbar_wait(done, 0, a.err, 36);
    } else if ((warp & 3) < 3) {
        const int row = 32 * (warp & 3) + lane, dy = row >> 5, ch = lane;  // row (dy, a)
        const int dz = (warp - 2) >> 2;
        float sum[L::kCols];
#pragma unroll
        for (int c = 0; c < L::kCols; ++c) sum[c] = 0.f;
        int chains = 0;
        for (long long u = blockIdx.x; u < U; u += gridDim.x) {
            const Unit w = unit_of(a.N, a.tiles_x, a.unit_z, u);
            chains = BP == 2 ? chains + w.z1 - w.z0 : chains < 2 ? chains + 1 : 2;
        }
        for (int f = 0; f < chains; ++f) {
            const int set = f % L::kSets;
            if (!mbar_wait(&sfull[set], (f / L::kSets) & 1, a.err, 38, 1 << 26)) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < L::kCols; c += 16) {
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(32 * dy) << 16) + (uint32_t)(128 * dz + 64 * set + c), v);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 16; ++e) sum[c + e] += __uint_as_float(v[e]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sread[set]);
        }
        float* out = a.partial + (size_t)blockIdx.x * (27 * 256 * BP) + ch;
#pragma unroll
        for (int c = 0; c < L::kCols; ++c)  // column (dx, b)
            out[((9 * dz + 3 * dy + c / (8 * BP)) * (8 * BP) + c % (8 * BP)) * 32] = sum[c];
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// Sums of per-block partials in a fixed order (the result does not depend on scheduling).  A block takes 32
// entries; its 8 warps add every eighth block each, 4 loads in flight, then the warps' sums are added in
// order.  (One thread per entry over all blocks in turn waited on 148 dependent loads: 25 us.)
__device__ __forceinline__ float partial_sum(const float* partial, int blocks, long long stride, int i, bool in) {
    __shared__ float red[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    for (int b0 = w; b0 < blocks; b0 += 32)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (in && b0 + 8 * k < blocks) s[k] += partial[(b0 + 8 * k) * stride + i];
    red[w][lane] = (s[0] + s[1]) + (s[2] + s[3]);
    __syncthreads();
    float t = 0.f;
    for (int k = 0; k < 8; ++k) t += red[k][lane];
    return t;
}
// out[i] = sum_b partial[b * stride + i]
__global__ void __launch_bounds__(256) k_sum_partials(const float* partial, int blocks, int n, int stride, float* out) {
    const int i = blockIdx.x * 32 + (threadIdx.x & 31);
    const float t = partial_sum(partial, blocks, stride, i, i < n);
    if (threadIdx.x < 32 && i < n) out[i] = t;
}
// The same for k_wgrad's partial sums [t][b][a] (BC channels b, 32 channels a), into the layer's order
// [cout][cin][27]: co = b, ci = a, tap = t, or the other way round and mirrored (`gradient_a`).
__global__ void __launch_bounds__(256) k_sum_wgrad(const float* partial, int blocks, int BC, int cout, int cin, int gradient_a, float* out) {
    const int n = 27 * BC * 32, i = blockIdx.x * 32 + (threadIdx.x & 31);
    const float s = partial_sum(partial, blocks, n, i, i < n);
    const int ca = i & 31, cb = i / 32 % BC, t = i / (32 * BC);
    const int co = gradient_a ? ca : cb, ci = gradient_a ? cb : ca, tap = gradient_a ? 26 - t : t;
    if (threadIdx.x < 32 && i < n && co < cout && ci < cin) out[((size_t)co * cin + ci) * 27 + tap] = s;
}

// Per-channel sums over the voxels of a planes tensor (bias gradients): block partials [block][C].
__global__ void k_channel_sums(const uint4* G, int planes, long long nvox, float* partial) {
    __shared__ float red[8][32];
    const int C = planes * 8;
    for (int pl = 0; pl < planes; ++pl) {
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nvox; v += (long long)gridDim.x * blockDim.x) {
            const uint4 u = G[pl * nvox + v];
            const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = unpack_bf16(w4[j]);
                s[2 * j] += f.x;
                s[2 * j + 1] += f.y;
            }
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            float t = s[e];
            for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(FULL, t, o);
            if ((threadIdx.x & 31) == 0) red[e][threadIdx.x >> 5] = t;
        }
        __syncthreads();
        if (threadIdx.x < 8) {
            float t = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
            partial[(size_t)blockIdx.x * C + pl * 8 + threadIdx.x] = t;
        }
        __syncthreads();
    }
}

// Input planes of the operator: plane 0 = (p / b, rate * rate_scale, shell, 0, ...); plane 1 stays
// zero (the first convolution reads 16 input channels).
__global__ void k_pack_input(const float* p, const float* rate, Geom g, float inv_b, float rate_scale, uint4* out) {
    const long long nvox = (long long)g.N * g.N * g.N;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nvox;
         v += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(v % g.N);
        const long long yz = v / g.N;
        const int y = (int)(yz % g.N), z = (int)(yz / g.N);
        const long long pi = x + (long long)g.P * y + g.PN * z;
        const int N = g.N;
        const bool shell = x < 2 || x > N - 3 || y < 2 || y > N - 3 || z < 2 || z > N - 3;
        out[v] = make_uint4(pack_bf16(__fmul_rn(p[pi], inv_b), __fmul_rn(rate[pi], rate_scale)),
                            pack_bf16(shell ? 1.f : 0.f, 0.f), 0u, 0u);
    }
}

// Input planes of the delta form: channel 0 = (p1 - p0) / m (the change of one plain substep,
// normalised by its largest magnitude inside the shell), channel 1 = rate * rate_scale, channel 2
// = the shell mask.
__global__ void k_pack_input_delta(const float* p1, const float* p0, const float* rate, Geom g, float inv_m,
                                   float rate_scale, uint4* out) {
    const long long nvox = (long long)g.N * g.N * g.N;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nvox;
         v += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(v % g.N);
        const long long yz = v / g.N;
        const int y = (int)(yz % g.N), z = (int)(yz / g.N);
        const long long pi = x + (long long)g.P * y + g.PN * z;
        const int N = g.N;
        const bool shell = x < 2 || x > N - 3 || y < 2 || y > N - 3 || z < 2 || z > N - 3;
        const float d = shell ? 0.f : __fmul_rn(__fsub_rn(p1[pi], p0[pi]), inv_m);
        out[v] = make_uint4(pack_bf16(d, __fmul_rn(rate[pi], rate_scale)), pack_bf16(shell ? 1.f : 0.f, 0.f), 0u, 0u);
    }
}

// max |a - b| over the voxels inside the shell (the values the next substep carries forward), as
// the bits of a non-negative float (ordered like the floats).
__global__ void k_absdiff_max(const float* a, const float* b, Geom g, unsigned* out) {
    const int N = g.N, M = N - 4;
    const long long n = (long long)M * M * M;
    float m = 0.f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % M) + 2;
        const long long yz = i / M;
        const int y = (int)(yz % M) + 2, z = (int)(yz / M) + 2;
        const long long pi = x + (long long)g.P * y + g.PN * z;
        m = fmaxf(m, fabsf(a[pi] - b[pi]));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

// ---------------------------------------------------------------- training: packing, loss, Adam

// Weight images from the fp32 master weights W[cout][cin][27] of one layer (device-side packing, so
// a training step never leaves the GPU): the forward image (input channel 16h + 8kc + e, output
// channel n, as pack_layer) or, with `transpose`, the image of the convolution that maps the
// gradient of the layer's output to the gradient of its input: input channels = the layer's
// outputs, output channels = the layer's inputs, taps mirrored (tap -> 26 - tap).
struct PackJob {
    const float* W;  // the layer's weights; its bias follows them
    int cin, cout, cin8, nout, transpose;
    __nv_bfloat16* img;
    float* bias;     // forward images only: the bias padded to nout
};
struct PackArgs {
    PackJob job[2 * kLayers];
};
__global__ void k_pack_w(const __grid_constant__ PackArgs a) {
    const PackJob& j = a.job[blockIdx.y];
    const int cin = j.cin, cout = j.cout, nout = j.nout;
    const int halves = j.cin8 / 2;
    const int n_img = 27 * halves * 2 * nout * 8;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_img; i += gridDim.x * blockDim.x) {
        const int e = i % 8, n = (i / 8) % nout, dz = 2 - (i / (8 * nout)) % 3, kc = (i / (24 * nout)) % 2;
        const int h = (i / (48 * nout)) % halves, r = i / (48 * nout * halves);  // r = 3 dy + dx
        const int tap = 9 * dz + r;
        const int k = 16 * h + 8 * kc + e;  // input channel of the packed convolution
        float v = 0.f;
        if (!j.transpose) {
            if (n < cout && k < cin) v = j.W[((size_t)n * cin + k) * 27 + tap];
        } else {
            if (k < cout && n < cin) v = j.W[((size_t)k * cin + n) * 27 + (26 - tap)];
        }
        j.img[i] = __float2bfloat16_rn(v);
    }
    if (j.bias && blockIdx.x == 0 && threadIdx.x < nout)
        j.bias[threadIdx.x] = threadIdx.x < cout ? j.W[(size_t)cout * cin * 27 + threadIdx.x] : 0.f;
}

// Gradient of the loss L = mean over the voxels inside the shell of ((q - y) / b)^2 with respect to
// the last convolution's output d (q = p + b d inside): 2 (q - y) / (b n), in channel 0 of plane 0
// of the gradient planes; zero on the shell.  Block partial sums of ((q - y) / b)^2 go to `loss`.
__global__ void k_loss_grad(const float* q, const float* y, Geom g, float b, float inv_n, uint4* gd, float* loss) {
    __shared__ float red[32];
    const int N = g.N;
    const long long nvox = (long long)N * N * N;
    float acc = 0.f;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nvox; v += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(v % N);
        const long long yz = v / N;
        const int yy = (int)(yz % N), zz = (int)(yz / N);
        const bool shell = x < 2 || x > N - 3 || yy < 2 || yy > N - 3 || zz < 2 || zz > N - 3;
        float gr = 0.f;
        if (!shell) {
            const long long pi = x + (long long)g.P * yy + g.PN * zz;
            const float e = (q[pi] - y[pi]) / b;
            acc = __fmaf_rn(e, e, acc);
            gr = 2.f * e * inv_n;
        }
        gd[v] = make_uint4(pack_bf16(gr, 0.f), 0u, 0u, 0u);
    }
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        loss[blockIdx.x] = t;
    }
}

// Sum of squares of the gradient (for clipping by its global norm): one block, 8 loads in flight per thread.
__global__ void __launch_bounds__(1024) k_sumsq(const float* g, long long n, float* out) {
    __shared__ float red[32];
    float a8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (long long i = threadIdx.x; i < n; i += 8 * 1024) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = i + k * 1024 < n ? g[i + k * 1024] : 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) a8[k] = __fmaf_rn(v[k], v[k], a8[k]);
    }
    float acc = ((a8[0] + a8[1]) + (a8[2] + a8[3])) + ((a8[4] + a8[5]) + (a8[6] + a8[7]));
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < 32; ++w) t += red[w];
        *out = t;
    }
}

// Adam (Kingma & Ba, ICLR 2015) with bias correction, on the gradient scaled to global norm
// <= clip: m = b1 m + (1 - b1) g; v = b2 v + (1 - b2) g^2; w -= lr (m / bc1) / (sqrt(v / bc2) + eps).
__global__ void k_adam(float* w, const float* g, float* m, float* v, long long n, const float* sumsq, float clip,
                       float lr, float b1, float b2, float eps, float bc1, float bc2) {
    const float norm = sqrtf(*sumsq);
    const float sc = norm > clip ? clip / norm : 1.f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i] * sc;
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    }
}

// Layer table: input planes, output channels (padded), mode.
struct LayerShape {
    int cin, cout, cin8, nout;
};
constexpr LayerShape kShape[kLayers] = {
    {kInCh, kHidden, 2, 32},   {kHidden, kHidden, 4, 32}, {kHidden, kHidden, 4, 32}, {kHidden, kHidden, 4, 32},
    {kHidden, kHidden, 4, 32}, {kHidden, kHidden, 4, 32}, {kHidden, kHidden, 4, 32}, {kHidden, kHidden, 4, 32},
    {kHidden, kHidden, 4, 32}, {kHidden, 1, 4, 32}};

}  // namespace

// ---------------------------------------------------------------- host state

// Training state of one substrate's operator (gell_surrogate_train_*): fp32 master weights in the
// layout of gell_surrogate_load, their gradient and Adam moments, the images of the data-gradient
// convolutions, every activation of the forward pass and the gradient planes.
struct TrainState {
    long long count = 0;
    long long off_w[kLayers] = {}, off_b[kLayers] = {};
    float *master = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
    float* partial = nullptr;    // block partial sums
    long long partial_n = 0;
    float* zero_bias = nullptr;  // 32 zeros
    float* scal = nullptr;       // [0] gradient sum of squares, [1] loss, [2..] loss partials
    float* hloss = nullptr;      // pinned
    uint8_t* wt[kLayers] = {};   // data-gradient images (layers 1..9)
    uint4* hb[5] = {};
    uint4* tb[4] = {};
    uint4 *gh = nullptr, *gu = nullptr, *gd = nullptr;
    float* tgt = nullptr;        // the plain solver's field after the substeps (pitched)
    PlaneMaps mh[5], mt[4], mgd, mgh, mgu;
    int step = 0;
};

struct SurrogateState {
    int substeps = 0;
    float rate_scale = 0.f, threshold = 0.f;
    // input channel 0: 0 = the field p / b; 1 = the change of one plain substep, (L(p) - p) / m with
    // m = its largest magnitude inside the shell, and the output scaled by m instead of b
    int input_kind = 0;
    float* p0 = nullptr;        // field before the step (pitched), delta input
    uint8_t* w[kLayers] = {};   // packed weight images
    float* bias[kLayers] = {};  // padded to the layer's NOUT
    uint4* in = nullptr;        // 2 planes
    uint4* h = nullptr;         // 4 planes
    uint4* t = nullptr;         // 4 planes
    float* ph = nullptr;        // surrogate output field (pitched)
    float* backup = nullptr;    // field before the step (pitched)
    unsigned* dmax = nullptr;   // judge scratch
    unsigned* hmax = nullptr;   // pinned host copy
    PlaneMaps map_in, map_h, map_t;
    struct TrainState* train = nullptr;
};

void surrogate_free(gell_ctx* c) {
    for (auto*& s : c->sur) {
        if (!s) continue;
        for (int l = 0; l < kLayers; ++l) {
            if (s->w[l]) cudaFree(s->w[l]);
            if (s->bias[l]) cudaFree(s->bias[l]);
        }
        for (void* p : {(void*)s->in, (void*)s->h, (void*)s->t, (void*)s->ph, (void*)s->backup, (void*)s->dmax,
                        (void*)s->p0})
            if (p) cudaFree(p);
        if (s->hmax) cudaFreeHost(s->hmax);
        if (TrainState* t = s->train) {
            for (void* p : {(void*)t->master, (void*)t->grad, (void*)t->m, (void*)t->v, (void*)t->partial,
                            (void*)t->zero_bias, (void*)t->scal, (void*)t->gh, (void*)t->gu, (void*)t->gd, (void*)t->tgt})
                if (p) cudaFree(p);
            for (auto* p : t->wt) if (p) cudaFree(p);
            for (auto* p : t->hb) if (p) cudaFree(p);
            for (auto* p : t->tb) if (p) cudaFree(p);
            if (t->hloss) cudaFreeHost(t->hloss);
            delete t;
        }
        delete s;
        s = nullptr;
    }
}

static gell_status plane_map(gell_ctx* c, PlaneMaps* m, void* base, int planes) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        cudaDriverEntryPointQueryResult q;
        void* fn = nullptr;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn)
            return fail(c, GELL_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
        encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    const cuuint64_t N = (cuuint64_t)c->g.N;
    // half voxels (8 bytes) as elements: a run of 128 voxels is one row of a box, 256 elements
    const cuuint64_t dims[4] = {2 * N, N, N, (cuuint64_t)planes};
    const cuuint64_t strides[3] = {16 * N, 16 * N * N, 16 * N * N * N};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    CUresult r = CUDA_SUCCESS;
    for (int k = 0; k < 3 && r == CUDA_SUCCESS; ++k) {
        const cuuint32_t box[4] = {k == 1 ? 4u : 2u * kTileM, 1, 1, k == 2 ? (cuuint32_t)planes : 1u};
        r = encode(k == 0 ? &m->run : k == 1 ? &m->tail : &m->all, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, base, dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (r != CUDA_SUCCESS) return fail(c, GELL_ERR_CUDA, "cuTensorMapEncodeTiled (planes) failed (" + std::to_string((int)r) + ")");
    return GELL_OK;
}

// Pack one layer's fp32 weights W[cout][cin][3][3][3] (PyTorch conv3d order, kz kz ky kx = dz dy dx
// + 1) into the shared-memory image: block (dy, dx, half) holds [kc][2 - dz][n][8] with input channel
// 16*half + 8*kc + e and output channel n; padding channels are zero.
static void pack_layer(const float* W, const LayerShape& s, std::vector<uint16_t>& img) {
    const int halves = s.cin8 / 2;
    img.assign((size_t)27 * halves * 2 * s.nout * 8, 0);
    auto bf = [](float f) {
        uint32_t u;
        std::memcpy(&u, &f, 4);
        if ((u & 0x7fffffffu) > 0x7f800000u) return (uint16_t)0x7fc0u;
        u += 0x7fffu + ((u >> 16) & 1u);  // round to nearest even
        return (uint16_t)(u >> 16);
    };
    for (int tap = 0; tap < 27; ++tap)
        for (int h = 0; h < halves; ++h)
            for (int kc = 0; kc < 2; ++kc)
                for (int n = 0; n < s.nout; ++n)
                    for (int e = 0; e < 8; ++e) {
                        const int ci = 16 * h + 8 * kc + e;
                        float v = 0.f;
                        if (n < s.cout && ci < s.cin) v = W[((size_t)n * s.cin + ci) * 27 + tap];
                        img[(((((size_t)(tap % 9) * halves + h) * 2 + kc) * 3 + 2 - tap / 9) * s.nout + n) * 8 + e] = bf(v);
                    }
}

// Lines per unit: as many as possible (a unit loads two row groups more than it has lines), but few enough
// that the units fill the last round of CTAs; the cost of a round is its lines plus those two groups.
// The last unit along z can be of any length from one line on.
static int unit_lines(int N, int sms) {
    int best = kUnitZ;
    long long cost = -1;
    for (int y = kUnitZ; y >= 4; --y) {
        const long long units = (long long)((N + kTileM - 1) / kTileM) * ((N + y - 1) / y) * N, rounds = (units + sms - 1) / sms;
        if (cost < 0 || rounds * (y + 2) < cost) {
            cost = rounds * (y + 2);
            best = y;
        }
    }
    return best;
}

// Lines per unit and CTAs of a k_conv3 or k_wgrad launch (or what gell_debug_conv_units asks for).
struct UnitPlan {
    int tiles_x, unit_z, grid;
};
static gell_status unit_plan(gell_ctx* c, UnitPlan* p) {
    const int N = c->g.N;
    int sms = 0;
    GELL_CUDA(c, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
    p->tiles_x = (N + kTileM - 1) / kTileM;
    p->unit_z = c->conv_unit_lines > 0 ? c->conv_unit_lines : unit_lines(N, sms);
    const long long units = (long long)p->tiles_x * ((N + p->unit_z - 1) / p->unit_z) * N;
    const int most = c->conv_ctas > 0 && c->conv_ctas < sms ? c->conv_ctas : sms;
    p->grid = (int)(units < most ? units : most);
    return GELL_OK;
}

template <int CIN8, int NOUT, int MODE>
static gell_status launch_conv(gell_ctx* c, const char* name, const PlaneMaps& in, const uint8_t* w, const float* bias,
                               uint4* out, const uint4* res, const uint4* aux, float* fout, const float* fin, float scale,
                               float bval) {
    using L = ConvSmem<CIN8, NOUT>;
    // the shared-memory opt-in is a per-device attribute; setting it is cheap, so every launch does
    GELL_CUDA(c, cudaFuncSetAttribute(k_conv3<CIN8, NOUT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes));
    ConvArgs a{};
    a.in = in;
    a.w = w;
    a.bias = bias;
    a.out = out;
    a.res = res;
    a.aux = aux;
    a.field_out = fout;
    a.field_in = fin;
    a.N = c->g.N;
    a.P = c->g.P;
    a.PN = c->g.PN;
    a.nvox = c->nvox;
    a.scale = scale;
    a.bval = bval;
    a.err = c->dev_err;
    UnitPlan plan{};
    if (gell_status st = unit_plan(c, &plan)) return st;
    a.tiles_x = plan.tiles_x;
    a.unit_z = plan.unit_z;
    GELL_KERNEL(c, name, (k_conv3<CIN8, NOUT, MODE><<<plan.grid, kConvThreads, L::kBytes, c->stream>>>(a)));
    return GELL_OK;
}

// The input packing and the first `layers` convolutions of one inference of substrate `sub`:
//   layer 0        h  = relu(conv_in(input))
//   layer 2k+1     t  = relu(conv_a(h))          (k = 0..3)
//   layer 2k+2     h += conv_b(t)
//   layer 9        S->ph = p + b * conv_out(h) inside the shell, b on it
// The delta form's input planes: one plain substep from the field p0 (kept in S->p0), the largest
// change m inside the shell (read back to the host), the planes packed from (L(p0) - p0) / m, and
// the field put back to p0.  *m_out = m.
static gell_status delta_input(gell_ctx* c, int sub, SurrogateState* S, float* m_out) {
    Substrate& Su = c->subs[sub];
    const size_t fb = (size_t)c->nvox_p * 4;
    GELL_CUDA(c, cudaMemcpyAsync(S->p0, Su.p, fb, cudaMemcpyDeviceToDevice, c->stream));
    gell_status st = lod_solver(c, sub, 1);
    if (st != GELL_OK) return st;
    GELL_CUDA(c, cudaMemsetAsync(S->dmax, 0, 4, c->stream));
    GELL_KERNEL(c, "k_absdiff_max", (k_absdiff_max<<<148 * 8, 256, 0, c->stream>>>(Su.p, S->p0, c->g, S->dmax)));
    GELL_CUDA(c, cudaMemcpyAsync(S->hmax, S->dmax, 4, cudaMemcpyDeviceToHost, c->stream));
    GELL_CUDA(c, cudaStreamSynchronize(c->stream));
    float m;
    std::memcpy(&m, S->hmax, 4);
    const int pb = blocks_for(c->nvox, 256);
    GELL_KERNEL(c, "k_pack_input",
                (k_pack_input_delta<<<pb < 148 * 16 ? pb : 148 * 16, 256, 0, c->stream>>>(
                    Su.p, S->p0, Su.rate, c->g, m > 0.f ? 1.f / m : 0.f, S->rate_scale, S->in)));
    GELL_CUDA(c, cudaMemcpyAsync(Su.p, S->p0, fb, cudaMemcpyDeviceToDevice, c->stream));
    *m_out = m;
    return GELL_OK;
}

static gell_status run_layers(gell_ctx* c, int sub, SurrogateState* S, int layers) {
    Substrate& Su = c->subs[sub];
    const float b = Su.s.boundary;
    const int pb = blocks_for(c->nvox, 256);
    float scale = b;  // the output's scale: b, or m in the delta form
    if (S->input_kind == 1) {
        if (gell_status sd = delta_input(c, sub, S, &scale)) return sd;
    } else {
        GELL_KERNEL(c, "k_pack_input",
                    (k_pack_input<<<pb < 148 * 16 ? pb : 148 * 16, 256, 0, c->stream>>>(Su.p, Su.rate, c->g, 1.f / b,
                                                                                     S->rate_scale, S->in)));
    }
    gell_status st = GELL_OK;
    for (int l = 0; l < layers && st == GELL_OK; ++l) {
        const uint8_t* w = S->w[l];
        const float* bi = S->bias[l];
        if (l == 0)
            st = launch_conv<2, 32, kRelu>(c, "k_conv3_in", S->map_in, w, bi, S->h, nullptr, nullptr, nullptr, nullptr, 0.f, 0.f);
        else if (l == kLayers - 1)
            st = launch_conv<4, 32, kField>(c, "k_conv3_out", S->map_h, w, bi, nullptr, nullptr, nullptr, S->ph, Su.p, scale, b);
        else if (l & 1)
            st = launch_conv<4, 32, kRelu>(c, "k_conv3_hidden", S->map_h, w, bi, S->t, nullptr, nullptr, nullptr, nullptr, 0.f, 0.f);
        else
            st = launch_conv<4, 32, kResidual>(c, "k_conv3_hidden", S->map_t, w, bi, S->h, S->h, nullptr, nullptr, nullptr, 0.f, 0.f);
    }
    return st;
}
static gell_status infer(gell_ctx* c, int sub, SurrogateState* S) { return run_layers(c, sub, S, kLayers); }

// Input planes of the data-gradient convolution of layer l (the layer's outputs, padded to 16 channels).
static int dgrad_cin8(int l) { return kShape[l].cout <= 16 ? 2 : 4; }

static gell_status repack(gell_ctx* c, SurrogateState* S) {
    TrainState* T = S->train;
    PackArgs a{};
    int n = 0;
    for (int l = 0; l < kLayers; ++l) {
        const LayerShape& sh = kShape[l];
        const float* W = T->master + T->off_w[l];
        a.job[n++] = PackJob{W, sh.cin, sh.cout, sh.cin8, sh.nout, 0, (__nv_bfloat16*)S->w[l], S->bias[l]};
        if (l >= 1) a.job[n++] = PackJob{W, sh.cin, sh.cout, dgrad_cin8(l), kHidden, 1, (__nv_bfloat16*)T->wt[l], nullptr};
    }
    GELL_KERNEL(c, "k_pack_w", (k_pack_w<<<dim3(16, n), 256, 0, c->stream>>>(a)));
    return GELL_OK;
}

template <int BP>
static gell_status launch_wgrad(gell_ctx* c, TrainState* T, const LayerShape& sh, const PlaneMaps& A, const PlaneMaps& B,
                                bool gradient_a, float* out) {
    using L = WgradSmem<BP>;
    WgradArgs a{};
    a.a = A.all;
    a.b = B.all;
    a.partial = T->partial;
    a.N = c->g.N;
    a.err = c->dev_err;
    UnitPlan plan{};
    if (gell_status st = unit_plan(c, &plan)) return st;
    a.tiles_x = plan.tiles_x;
    a.unit_z = plan.unit_z;
    const int grid = plan.grid < kWgCtas ? plan.grid : kWgCtas;
    GELL_CUDA(c, cudaFuncSetAttribute(k_wgrad<BP>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes));
    GELL_KERNEL(c, BP == 2 ? "k_wgrad_thin" : "k_wgrad", (k_wgrad<BP><<<grid, kWgThreads, L::kBytes, c->stream>>>(a)));
    const int n = 27 * 256 * BP;
    GELL_KERNEL(c, "k_sum_partials", (k_sum_wgrad<<<n / 32, 256, 0, c->stream>>>(T->partial, grid, 8 * BP, sh.cout, sh.cin, gradient_a, out)));
    return GELL_OK;
}

// Weight gradient of layer l into T->grad (the layer's block); bias gradient = per-channel sums of G.
static gell_status wgrad_layer(gell_ctx* c, SurrogateState* S, int l, const PlaneMaps& x, const PlaneMaps& g, const uint4* G) {
    TrainState* T = S->train;
    const LayerShape& sh = kShape[l];
    float* out = T->grad + T->off_w[l];
    const gell_status st = l == 0           ? launch_wgrad<2>(c, T, sh, g, x, true, out)
                           : l == kLayers - 1 ? launch_wgrad<2>(c, T, sh, x, g, false, out)
                                              : launch_wgrad<4>(c, T, sh, x, g, false, out);
    if (st != GELL_OK) return st;
    const int planes = (sh.cout + 7) / 8, blocks = 148 * 4;
    GELL_KERNEL(c, "k_channel_sums", (k_channel_sums<<<blocks, 256, 0, c->stream>>>(G, planes, c->nvox, T->partial)));
    GELL_KERNEL(c, "k_sum_partials", (k_sum_partials<<<1, 256, 0, c->stream>>>(T->partial, blocks, sh.cout, 8 * planes, T->grad + T->off_b[l])));
    return GELL_OK;
}

// One training pair: the plain solver advances the field by the operator's substeps (the target),
// the operator runs from the field before them with every activation kept, the loss gradient goes
// back through the ten layers (data gradients on tcgen05, weight gradients as above), Adam updates
// the master weights, the images are repacked, and the field is left at the target.
static gell_status train_pair(gell_ctx* c, int sub, SurrogateState* S, float lr, float* loss_out) {
    TrainState* T = S->train;
    Substrate& Su = c->subs[sub];
    const float b = Su.s.boundary;
    const size_t fb = (size_t)c->nvox_p * 4;
    GELL_CUDA(c, cudaMemcpyAsync(S->backup, Su.p, fb, cudaMemcpyDeviceToDevice, c->stream));
    // delta form: the input planes from one plain substep first (the field is put back), the output
    // and the loss in units of m, the substep's largest change (a fixed point, m = 0, has q = p = y)
    float scale = b, loss_unit = b;
    gell_status st = GELL_OK;
    if (S->input_kind == 1) {
        if ((st = delta_input(c, sub, S, &scale)) != GELL_OK) return st;
        loss_unit = scale > 0.f ? scale : b;
    }
    st = lod_solver(c, sub, S->substeps);
    if (st != GELL_OK) return st;
    GELL_CUDA(c, cudaMemcpyAsync(T->tgt, Su.p, fb, cudaMemcpyDeviceToDevice, c->stream));
    GELL_CUDA(c, cudaMemcpyAsync(Su.p, S->backup, fb, cudaMemcpyDeviceToDevice, c->stream));

    // forward, every activation kept
    const int pb = blocks_for(c->nvox, 256);
    if (S->input_kind == 0)
        GELL_KERNEL(c, "k_pack_input", (k_pack_input<<<pb < 148 * 16 ? pb : 148 * 16, 256, 0, c->stream>>>(
                                            Su.p, Su.rate, c->g, 1.f / b, S->rate_scale, S->in)));
    st = launch_conv<2, 32, kRelu>(c, "k_conv3_in", S->map_in, S->w[0], S->bias[0], T->hb[0], nullptr, nullptr, nullptr,
                                   nullptr, 0.f, 0.f);
    for (int k = 0; k < 4 && st == GELL_OK; ++k) {
        st = launch_conv<4, 32, kRelu>(c, "k_conv3_hidden", T->mh[k], S->w[2 * k + 1], S->bias[2 * k + 1], T->tb[k],
                                       nullptr, nullptr, nullptr, nullptr, 0.f, 0.f);
        if (st == GELL_OK)
            st = launch_conv<4, 32, kResidual>(c, "k_conv3_hidden", T->mt[k], S->w[2 * k + 2], S->bias[2 * k + 2],
                                               T->hb[k + 1], T->hb[k], nullptr, nullptr, nullptr, 0.f, 0.f);
    }
    if (st == GELL_OK)
        st = launch_conv<4, 32, kField>(c, "k_conv3_out", T->mh[4], S->w[9], S->bias[9], nullptr, nullptr, nullptr, S->ph,
                                        Su.p, scale, b);
    if (st != GELL_OK) return st;

    // loss and its gradient
    const long long inner = (long long)(c->g.N - 4) * (c->g.N - 4) * (c->g.N - 4);
    const int lb = 148 * 8;
    GELL_KERNEL(c, "k_loss_grad", (k_loss_grad<<<lb, 256, 0, c->stream>>>(S->ph, T->tgt, c->g, loss_unit, 1.f / (float)inner, T->gd,
                                                                          T->scal + 2)));
    GELL_KERNEL(c, "k_sum_partials", (k_sum_partials<<<1, 256, 0, c->stream>>>(T->scal + 2, lb, 1, 1, T->scal + 1)));

    // backward
    if ((st = wgrad_layer(c, S, 9, T->mh[4], T->mgd, T->gd)) != GELL_OK) return st;
    st = launch_conv<2, 32, kLinear>(c, "k_conv3_dgrad", T->mgd, T->wt[9], T->zero_bias, T->gh, nullptr, nullptr, nullptr,
                                     nullptr, 0.f, 0.f);
    for (int k = 3; k >= 0 && st == GELL_OK; --k) {
        if ((st = wgrad_layer(c, S, 2 * k + 2, T->mt[k], T->mgh, T->gh)) != GELL_OK) return st;
        st = launch_conv<4, 32, kMask>(c, "k_conv3_dgrad", T->mgh, T->wt[2 * k + 2], T->zero_bias, T->gu, nullptr,
                                       T->tb[k], nullptr, nullptr, 0.f, 0.f);
        if (st != GELL_OK) return st;
        if ((st = wgrad_layer(c, S, 2 * k + 1, T->mh[k], T->mgu, T->gu)) != GELL_OK) return st;
        if (k > 0)
            st = launch_conv<4, 32, kResidual>(c, "k_conv3_dgrad", T->mgu, T->wt[2 * k + 1], T->zero_bias, T->gh, T->gh,
                                               nullptr, nullptr, nullptr, 0.f, 0.f);
        else
            st = launch_conv<4, 32, kResMask>(c, "k_conv3_dgrad", T->mgu, T->wt[1], T->zero_bias, T->gh, T->gh, T->hb[0],
                                              nullptr, nullptr, 0.f, 0.f);
    }
    if (st != GELL_OK) return st;
    if ((st = wgrad_layer(c, S, 0, S->map_in, T->mgh, T->gh)) != GELL_OK) return st;

    // Adam on the clipped gradient, new images
    GELL_KERNEL(c, "k_sumsq", (k_sumsq<<<1, 1024, 0, c->stream>>>(T->grad, T->count, T->scal)));
    T->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float bc1 = 1.f - powf(b1, (float)T->step), bc2 = 1.f - powf(b2, (float)T->step);
    GELL_KERNEL(c, "k_adam", (k_adam<<<64, 256, 0, c->stream>>>(T->master, T->grad, T->m, T->v, T->count, T->scal, 1.f, lr,
                                                                b1, b2, 1e-8f, bc1, bc2)));
    if ((st = repack(c, S)) != GELL_OK) return st;
    GELL_CUDA(c, cudaMemcpyAsync(Su.p, T->tgt, fb, cudaMemcpyDeviceToDevice, c->stream));
    if (loss_out) {
        GELL_CUDA(c, cudaMemcpyAsync(T->hloss, T->scal + 1, 4, cudaMemcpyDeviceToHost, c->stream));
        GELL_CUDA(c, cudaStreamSynchronize(c->stream));
        *loss_out = *T->hloss / (float)inner;
    }
    return GELL_OK;
}

}  // namespace gell

using namespace gell;

static long long weight_count() {
    long long n = 0;
    for (const auto& s : kShape) n += (long long)s.cout * s.cin * 27 + s.cout;
    return n;
}

extern "C" {

long long gell_surrogate_weight_count(void) { return weight_count(); }

gell_status gell_surrogate_load(gell_ctx* c, int sub, const float* weights, long long count, int substeps,
                                float rate_scale, float threshold) {
    GELL_RANGE("gell_surrogate_load");
    if (!c || !weights || sub < 0 || sub >= (int)c->subs.size() || substeps < 1) return GELL_ERR_INVALID_ARG;
    if (count != weight_count()) return fail(c, GELL_ERR_INVALID_ARG, "surrogate weight count does not match the operator");
    if (!(c->subs[sub].s.boundary != 0.f)) return fail(c, GELL_ERR_UNSUPPORTED, "the surrogate scales by the boundary value, which is 0");
    if (c->g.N < 8 || c->g.N > 1023) return fail(c, GELL_ERR_UNSUPPORTED, "grid edge outside the surrogate's range");
    SurrogateState* S = c->sur[sub];  // reloading keeps the buffers and replaces the weights
    const bool fresh = S == nullptr;
    if (fresh) S = new SurrogateState();
    S->substeps = substeps;
    S->rate_scale = rate_scale;
    S->threshold = threshold;
    S->input_kind = c->sur_input;
    const float* W = weights;
    for (int l = 0; l < kLayers; ++l) {
        const LayerShape& s = kShape[l];
        std::vector<uint16_t> img;
        pack_layer(W, s, img);
        W += (size_t)s.cout * s.cin * 27;
        std::vector<float> bias(s.nout, 0.f);
        for (int n = 0; n < s.cout; ++n) bias[n] = W[n];
        W += s.cout;
        if (!S->w[l]) {
            c->sur[sub] = S;  // owned by the context from here on (freed with it)
            if (cudaMalloc(&S->w[l], img.size() * 2) != cudaSuccess || cudaMalloc(&S->bias[l], bias.size() * 4) != cudaSuccess)
                return fail(c, GELL_ERR_ALLOC, "surrogate weights");
        }
        // copies on the context's stream (a non-blocking stream: a plain cudaMemcpy would not be
        // ordered before the kernels that read these buffers), finished before the vectors go away
        GELL_CUDA(c, cudaMemcpyAsync(S->w[l], img.data(), img.size() * 2, cudaMemcpyHostToDevice, c->stream));
        GELL_CUDA(c, cudaMemcpyAsync(S->bias[l], bias.data(), bias.size() * 4, cudaMemcpyHostToDevice, c->stream));
        GELL_CUDA(c, cudaStreamSynchronize(c->stream));
    }
    c->sur[sub] = S;
    if (fresh) {
        const size_t plane = (size_t)c->nvox * 16, field = (size_t)c->nvox_p * 4;
        if (cudaMalloc(&S->in, 2 * plane) != cudaSuccess || cudaMalloc(&S->h, 4 * plane) != cudaSuccess ||
            cudaMalloc(&S->t, 4 * plane) != cudaSuccess || cudaMalloc(&S->ph, field) != cudaSuccess ||
            cudaMalloc(&S->backup, field) != cudaSuccess || cudaMalloc(&S->dmax, 4) != cudaSuccess ||
            cudaMallocHost(&S->hmax, 4) != cudaSuccess)
            return fail(c, GELL_ERR_ALLOC, "surrogate activations (10 planes of 16 bytes per voxel)");
        GELL_CUDA(c, cudaMemsetAsync(S->in, 0, 2 * plane, c->stream));
        gell_status st = GELL_OK;
        if (cudaMalloc(&S->p0, field) != cudaSuccess) return fail(c, GELL_ERR_ALLOC, "surrogate field copy");
        st = plane_map(c, &S->map_in, S->in, 2);
        if (st == GELL_OK) st = plane_map(c, &S->map_h, S->h, 4);
        if (st == GELL_OK) st = plane_map(c, &S->map_t, S->t, 4);
        if (st != GELL_OK) return st;
    }
    return GELL_OK;
}

gell_status gell_surrogate_infer(gell_ctx* c, int sub) {
    GELL_RANGE("gell_surrogate_infer");
    if (!c || sub < 0 || sub >= (int)c->subs.size()) return GELL_ERR_INVALID_ARG;
    SurrogateState* S = c->sur[sub];
    if (!S) return fail(c, GELL_ERR_INVALID_ARG, "no surrogate loaded for this substrate");
    gell_status st = infer(c, sub, S);
    if (st != GELL_OK) return st;
    GELL_CUDA(c, cudaMemcpyAsync(c->subs[sub].p, S->ph, (size_t)c->nvox_p * 4, cudaMemcpyDeviceToDevice, c->stream));
    return GELL_OK;
}

gell_status gell_lod_surrogate(gell_ctx* c, int sub, int* accepted, float* residual) {
    GELL_RANGE("gell_lod_surrogate");
    if (!c || sub < 0 || sub >= (int)c->subs.size()) return GELL_ERR_INVALID_ARG;
    SurrogateState* S = c->sur[sub];
    if (!S) return fail(c, GELL_ERR_INVALID_ARG, "no surrogate loaded for this substrate");
    Substrate& Su = c->subs[sub];
    const size_t fb = (size_t)c->nvox_p * 4;
    GELL_CUDA(c, cudaMemcpyAsync(S->backup, Su.p, fb, cudaMemcpyDeviceToDevice, c->stream));
    gell_status st = infer(c, sub, S);
    if (st != GELL_OK) return st;
    // judge: one plain substep from the surrogate's field; a field on the solver's trajectory moves
    // little in one substep
    GELL_CUDA(c, cudaMemcpyAsync(Su.p, S->ph, fb, cudaMemcpyDeviceToDevice, c->stream));
    st = lod_solver(c, sub, 1);
    if (st != GELL_OK) return st;
    GELL_CUDA(c, cudaMemsetAsync(S->dmax, 0, 4, c->stream));
    GELL_KERNEL(c, "k_absdiff_max", (k_absdiff_max<<<148 * 8, 256, 0, c->stream>>>(Su.p, S->ph, c->g, S->dmax)));
    GELL_CUDA(c, cudaMemcpyAsync(S->hmax, S->dmax, 4, cudaMemcpyDeviceToHost, c->stream));
    GELL_CUDA(c, cudaStreamSynchronize(c->stream));
    float r;
    std::memcpy(&r, S->hmax, 4);
    r /= Su.s.boundary;
    if (residual) *residual = r;
    const bool ok = r <= S->threshold;
    if (accepted) *accepted = ok ? 1 : 0;
    if (ok) {
        GELL_CUDA(c, cudaMemcpyAsync(Su.p, S->ph, fb, cudaMemcpyDeviceToDevice, c->stream));
        return GELL_OK;
    }
    GELL_CUDA(c, cudaMemcpyAsync(Su.p, S->backup, fb, cudaMemcpyDeviceToDevice, c->stream));
    return lod_solver(c, sub, S->substeps);
}

gell_status gell_surrogate_train_init(gell_ctx* c, int sub, const float* weights, long long count, int substeps,
                                      float rate_scale) {
    GELL_RANGE("gell_surrogate_train_init");
    gell_status st = gell_surrogate_load(c, sub, weights, count, substeps, rate_scale, 0.f);
    if (st != GELL_OK) return st;
    SurrogateState* S = c->sur[sub];
    if (!S->train) {
        TrainState* T = new TrainState();
        S->train = T;
        T->count = count;
        long long off = 0;
        for (int l = 0; l < kLayers; ++l) {
            T->off_w[l] = off;
            off += (long long)kShape[l].cout * kShape[l].cin * 27;
            T->off_b[l] = off;
            off += kShape[l].cout;
        }
        const size_t plane = (size_t)c->nvox * 16, field = (size_t)c->nvox_p * 4;
        T->partial_n = (long long)kWgCtas * kWgPart;
        bool ok = cudaMalloc(&T->master, count * 4) == cudaSuccess && cudaMalloc(&T->grad, count * 4) == cudaSuccess &&
                  cudaMalloc(&T->m, count * 4) == cudaSuccess && cudaMalloc(&T->v, count * 4) == cudaSuccess &&
                  cudaMalloc(&T->partial, T->partial_n * 4) == cudaSuccess &&
                  cudaMalloc(&T->zero_bias, 32 * 4) == cudaSuccess &&
                  cudaMalloc(&T->scal, (2 + 148 * 8) * 4) == cudaSuccess && cudaMallocHost(&T->hloss, 4) == cudaSuccess &&
                  cudaMalloc(&T->gh, 4 * plane) == cudaSuccess && cudaMalloc(&T->gu, 4 * plane) == cudaSuccess &&
                  cudaMalloc(&T->gd, 2 * plane) == cudaSuccess && cudaMalloc(&T->tgt, field) == cudaSuccess;
        for (int k = 0; ok && k < 5; ++k) ok = cudaMalloc(&T->hb[k], 4 * plane) == cudaSuccess;
        for (int k = 0; ok && k < 4; ++k) ok = cudaMalloc(&T->tb[k], 4 * plane) == cudaSuccess;
        for (int l = 1; ok && l < kLayers; ++l)
            ok = cudaMalloc(&T->wt[l], (size_t)27 * (dgrad_cin8(l) / 2) * 2 * kHidden * 8 * 2) == cudaSuccess;
        if (!ok) return fail(c, GELL_ERR_ALLOC, "surrogate training buffers (46 planes of 16 bytes per voxel)");
        GELL_CUDA(c, cudaMemsetAsync(T->zero_bias, 0, 32 * 4, c->stream));
        GELL_CUDA(c, cudaMemsetAsync(T->gd, 0, 2 * plane, c->stream));
        for (int k = 0; k < 5 && st == GELL_OK; ++k) st = plane_map(c, &T->mh[k], T->hb[k], 4);
        for (int k = 0; k < 4 && st == GELL_OK; ++k) st = plane_map(c, &T->mt[k], T->tb[k], 4);
        if (st == GELL_OK) st = plane_map(c, &T->mgd, T->gd, 2);
        if (st == GELL_OK) st = plane_map(c, &T->mgh, T->gh, 4);
        if (st == GELL_OK) st = plane_map(c, &T->mgu, T->gu, 4);
        if (st != GELL_OK) return st;
    }
    TrainState* T = S->train;
    T->step = 0;
    GELL_CUDA(c, cudaMemcpyAsync(T->master, weights, count * 4, cudaMemcpyHostToDevice, c->stream));
    GELL_CUDA(c, cudaMemsetAsync(T->m, 0, count * 4, c->stream));
    GELL_CUDA(c, cudaMemsetAsync(T->v, 0, count * 4, c->stream));
    if ((st = repack(c, S)) != GELL_OK) return st;
    GELL_CUDA(c, cudaStreamSynchronize(c->stream));  // `weights` may go away after the return
    return GELL_OK;
}

gell_status gell_surrogate_train_pair(gell_ctx* c, int sub, float lr, float* loss) {
    GELL_RANGE("gell_surrogate_train_pair");
    if (!c || sub < 0 || sub >= (int)c->subs.size() || !c->sur[sub] || !c->sur[sub]->train) return GELL_ERR_INVALID_ARG;
    return train_pair(c, sub, c->sur[sub], lr, loss);
}

gell_status gell_surrogate_train_read(gell_ctx* c, int sub, int which, float* host, long long count) {
    if (!c || !host || sub < 0 || sub >= (int)c->subs.size() || !c->sur[sub] || !c->sur[sub]->train)
        return GELL_ERR_INVALID_ARG;
    TrainState* T = c->sur[sub]->train;
    if (which == 2) {
        if (count != c->nvox_p) return GELL_ERR_INVALID_ARG;
        GELL_CUDA(c, cudaMemcpyAsync(host, T->tgt, (size_t)count * 4, cudaMemcpyDeviceToHost, c->stream));
    } else {
        if (count != T->count || (which != 0 && which != 1)) return GELL_ERR_INVALID_ARG;
        GELL_CUDA(c, cudaMemcpyAsync(host, which == 0 ? T->master : T->grad, (size_t)count * 4, cudaMemcpyDeviceToHost,
                                     c->stream));
    }
    GELL_CUDA(c, cudaStreamSynchronize(c->stream));
    return GELL_OK;
}

gell_status gell_surrogate_run_layers(gell_ctx* c, int sub, int layers) {
    if (!c || sub < 0 || sub >= (int)c->subs.size() || layers < 0 || layers > kLayers) return GELL_ERR_INVALID_ARG;
    SurrogateState* S = c->sur[sub];
    if (!S) return fail(c, GELL_ERR_INVALID_ARG, "no surrogate loaded for this substrate");
    return run_layers(c, sub, S, layers);
}

gell_status gell_debug_conv_units(gell_ctx* c, int lines, int ctas) {
    if (!c) return GELL_ERR_INVALID_ARG;
    if (lines < 0 || lines > kUnitZ || ctas < 0) return fail(c, GELL_ERR_INVALID_ARG, "convolution units outside 0..16 lines");
    c->conv_unit_lines = lines;
    c->conv_ctas = ctas;
    return GELL_OK;
}

gell_status gell_surrogate_read(gell_ctx* c, int sub, int which, void* host, long long bytes) {
    if (!c || !host || sub < 0 || sub >= (int)c->subs.size() || !c->sur[sub]) return GELL_ERR_INVALID_ARG;
    SurrogateState* S = c->sur[sub];
    const long long plane = c->nvox * 16;
    const void* src = which == 0 ? (const void*)S->in : which == 1 ? (const void*)S->h : which == 2 ? (const void*)S->t
                    : which == 3 ? (const void*)S->ph : nullptr;
    const long long need = which == 0 ? 2 * plane : which == 3 ? c->nvox_p * 4 : 4 * plane;
    if (!src || bytes != need) return GELL_ERR_INVALID_ARG;
    GELL_CUDA(c, cudaMemcpyAsync(host, src, (size_t)bytes, cudaMemcpyDeviceToHost, c->stream));
    GELL_CUDA(c, cudaStreamSynchronize(c->stream));
    return GELL_OK;
}

}  // extern "C"
