// sf_conv_tc.cuh -- 3x3x3 convolution forward on the 5th-generation tensor cores (tcgen05 + TMA, sm_103a).
//
// Implicit GEMM per CTA: MT tiles of M = 128 output voxels (a 32 (z) x 4 MT (y) x 1 (x) brick), N = Cout,
// K = 27 taps x Cin.  Operands are staged by TMA in the no-swizzle K-major "core matrix" layout: one 4-D box of
// 8 channels x (32 x 4 MT x 1) voxels per 8-channel chunk and tap lands as 128 MT rows x 16 B, i.e. 8-row x 16-B
// core matrices with a 128-B stride along M, one tile per 2 KB and one (2 MT)-KB chunk per 8 channels along K;
// taps outside the grid are filled with zeros by the TMA unit (the convolution's zero padding).  Weights
// [tap][Cout][Cin] are staged the same way, once per tap for all MT tiles.  Lane 0 of warp 1 issues the TMA loads
// and lane 0 of warp 0 the tcgen05.mma (M=128, N=Cout, K=16, BF16 in, FP32 accumulate in TMEM, one accumulator of
// Cout columns per tile) through a ring of stages guarded by mbarriers; all four warps read the accumulators back
// with tcgen05.ld and apply bias + ReLU + BF16 conversion.  Every wait is bounded: on timeout the CTA records an error code and
// returns after releasing its tensor memory.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "sf_internal.cuh"
#include "sf_tma.cuh"

namespace sf {
namespace tc {

constexpr int kMaxStages = 4;
// Shared-memory matrix descriptor, no swizzle, K-major: start, leading (K) and stride (M/N) byte offsets in
// 16-byte units, descriptor version 1 (bits 46..48 = 0b001), swizzle mode 0.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// The same descriptor for the 32-byte swizzled K-major layout (layout type 6): rows of 32 bytes (16 BF16 along K)
// whose two 16-byte halves swap in rows 4-7 of every 8-row, 256-byte atom, as TMA writes them with
// CU_TENSOR_MAP_SWIZZLE_32B; the stride (M/N) byte offset is the 256-byte atom, the leading offset is unused.
__device__ __forceinline__ uint64_t smem_desc_sw32(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(256u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)6 << 61;
    return d;
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M = m (128 or 64), N = n.
__host__ __device__ constexpr uint32_t instr_desc_bf16(int n, int m = 128) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

template <int N>
__device__ __forceinline__ void tmem_ld_x16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = __uint_as_float(r[q]);
}

constexpr int kTileZ = 32, kTileY = 4;

// M tiles per CTA: four (the weights of a tap staged once for 512 voxels), two for 64 input channels, whose
// stages are twice as large
template <int CI, int CO>
constexpr int tiles_per_cta() {
    return CI == 64 ? 2 : 4;
}

template <int CI, int CO, int MT>
struct Layout {
    static constexpr int kChunks = CI / 8;
    static constexpr uint32_t kChunkBytes = 128u * 16u * MT;  // 128 MT rows x 16 B per 8-channel chunk
    static constexpr uint32_t kABytes = kChunkBytes * kChunks;
    static constexpr uint32_t kBBytes = (uint32_t)CO * 16u * kChunks;
    static constexpr uint32_t kStageBytes = kABytes + kBBytes;
    // stages within about 100 KB, so that two or more CTAs share an SM where the stages are small
    static constexpr int kStages = (int)(100u * 1024u / kStageBytes) > kMaxStages ? kMaxStages
                                   : (int)(100u * 1024u / kStageBytes) < 2    ? 2
                                                                              : (int)(100u * 1024u / kStageBytes);
    // accumulator columns: one Cout-wide block per tile, allocated as a power of two >= 32
    static constexpr uint32_t kCols = (uint32_t)(MT * CO) <= 32u    ? 32u
                                      : (uint32_t)(MT * CO) <= 64u  ? 64u
                                      : (uint32_t)(MT * CO) <= 128u ? 128u
                                      : (uint32_t)(MT * CO) <= 256u ? 256u
                                                                    : 512u;
    static constexpr uint32_t kNeed = kStages * kStageBytes + 1024 /* alignment */ + 256 /* barriers */;
    // enough shared memory that at most 512 / kCols CTAs share an SM, so every CTA's TMEM allocation fits
    static constexpr uint32_t kMinSmem = 233472u / (512u / kCols + 1u) + 1024u;
    static constexpr uint32_t kSmemBytes = kNeed > kMinSmem ? kNeed : kMinSmem;
    static_assert(kSmemBytes <= 227u * 1024u, "shared memory");
    static_assert(MT * CO <= 512, "TMEM columns");
};

// err: first error code of any CTA (1 = TMA/MMA wait timed out).
// EPI 0: + bias, ReLU, BF16 out (forward).  EPI 1: FP32 out, no bias (input gradient, with the mirrored and
// transposed weights).
template <int CI, int CO, int EPI = 0, int MT = tiles_per_cta<CI, CO>()>
__global__ void __launch_bounds__(128, 1) k_conv_tc(const __grid_constant__ CUtensorMap tmap_x,
                                                    const __grid_constant__ CUtensorMap tmap_w, Dims d,
                                                    const float *__restrict__ bias, void *__restrict__ yout,
                                                    int *err) {
    static_assert(CI % 16 == 0 && CO % 16 == 0 && CO <= 256, "shape");
    using L = Layout<CI, CO, MT>;
    constexpr int kStages = L::kStages;
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte aligned stage buffers, barriers after them
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kStages * L::kStageBytes);
    // sh: [0] TMEM base, [1] status, [2] MMA side ok, [3] stages waited, [4] TMA side ok, [5] stages issued
    volatile uint32_t *sh = reinterpret_cast<volatile uint32_t *>(bars + 2 * kStages + 1);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + kStages), done = smem_u32(bars + 2 * kStages);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const int tiles_z = (d.nz + kTileZ - 1) / kTileZ, tiles_y = (d.ny + kTileY * MT - 1) / (kTileY * MT);
    const int bz = blockIdx.x % tiles_z, by = (blockIdx.x / tiles_z) % tiles_y, bx = blockIdx.x / (tiles_z * tiles_y);
    const int z0 = bz * kTileZ, y0 = by * kTileY * MT, x0 = bx;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(done, 1);
        for (int k = 1; k < 6; k++) sh[k] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<uint32_t *>(sh))),
                     "r"(L::kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh[0];

    // warp specialised: lane 0 of warp 1 issues the TMA loads of the 27 taps through the ring of stages, lane 0 of
    // warp 0 the MMAs, so a stage is refilled as soon as its MMAs complete without holding up the next MMAs
    constexpr int T = 27;
    if (warp == 1 && lane == 0) {
        bool ok = true;
        int issued = 0;
        for (int t = 0; t < T; t++) {
            const int s = t % kStages;
            if (t >= kStages && !mbar_wait(empty0 + 8 * s, (uint32_t)(t / kStages - 1) & 1u)) {
                ok = false;
                break;
            }
            const uint32_t a = smem_u32(smem + s * L::kStageBytes), b = a + L::kABytes;
            const uint32_t bar = full0 + 8 * s;
            mbar_expect_tx(bar, L::kStageBytes);
            const int dx = t / 9 - 1, dy = (t / 3) % 3 - 1, dz = t % 3 - 1;
#pragma unroll
            for (int c = 0; c < L::kChunks; c++) {
                tma_load_4d(a + c * L::kChunkBytes, &tmap_x, bar, 8 * c, z0 + dz, y0 + dy, x0 + dx);
                tma_load_3d(b + c * (uint32_t)CO * 16u, &tmap_w, bar, 8 * c, 0, t);
            }
            issued = t + 1;
        }
        sh[4] = ok ? 1u : 0u;
        sh[5] = (uint32_t)issued;
    } else if (warp == 0 && lane == 0) {
        constexpr uint32_t idesc = instr_desc_bf16(CO);
        bool ok = true;
        int waited = 0;
        for (int t = 0; t < T; t++) {
            const int s = t % kStages;
            if (!mbar_wait(full0 + 8 * s, (uint32_t)(t / kStages) & 1u)) {
                ok = false;
                break;
            }
            waited = t + 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = smem_u32(smem + s * L::kStageBytes), b = a + L::kABytes;
            // K = 16 spans two 8-channel chunks: leading (K) offset = one chunk, stride (M/N) = 8 rows; tile m's rows
            // start 2 KB further into each chunk, its accumulator CO columns further.  The descriptors are bases plus
            // compile-time offsets in 16-byte units (no carry: shared addresses stay below 256 KB).
            const uint64_t ad0 = smem_desc(a, L::kChunkBytes, 128u), bd0 = smem_desc(b, (uint32_t)CO * 16u, 128u);
            const uint32_t acc0 = t > 0 ? 1u : 0u;
#pragma unroll
            for (int j = 0; j < CI / 16; j++) {
                const uint64_t bd = bd0 + (uint64_t)(j * 2 * CO);
#pragma unroll
                for (int m = 0; m < MT; m++) {
                    const uint64_t ad = ad0 + (uint64_t)((j * 2 * L::kChunkBytes + m * 2048u) >> 4);
                    mma_bf16(tmem + (uint32_t)(m * CO), ad, bd, idesc, j > 0 ? 1u : acc0);
                }
            }
            mma_commit(empty0 + 8 * s);
        }
        if (waited > 0) {  // completion of every MMA issued (also on the error path, before TMEM is released)
            mma_commit(done);
            if (!mbar_wait(done, 0)) ok = false;
        }
        sh[2] = ok ? 1u : 0u;
        sh[3] = (uint32_t)waited;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const bool ok = sh[2] && sh[4];
        if (!ok) {  // drain loads still in flight into this CTA's shared memory (bounded)
            for (uint32_t t = sh[3]; t < sh[5]; t++) mbar_wait(full0 + 8 * (t % kStages), (t / kStages) & 1u);
            atomicCAS(err, 0, 1);
        }
        sh[1] = ok ? 1u : 0u;
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (sh[1]) {  // uniform across the CTA
#pragma unroll 1
        for (int m = 0; m < MT; m++) {
        const int r = 32 * warp + lane;  // TMEM lane = tile row
        const int z = z0 + (r % kTileZ), yy = y0 + kTileY * m + r / kTileZ;
        const bool inb = z < d.nz && yy < d.ny && x0 < d.nx;
        const long long v = inb ? cid(d, x0, yy, z) : 0;
#pragma unroll
        for (int c0 = 0; c0 < CO; c0 += 16) {
            float acc[16];
            tmem_ld_x16<16>(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(m * CO + c0), acc);
            if (inb && EPI == 0) {
                uint32_t pk[8];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const float a0 = fmaxf(acc[2 * q] + bias[c0 + 2 * q], 0.f);
                    const float a1 = fmaxf(acc[2 * q + 1] + bias[c0 + 2 * q + 1], 0.f);
                    __nv_bfloat162 h2 = __floats2bfloat162_rn(a0, a1);
                    pk[q] = *reinterpret_cast<uint32_t *>(&h2);
                }
                uint4 *dst = reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(yout) + v * CO + c0);
                dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
            } else if (inb) {
                float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(yout) + v * CO + c0);
#pragma unroll
                for (int q = 0; q < 4; q++) dst[q] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
            }
        }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::kCols) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------ z lines
// Forward (and input gradient) for Cin = 16 or 32, Cout <= 32, on grids with nz >= 128: a persistent CTA per SM
// takes bricks of 128 (z) x Y (y) x 2 (x) voxels (Y = 4, or 8 for 16 output channels where that costs less), 2 Y M tiles
// of one z line of 128 voxels each.  A pipeline stage is one z shift dz, one group of 16 channels (K = 16) and one of
// the four x planes the brick's taps reach: one TMA box, (16 channels, 128 z, Y + 2 y) from (z0 + dz, y0 - 1) of plane
// x0 - 1 + xb, lands as 32-byte rows in the 32-byte swizzled K-major layout and carries the tile rows of all its (dx, dy)
// taps: tile (yy, xx = xb - 1 - dx) of tap (dx, dy) starts 4 KB x (yy + 1 + dy) into the box, so each box is read once
// for up to six taps (the 27-box kernel above reads a box a tap, of 16-byte rows, each half of a 32-byte sector).  The 27
// taps' weights stay in shared memory, swizzled the same way and ordered (dz, dx, dy), for the CTA's whole run.
// One line of the box meets up to three tiles along y, through the taps dy = -1, 0, 1; their weights are consecutive rows
// and the accumulators stand by descending y, so one MMA of N = 3 Cout does the three: an M = 128 operand costs 4 KB of
// shared memory reads whatever N is (64 clocks as measured), and those reads bound a tap at a time.  The order of an
// accumulator's sums, (dz, channels, dx, dy), is the same.  16 to 16 channels at 256^3: 795 us a tap at a time, 626 with
// three taps an MMA (boxes of four planes, two stages: copies and MMAs half overlapped), 515 with a plane a stage and
// Y = 8, which reads 2.5 lines a voxel and z shift instead of 3.  What bounds it now is shared memory: a brick's 194 MMAs read
// 16 k clocks' worth at 64 bytes a clock, the copies write 3.8 k at 128, 19.9 k measured.
// Warp 1 lane 0 issues the TMA loads through the stages, warp 0 lane 0 the MMAs (M = 128, N up to 3 Cout, K = 16) into
// one of two TMEM accumulator sets, and warps 2-5 read the other set back (bias + ReLU + BF16, or FP32), so the epilogue
// of a brick overlaps the MMAs of the next.  Every wait is bounded; a
// timeout stops all roles, drains the copies in flight and sets the error flag.
constexpr int kLineZ = 128, kLineY = 4;

constexpr int kLineX = 2;

template <int CI, int CO, int Y>
struct LineLayout {
    static constexpr int kTiles = Y * kLineX, KP = CI / 16;  // 16-channel groups
    static constexpr uint32_t kStageBytes = kLineZ * (Y + 2) * 32u;  // one x plane of one z shift and channel group
    static constexpr uint32_t kWChunkRaw = 27u * CO * 32u;  // [tap][co] rows of 16 channels
    static constexpr uint32_t kWChunk = (kWChunkRaw + 1023u) & ~1023u;
    static constexpr uint32_t kRest = 1024u + KP * kWChunk + 256u;
    static constexpr int kStagesRaw = (int)((227u * 1024u - kRest) / kStageBytes);
    static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
    static constexpr uint32_t kCols = kTiles * CO;  // one accumulator set
    static constexpr uint32_t kAlloc = 2u * kCols <= 256u ? 256u : 512u;
    static constexpr uint32_t kNeed = kRest + kStages * kStageBytes;
    // at least 116 KB: one CTA per SM, whose TMEM columns are then always free
    static constexpr uint32_t kSmemBytes = kNeed > 116u * 1024u ? kNeed : 116u * 1024u;
    static_assert(CI % 16 == 0 && 2u * kCols <= 512u && kStages >= 3 && kSmemBytes <= 227u * 1024u, "line layout");
};

// EPI 2: as 0, and the 2x2x2 average pooling of y besides (a brick holds whole 2x2x2 cells; sums in k_pool's order).
// EPI 3 (Cout = 16): the 1x1 head applied to y, which is not stored.  256^3: pooling and head by themselves read the 537
// MB again, 92 and 87 us; in these epilogues, which run beside the next brick's MMAs, the convolutions take 514 and 474
// us (515 without either).
// (The upsampling and skip sum in the epilogue of the layer before it: 280 us, 131 and 165 by themselves.)
struct LineEpi {
    __nv_bfloat16 *pool;
    Dims dc;               // of the pooled grid
    const float *hw, *hb;  // head
    float *out;
};

template <int CI, int CO, int EPI, int Y>
__global__ void __launch_bounds__(192, 1) k_conv_tc_line(const __grid_constant__ CUtensorMap tmap_x,
                                                         const __grid_constant__ CUtensorMap tmap_w, Dims d,
                                                         const float *__restrict__ bias, void *__restrict__ yout,
                                                         int *err, LineEpi ep) {
    static_assert(EPI != 3 || CO == 16, "head");
    using L = LineLayout<CI, CO, Y>;
    constexpr int LX = kLineX, kTiles = L::kTiles, KP = L::KP, S = L::kStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *wbuf = smem + S * L::kStageBytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(wbuf + KP * L::kWChunk);
    // barriers: [0,S) stage full, [S,2S) stage empty, then weights, two accumulators full, two accumulators
    // empty (four epilogue warps), done
    volatile uint32_t *sh = reinterpret_cast<volatile uint32_t *>(bars + 2 * S + 6);
    // sh: [0] TMEM base, [1] abort, [2] stage jobs issued, [3] stage jobs waited, [4] weights waited
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + S), wfull = smem_u32(bars + 2 * S),
                   tfull0 = smem_u32(bars + 2 * S + 1), tempty0 = smem_u32(bars + 2 * S + 3),
                   done = smem_u32(bars + 2 * S + 5);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bz_n = (d.nz + kLineZ - 1) / kLineZ, by_n = (d.ny + Y - 1) / Y;
    const long long nbricks = (long long)bz_n * by_n * ((d.nx + LX - 1) / LX);
    const int nb = nbricks > blockIdx.x ? (int)((nbricks - 1 - blockIdx.x) / gridDim.x + 1) : 0;
    auto brick = [&](int bi, int &z0, int &y0, int &x0) {
        const long long br = blockIdx.x + (long long)bi * gridDim.x;
        z0 = kLineZ * (int)(br % bz_n);
        y0 = Y * (int)((br / bz_n) % by_n);
        x0 = LX * (int)(br / ((long long)bz_n * by_n));
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(tfull0 + 8 * s, 1);
            mbar_init(tempty0 + 8 * s, 4);
        }
        mbar_init(wfull, 1);
        mbar_init(done, 1);
        for (int k = 1; k < 5; k++) sh[k] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<uint32_t *>(sh))),
                     "r"(L::kAlloc)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh[0];

    if (warp == 1 && lane == 0 && nb > 0) {  // TMA producer
        mbar_expect_tx(wfull, KP * L::kWChunkRaw);
        for (int c = 0; c < KP; c++) tma_load_3d(smem_u32(wbuf + c * L::kWChunk), &tmap_w, wfull, 16 * c, 0, 0);
        int q = 0;
        for (int bi = 0; bi < nb && !sh[1]; bi++) {
            int z0, y0, x0;
            brick(bi, z0, y0, x0);
            for (int p = 0; p < 3 * KP * (LX + 2) && !sh[1]; p++, q++) {  // (dz, 16-channel group, x plane)
                const int xb = p % (LX + 2), st = p / (LX + 2), dz = st / KP, jp = st % KP, s = q % S;
                if (q >= S && !mbar_wait(empty0 + 8 * s, (uint32_t)(q / S - 1) & 1u)) {
                    sh[1] = 1;
                    break;
                }
                mbar_expect_tx(full0 + 8 * s, L::kStageBytes);
                tma_load_4d(smem_u32(smem + s * L::kStageBytes), &tmap_x, full0 + 8 * s, 16 * jp, z0 + dz - 1, y0 - 1,
                            x0 - 1 + xb);
                sh[2] = (uint32_t)(q + 1);
            }
        }
    } else if (warp == 0 && lane == 0 && nb > 0) {  // MMA issuer
        bool any = false;
        if (!mbar_wait(wfull, 0)) sh[1] = 1;
        else sh[4] = 1;
        int q = 0;
        for (int bi = 0; bi < nb && !sh[1]; bi++) {
            const int tb = bi & 1;
            if (bi >= 2 && !mbar_wait(tempty0 + 8 * tb, (uint32_t)((bi - 2) >> 1) & 1u)) {
                sh[1] = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int st = 0; st < 3 * KP && !sh[1]; st++) {
                const int dz = st / KP, jp = st % KP;
                // weights of this z shift and channel group; every MMA below adds a compile-time offset in 16-byte units
                // (the start field cannot carry: shared addresses stay below 256 KB)
                const uint64_t bd0 = smem_desc_sw32(smem_u32(wbuf) + jp * L::kWChunk + (uint32_t)dz * 9u * CO * 32u);
                const uint32_t tacc = tmem + (uint32_t)(tb * L::kCols);
#pragma unroll
                for (int xb = 0; xb < LX + 2; xb++, q++) {
                    const int s = q % S;
                    if (!mbar_wait(full0 + 8 * s, (uint32_t)(q / S) & 1u)) {
                        sh[1] = 1;
                        break;
                    }
                    sh[3] = (uint32_t)(q + 1);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad0 = smem_desc_sw32(smem_u32(smem + s * L::kStageBytes));
#pragma unroll
                    for (int xx = 0; xx < LX; xx++) {
                        const int dx = xb - xx;  // this plane is tap dx of the tiles of column xx
                        if (dx < 0 || dx > 2) continue;
                        const uint64_t bd = bd0 + (uint64_t)(3 * dx * CO * 2);
                        const bool first = dx == 0 && st == 0;
                        if (first) {  // the brick's first tap overwrites its accumulator: by itself
#pragma unroll
                            for (int yb = 0; yb < Y; yb++)
                                mma_bf16(tacc + (uint32_t)((xx * Y + Y - 1 - yb) * CO), ad0 + (uint64_t)(256 * yb), bd,
                                         instr_desc_bf16(CO), 0u);
                        }
#pragma unroll
                        for (int yb = 0; yb < Y + 2; yb++) {  // line yb meets the tiles yb - dy, dy0 <= dy <= dy1
                            const int lo = yb < Y ? 0 : yb - Y + 1, dy1 = yb < 2 ? yb : 2;
                            const int dy0 = first && lo == 0 ? 1 : lo;
                            if (dy0 > dy1) continue;
                            mma_bf16(tacc + (uint32_t)((xx * Y + Y - 1 - (yb - dy0)) * CO), ad0 + (uint64_t)(256 * yb),
                                     bd + (uint64_t)(dy0 * CO * 2), instr_desc_bf16((dy1 - dy0 + 1) * CO), 1u);
                        }
                    }
                    any = true;
                    mma_commit(empty0 + 8 * s);
                }
            }
            if (sh[1]) break;
            mma_commit(tfull0 + 8 * tb);
        }
        if (any) {  // completion of every MMA issued (also on the error path, before TMEM is released)
            mma_commit(done);
            if (!mbar_wait(done, 0)) sh[1] = 1;
        }
    } else if (warp >= 2 && nb > 0) {  // epilogue
        const int q4 = warp & 3;  // TMEM lane quarter of this warp
        float hw[EPI == 3 ? 16 : 1], hb = 0.f;
        if (EPI == 3) {
#pragma unroll
            for (int c = 0; c < 16; c++) hw[EPI == 3 ? c : 0] = ep.hw[c];
            hb = ep.hb[0];
        }
        float bs[EPI == 1 ? 1 : CO];
#pragma unroll
        for (int c = 0; c < (EPI == 1 ? 0 : CO); c++) bs[c] = bias[c];
        for (int bi = 0; bi < nb; bi++) {
            const int tb = bi & 1;
            const uint32_t par = (uint32_t)(bi >> 1) & 1u;
            int z0, y0, x0;
            brick(bi, z0, y0, x0);
            const int z = z0 + 32 * q4 + lane;
            // lane 0 decides for the warp, so that the warp-collective TMEM loads below are never divergent
            int go = 0;
            if (lane == 0) go = (!sh[1] && mbar_wait(tfull0 + 8 * tb, par)) ? 1 : 0;
            go = __shfl_sync(0xffffffffu, go, 0);
            if (!go) {
                if (lane == 0) sh[1] = 1;
                break;
            }
            mbar_wait(tfull0 + 8 * tb, par);  // completed: returns at once, with this thread's acquire
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // 16 channels c0 .. of tile (yy, xx), after bias and ReLU, as BF16 pairs
            auto relu16 = [&](int yy, int xx, int c0, uint32_t(&pk)[8]) {
                float acc[16];
                tmem_ld_x16<16>(tmem + ((uint32_t)(32 * q4) << 16) +
                                    (uint32_t)(tb * L::kCols + (xx * Y + Y - 1 - yy) * CO + c0),
                                acc);  // accumulators by descending y
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const float a0 = fmaxf(acc[2 * k] + bs[EPI == 1 ? 0 : c0 + 2 * k], 0.f);
                    const float a1 = fmaxf(acc[2 * k + 1] + bs[EPI == 1 ? 0 : c0 + 2 * k + 1], 0.f);
                    __nv_bfloat162 h2 = __floats2bfloat162_rn(a0, a1);
                    pk[k] = *reinterpret_cast<uint32_t *>(&h2);
                }
            };
            auto put16 = [&](long long v, int c0, const uint32_t(&pk)[8]) {
                uint4 *dst = reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(yout) + v * CO + c0);
                dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
            };
            if constexpr (EPI == 2) {
                // lanes 2K and 2K + 1 hold the two z of coarse cell K: the even one takes channels 0-7 of both, the odd
                // one 8-15; the lower z of the four columns first, then the upper (held in up)
                const bool odd = lane & 1;
#pragma unroll 1
                for (int yp = 0; yp < Y; yp += 2) {
#pragma unroll
                    for (int c0 = 0; c0 < CO; c0 += 16) {
                        float sum[8];
                        uint32_t up[4][4];
#pragma unroll
                        for (int q = 0; q < 8; q++) sum[q] = 0.f;
                        auto add = [&](const uint32_t(&w)[4]) {
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                sum[2 * q] += __uint_as_float(w[q] << 16);
                                sum[2 * q + 1] += __uint_as_float(w[q] & 0xffff0000u);
                            }
                        };
#pragma unroll
                        for (int t = 0; t < 4; t++) {
                            const int xx = t & 1, yy = yp + (t >> 1);
                            uint32_t pk[8], lo[4];
                            relu16(yy, xx, c0, pk);
                            if (z < d.nz && y0 + yy < d.ny && x0 + xx < d.nx) {
                                put16(cid(d, x0 + xx, y0 + yy, z), c0, pk);
                            } else {  // absent
#pragma unroll
                                for (int q = 0; q < 8; q++) pk[q] = 0u;
                            }
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? pk[q] : pk[4 + q], 1);
                                lo[q] = odd ? got : pk[q];
                                up[t][q] = odd ? pk[4 + q] : got;
                            }
                            add(lo);
                        }
#pragma unroll
                        for (int t = 0; t < 4; t++) add(up[t]);
                        const int I = x0 >> 1, J = (y0 + yp) >> 1, K = z >> 1;
                        if (I < ep.dc.nx && J < ep.dc.ny && K < ep.dc.nz) {
                            uint32_t w[4];
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                __nv_bfloat162 h2 = __floats2bfloat162_rn(sum[2 * q] * 0.125f, sum[2 * q + 1] * 0.125f);
                                w[q] = *reinterpret_cast<uint32_t *>(&h2);
                            }
                            *reinterpret_cast<uint4 *>(ep.pool + cid(ep.dc, I, J, K) * CO + c0 + (odd ? 8 : 0)) =
                                make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
            } else {
#pragma unroll 1
                for (int tile = 0; tile < kTiles; tile++) {
                    const int yt = tile % Y, xt = tile / Y, yy = y0 + yt, xx = x0 + xt;
                    const bool inb = z < d.nz && yy < d.ny && xx < d.nx;
                    const long long v = inb ? cid(d, xx, yy, z) : 0;
#pragma unroll
                    for (int c0 = 0; c0 < CO; c0 += 16) {
                        if constexpr (EPI == 1) {
                            float acc[16];
                            tmem_ld_x16<16>(tmem + ((uint32_t)(32 * q4) << 16) +
                                                (uint32_t)(tb * L::kCols + (xt * Y + Y - 1 - yt) * CO + c0),
                                            acc);
                            if (!inb) continue;
                            float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(yout) + v * CO + c0);
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                dst[k] = make_float4(acc[4 * k], acc[4 * k + 1], acc[4 * k + 2], acc[4 * k + 3]);
                        } else {
                            uint32_t pk[8];
                            relu16(yt, xt, c0, pk);
                            if (!inb) continue;
                            if constexpr (EPI == 3) {
                                float s = hb;
#pragma unroll
                                for (int k = 0; k < 8; k++) {
                                    s += hw[2 * k] * __uint_as_float(pk[k] << 16);
                                    s += hw[2 * k + 1] * __uint_as_float(pk[k] & 0xffff0000u);
                                }
                                ep.out[v] = s;
                            } else {
                                put16(v, c0, pk);
                            }
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tempty0 + 8 * tb) : "memory");
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && sh[1]) {  // drain copies still in flight into this CTA's shared memory (bounded)
        for (uint32_t q = sh[3]; q < sh[2]; q++) mbar_wait(full0 + 8 * (q % S), (q / S) & 1u);
        if (!sh[4] && nb > 0) mbar_wait(wfull, 0);
        atomicCAS(err, 0, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::kAlloc) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------ 64-long z lines
// The z-line kernel for grids with 64 <= nz (the 64^3 level of a 256^3 network), any of 16, 32, 64 channels in and
// out: bricks of 64 (z) x 4 (y) x 2 (x) voxels, four M tiles of 64 z x 2 y (128 rows: two z lines).  A stage is one z
// shift dz and one group of 16 input channels: the halo'd box (16 channels, 64 z, 6 y, 4 x) from
// (z0 + dz - 1, y0 - 1, x0 - 1), 32-byte swizzled, whose tile (ty, xx) of tap (dx, dy) starts 2 KB x
// ((2 ty + 1 + dy) + 6 (xx + 1 + dx)) into it, and the weights of the nine taps (dx, dy, dz) for those 16 channels,
// one box (16 channels, Cout, 9) of a copy of the weights whose taps are ordered (dz, dx, dy) (the weights of a
// 64-channel layer do not fit in shared memory whole).  Three stages; otherwise as k_conv_tc_line.
constexpr int kL64Z = 64, kL64Y = 4, kL64X = 2, kL64Stages = 3;

template <int CI, int CO>
struct Line64Layout {
    static constexpr int KP = CI / 16, kTiles = (kL64Y / 2) * kL64X;
    static constexpr uint32_t kABytes = kL64Z * (kL64Y + 2) * (kL64X + 2) * 32u;  // 48 KB
    static constexpr uint32_t kWRaw = 9u * CO * 32u;
    static constexpr uint32_t kWBytes = (kWRaw + 1023u) & ~1023u;
    static constexpr uint32_t kStageBytes = kABytes + kWBytes;
    static constexpr uint32_t kCols = kTiles * CO;
    static constexpr uint32_t kAlloc = 2u * kCols <= 32u ? 32u : 2u * kCols <= 64u ? 64u : 2u * kCols <= 128u ? 128u
                                                                                    : 2u * kCols <= 256u ? 256u
                                                                                                         : 512u;
    static constexpr uint32_t kSmemBytes = 1024u + kL64Stages * kStageBytes + 256u;
    static_assert(CI % 16 == 0 && CO % 16 == 0 && 2u * kCols <= 512u && kSmemBytes <= 227u * 1024u, "layout");
};

template <int CI, int CO, int EPI>
__global__ void __launch_bounds__(192, 1) k_conv_tc_line64(const __grid_constant__ CUtensorMap tmap_x,
                                                           const __grid_constant__ CUtensorMap tmap_wp, Dims d,
                                                           const float *__restrict__ bias, void *__restrict__ yout,
                                                           int *err) {
    using L = Line64Layout<CI, CO>;
    constexpr int KP = L::KP, S = kL64Stages, kTiles = L::kTiles;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + S * L::kStageBytes);
    // barriers: [0,S) stage full, [S,2S) stage empty, [2S,2S+2) accumulators full, [2S+2,2S+4) accumulators empty
    // (four epilogue warps), 2S+4 done
    volatile uint32_t *sh = reinterpret_cast<volatile uint32_t *>(bars + 2 * S + 5);
    // sh: [0] TMEM base, [1] abort, [2] stage jobs issued, [3] stage jobs waited
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + S), tfull0 = smem_u32(bars + 2 * S),
                   tempty0 = smem_u32(bars + 2 * S + 2), done = smem_u32(bars + 2 * S + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bz_n = (d.nz + kL64Z - 1) / kL64Z, by_n = (d.ny + kL64Y - 1) / kL64Y;
    const long long nbricks = (long long)bz_n * by_n * ((d.nx + kL64X - 1) / kL64X);
    const int nb = nbricks > blockIdx.x ? (int)((nbricks - 1 - blockIdx.x) / gridDim.x + 1) : 0;
    auto brick = [&](int bi, int &z0, int &y0, int &x0) {
        const long long br = blockIdx.x + (long long)bi * gridDim.x;
        z0 = kL64Z * (int)(br % bz_n);
        y0 = kL64Y * (int)((br / bz_n) % by_n);
        x0 = kL64X * (int)(br / ((long long)bz_n * by_n));
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(tfull0 + 8 * s, 1);
            mbar_init(tempty0 + 8 * s, 4);
        }
        mbar_init(done, 1);
        for (int k = 1; k < 4; k++) sh[k] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<uint32_t *>(sh))),
                     "r"(L::kAlloc)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh[0];

    if (warp == 1 && lane == 0 && nb > 0) {  // TMA producer
        int q = 0;
        for (int bi = 0; bi < nb && !sh[1]; bi++) {
            int z0, y0, x0;
            brick(bi, z0, y0, x0);
            for (int st = 0; st < 3 * KP && !sh[1]; st++, q++) {  // stage = (dz, 16-channel group)
                const int dz = st / KP, jp = st % KP, s = q % S;
                if (q >= S && !mbar_wait(empty0 + 8 * s, (uint32_t)(q / S - 1) & 1u)) {
                    sh[1] = 1;
                    break;
                }
                const uint32_t a = smem_u32(smem + s * L::kStageBytes);
                mbar_expect_tx(full0 + 8 * s, L::kABytes + L::kWRaw);
                tma_load_4d(a, &tmap_x, full0 + 8 * s, 16 * jp, z0 + dz - 1, y0 - 1, x0 - 1);
                tma_load_3d(a + L::kABytes, &tmap_wp, full0 + 8 * s, 16 * jp, 0, 9 * dz);
                sh[2] = (uint32_t)(q + 1);
            }
        }
    } else if (warp == 0 && lane == 0 && nb > 0) {  // MMA issuer
        constexpr uint32_t idesc = instr_desc_bf16(CO);
        bool any = false;
        int q = 0;
        for (int bi = 0; bi < nb && !sh[1]; bi++) {
            const int tb = bi & 1;
            if (bi >= 2 && !mbar_wait(tempty0 + 8 * tb, (uint32_t)((bi - 2) >> 1) & 1u)) {
                sh[1] = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int st = 0; st < 3 * KP; st++, q++) {
                const int s = q % S;
                if (!mbar_wait(full0 + 8 * s, (uint32_t)(q / S) & 1u)) {
                    sh[1] = 1;
                    break;
                }
                sh[3] = (uint32_t)(q + 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // descriptor bases of this stage plus compile-time offsets in 16-byte units (no carry: shared
                // addresses stay below 256 KB)
                const uint32_t a = smem_u32(smem + s * L::kStageBytes);
                const uint64_t ad0 = smem_desc_sw32(a), bd0 = smem_desc_sw32(a + L::kABytes);
                const uint32_t tacc = tmem + (uint32_t)(tb * L::kCols);
                const uint32_t acc0 = st > 0 ? 1u : 0u;
#pragma unroll
                for (int pr = 0; pr < 9; pr++) {
                    const int dx = pr / 3 - 1, dy = pr % 3 - 1;
                    const uint64_t bd = bd0 + (uint64_t)(pr * CO * 2);
#pragma unroll
                    for (int tile = 0; tile < kTiles; tile++) {
                        const int ty = tile % (kL64Y / 2), xx = tile / (kL64Y / 2);
                        const uint64_t ad = ad0 + (uint64_t)(128 * ((2 * ty + 1 + dy) + (kL64Y + 2) * (xx + 1 + dx)));
                        mma_bf16(tacc + (uint32_t)(tile * CO), ad, bd, idesc, pr > 0 ? 1u : acc0);
                    }
                }
                any = true;
                mma_commit(empty0 + 8 * s);
            }
            if (sh[1]) break;
            mma_commit(tfull0 + 8 * tb);
        }
        if (any) {  // completion of every MMA issued (also on the error path, before TMEM is released)
            mma_commit(done);
            if (!mbar_wait(done, 0)) sh[1] = 1;
        }
    } else if (warp >= 2 && nb > 0) {  // epilogue
        const int q4 = warp & 3;  // TMEM lane quarter of this warp
        for (int bi = 0; bi < nb; bi++) {
            const int tb = bi & 1;
            const uint32_t par = (uint32_t)(bi >> 1) & 1u;
            // lane 0 decides for the warp, so that the warp-collective TMEM loads below are never divergent
            int go = 0;
            if (lane == 0) go = (!sh[1] && mbar_wait(tfull0 + 8 * tb, par)) ? 1 : 0;
            go = __shfl_sync(0xffffffffu, go, 0);
            if (!go) {
                if (lane == 0) sh[1] = 1;
                break;
            }
            mbar_wait(tfull0 + 8 * tb, par);  // completed: returns at once, with this thread's acquire
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            int z0, y0, x0;
            brick(bi, z0, y0, x0);
            const int m = 32 * q4 + lane;  // TMEM lane = tile row: z = m % 64, y = m / 64
            const int z = z0 + (m & (kL64Z - 1));
#pragma unroll 1
            for (int tile = 0; tile < kTiles; tile++) {
                const int yy = y0 + 2 * (tile % (kL64Y / 2)) + (m >> 6), xx = x0 + tile / (kL64Y / 2);
                const bool inb = z < d.nz && yy < d.ny && xx < d.nx;
                const long long v = inb ? cid(d, xx, yy, z) : 0;
#pragma unroll
                for (int c0 = 0; c0 < CO; c0 += 16) {
                    float acc[16];
                    tmem_ld_x16<16>(tmem + ((uint32_t)(32 * q4) << 16) + (uint32_t)(tb * L::kCols + tile * CO + c0),
                                    acc);
                    if (inb && EPI == 0) {
                        uint32_t pk[8];
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            const float a0 = fmaxf(acc[2 * k] + bias[c0 + 2 * k], 0.f);
                            const float a1 = fmaxf(acc[2 * k + 1] + bias[c0 + 2 * k + 1], 0.f);
                            __nv_bfloat162 h2 = __floats2bfloat162_rn(a0, a1);
                            pk[k] = *reinterpret_cast<uint32_t *>(&h2);
                        }
                        uint4 *dst = reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(yout) + v * CO + c0);
                        dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                        dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
                    } else if (inb) {
                        float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(yout) + v * CO + c0);
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            dst[k] = make_float4(acc[4 * k], acc[4 * k + 1], acc[4 * k + 2], acc[4 * k + 3]);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tempty0 + 8 * tb) : "memory");
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && sh[1]) {  // drain copies still in flight into this CTA's shared memory (bounded)
        for (uint32_t q = sh[3]; q < sh[2]; q++) mbar_wait(full0 + 8 * (q % S), (q / S) & 1u);
        atomicCAS(err, 0, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::kAlloc) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------ weight gradient
// dW[tap][co][ci] = sum over voxels v of dY[v][co] X[v + off(tap)][ci]: GEMMs with M = Cout, K = voxels and
// N = (dz, Cin), both operands K-major with 8 consecutive z per 16-byte row.  k_to_chmajor makes channel-major copies
// with z split into 8-voxel rows: dYT[zh][x][y][co][zl] and XT[zh][x][y][s][ci][zl] = X[x][y][8 zh + zl + s - 1][ci]
// (zero outside), the three z shifts s = dz + 1 interleaved per row so that one TMA box starting on a row boundary
// carries all three.  A job is one (dx, dy) pair over one brick of 32 (z) x 4 (y) x BX (x) voxels: one TMA box
// of 8 z x C x 4 y x BX x x 4 zh lands as rows c + C k of 16 B, k = y + 4 (x + BX zh) the K index of the 8-voxel core
// matrices, so consecutive K steps are C x 16 B apart (LBO) and 8-row groups 128 B (SBO); the y and x shifts are box
// coordinates (outside the grid: zero fill).  One MMA (K = 16) then accumulates the three taps (dx, dy, -1..1) into
// 3 Cin TMEM columns.  M = 64 rows of which the first Cout are dY channels; the rows past them read the next K
// steps' rows (or a zeroed slack after the buffer) and land in accumulator lanes that are never read (M = 128 reads
// twice the shared memory for nothing).
// HALO (16 input channels, grids that hold the box): a job is one zh of a brick with all nine pairs: the box with its
// halo, 6 y x (BX + 2) x, is read once for them, and as the rows of y, y + 1 and y + 2 follow one another one MMA of
// N = 144 does the three dy.  16 to 16 channels at 128^3: 405 us with a box a pair and M = 128, 126 so
// (the 6.5 KB an MMA reads, at 64 bytes a clock).
// The maps take the contiguous (8 z, channels) as long rows: a row of 16 bytes costs the copy unit as much as one of 512.
// One CTA (one per SM, 512 TMEM columns) runs a group of (dx, dy) pairs over a strided set of bricks, warp
// specialised: lane 0 of warp 1 issues the TMA loads (dY of a brick once, into one of two buffers; X per pair through
// a ring of stages), lane 0 of warp 0 the MMAs, so neither waits on the other's latency.  The CTA writes its partial
// sums part[chunk][tap][co][ci] (FP32), reduced over chunks in fixed order afterwards.  Every wait is bounded as in
// k_conv_tc.
constexpr uint32_t kWgSlack = 2048;

template <int CI>
__host__ __device__ constexpr int wg_bx() {  // x extent of a brick
    return CI == 16 ? 2 : 1;
}
// (dx, dy) pairs per CTA: 3 CI columns each, at most 512
template <int CI>
__host__ __device__ constexpr int wg_pairs_per_cta() {
    return CI == 16 ? 9 : CI == 32 ? 5 : 2;
}

// channels of one row of a box (8 z each, at most 256 elements)
__host__ __device__ constexpr int wg_row_channels(int c) { return c <= 32 ? c : c % 32 == 0 ? 32 : 24; }

template <int CI, int CO, bool HALO>
struct WgLayout {
    static constexpr int BX = wg_bx<CI>();
    static constexpr uint32_t kABytes = 256u * CO * BX;  // 8 z x CO x 4 y x BX x x 4 zh, BF16
    // 8 z x 3 CI x 4 y x BX x x 4 zh, or x 6 y x (BX + 2) x
    static constexpr uint32_t kBBytes = HALO ? 48u * CI * 6u * (BX + 2) : 768u * CI * BX;
    static constexpr uint32_t kAStride = kABytes + kWgSlack;
    static constexpr int kStagesRaw = (int)((216u * 1024u - 2u * kAStride) / kBBytes);
    static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
    static constexpr uint32_t kNeed = 2u * kAStride + kStages * kBBytes + 1024u + 512u;
    // at least 116 KB: one CTA per SM, whose 512 TMEM columns are then always free
    static constexpr uint32_t kSmemBytes = kNeed > 116u * 1024u ? kNeed : 116u * 1024u;
    static_assert(kStages >= 2 && kSmemBytes <= 227u * 1024u, "shared memory");
};

// dst[zh][x][y][s][c][zl] = src[x][y][8 zh + zl + s - 1][c] where 8 zh + zl < nz and the shifted z lies in
// the grid, else 0; s < 3, zh < nzh = ceil(nz / 8).  A thread takes two channels of one (zh, x, y): each z is
// read once, in 4-byte words, for all its shifts, and 32 bytes are stored per shift (a channel a thread and a read per
// shift: 76 us for 16 channels at 128^3, 56 now).
template <int C>
__global__ void __launch_bounds__(256) k_to_chmajor(Dims d, const __nv_bfloat16 *__restrict__ src,
                                                    __nv_bfloat16 *__restrict__ dst) {
    constexpr int P = C / 2, NS = 3;
    const long long m = (long long)((d.nz + 7) / 8) * d.nx * d.ny * P;
    const uint32_t *s32 = reinterpret_cast<const uint32_t *>(src);
    for (long long e = blockIdx.x * 256LL + threadIdx.x; e < m; e += gridDim.x * 256LL) {
        const int cp = (int)(e % P);
        const unsigned r = (unsigned)(e / P), t = r / (unsigned)d.ny;  // r = (zh nx + x) ny + y
        const int y = (int)(r - t * d.ny), zh = (int)(t / (unsigned)d.nx), x = (int)(t - (unsigned)zh * d.nx);
        const uint32_t *row = s32 + ((long long)x * d.ny + y) * d.nz * P + cp;
        uint32_t v[7 + NS];
#pragma unroll
        for (int q = 0; q < 7 + NS; q++) {
            const int z = 8 * zh + q - 1;
            v[q] = z >= 0 && z < d.nz ? row[(long long)z * P] : 0u;
        }
        const int nv = d.nz - 8 * zh;  // voxels of this 8-voxel row inside the grid
#pragma unroll
        for (int s = 0; s < NS; s++) {
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t a = 2 * q < nv ? v[2 * q + s] : 0u, b = 2 * q + 1 < nv ? v[2 * q + 1 + s] : 0u;
                lo[q] = __byte_perm(a, b, 0x5410);
                hi[q] = __byte_perm(a, b, 0x7632);
            }
            uint4 *out = reinterpret_cast<uint4 *>(dst) + ((long long)r * NS + s) * C + 2 * cp;
            out[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            out[1] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        }
    }
}

// dY = dpost (post > 0) as BF16 [voxel][C], and its channel-major copy [zh][x][y][c][zl], zero past nz, in one pass (37
// and 23 us for 16 channels at 128^3 by themselves, 52 together).
template <int C>
__global__ void __launch_bounds__(256) k_relu_chmajor(Dims d, const float *__restrict__ dpost,
                                                      const __nv_bfloat16 *__restrict__ post,
                                                      __nv_bfloat16 *__restrict__ dy, __nv_bfloat16 *__restrict__ dyT) {
    constexpr int P = C / 2;
    const long long m = (long long)((d.nz + 7) / 8) * d.nx * d.ny * P;
    for (long long e = blockIdx.x * 256LL + threadIdx.x; e < m; e += gridDim.x * 256LL) {
        const int cp = (int)(e % P);
        const unsigned r = (unsigned)(e / P), t = r / (unsigned)d.ny;  // r = (zh nx + x) ny + y
        const int y = (int)(r - t * d.ny), zh = (int)(t / (unsigned)d.nx), x = (int)(t - (unsigned)zh * d.nx);
        const long long row = (((long long)x * d.ny + y) * d.nz + 8 * zh) * P + cp;  // in channel pairs
        const int nv = d.nz - 8 * zh;
        uint32_t v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            v[q] = 0u;
            if (q < nv) {
                const float2 g = reinterpret_cast<const float2 *>(dpost)[row + q * P];
                const uint32_t a = reinterpret_cast<const uint32_t *>(post)[row + q * P];
                __nv_bfloat162 h2 = __floats2bfloat162_rn(__uint_as_float(a << 16) > 0.f ? g.x : 0.f,
                                                          __uint_as_float(a & 0xffff0000u) > 0.f ? g.y : 0.f);
                v[q] = *reinterpret_cast<uint32_t *>(&h2);
                reinterpret_cast<uint32_t *>(dy)[row + q * P] = v[q];
            }
        }
        uint4 *out = reinterpret_cast<uint4 *>(dyT) + (long long)r * C + 2 * cp;
        out[0] = make_uint4(__byte_perm(v[0], v[1], 0x5410), __byte_perm(v[2], v[3], 0x5410),
                            __byte_perm(v[4], v[5], 0x5410), __byte_perm(v[6], v[7], 0x5410));
        out[1] = make_uint4(__byte_perm(v[0], v[1], 0x7632), __byte_perm(v[2], v[3], 0x7632),
                            __byte_perm(v[4], v[5], 0x7632), __byte_perm(v[6], v[7], 0x7632));
    }
}

template <int CI, int CO, bool HALO>
__global__ void __launch_bounds__(128, 1) k_wgrad_tc(const __grid_constant__ CUtensorMap tmap_dy,
                                                     const __grid_constant__ CUtensorMap tmap_x, Dims d,
                                                     float *__restrict__ part, int *err) {
    constexpr int NP = wg_pairs_per_cta<CI>();
    constexpr int N = 3 * CI;
    static_assert(NP * N <= 512 && CO <= 64 && CI % 16 == 0 && CO % 16 == 0 && N <= 256, "shape");
    static_assert(!HALO || (NP == 9 && 3 * N <= 256), "halo form: every pair in one CTA, three of them an MMA");
    using L = WgLayout<CI, CO, HALO>;
    constexpr int S = L::kStages, BX = L::BX;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *abuf = smem, *bbuf = smem + 2 * L::kAStride;
    uint64_t *bars = reinterpret_cast<uint64_t *>(bbuf + S * L::kBBytes);
    // [0, 2) dY full, [2, 4) dY empty, [4, 4 + S) X full, [4 + S, 4 + 2S) X empty, then done
    // sh: [0] TMEM base, [1] status, [2] MMA side ok, [3] X jobs waited, [4] bricks waited, [5] TMA side ok,
    //     [6] X jobs issued, [7] bricks issued
    volatile uint32_t *sh = reinterpret_cast<volatile uint32_t *>(bars + 4 + 2 * S + 1);
    const uint32_t afull0 = smem_u32(bars), aempty0 = smem_u32(bars + 2), bfull0 = smem_u32(bars + 4),
                   bempty0 = smem_u32(bars + 4 + S), done = smem_u32(bars + 4 + 2 * S);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pair0 = blockIdx.y * NP, npair = min(NP, 9 - pair0);
    const int bz_n = (d.nz + 31) / 32, by_n = (d.ny + 3) / 4, bx_n = (d.nx + BX - 1) / BX;
    const long long nbricks = (long long)bz_n * by_n * bx_n;
    const int nb = nbricks > blockIdx.x ? (int)((nbricks - 1 - blockIdx.x) / gridDim.x + 1) : 0;
    const int JB = HALO ? 4 : npair, J = nb * JB;  // jobs per brick

    // zero the slack after each dY buffer (read by the MMA rows past Cout)
    for (uint32_t i = threadIdx.x; i < kWgSlack / 16; i += blockDim.x) {
        reinterpret_cast<uint4 *>(abuf + L::kABytes)[i] = make_uint4(0, 0, 0, 0);
        reinterpret_cast<uint4 *>(abuf + L::kAStride + L::kABytes)[i] = make_uint4(0, 0, 0, 0);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(afull0 + 8 * s, 1);
            mbar_init(aempty0 + 8 * s, 1);
        }
        for (int s = 0; s < S; s++) {
            mbar_init(bfull0 + 8 * s, 1);
            mbar_init(bempty0 + 8 * s, 1);
        }
        mbar_init(done, 1);
        for (int k = 1; k < 8; k++) sh[k] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<uint32_t *>(sh))),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh[0];

    auto brick = [&](int bi, int &z0, int &y0, int &x0) {
        const long long br = blockIdx.x + (long long)bi * gridDim.x;
        z0 = 32 * (int)(br % bz_n);
        y0 = 4 * (int)((br / bz_n) % by_n);
        x0 = BX * (int)(br / ((long long)bz_n * by_n));
    };
    if (warp == 1 && lane == 0) {  // TMA producer
        bool ok = true;
        int a_issued = 0, b_issued = 0;
        for (int q = 0; q < J && ok; q++) {
            const int bi = q / JB, jj = q % JB;
            int z0, y0, x0;
            brick(bi, z0, y0, x0);
            if (jj == 0) {
                const int ab = bi & 1;
                if (bi >= 2 && !mbar_wait(aempty0 + 8 * ab, (uint32_t)((bi - 2) >> 1) & 1u)) {
                    ok = false;
                    break;
                }
                mbar_expect_tx(afull0 + 8 * ab, L::kABytes);
                tma_load_5d(smem_u32(abuf + ab * L::kAStride), &tmap_dy, afull0 + 8 * ab, 0, 0, y0, x0, z0 / 8);
                a_issued = bi + 1;
            }
            const int pr = pair0 + jj, dx = pr / 3 - 1, dy = pr % 3 - 1;
            const int s = q % S;
            if (q >= S && !mbar_wait(bempty0 + 8 * s, (uint32_t)(q / S - 1) & 1u)) {
                ok = false;
                break;
            }
            mbar_expect_tx(bfull0 + 8 * s, L::kBBytes);
            if (HALO)
                tma_load_5d(smem_u32(bbuf + s * L::kBBytes), &tmap_x, bfull0 + 8 * s, 0, 0, y0 - 1, x0 - 1, z0 / 8 + jj);
            else
                tma_load_5d(smem_u32(bbuf + s * L::kBBytes), &tmap_x, bfull0 + 8 * s, 0, 0, y0 + dy, x0 + dx, z0 / 8);
            b_issued = q + 1;
        }
        sh[5] = ok ? 1u : 0u;
        sh[6] = (uint32_t)b_issued;
        sh[7] = (uint32_t)a_issued;
    } else if (warp == 0 && lane == 0) {  // MMA issuer
        constexpr uint32_t idesc = instr_desc_bf16(HALO ? 3 * N : N, 64);
        bool ok = true;
        int a_waited = 0, b_waited = 0;
        for (int q = 0; q < J; q++) {
            const int bi = q / JB, jj = q % JB, ab = bi & 1, s = q % S;
            if (jj == 0) {
                if (!mbar_wait(afull0 + 8 * ab, (uint32_t)(bi >> 1) & 1u)) {
                    ok = false;
                    break;
                }
                a_waited = bi + 1;
            }
            if (!mbar_wait(bfull0 + 8 * s, (uint32_t)(q / S) & 1u)) {
                ok = false;
                break;
            }
            b_waited = q + 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t ad0 = smem_desc(smem_u32(abuf + ab * L::kAStride), (uint32_t)CO * 16u, 128u);
            const uint64_t bd0 = smem_desc(smem_u32(bbuf + s * L::kBBytes), (uint32_t)N * 16u, 128u);
            // start addresses advance in 16-byte units (no carry: < 256 KB)
            if (HALO) {
                const uint64_t ad = ad0 + (uint64_t)(jj * 4 * BX * CO);
#pragma unroll
                for (int dx = 0; dx < 3; dx++)
#pragma unroll
                    for (int p = 0; p < 2 * BX; p++)  // p = y / 2 + 2 x
                        mma_bf16(tmem + (uint32_t)(3 * dx * N), ad + (uint64_t)(2 * p * CO),
                                 bd0 + (uint64_t)((2 * (p % 2) + 6 * (p / 2 + dx)) * N), idesc, (q > 0 || p > 0) ? 1u : 0u);
            } else {
#pragma unroll
                for (int p = 0; p < 8 * BX; p++)
                    mma_bf16(tmem + (uint32_t)(jj * N), ad0 + (uint64_t)(2 * p * CO), bd0 + (uint64_t)(2 * p * N), idesc,
                             (bi > 0 || p > 0) ? 1u : 0u);
            }
            mma_commit(bempty0 + 8 * s);
            if (jj == JB - 1) mma_commit(aempty0 + 8 * ab);
        }
        if (b_waited > 0) {  // completion of every MMA issued (also on the error path, before TMEM is released)
            mma_commit(done);
            if (!mbar_wait(done, 0)) ok = false;
        }
        sh[2] = ok ? 1u : 0u;
        sh[3] = (uint32_t)b_waited;
        sh[4] = (uint32_t)a_waited;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const bool ok = sh[2] && sh[5];
        if (!ok) {  // drain copies still in flight into this CTA's shared memory (bounded)
            for (uint32_t q = sh[3]; q < sh[6]; q++) mbar_wait(bfull0 + 8 * (q % S), (q / S) & 1u);
            for (uint32_t q = sh[4]; q < sh[7]; q++) mbar_wait(afull0 + 8 * (q & 1), (q >> 1) & 1u);
            atomicCAS(err, 0, 1);
        }
        sh[1] = ok ? (J > 0 ? 1u : 2u) : 0u;
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t st = sh[1];
    if (st != 0 && 16 * warp < CO) {  // 1: the accumulators hold this CTA's sums; 2: no brick, the sums are zero
        const int co = lane < 16 ? 16 * warp + lane : CO;  // an M = 64 accumulator: 16 rows in each lane quarter
        for (int jj = 0; jj < npair; jj++) {
#pragma unroll
            for (int sz = 0; sz < 3; sz++) {
                float *out = part + (((long long)blockIdx.x * 27 + 3 * (pair0 + jj) + sz) * CO) * CI;
#pragma unroll
                for (int c0 = 0; c0 < CI; c0 += 16) {
                    float acc[16];
                    if (st == 1) {
                        tmem_ld_x16<16>(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(jj * N + sz * CI + c0), acc);
                    } else {
#pragma unroll
                        for (int q = 0; q < 16; q++) acc[q] = 0.f;
                    }
                    if (co < CO) {
                        float4 *dst = reinterpret_cast<float4 *>(out + (long long)co * CI + c0);
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            dst[q] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

}  // namespace tc
}  // namespace sf
