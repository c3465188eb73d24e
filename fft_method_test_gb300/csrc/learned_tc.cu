// learned_tc.cu -- the 3x3x3 convolution of the learned warm start on the
// fifth-generation tensor cores: tcgen05.mma with the accumulator in tensor
// memory (TMEM), operands staged in shared memory.  No counterpart in the
// reference (its MinresSolver::solve takes an initial guess,
// src/solver/MinresSolver.hpp:23, that nothing fills).
//
// Implicit GEMM, one CTA per 128 voxels (the MMA's M), in two forms: k_conv_halo
// below (dilation 1, up to 64 input channels) and k_conv_tc; conv_rules.h chooses
// the form, the output channels of a CTA and k_conv_tc's buffers by size:
//   y[v][o] = sum_tap sum_i x[v + sign*dil*off(tap)][i] W[tap][o][i]
// Activations are channels-last BF16 [voxel][channel], weights BF16
// [27][cout][cin] (the data gradient passes the per-tap transposed weights
// and sign -1), periodic wrap, FP32 accumulation.  Per tap the 128 shifted
// input rows (A, 128 x cin) and the tap's weights (B, cout x cin) are
// copied into one of STAGES shared-memory buffers with cp.async, in the
// canonical K-major layout without swizzle: 8 x 16-byte core matrices, the
// two core matrices of a 16-channel chunk side by side (leading byte offset
// 128), 8-row groups 256 bytes apart (stride byte offset).  One thread issues
// cin/16 MMAs of 128 x cout x 16 per tap and commits them to the buffer's
// mbarrier; the 128 threads meanwhile gather the rows of tap t + STAGES - 1, so
// the latency of a gather is hidden by STAGES - 1 taps (128 -> 128 channels on
// four 8^3 cells: 77 us with two buffers and all channels in a CTA, 48 with four
// and sixteen channels).  A grid of few voxels splits the output channels over
// blockIdx.y.  The epilogue reads the accumulator rows back with tcgen05.ld (warp w
// owns TMEM lanes 32w..32w+31 = voxel rows), adds the bias, applies ReLU and
// stores FP32 and/or BF16.
//
// Every wait is bounded (the mbarrier helpers of tma.cuh): on a timeout the
// CTA raises the file-scope error flag (fp_nn_tc_error), frees its TMEM and
// returns.  The dynamic shared memory of a CTA is at least its share of the
// SM for the TMEM columns it holds, so the CTAs resident on an SM never ask
// for more than the 512 TMEM columns there are.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/fftperm.h"
#include "common.cuh"
#include "conv_rules.h"
#include "tma.cuh"

#ifndef FP_TC_LBO
#define FP_TC_LBO 128  // bytes between the two core matrices of a 16-channel chunk
#endif
#ifndef FP_TC_SBO
#define FP_TC_SBO 256  // bytes between 8-row groups
#endif

namespace fp {
namespace {

constexpr int kTcM = 128;  // voxels per CTA = MMA M = TMEM lanes
constexpr int kTcThreads = 128;

__device__ int g_tc_err = 0;

struct TcConv {
    int nx, ny, nz;
    long long n;      // voxels per sample
    long long total;  // voxels of all samples
    int dil, sign;
    const __nv_bfloat16* in;
    int cin;
    int cout;  // all output channels (a CTA computes COUT of them)
    const __nv_bfloat16* w;
    const float* bias;
    int relu;
    float* out32;
    __nv_bfloat16* out16;
};

__device__ __forceinline__ void cp_async16_zfill(void* smem, const void* gmem, bool valid) {
    const int n = valid ? 16 : 0;  // src-size 0: the 16 bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem)), "l"(gmem),
                 "r"(n)
                 : "memory");
}

// shared-memory matrix descriptor: K-major, no swizzle
__device__ __forceinline__ uint64_t smem_desc(const void* p) {
    const uint32_t a = smem_u32(p);
    return (uint64_t)((a >> 4) & 0x3FFF) | ((uint64_t)((FP_TC_LBO >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((FP_TC_SBO >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

// the same for rows 16 bytes apart (eight-row groups 128 bytes apart) and core
// matrices of neighbouring eight-channel groups `rows` such rows apart
__device__ __forceinline__ uint64_t smem_desc_rows(const void* p, uint32_t rows) {
    const uint32_t a = smem_u32(p);
    return (uint64_t)((a >> 4) & 0x3FFF) | ((uint64_t)(rows & 0x3FFF) << 16) | ((uint64_t)(128 >> 4) << 32) |
           (1ull << 46);
}

// instruction descriptor of kind::f16: BF16 A and B, FP32 D, K-major both,
// N = cout, M = 128
template <int N>
__device__ __forceinline__ constexpr uint32_t idesc_bf16() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(kTcM >> 4) << 24);
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// core-matrix position of element row m, 8-element group q (k = 8q..8q+7)
// inside a tile of `rows` rows: chunk q / 2 of rows * 32 bytes, core matrix
// ((m / 8) * 2 + q % 2) of 128 bytes, row m % 8 of 16 bytes
__device__ __forceinline__ uint32_t core_offset(int m, int q, int rows) {
    return (uint32_t)((q >> 1) * rows * 32 + ((m >> 3) * 2 + (q & 1)) * 128 + (m & 7) * 16);
}

// Sixteen output channels c0.. of a warp's 32 accumulator rows (TMEM lanes from
// trow): bias, ReLU and the stores of voxel v.
__device__ __forceinline__ void store_rows(uint32_t trow, int c0, int o0, const float* bias, int relu, bool valid,
                                           long long v, int cout, float* out32, __nv_bfloat16* out16) {
    uint32_t rr[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
        "%13,%14,%15}, [%16];"
        : "=r"(rr[0]), "=r"(rr[1]), "=r"(rr[2]), "=r"(rr[3]), "=r"(rr[4]), "=r"(rr[5]),
          "=r"(rr[6]), "=r"(rr[7]), "=r"(rr[8]), "=r"(rr[9]), "=r"(rr[10]), "=r"(rr[11]),
          "=r"(rr[12]), "=r"(rr[13]), "=r"(rr[14]), "=r"(rr[15])
        : "r"(trow + (uint32_t)c0));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (!valid) return;
    float f[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        f[j] = __uint_as_float(rr[j]);
        if (bias) f[j] += bias[o0 + c0 + j];
        if (relu) f[j] = fmaxf(f[j], 0.f);
    }
    if (out32) {
        float4* o = reinterpret_cast<float4*>(out32 + v * cout + o0 + c0);
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = make_float4(f[4 * j], f[4 * j + 1], f[4 * j + 2], f[4 * j + 3]);
    }
    if (out16) {
        uint32_t pk[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t lo = __bfloat16_as_ushort(__float2bfloat16(f[2 * j]));
            const uint32_t hi = __bfloat16_as_ushort(__float2bfloat16(f[2 * j + 1]));
            pk[j] = lo | (hi << 16);
        }
        uint4* o = reinterpret_cast<uint4*>(out16 + v * cout + o0 + c0);
        o[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        o[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
    }
}

template <int COUT, int STAGES>
__global__ void __launch_bounds__(kTcThreads) k_conv_tc(TcConv p) {
    constexpr int NCOLS = COUT < 32 ? 32 : COUT;  // TMEM columns (power of two, >= 32)
    extern __shared__ __align__(1024) unsigned char sm[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + 64);
    volatile int* failed = reinterpret_cast<volatile int*>(sm + 72);
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int cin = p.cin;
    const int kc = cin / 16;
    const int o0 = blockIdx.y * COUT;
    const uint32_t abytes = (uint32_t)kTcM * cin * 2;
    const uint32_t bbytes = (uint32_t)COUT * cin * 2;
    unsigned char* buf0 = sm + 1024;
    auto abuf = [&](int b) { return buf0 + (size_t)b * (abytes + bbytes); };
    auto bbuf = [&](int b) { return buf0 + (size_t)b * (abytes + bbytes) + abytes; };

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tslot)),
                     "r"(NCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int b = 0; b < STAGES; ++b) mbar_init(&bars[b], 1);
        fence_mbar_init();
        *failed = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    // this thread's voxel (A row tid) and its wrapped neighbours along each axis
    const long long v = (long long)blockIdx.x * kTcM + tid;
    const bool valid = v < p.total;
    const long long vv = valid ? v : 0;
    const long long smp = vv / p.n;
    const long long r = vv - smp * p.n;
    const int x = (int)(r % p.nx);
    const long long q0 = r / p.nx;
    const int y = (int)(q0 % p.ny);
    const int z = (int)(q0 / p.ny);
    const int step = p.sign * p.dil;
    auto wrap = [](int i, int n) {
        i %= n;
        return i < 0 ? i + n : i;
    };
    const int xm = wrap(x - step, p.nx), xp = wrap(x + step, p.nx);
    const int ym = wrap(y - step, p.ny), yp = wrap(y + step, p.ny);
    const int zm = wrap(z - step, p.nz), zp = wrap(z + step, p.nz);
    const __nv_bfloat16* in = p.in + smp * p.n * cin;

    auto issue = [&](int tap) {
        const int b = tap % STAGES;
        // A: the shifted input row of this voxel
        {
            const int dz = tap / 9, dy = tap / 3 % 3, dx = tap % 3;
            const int zz = dz == 0 ? zm : (dz == 1 ? z : zp);
            const int yy = dy == 0 ? ym : (dy == 1 ? y : yp);
            const int xx = dx == 0 ? xm : (dx == 1 ? x : xp);
            const __nv_bfloat16* src = in + (((long long)zz * p.ny + yy) * p.nx + xx) * cin;
            unsigned char* a = abuf(b);
            for (int q = 0; q < cin / 8; ++q)
                cp_async16_zfill(a + core_offset(tid, q, kTcM), src + q * 8, valid);
        }
        // B: the tap's weights [cout][cin]
        {
            const int per = cin / 8;
            const __nv_bfloat16* wt = p.w + ((size_t)tap * p.cout + o0) * cin;
            unsigned char* bm = bbuf(b);
            for (int i = tid; i < COUT * per; i += kTcThreads) {
                const int co = i / per;
                const int q = i - co * per;
                cp_async16_zfill(bm + core_offset(co, q, COUT), wt + (size_t)co * cin + q * 8, true);
            }
        }
    };

    bool ok = true;
#pragma unroll
    for (int tap = 0; tap < STAGES - 1; ++tap) {
        issue(tap);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int tap = 0; tap < 27; ++tap) {
        const int b = tap % STAGES;
        // this thread's copies of the tap, then everybody's
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        fence_proxy_async_smem();
        __syncthreads();
        if (*failed) {
            ok = false;
            break;
        }
        if (tid == 0) {
            tc_fence_after();
            const unsigned char* a = abuf(b);
            const unsigned char* bm = bbuf(b);
            for (int k = 0; k < kc; ++k) {
                const uint64_t ad = smem_desc(a + (size_t)k * kTcM * 32);
                const uint64_t bd = smem_desc(bm + (size_t)k * COUT * 32);
                const uint32_t acc = (tap | k) != 0;
                asm volatile(
                    "{\n"
                    " .reg .pred p;\n"
                    " setp.ne.b32 p, %4, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
                    "}\n" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(idesc_bf16<COUT>()), "r"(acc)
                    : "memory");
            }
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                    smem_u32(&bars[b]))
                : "memory");
        }
        // tap + STAGES - 1 goes where the MMAs of tap - 1 read
        const int nt = tap + STAGES - 1;
        if (nt < 27) {
            if (tap >= 1 &&
                !mbar_wait_bounded(&bars[(tap - 1) % STAGES], (uint32_t)(((tap - 1) / STAGES) & 1)))
                *failed = 1;  // every thread sees it after the next barrier
            else
                issue(nt);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // the last commit covers every MMA issued before it
    if (ok) ok = mbar_wait_bounded(&bars[26 % STAGES], (uint32_t)((26 / STAGES) & 1));
    if (__syncthreads_or(!ok)) {
        ok = false;
        if (tid == 0) atomicExch(&g_tc_err, 1);
    }
    tc_fence_after();
    if (ok) {
        // epilogue: TMEM lanes 32w..32w+31 are the rows of warp w
        const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
        for (int c0 = 0; c0 < COUT; c0 += 16) store_rows(trow, c0, o0, p.bias, p.relu, valid, v, p.cout, p.out32, p.out16);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOLS)
                     : "memory");
}

// The same convolution (dilation 1) with the neighbourhood loaded once per tile.
// Positions are linear in a sample's volume padded by one voxel along x and y
// (rows of nx + 2, planes of ny + 2 rows), so the neighbours of 128 consecutive
// positions in one plane are the same positions shifted by dy (nx + 2) + dx: a
// CTA copies the 128 + 2 (nx + 3) voxel rows of the three planes z - 1, z, z + 1
// into shared memory as K-major core matrices with the rows 16 bytes apart
// (stride byte offset 128, one plane per eight channels), and each tap's A
// operand is the start address moved by its shift.  All 27 taps' MMAs issue
// without another barrier, and a voxel's row is read about 4 times per tile
// position instead of 27 times.  Positions on the padding compute values nobody
// reads.  The weights stay in shared memory over a CTA's tiles.  Against the per-tap
// form: four 32^3 cells 16 -> 32 channels 77 -> 35 us, 32 -> 16 116 -> 42, four 64^3
// cells 16 -> 16 326 -> 126 (the copies into shared memory bound it).
struct HaloConv {
    int nx, ny, nz, samples;
    long long n;
    int sign;
    const __nv_bfloat16* in;
    int cin, cout;
    const __nv_bfloat16* w;
    const float* bias;
    int relu;
    float* out32;
    __nv_bfloat16* out16;
    int pitch, plane;       // nx + 2, (nx + 2) (ny + 2)
    int rows;               // voxel rows of one plane segment: 128 + 2 (pitch + 1)
    int tiles;              // tiles per sample
    long long ntiles;
};

template <int COUT>
__global__ void __launch_bounds__(kTcThreads) k_conv_halo(const __grid_constant__ HaloConv p) {
    constexpr int NCOLS = COUT < 32 ? 32 : COUT;
    extern __shared__ __align__(1024) unsigned char sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + 64);
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int cin = p.cin;
    const int kc = cin / 16, per = cin / 8;
    const int o0 = blockIdx.y * COUT;
    unsigned char* wsm = sm + 1024;                          // [27][cin/16][COUT * 32 bytes]
    unsigned char* asm_ = wsm + (size_t)27 * COUT * cin * 2;  // [cin/8][3][rows] 16-byte rows
    const int seg_rows = 3 * p.rows;
    const int last = p.nz * p.plane;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tslot)),
                     "r"(NCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    // the weights of this CTA's output channels
    for (int i = tid; i < 27 * COUT * per; i += kTcThreads) {
        const int tap = i / (COUT * per), e = i - tap * COUT * per;
        const int co = e / per, q = e - co * per;
        cp_async16_zfill(wsm + (size_t)tap * COUT * cin * 2 + core_offset(co, q, COUT),
                         p.w + ((size_t)tap * p.cout + o0 + co) * cin + q * 8, true);
    }
    auto load = [&](long long tile) {
        const int smp = (int)(tile / p.tiles);
        const int j0 = (int)(tile - (long long)smp * p.tiles) * kTcM;
        const __nv_bfloat16* in = p.in + (size_t)smp * p.n * cin;
        for (int r = tid; r < seg_rows; r += kTcThreads) {
            const int seg = r / p.rows, t = r - seg * p.rows;
            const int j = j0 - (p.pitch + 1) + t;
            const bool ok = j >= 0 && j < last;
            const int jj = ok ? j : 0;
            int z = jj / p.plane;
            const int rem = jj - z * p.plane;
            const int yp = rem / p.pitch, xp = rem - yp * p.pitch;
            const int y = yp == 0 ? p.ny - 1 : (yp > p.ny ? 0 : yp - 1);
            const int x = xp == 0 ? p.nx - 1 : (xp > p.nx ? 0 : xp - 1);
            z += seg - 1;
            z = z < 0 ? p.nz - 1 : (z >= p.nz ? 0 : z);
            const __nv_bfloat16* src = in + ((size_t)((long long)z * p.ny + y) * p.nx + x) * cin;
            for (int q = 0; q < per; ++q)
                cp_async16_zfill(asm_ + ((size_t)q * seg_rows + r) * 16, src + q * 8, ok);
        }
    };
    long long tile = blockIdx.x;
    if (tile < p.ntiles) load(tile);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    bool ok = true;
    for (uint32_t it = 0; tile < p.ntiles; tile += gridDim.x, ++it) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        fence_proxy_async_smem();
        tc_fence_before();  // the epilogue's TMEM reads of the tile before
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            for (int tap = 0; tap < 27; ++tap) {
                const int dz = p.sign * (tap / 9 - 1), sh = p.sign * ((tap / 3 % 3 - 1) * p.pitch + tap % 3 - 1);
                const unsigned char* a = asm_ + ((size_t)(dz + 1) * p.rows + p.pitch + 1 + sh) * 16;
                const unsigned char* bm = wsm + (size_t)tap * COUT * cin * 2;
                for (int k = 0; k < kc; ++k) {
                    const uint64_t ad = smem_desc_rows(a + (size_t)2 * k * seg_rows * 16, (uint32_t)seg_rows);
                    const uint64_t bd = smem_desc(bm + (size_t)k * COUT * 32);
                    const uint32_t acc = (tap | k) != 0;
                    asm volatile(
                        "{\n"
                        " .reg .pred p;\n"
                        " setp.ne.b32 p, %4, 0;\n"
                        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
                        "}\n" ::"r"(tmem),
                        "l"(ad), "l"(bd), "r"(idesc_bf16<COUT>()), "r"(acc)
                        : "memory");
                }
            }
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                : "memory");
        }
        // the position of this thread's accumulator row, while the MMAs run
        const int smp = (int)(tile / p.tiles);
        const int j = (int)(tile - (long long)smp * p.tiles) * kTcM + tid;
        const int z = j / p.plane, rem = j - z * p.plane;
        const int yp = rem / p.pitch, xp = rem - yp * p.pitch;
        const bool valid = j < last && yp >= 1 && yp <= p.ny && xp >= 1 && xp <= p.nx;
        const long long v = smp * p.n + ((long long)z * p.ny + yp - 1) * p.nx + xp - 1;
        ok = mbar_wait_bounded(bar, it & 1u);
        if (__syncthreads_or(!ok)) {
            ok = false;
            if (tid == 0) atomicExch(&g_tc_err, 1);
            break;
        }
        tc_fence_after();
        if (tile + gridDim.x < p.ntiles) load(tile + gridDim.x);  // the MMAs have read this tile's rows
        const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
        for (int c0 = 0; c0 < COUT; c0 += 16) store_rows(trow, c0, o0, p.bias, p.relu, valid, v, p.cout, p.out32, p.out16);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOLS)
                     : "memory");
}

// the largest dynamic shared memory a CTA may use, set once per kernel and device
template <typename K>
void ensure_smem_limit(K kern, std::atomic<unsigned long long>& done) {
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(done.load(std::memory_order_acquire) & bit)) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
        done.fetch_or(bit, std::memory_order_release);
    }
}

}  // namespace
}  // namespace fp

extern "C" int fp_nn_conv_tc(int nx, int ny, int nz, int64_t total, int dilation, int sign,
                             const void* in_bf16, int cin, const void* w_bf16, const float* bias,
                             int cout, int relu, float* out_f32, void* out_bf16, void* stream) {
    if (nx <= 0 || ny <= 0 || nz <= 0 || total <= 0 || cin <= 0 || cin % 16 || cin > 128 ||
        !in_bf16 || !w_bf16 || (!out_f32 && !out_bf16))
        return FP_ERR_INVALID;
    if (dilation < 1 || (sign != 1 && sign != -1)) return FP_ERR_INVALID;
    fp::TcConv p{nx, ny, nz, (long long)nx * ny * nz, (long long)total, dilation, sign,
                 static_cast<const __nv_bfloat16*>(in_bf16), cin, cout,
                 static_cast<const __nv_bfloat16*>(w_bf16), bias, relu, out_f32,
                 static_cast<__nv_bfloat16*>(out_bf16)};
    if (p.total % p.n) return FP_ERR_INVALID;
    const long long blocks = (p.total + fp::kTcM - 1) / fp::kTcM;
    if (blocks > 0x7fffffffLL) return FP_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (cout != 16 && cout != 32 && cout != 64 && cout != 128) return FP_ERR_INVALID;
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const fp::ConvCall call{nx, ny, nz, p.total / p.n, dilation, cin, cout, sms};
    const fp::ConvPlan plan = fp::conv_plan(call);
    const unsigned splits = (unsigned)(cout / plan.tile);
    if (plan.halo) {
        fp::HaloConv h{};
        h.nx = nx;
        h.ny = ny;
        h.nz = nz;
        h.samples = (int)call.samples;
        h.n = p.n;
        h.sign = sign;
        h.in = p.in;
        h.cin = cin;
        h.cout = cout;
        h.w = p.w;
        h.bias = bias;
        h.relu = relu;
        h.out32 = p.out32;
        h.out16 = p.out16;
        h.pitch = nx + 2;
        h.plane = (nx + 2) * (ny + 2);
        h.rows = (int)fp::conv_halo_rows(nx);
        h.ntiles = fp::conv_halo_tiles(call);
        h.tiles = (int)(h.ntiles / h.samples);
        const size_t smem = fp::conv_halo_smem(nx, cin, plan.tile);
        const unsigned gx = (unsigned)fp::conv_halo_grid(call, plan.tile);
#define FP_HALO_LAUNCH(C)                                                                \
    {                                                                                    \
        static std::atomic<unsigned long long> done_{0};                                 \
        fp::ensure_smem_limit(fp::k_conv_halo<C>, done_);                                \
        FP_LAUNCHED();                                                                   \
        fp::k_conv_halo<C><<<dim3(gx, splits), fp::kTcThreads, smem, s>>>(h);            \
    }
        switch (plan.tile) {
            case 16: FP_HALO_LAUNCH(16) break;
            case 32: FP_HALO_LAUNCH(32) break;
            case 64: FP_HALO_LAUNCH(64) break;
            default: FP_HALO_LAUNCH(128) break;
        }
#undef FP_HALO_LAUNCH
        return cudaGetLastError() == cudaSuccess ? FP_OK : FP_ERR_CUDA;
    }
    const size_t smem = fp::conv_tap_smem(cin, plan.tile, plan.stages);
#define FP_TC_LAUNCH(C, S)                                                                        \
    case C * 10 + S: {                                                                            \
        static std::atomic<unsigned long long> done_{0};                                          \
        fp::ensure_smem_limit(fp::k_conv_tc<C, S>, done_);                                        \
        FP_LAUNCHED();                                                                            \
        fp::k_conv_tc<C, S><<<dim3((unsigned)blocks, splits), fp::kTcThreads, smem, s>>>(p);      \
    } break;
    switch (plan.tile * 10 + plan.stages) {
        FP_TC_LAUNCH(16, 2) FP_TC_LAUNCH(16, 3) FP_TC_LAUNCH(16, 4)
        FP_TC_LAUNCH(32, 2) FP_TC_LAUNCH(32, 3) FP_TC_LAUNCH(32, 4)
        FP_TC_LAUNCH(64, 2) FP_TC_LAUNCH(64, 3) FP_TC_LAUNCH(64, 4)
        FP_TC_LAUNCH(128, 2) FP_TC_LAUNCH(128, 3) FP_TC_LAUNCH(128, 4)
        default: return FP_ERR_INVALID;
    }
#undef FP_TC_LAUNCH
    return cudaGetLastError() == cudaSuccess ? FP_OK : FP_ERR_CUDA;
}

extern "C" int fp_nn_tc_error(int* flag, int reset) {
    int h = 0;
    if (cudaMemcpyFromSymbol(&h, fp::g_tc_err, sizeof(int)) != cudaSuccess) return FP_ERR_CUDA;
    if (flag) *flag = h;
    if (reset) {
        const int z = 0;
        if (cudaMemcpyToSymbol(fp::g_tc_err, &z, sizeof(int)) != cudaSuccess) return FP_ERR_CUDA;
    }
    return FP_OK;
}
