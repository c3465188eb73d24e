// wgrad.cuh -- the weight gradient of a 3x3x3 convolution as per-tap GEMMs over
// voxels, dW[tap][o][i] = sum_v dy[v][o] x[v + off(tap)][i], on mma.sync
// (learned.cu, learned_unet.cu).
//
// A CTA of eight warps takes one voxel chunk, TAPS neighbouring taps (along x)
// and an MB x NB block of channels.  The warps share out the chunk's 16-voxel
// steps; each keeps its own three-stage cp.async ring of voxel rows (one dy row
// for all taps, one x row per tap), read back transposed by ldmatrix, and its
// own FP32 accumulators, which are summed over the warps in a fixed order.  A
// lane always copies the same row of a step, so the voxel's coordinates advance
// by additions.  The loads bound it, not the MMAs: the former kernel (one warp
// per tap and chunk, two-byte loads, four coordinate divisions per step and
// lane) made a layer's training step (four 32^3 cells, 16 -> 32 channels: forward,
// data, weight and bias gradients) 831 us, with this one and the bias gradient's
// cluster 234.
// Needs channel counts that are multiples of 16 and 16-byte aligned tensors.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "tma.cuh"

namespace fp {

struct WgradArgs {
    int nx, ny, nz;
    long long n, total;  // voxels per sample, voxels of all samples
    int dil;
    const __nv_bfloat16* dy;
    int cout;
    const __nv_bfloat16* x;
    int cin;
    long long chunk;
    float* partial;  // [chunk][tap][cout][cin]
    float* dw;       // [tap][cout][cin]
};

constexpr int kWgWarps = 8;
constexpr int kWgStages = 3;

template <int MB, int NB, int TAPS>
__host__ __device__ constexpr int wg_stage_bytes() {
    return 16 * (MB * 2 + 16) + TAPS * 16 * (NB * 2 + 16);  // rows padded by 16 bytes (banks)
}
template <int MB, int NB, int TAPS>
__host__ __device__ constexpr int wg_smem_bytes() {
    constexpr int ring = kWgWarps * kWgStages * wg_stage_bytes<MB, NB, TAPS>();
    constexpr int sums = kWgWarps * TAPS * MB * NB * 4;
    return ring > sums ? ring : sums;
}

__device__ __forceinline__ void wg_copy16(void* smem, const void* gmem, bool valid) {
    const int n = valid ? 16 : 0;  // src-size 0: zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem)), "l"(gmem), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void wg_ldmatrix_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void wg_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int MB, int NB, int TAPS>
__global__ void __launch_bounds__(32 * kWgWarps) k_wgrad_ring(const __grid_constant__ WgradArgs p) {
    constexpr int MT = MB / 16, NT = NB / 8;
    constexpr int DYS = MB * 2 + 16, XS = NB * 2 + 16;  // row strides in bytes
    constexpr int STAGE = wg_stage_bytes<MB, NB, TAPS>();
    extern __shared__ __align__(128) unsigned char sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* ring = sm + warp * kWgStages * STAGE;
    const long long ck = blockIdx.x;
    const int tap0 = blockIdx.y * TAPS;
    const int nbi = p.cin / NB;
    const int o0 = (blockIdx.z / nbi) * MB, i0 = (blockIdx.z % nbi) * NB;
    const long long v_begin = ck * p.chunk;
    const long long v_end = v_begin + p.chunk < p.total ? v_begin + p.chunk : p.total;
    const int steps = (int)((v_end - v_begin + 15) / 16);

    // this lane's row of a step, its coordinates, and their increment per turn
    const int row = lane >> 1, piece = lane & 1;
    long long v = v_begin + 16LL * warp + row;
    long long b = v / p.n;
    int x, y, z, sx, sy, sz;
    long long sb;
    {
        const int r = (int)(v - b * p.n);
        x = r % p.nx;
        y = r / p.nx % p.ny;
        z = r / p.nx / p.ny;
        const long long st = 16LL * kWgWarps;
        sb = st / p.n;
        const int q = (int)(st - sb * p.n);
        sx = q % p.nx;
        sy = q / p.nx % p.ny;
        sz = q / p.nx / p.ny;
    }
    auto wrap = [](int d, int n) { return ((d % n) + n) % n; };
    const int oz = wrap(p.dil * (tap0 / 9 - 1), p.nz), oy = wrap(p.dil * (tap0 / 3 % 3 - 1), p.ny);
    int ox[TAPS];
#pragma unroll
    for (int t = 0; t < TAPS; ++t) ox[t] = wrap(p.dil * ((tap0 + t) % 3 - 1), p.nx);

    auto issue = [&](int st) {
        unsigned char* d = ring + st * STAGE + row * DYS;
        const bool ok = v < v_end;
        const __nv_bfloat16* src = p.dy + (ok ? v : 0) * p.cout + o0;
#pragma unroll
        for (int i = 0; i < MT; ++i) wg_copy16(d + (piece + 2 * i) * 16, src + (piece + 2 * i) * 8, ok);
        const int zz = z + oz < p.nz ? z + oz : z + oz - p.nz;
        const int yy = y + oy < p.ny ? y + oy : y + oy - p.ny;
        const long long line = ((b * p.nz + zz) * p.ny + yy) * p.nx;
#pragma unroll
        for (int t = 0; t < TAPS; ++t) {
            const int xx = x + ox[t] < p.nx ? x + ox[t] : x + ox[t] - p.nx;
            const __nv_bfloat16* xs = p.x + (ok ? line + xx : 0) * p.cin + i0;
            unsigned char* e = ring + st * STAGE + 16 * DYS + (t * 16 + row) * XS;
#pragma unroll
            for (int i = 0; i < NB / 16; ++i) wg_copy16(e + (piece + 2 * i) * 16, xs + (piece + 2 * i) * 8, ok);
        }
        // the next step of this warp
        v += 16LL * kWgWarps;
        x += sx;
        if (x >= p.nx) x -= p.nx, ++y;
        y += sy;
        if (y >= p.ny) y -= p.ny, ++z;
        z += sz;
        if (z >= p.nz) z -= p.nz, ++b;
        b += sb;
    };

    float acc[TAPS][MT][NT][4] = {};
    const int mine = warp < steps ? (steps - 1 - warp) / kWgWarps + 1 : 0;
#pragma unroll
    for (int s = 0; s < kWgStages - 1; ++s) {
        if (s < mine) issue(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int s = 0; s < mine; ++s) {
        if (s + kWgStages - 1 < mine) issue((s + kWgStages - 1) % kWgStages);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group %0;" ::"n"(kWgStages - 1) : "memory");
        __syncwarp();
        const uint32_t base = smem_u32(ring + (s % kWgStages) * STAGE);
        uint32_t a[MT][4];
        // dy^T: matrices (k 0-7 | 8-15) x (m 0-7 | 8-15)
#pragma unroll
        for (int m = 0; m < MT; ++m)
            wg_ldmatrix_trans(a[m], base + ((lane & 7) + (lane >> 4) * 8) * DYS + (m * 16 + ((lane >> 3) & 1) * 8) * 2);
#pragma unroll
        for (int t = 0; t < TAPS; ++t)
#pragma unroll
            for (int q = 0; q < NT / 2; ++q) {
                uint32_t bb[4];
                wg_ldmatrix_trans(bb, base + 16 * DYS + (t * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * XS +
                                          (q * 16 + (lane >> 4) * 8) * 2);
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    wg_mma(acc[t][m][2 * q], a[m], bb[0], bb[1]);
                    wg_mma(acc[t][m][2 * q + 1], a[m], bb[2], bb[3]);
                }
            }
        __syncwarp();  // the stage is refilled by the next issue
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // sums over the warps, in warp order
    float* sums = reinterpret_cast<float*>(sm);
#pragma unroll
    for (int t = 0; t < TAPS; ++t)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int q = 0; q < NT; ++q)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int o = m * 16 + (lane >> 2) + (r >> 1) * 8, i = q * 8 + (lane & 3) * 2 + (r & 1);
                    sums[((warp * TAPS + t) * MB + o) * NB + i] = acc[t][m][q][r];
                }
    __syncthreads();
    for (int e = threadIdx.x; e < TAPS * MB * NB; e += 32 * kWgWarps) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < kWgWarps; ++w) s += sums[w * TAPS * MB * NB + e];
        const int t = e / (MB * NB), o = e / NB % MB, i = e % NB;
        p.partial[((ck * 27 + tap0 + t) * p.cout + o0 + o) * p.cin + i0 + i] = s;
    }
}

// dW[e] = sum over the chunks' partial sums: a CTA of 256 threads takes 32
// entries, eight threads each over every eighth chunk (fixed order).
static __global__ void __launch_bounds__(256) k_wgrad_sum(const float* __restrict__ partial, long long nchunks,
                                                          long long m, float* __restrict__ dw) {
    __shared__ float red[8][32];
    const int part = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long e = blockIdx.x * 32LL + lane;
    float s = 0.f;
    if (e < m)
        for (long long c = part; c < nchunks; c += 8) s += partial[c * m + e];
    red[part][lane] = s;
    __syncthreads();
    if (part == 0 && e < m) {
#pragma unroll
        for (int q = 1; q < 8; ++q) s += red[q][lane];
        dw[e] = s;
    }
}

template <int MB, int NB, int TAPS>
inline cudaError_t wgrad_launch(const WgradArgs& p, long long nchunks, cudaStream_t s) {
    constexpr int smem = wg_smem_bytes<MB, NB, TAPS>();
    static_assert(smem <= 227 * 1024, "shared memory");
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(done.load(std::memory_order_acquire) & bit)) {
        const cudaError_t e =
            cudaFuncSetAttribute(k_wgrad_ring<MB, NB, TAPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        done.fetch_or(bit, std::memory_order_release);
    }
    FP_LAUNCHED();
    k_wgrad_ring<MB, NB, TAPS><<<dim3((unsigned)nchunks, 27 / TAPS, (unsigned)((p.cout / MB) * (p.cin / NB))),
                                 32 * kWgWarps, smem, s>>>(p);
    const long long m = 27LL * p.cout * p.cin;
    FP_LAUNCHED();
    k_wgrad_sum<<<(unsigned)((m + 31) / 32), 256, 0, s>>>(p.partial, nchunks, m, p.dw);
    return cudaGetLastError();
}

// The channel block is the largest of 64, 32, 16 that divides each count; three
// taps share a dy row where their accumulators fit the registers (MB * NB <= 1024).
inline cudaError_t wgrad_ring(const WgradArgs& p, cudaStream_t s) {
    const long long nchunks = (p.total + p.chunk - 1) / p.chunk;
    const int mb = p.cout % 64 == 0 ? 64 : (p.cout % 32 == 0 ? 32 : 16);
    const int nb = p.cin % 64 == 0 ? 64 : (p.cin % 32 == 0 ? 32 : 16);
    switch (mb * 100 + nb) {
        case 1616: return wgrad_launch<16, 16, 3>(p, nchunks, s);
        case 1632: return wgrad_launch<16, 32, 3>(p, nchunks, s);
        case 1664: return wgrad_launch<16, 64, 3>(p, nchunks, s);
        case 3216: return wgrad_launch<32, 16, 3>(p, nchunks, s);
        case 3232: return wgrad_launch<32, 32, 3>(p, nchunks, s);
        case 3264: return wgrad_launch<32, 64, 1>(p, nchunks, s);
        case 6416: return wgrad_launch<64, 16, 3>(p, nchunks, s);
        case 6432: return wgrad_launch<64, 32, 1>(p, nchunks, s);
        default: return wgrad_launch<64, 64, 1>(p, nchunks, s);
    }
}

// the rule of the entry points: rows and tensors of whole 16-byte pieces, and
// samples of at most 2^31 voxels
inline bool wgrad_ring_ok(const WgradArgs& p) {
    return p.cout % 16 == 0 && p.cin % 16 == 0 && p.n <= 0x7fffffffLL &&
           ((reinterpret_cast<uintptr_t>(p.dy) | reinterpret_cast<uintptr_t>(p.x)) & 15) == 0;
}

}  // namespace fp
