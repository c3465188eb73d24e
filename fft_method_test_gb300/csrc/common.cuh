// common.cuh -- shared device helpers for the GB300 permeability kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace fp {

// Process-wide count of this library's kernel launches (all devices and
// streams), read by fp_kernel_launch_count.  Every launch site bumps it.
extern std::atomic<long long> g_kernel_launches;
// The calling thread's own launches (a stream capture subtracts what it
// recorded: other threads keep launching meanwhile).
extern thread_local long long g_thread_launches;
#define FP_LAUNCHED() \
    (++::fp::g_thread_launches, ::fp::g_kernel_launches.fetch_add(1, std::memory_order_relaxed))

// ---- programmatic dependent launch ----
// Kernels of a chain (operator passes, MINRES and Brinkman iterations) start
// with pdl_wait(): everything before this kernel in the stream has completed
// and its writes are visible.  Their launch and block start-up overlap the end
// of the kernel before; with pdl_trigger() near the end of a block's work the
// next kernel's blocks are placed that much earlier.  Measured per mixed apply
// with its reduction to alpha (fp_time_apply, without | with the launch attribute):
// 48^3 28.7 | 17.4 us, 64^3 30.8 | 21.9, 96^3 55.2 | 45.1, 128^3 76.4 | 65.2, 256^3
// 456 | 443.  (A caller who launches one apply at a time waits for the host: 40 us
// at 48^3 either way.)
// Only the FP32 forward x, y and z passes trigger.  A kernel whose successor is
// bound by the FP64 pipe must not: blocks placed while other blocks still run
// go to the SMs that have room, and the fullest SM's pipe sets the time (FP64
// apply at 64^3: 114 us without, 166 us with triggers).  Nor may a trigger come
// at the start of a kernel: several waiting kernels then pile up on the SMs
// (64^3 solve 58 -> 123 ms).
// Every kernel launched through launch_pdl calls pdl_wait before its first
// access to memory that another kernel writes and before any return, and none
// of its parameters is `const __restrict__`: loads through such a pointer count
// as invariant and may be moved above the wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    FP_LAUNCHED();
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

// ---- device memory vs graph capture (capi.cu) ----
// cudaMalloc / cudaFree may synchronise the whole device, which invalidates a
// stream capture running in another host thread.  Every allocation or free
// site holds DeviceMemGuard (exclusive, re-entrant within a thread); every
// capture holds CaptureGuard (shared: captures in different threads overlap).
struct DeviceMemGuard {
    DeviceMemGuard();
    ~DeviceMemGuard();
    DeviceMemGuard(const DeviceMemGuard&) = delete;
    DeviceMemGuard& operator=(const DeviceMemGuard&) = delete;
};
struct CaptureGuard {
    CaptureGuard();
    ~CaptureGuard();
    CaptureGuard(const CaptureGuard&) = delete;
    CaptureGuard& operator=(const CaptureGuard&) = delete;
};


template <typename T>
struct Cplx;
template <>
struct Cplx<double> {
    using type = double2;
};
template <>
struct Cplx<float> {
    using type = float2;
};
template <typename T>
using c_t = typename Cplx<T>::type;

template <typename T2>
__device__ __forceinline__ T2 cmk(decltype(T2::x) a, decltype(T2::x) b) {
    T2 r;
    r.x = a;
    r.y = b;
    return r;
}
template <typename T2>
__device__ __forceinline__ T2 cadd(T2 a, T2 b) {
    return cmk<T2>(a.x + b.x, a.y + b.y);
}
template <typename T2>
__device__ __forceinline__ T2 csub(T2 a, T2 b) {
    return cmk<T2>(a.x - b.x, a.y - b.y);
}
template <typename T2>
__device__ __forceinline__ T2 cmul(T2 a, T2 b) {
    return cmk<T2>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// FP32 complex values as packed pairs: one f32x2 instruction does both parts
// (each rounded as the scalar operation rounds).  The FP32 passes are bound by
// instruction issue as much as by memory, and the packed form takes half the
// issue slots at the same FP32 rate (measured: 120 lane operations per clock
// and SM either way, 60 packed instructions).
__device__ __forceinline__ unsigned long long f2_bits(float2 a) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 bits_f2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
template <>
__device__ __forceinline__ float2 cadd<float2>(float2 a, float2 b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
    return bits_f2(r);
}
template <>
__device__ __forceinline__ float2 csub<float2>(float2 a, float2 b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
    return bits_f2(r);
}
template <typename T2>
__device__ __forceinline__ T2 cscale(T2 a, decltype(T2::x) s) {
    return cmk<T2>(a.x * s, a.y * s);
}
template <>
__device__ __forceinline__ float2 cscale<float2>(float2 a, float s) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(make_float2(s, s))));
    return bits_f2(r);
}

// a + sign*i*b and a - sign*i*b as two scalar additions: the rotated operand is
// never formed (a packed addition would have to swap its halves first)
template <int SIGN, typename T2>
__device__ __forceinline__ T2 cadd_si(T2 a, T2 b) {
    return SIGN < 0 ? cmk<T2>(a.x + b.y, a.y - b.x) : cmk<T2>(a.x - b.y, a.y + b.x);
}
template <int SIGN, typename T2>
__device__ __forceinline__ T2 csub_si(T2 a, T2 b) {
    return cadd_si<-SIGN>(a, b);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double pick(bool c, double a, double b) { return c ? a : b; }

// Sums over a warp of NV (1, 2 or 4) doubles per lane in the order of warp_sum
// (xor 16, 8, 4, 2, 1).  GB300 issues one FP64 warp instruction per 16 clocks
// and SM, so with several values the lanes split them at the first steps: 6
// additions for four values instead of 20 (5 instead of 10 for two), with the
// same bits.  Lane l returns the sum of value l / (32 / NV).
template <int NV>
__device__ __forceinline__ double warp_sum_split(const double (&v)[NV], int lane) {
    static_assert(NV == 1 || NV == 2 || NV == 4, "values per lane");
    constexpr unsigned kAll = 0xffffffffu;
    double a;
    if constexpr (NV == 4) {
        const bool h = lane & 16;
        const double a0 = pick(h, v[2], v[0]) + __shfl_xor_sync(kAll, pick(h, v[0], v[2]), 16);
        const double a1 = pick(h, v[3], v[1]) + __shfl_xor_sync(kAll, pick(h, v[1], v[3]), 16);
        const bool q = lane & 8;
        a = pick(q, a1, a0) + __shfl_xor_sync(kAll, pick(q, a0, a1), 8);
    } else if constexpr (NV == 2) {
        const bool h = lane & 16;
        a = pick(h, v[1], v[0]) + __shfl_xor_sync(kAll, pick(h, v[0], v[1]), 16);
        a += __shfl_xor_sync(kAll, a, 8);
    } else {
        a = v[0] + __shfl_xor_sync(kAll, v[0], 16);
        a += __shfl_xor_sync(kAll, a, 8);
    }
    a += __shfl_xor_sync(kAll, a, 4);
    a += __shfl_xor_sync(kAll, a, 2);
    a += __shfl_xor_sync(kAll, a, 1);
    return a;
}

// Second stage of a block reduction: the first warp sums scratch[32 * j + w]
// over the block's warps w; every lane of it gets the totals.  Callers put a
// barrier before it.
template <int NV>
__device__ __forceinline__ void sum_warps(const double* scratch, double (&out)[NV]) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int nwarp = (blockDim.x + 31) >> 5;
    if (nwarp <= 8) {  // eight lanes per value: the zeros of the wider tree change nothing
        const int j = lane >> 3, w = lane & 7;
        double v = (j < NV && w < nwarp) ? scratch[32 * j + w] : 0.0;
        v += __shfl_xor_sync(kAll, v, 4);
        v += __shfl_xor_sync(kAll, v, 2);
        v += __shfl_xor_sync(kAll, v, 1);
#pragma unroll
        for (int i = 0; i < NV; ++i) out[i] = __shfl_sync(kAll, v, 8 * i);
    } else {
#pragma unroll
        for (int i = 0; i < NV; ++i) out[i] = warp_sum(lane < nwarp ? scratch[32 * i + lane] : 0.0);
    }
}

// Deterministic block reduction of NV (1, 2 or 4) doubles per thread.  Every
// thread contributes vals[0..NV); the threads of the first warp get the block
// totals in out[0..NV).  scratch: shared array of at least NV * 32 doubles.
template <int NV>
__device__ __forceinline__ void block_sum(double (&vals)[NV], double* scratch, double (&out)[NV]) {
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const double v = warp_sum_split<NV>(vals, lane);
    if (lane % (32 / NV) == 0) scratch[32 * (lane / (32 / NV)) + warp] = v;
    __syncthreads();
    if (warp == 0) sum_warps<NV>(scratch, out);
    __syncthreads();
}

// Column sums of the first NV (1, 2 or 4) columns of `nparts` partial rows of
// STRIDE doubles that other blocks wrote, by one whole block: a thread adds one
// column over its rows.  The threads of the first warp get the totals.
template <int NV, int STRIDE>
__device__ __forceinline__ void sum_rows(const double* partials, int nparts, double* scratch, double (&out)[NV]) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int j = threadIdx.x % NV;
    double v = 0.0;
    for (int r = threadIdx.x / NV; r < nparts; r += blockDim.x / NV) v += __ldcg(partials + (long long)STRIDE * r + j);
#pragma unroll
    for (int o = 16; o >= NV; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
    if (lane < NV) scratch[32 * lane + warp] = v;
    __syncthreads();
    if (warp == 0) sum_warps<NV>(scratch, out);
    __syncthreads();
}

}  // namespace fp
