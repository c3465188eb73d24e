// fft_fast.cuh -- the five apply passes specialised at compile time for 36 grid
// edges (32, 48, 64, 80, 96, 128, 160, 256 and those of fft_edges.cuh; the three
// edges of a grid may differ), for compact-vector operator applies (scatter in,
// gather out).  The generic engine of fft_passes.cuh serves every other edge,
// source and destination.
//
// Each line of length N = R1 * R2 is transformed by TPL threads with the
// four-step decomposition, one vector component per thread (where TPL does not
// divide a radix, a thread's last owner may be idle):
//
//   x[R2*i + a]  (i < R1, a < R2)
//   stage A  threads owning a: DFT-R1 over i, times W_N^(S a k) -> Y[k][a]
//   stage B  threads owning k: DFT-R2 over a                     -> X[k + R1*m]
//
// The inverse runs the same two stages with the radices swapped (R2 first).
// Only the Y exchange between the stages (and the natural-order exchange
// around the Green multiply) goes through shared memory; every stage reads
// or writes HBM directly where its owner pattern is the natural one.
//
// Passes (kernels below):
//   k_fx_fwd   scatter of the compact vector (minus its mean) into real
//              x-lines, two real lines per complex FFT, half spectrum out
//   k_fcol_y   y pass, one component per CTA slice, TX kx columns per CTA
//   k_fz       z pass: forward, 3x3 Green multiply, inverse, all three
//              components in one CTA; persistent CTAs with a two-stage TMA
//              pipeline (cp.async.bulk.tensor boxes of the spectral and Green
//              tiles of the next (kx, ky) tile load while the current one is
//              transformed)
//   k_fx_inv   C2R x lines, gather to the support, 1/N scale, per-CTA partial
//              sums (component sums and the dot with a given vector)
//
// Shared-memory line strides are chosen so that the half-warp (FP32) or
// quarter-warp (FP64) of every exchange touches distinct banks.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "fft_edges.cuh"
#include "fft_engine.cuh"
#include "internal.h"
#include "minres_device.cuh"
#include "tma.cuh"

namespace fp {
namespace fast {

// N = R1 * R2; TPL threads per line.  For these eight edges TPL divides R1 and
// R2 (R2 for the powers of two, 4 for the edges with a factor 3 or 5);
// fft_edges.cuh lists the others.
template <int N>
struct Split;
template <>
struct Split<32> {
    static constexpr int R1 = 8, R2 = 4, TPL = 4;
};
template <>
struct Split<48> {
    static constexpr int R1 = 12, R2 = 4, TPL = 4;
};
template <>
struct Split<64> {
    static constexpr int R1 = 8, R2 = 8, TPL = 8;
};
template <>
struct Split<80> {
    static constexpr int R1 = 20, R2 = 4, TPL = 4;
};
template <>
struct Split<96> {
    static constexpr int R1 = 12, R2 = 8, TPL = 4;
};
template <>
struct Split<128> {
    static constexpr int R1 = 16, R2 = 8, TPL = 8;
};
template <>
struct Split<160> {
    static constexpr int R1 = 20, R2 = 8, TPL = 4;
};
template <>
struct Split<256> {
    static constexpr int R1 = 16, R2 = 16, TPL = 16;
};

#define FP_SPLIT(N, A, B, T)                               \
    template <>                                            \
    struct Split<N> {                                      \
        static constexpr int R1 = A, R2 = B, TPL = T;      \
        static_assert(A * B == N && 32 % T == 0, "split"); \
    };
FP_EDGES_SMALL(FP_SPLIT)
FP_EDGES_MIDDLE(FP_SPLIT)
FP_EDGES_LARGE(FP_SPLIT)
#undef FP_SPLIT

// ---- small DFTs in natural order -------------------------------------------

template <int P, int Q, int S, typename T2>
__device__ __forceinline__ void dft_pfa(T2 (&v)[P * Q]);

// DFT9 as 3 x 3: n = 3 n1 + n2, k = k1 + 3 k2, twiddles W9^(n2 k1).
template <int S, typename T2>
__device__ __forceinline__ void dft9(T2 (&v)[9]) {
    using T = decltype(T2::x);
    const T c1 = (T)0.76604444311897803520, s1 = (T)0.64278760968653932632;   // 2 pi / 9
    const T c2 = (T)0.17364817766693034885, s2 = (T)0.98480775301220805937;   // 4 pi / 9
    const T c4 = (T)-0.93969262078590838405, s4 = (T)0.34202014332566873304;  // 8 pi / 9
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) dft3<S>(v[n2], v[3 + n2], v[6 + n2]);  // v[3 k1 + n2]
    v[4] = mul_const<S>(v[4], c1, s1);
    v[5] = mul_const<S>(v[5], c2, s2);
    v[7] = mul_const<S>(v[7], c2, s2);
    v[8] = mul_const<S>(v[8], c4, s4);
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) dft3<S>(v[3 * k1], v[3 * k1 + 1], v[3 * k1 + 2]);  // X[k1 + 3 k2]
    const T2 t[9] = {v[0], v[3], v[6], v[1], v[4], v[7], v[2], v[5], v[8]};
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = t[k];
}

// Natural-order DFT of R values (S = -1 forward, +1 backward) with the
// radix kernels of fft_engine.cuh (2, 3, 4, 5, 8, 16) and dft9; 6, 10, 12, 15,
// 18 and 20 by the prime-factor algorithm.
template <int R, int S, typename T2>
__device__ __forceinline__ void dft_nat(T2 (&v)[R]) {
    if constexpr (R == 6) {
        dft_pfa<2, 3, S>(v);
    } else if constexpr (R == 9) {
        dft9<S>(v);
    } else if constexpr (R == 10) {
        dft_pfa<2, 5, S>(v);
    } else if constexpr (R == 15) {
        dft_pfa<3, 5, S>(v);
    } else if constexpr (R == 18) {
        dft_pfa<2, 9, S>(v);
    } else if constexpr (R == 12) {
        dft_pfa<4, 3, S>(v);
    } else if constexpr (R == 20) {
        dft_pfa<4, 5, S>(v);
    } else {
        T2 t[R];
#pragma unroll
        for (int i = 0; i < R; ++i) t[i] = v[i];
        dft_r<R, S>(t);
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = t[out_slot<R>(k)];
    }
}

// Prime-factor (Good-Thomas) DFT of R = P * Q values, P and Q coprime: input
// n = (Q n1 + P n2) mod R goes to a[n1][n2], length-Q DFTs along n2, then
// length-P DFTs along n1, and output k is a[k mod P][k mod Q].  No twiddles
// (Chinese-remainder index maps).
template <int P, int Q, int S, typename T2>
__device__ __forceinline__ void dft_pfa(T2 (&v)[P * Q]) {
    constexpr int R = P * Q;
    T2 a[P][Q];
#pragma unroll
    for (int n1 = 0; n1 < P; ++n1)
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) a[n1][n2] = v[(Q * n1 + P * n2) % R];
#pragma unroll
    for (int n1 = 0; n1 < P; ++n1) dft_nat<Q, S>(a[n1]);
#pragma unroll
    for (int n2 = 0; n2 < Q; ++n2) {
        T2 c[P];
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) c[n1] = a[n1][n2];
        dft_nat<P, S>(c);
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) a[n1][n2] = c[n1];
    }
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = a[k % P][k % Q];
}

// Twiddle W_N^(S a k) of output k of owner a between the two stages, N = RA*RB.
// The tables hold them in the order the threads read them, [k][a], so that the
// owners of one warp instruction read neighbouring entries: indexing one table
// of N roots by a*k touches up to RB cache lines per load, and the L1 data pipe
// is the busiest unit of these passes (65-87 % of its peak under ncu).  Measured
// at 256^3 FP32: 431.6 -> 425.0 us per apply.
// The forward table [R1][R2] is followed by the inverse one [R2][R1], conjugated.
template <int RA, int RB, int S, typename T2>
__device__ __forceinline__ T2 twiddle(const T2* __restrict__ tw, int k, int a) {
    return __ldg(tw + (S > 0 ? RA * RB : 0) + k * RB + a);
}

// ---- line strides ------------------------------------------------------------

// Positions used in a line: the natural N plus the Y layout k*(RB+1) + a of
// either direction (RB = R2 forward, R1 inverse).
template <int N>
__host__ __device__ constexpr int line_span() {
    return N + (Split<N>::R1 > Split<N>::R2 ? Split<N>::R1 : Split<N>::R2);
}

// Column passes (thread = column + TX * (owner + TPL * comp)): one
// shared-memory wavefront serves G = 128 / sizeof(complex) threads (a
// half-warp in FP32, a quarter-warp in FP64), TX columns x G / TX
// consecutive owners; every exchange steps owners by an odd number of
// elements, so a line stride of G / TX modulo G keeps them in distinct banks.
template <int N, typename T, int TX>
__host__ __device__ constexpr int col_ld() {
    constexpr int G = 128 / (2 * (int)sizeof(T));
    return ((line_span<N>() + G - 1) / G) * G + (G / TX) % G;
}

// x passes (thread = owner + TPL * line): the lines of one half-warp (FP32)
// or quarter-warp (FP64) must fall in distinct banks, so for a power-of-two
// TPL below the group size G the stride is TPL mod G.
template <int N, typename T>
__host__ __device__ constexpr int x_ld() {
    constexpr int G = sizeof(T) == 4 ? 16 : 8;
    constexpr int tpl = Split<N>::TPL;
    constexpr int base = ((line_span<N>() + G - 1) / G) * G;
    return tpl < G ? base + tpl : base;
}

// ---- barriers -------------------------------------------------------------------

// the whole CTA
struct CtaBarrier {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
// the `count` threads (a multiple of 32) of one named barrier `id` (1..15)
struct GroupBarrier {
    int id, count;
    __device__ __forceinline__ void operator()() const {
        asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
    }
};

// one warp: the threads of a line in the x passes (TPL divides 32)
struct WarpBarrier {
    __device__ __forceinline__ void operator()() const { __syncwarp(); }
};

template <class B>
__device__ __forceinline__ B make_group_barrier(int id, int count);
template <>
__device__ __forceinline__ GroupBarrier make_group_barrier<GroupBarrier>(int id, int count) {
    return GroupBarrier{id, count};
}
template <>
__device__ __forceinline__ CtaBarrier make_group_barrier<CtaBarrier>(int, int) {
    return CtaBarrier{};
}

// ---- four-step stages --------------------------------------------------------

// owners of a thread among R; with TPL not dividing R the last may be idle
template <int R, int TPL>
__host__ __device__ constexpr int owners() {
    return (R + TPL - 1) / TPL;
}
template <int R, int TPL>
__device__ __forceinline__ bool owned(int k) {
    return R % TPL == 0 || k < R;
}

// Stage A for owners a = t + TPL*j (a < RB): loads RA values through
// load(pos) (pos = RB*i + a), DFT-RA, twiddle W_N^(S a k), stores Y[k][a] at
// line[k*(RB+1) + a].  With SYNC, bar() runs between the loads and the
// stores (the loads read the same lines).
template <int RA, int RB, int S, int TPL, bool SYNC, typename T2, class Load,
          class Bar = CtaBarrier>
__device__ __forceinline__ void stage_a(T2* line, int t, bool active, const T2* __restrict__ tw,
                                        Load& load, Bar bar = Bar{}) {
    constexpr int J = owners<RB, TPL>();
    T2 v[J][RA];
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const bool on = active && owned<RB, TPL>(t + TPL * j);
#pragma unroll
        for (int i = 0; i < RA; ++i) v[j][i] = on ? load(RB * i + t + TPL * j) : T2{};
    }
    if (SYNC) bar();
    if (active) {
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int a = t + TPL * j;
            if (!owned<RB, TPL>(a)) continue;
            dft_nat<RA, S>(v[j]);
#pragma unroll
            for (int k = 0; k < RA; ++k) {
                T2 y = v[j][k];
                if (k > 0) y = cmul(y, twiddle<RA, RB, S>(tw, k, a));
                line[k * (RB + 1) + a] = y;
            }
        }
    }
}

// Stage B for owners k = t + TPL*j (k < RA): loads Y[k][a] (a < RB),
// DFT-RB, hands X[k + RA*m] to store(pos, value).  With SYNC, bar() runs
// between the loads and the stores.
template <int RA, int RB, int S, int TPL, bool SYNC, typename T2, class Store,
          class Bar = CtaBarrier>
__device__ __forceinline__ void stage_b(const T2* line, int t, bool active, Store& store,
                                        Bar bar = Bar{}) {
    constexpr int J = owners<RA, TPL>();
    T2 u[J][RB];
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const bool on = active && owned<RA, TPL>(t + TPL * j);
#pragma unroll
        for (int a = 0; a < RB; ++a) u[j][a] = on ? line[(t + TPL * j) * (RB + 1) + a] : T2{};
    }
    if (SYNC) bar();
    if (active) {
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int k = t + TPL * j;
            if (!owned<RA, TPL>(k)) continue;
            dft_nat<RB, S>(u[j]);
#pragma unroll
            for (int m = 0; m < RB; ++m) store(k + RA * m, u[j][m]);
        }
    }
}

// Stage A with its inputs already in registers (z[j][i] = x[RB*i + t + TPL*j]);
// the line is free to be written.
template <int RA, int RB, int S, int TPL, typename T2>
__device__ __forceinline__ void stage_a_regs(T2* line, int t, bool active, const T2* __restrict__ tw,
                                             T2 (&z)[RB / TPL][RA]) {
    if (!active) return;
#pragma unroll
    for (int j = 0; j < RB / TPL; ++j) {
        const int a = t + TPL * j;
        dft_nat<RA, S>(z[j]);
#pragma unroll
        for (int k = 0; k < RA; ++k) {
            T2 y = z[j][k];
            if (k > 0) y = cmul(y, twiddle<RA, RB, S>(tw, k, a));
            line[k * (RB + 1) + a] = y;
        }
    }
}

// Stage B leaving its outputs in registers: z[j][m] = X[t + TPL*j + RA*m].
template <int RA, int RB, int S, int TPL, typename T2>
__device__ __forceinline__ void stage_b_regs(const T2* line, int t, bool active, T2 (&z)[RA / TPL][RB]) {
#pragma unroll
    for (int j = 0; j < RA / TPL; ++j)
#pragma unroll
        for (int a = 0; a < RB; ++a) z[j][a] = active ? line[(t + TPL * j) * (RB + 1) + a] : T2{};
#pragma unroll
    for (int j = 0; j < RA / TPL; ++j) dft_nat<RB, S>(z[j]);
}

// ---- spectral layout -----------------------------------------------------------

// The spectral field between the specialised passes is blocked over kx in
// tiles of kt = 2^ktl columns: element (comp, kx, ky, kz) sits at
//   comp * nh + (kx / kt) * kts + (kz * ny + ky) * kt + kx % kt,  kts = kt * ny * nz,
// so a y line of a tile is one contiguous block and the lines of a z tile are
// ny * kt elements apart.  kt is the number of threads of an x line: a load or
// store of the x passes covers one tile row whole (with a narrower tile it
// touched a cache line per 32 bytes).  Measured per mixed apply, [kz][ky][kx]
// against this layout: 64^3 32.7 -> 30.4 us, 128^3 80.0 -> 74.9, 160^3 152.5 ->
// 140.2, 256^3 425 -> 431 (its y passes 72 -> 63 us, its x passes as much slower).
template <int N>
__host__ __device__ constexpr int kx_tile() {
    return Split<N>::TPL < 4 ? 4 : Split<N>::TPL;
}

// ---- kernel arguments ----------------------------------------------------------

struct FastArgs {
    int nx, ny, nz, nxh;
    long long nh, nrows, n;
    int ktl;        // log2 of the kx tile width
    long long kts;  // elements of one kx tile of a component
    const float2* tw32x;  // stage twiddles of the specialised edges (AxisPlan::fw32)
    const float2* tw32y;
    const float2* tw32z;
    const double2* tw64x;
    const double2* tw64y;
    const double2* tw64z;
    void* spec;
    const void* green;
    int* err;  // z pass: a bounded TMA wait gave up
    // x passes
    int rows;       // grid rows per tile (even)
    long long ntiles;
    const int* support;
    const int* row_ptr;
    const double* src;
    const double* src_sum;
    double inv_nb;
    double* dst;
    const double* dot_with;
    double scale;
    double* partials;
    const int* skip;
    // inverse x: the last block reduces the partial rows to the z mean and the
    // Lanczos alpha (null: the caller reduces them)
    MinresScalars* alpha_sc;
    unsigned int* alpha_ticket;
    double* sum_out;  // or to their four sums (null: the caller reduces them)
    // A group of problems of one grid in one launch per pass: when set, the
    // kernels (GROUP = true) take their member's arguments from group[p], p =
    // blockIdx.y (x and z passes) or blockIdx.z / 3 (y pass), and the z pass
    // its tensor maps from group_maps[2p] (spectral) and [2p + 1] (Green).
    const FastArgs* group;
    const CUtensorMap* group_maps;
    // members of a group whose z pass shares one Green table (group_maps[1]):
    // k_fz_shared loads each Green tile once for all of them (0 = not shared)
    int share;
};

template <typename T>
__device__ __forceinline__ const c_t<T>* tw_of(const FastArgs& a, int axis);
template <>
__device__ __forceinline__ const float2* tw_of<float>(const FastArgs& a, int axis) {
    return axis == 0 ? a.tw32x : (axis == 1 ? a.tw32y : a.tw32z);
}
template <>
__device__ __forceinline__ const double2* tw_of<double>(const FastArgs& a, int axis) {
    return axis == 0 ? a.tw64x : (axis == 1 ? a.tw64y : a.tw64z);
}

// A group member's arguments are copied out of the table into shared memory,
// where a single apply has them in the constant bank: kept in registers they
// cost the inverse x pass 109 instead of 80 registers per thread and half its
// warps (122 against 67 us per member at 256^3 FP32 under ncu), and through a
// reference to the table they would be reloaded after every global store.
template <bool GROUP>
struct ArgSlot {
    unsigned long long w[GROUP ? (sizeof(FastArgs) + 7) / 8 : 1];
};
template <bool GROUP>
__device__ __forceinline__ const FastArgs& member_args(const FastArgs& a0, int member, ArgSlot<GROUP>& slot) {
    if constexpr (GROUP) {
        static_assert(sizeof(FastArgs) % 8 == 0 && alignof(FastArgs) <= 8, "copied by 8-byte words");
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(a0.group + member);
        for (int i = threadIdx.x; i < (int)(sizeof(FastArgs) / 8); i += blockDim.x) slot.w[i] = src[i];
        __syncthreads();
        return *reinterpret_cast<const FastArgs*>(slot.w);
    } else {
        return a0;
    }
}

// ---- two real lines in one complex line --------------------------------------

// A thread t of a line's TPL threads holds Z[k] for k = t + TPL*j + R1*m in
// z[j][m] (j < R1/TPL, m < R2): the owners of the forward transform's stage B
// and of the inverse transform's stage A.  Z[N - k] then sits in register
// [J-1-j][R2-1-m] of thread (TPL - t) % TPL, except for t = 0, whose mirror
// images are its own registers: the two Hermitian halves meet through warp
// shuffles, without shared memory.

// That needs whole owners (TPL divides R1) and an even R2; other splits write
// the transformed line back and read the mirror images from shared memory.
template <int N>
__host__ __device__ constexpr bool mirrored() {
    return Split<N>::R1 % Split<N>::TPL == 0 && Split<N>::R2 % 2 == 0;
}

// the value of `v` in the mirror thread
template <int TPL>
__device__ __forceinline__ float2 shfl_mirror(float2 v, int t) {
    const int src = (TPL - t) & (TPL - 1);
    return make_float2(__shfl_sync(0xffffffffu, v.x, src, TPL), __shfl_sync(0xffffffffu, v.y, src, TPL));
}
template <int TPL>
__device__ __forceinline__ double2 shfl_mirror(double2 v, int t) {
    const int src = (TPL - t) & (TPL - 1);
    return make_double2(__shfl_sync(0xffffffffu, v.x, src, TPL), __shfl_sync(0xffffffffu, v.y, src, TPL));
}

template <class T2>
__device__ __forceinline__ T2 pick(bool c, T2 a, T2 b) {
    return cmk<T2>(c ? a.x : b.x, c ? a.y : b.y);
}

// Spectra of the two real lines of a forward line, each times two:
// store(k, 2 A[k], 2 B[k]) for this thread's k <= N/2.
template <int R1, int R2, int TPL, typename T2, class Store>
__device__ __forceinline__ void separate_lines(const T2 (&z)[R1 / TPL][R2], int t, Store& store) {
    static_assert(R2 % 2 == 0, "the half spectrum is the lower half of the outputs");
    constexpr int J = R1 / TPL;
#pragma unroll
    for (int m = 0; m < R2 / 2; ++m)
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const T2 own = j > 0 ? z[j > 0 ? J - j : 0][R2 - 1 - m] : z[0][(R2 - m) % R2];
            const T2 zn = pick(t == 0, own, shfl_mirror<TPL>(z[J - 1 - j][R2 - 1 - m], t));
            const T2 zk = z[j][m];
            store(t + TPL * j + R1 * m, cmk<T2>(zk.x + zn.x, zk.y - zn.y), cmk<T2>(zk.y + zn.y, zn.x - zk.x));
        }
    if (t == 0) {  // k = N/2 is its own mirror image
        using T = decltype(T2::x);
        const T2 zk = z[0][R2 / 2];
        store(R1 * R2 / 2, cmk<T2>(zk.x + zk.x, (T)0), cmk<T2>(zk.y + zk.y, (T)0));
    }
}

// The inverse: z[j][m] of Z = A + iB from the half spectra, load(k, A, B) for
// this thread's k <= N/2 (DC and Nyquist are real).
template <int R1, int R2, int TPL, typename T2, class Load>
__device__ __forceinline__ void join_lines(T2 (&z)[R1 / TPL][R2], int t, Load& load) {
    using T = decltype(T2::x);
    constexpr int J = R1 / TPL;
    constexpr int H = R2 / 2;
    T2 a[J][H], b[J][H], an{}, bn{};
#pragma unroll
    for (int m = 0; m < H; ++m)
#pragma unroll
        for (int j = 0; j < J; ++j) load(t + TPL * j + R1 * m, a[j][m], b[j][m]);
    if (t == 0) load(R1 * H, an, bn);
    if (t == 0) a[0][0].y = b[0][0].y = (T)0;
    T2 w[J][H];  // Z[N - k]
#pragma unroll
    for (int m = 0; m < H; ++m)
#pragma unroll
        for (int j = 0; j < J; ++j) {
            z[j][m] = cmk<T2>(a[j][m].x - b[j][m].y, a[j][m].y + b[j][m].x);
            w[j][m] = cmk<T2>(a[j][m].x + b[j][m].y, b[j][m].x - a[j][m].y);
        }
    const T2 nyq = cmk<T2>(an.x, bn.x);
#pragma unroll
    for (int m = 0; m < H; ++m)
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const T2 own = j + 1 < J ? w[j + 1 < J ? j + 1 : 0][m] : (m + 1 < H ? w[0][m + 1 < H ? m + 1 : 0] : nyq);
            z[J - 1 - j][R2 - 1 - m] = pick(t == 0, own, shfl_mirror<TPL>(w[j][m], t));
        }
}

// ---- P1: scatter + R2C x -------------------------------------------------------

// complex lines per tile of the x passes at most (3 * rows / 2, rows <= 32), and
// threads of a CTA
constexpr int kMaxXLines = 48;
constexpr int kMaxXThreads = 384;

// One line's threads share a warp, so the stages of a line exchange through
// shared memory with warp barriers, and the half spectra leave the registers
// for HBM directly (a store covers TPL neighbouring kx).  The two spectra are
// stored times two; the inverse pass takes the factor back with its 1/N.
// Against separating the spectra through shared memory: 49 -> 37 M warp
// instructions, 80.3 -> 63.0 us at 256^3 FP32 under ncu (tiles of four rows); L1
// bounds it (75 % of its peak; DRAM at 41 %, 25 warps per SM).
template <typename T, int N, bool GROUP>
__global__ void __launch_bounds__(kMaxXThreads) k_fx_fwd(const __grid_constant__ FastArgs a0) {
    pdl_wait();
    __shared__ ArgSlot<GROUP> slot;
    const FastArgs& a = member_args<GROUP>(a0, blockIdx.y, slot);
    if (a.skip && *a.skip) return;
    using T2 = c_t<T>;
    constexpr int R1 = Split<N>::R1, R2 = Split<N>::R2, TPL = Split<N>::TPL;
    constexpr int KT = kx_tile<N>();
    static_assert(32 % TPL == 0, "the threads of a line share a warp");
    constexpr int LD = x_ld<N, T>();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T2* lines = reinterpret_cast<T2*>(smem_raw);
    const int RB = a.rows;
    const int nq = 3 * RB / 2;
    const int tid = threadIdx.x;
    const int nthr = blockDim.x;
    const int q = tid / TPL;
    const int t = tid - q * TPL;
    const T2* tw = tw_of<T>(a, 0);
    T2* spec = reinterpret_cast<T2*>(a.spec);
    const T mean[3] = {a.src_sum ? (T)(a.src_sum[0] * a.inv_nb) : (T)0,
                       a.src_sum ? (T)(a.src_sum[1] * a.inv_nb) : (T)0,
                       a.src_sum ? (T)(a.src_sum[2] * a.inv_nb) : (T)0};
    const int La = 2 * q, rla = La / 3, ca = La - 3 * rla;
    const int Lb = La + 1, rlb = Lb / 3, cb = Lb - 3 * rlb;
    for (long long tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
        const long long r0 = tile * RB;
        const int rows = (int)min((long long)RB, a.nrows - r0);
        const int nreal = 3 * rows;
        const int nqa = (nreal + 1) / 2;
        // 1) zero the lines
        for (int i = tid; i < nq * LD; i += nthr) lines[i] = T2{};
        __syncthreads();
        // 2) scatter the compact vector minus its mean (support voxels only)
        {
            const int s0 = a.row_ptr[r0];
            const int s1 = a.row_ptr[r0 + rows];
            for (int s = s0 + tid; s < s1; s += nthr) {
                const int idx = a.support[s];
                const int row = idx / N;
                const int x = idx - row * N;
                const int rl = row - (int)r0;
                const double c0 = a.src[3LL * s], c1 = a.src[3LL * s + 1], c2 = a.src[3LL * s + 2];
                const T v3[3] = {(T)c0 - mean[0], (T)c1 - mean[1], (T)c2 - mean[2]};
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int L = 3 * rl + c;
                    T2* p = &lines[(L >> 1) * LD + x];
                    if (L & 1) p->y = v3[c]; else p->x = v3[c];
                }
            }
        }
        __syncthreads();
        // 3) forward FFT of every complex line (stage A reads the natural line,
        //    stage B leaves X in registers), half spectra to HBM
        const bool act = q < nqa;
        T2* my = lines + (act ? q : 0) * LD;
        auto ld_nat = [&](int pos) { return my[pos]; };
        stage_a<R1, R2, -1, TPL, true>(my, t, act, tw, ld_nat, WarpBarrier{});
        __syncwarp();
        if constexpr (mirrored<N>()) {
            T2 z[R1 / TPL][R2];
            stage_b_regs<R1, R2, -1, TPL>(my, t, act, z);
            if (sizeof(T) == 4 && tile + gridDim.x >= a.ntiles) pdl_trigger();
            T2* pa = spec + ca * a.nh + (r0 + rla) * KT;
            T2* pb = spec + cb * a.nh + (r0 + rlb) * KT;
            const bool hasb = act && Lb < nreal;
            auto st = [&](int k, T2 A, T2 B) {
                const long long o = (k / KT) * a.kts + k % KT;
                if (act) pa[o] = A;
                if (hasb) pb[o] = B;
            };
            separate_lines<R1, R2, TPL>(z, t, st);
        } else {
            auto st_nat = [&](int pos, T2 v) { my[pos] = v; };
            stage_b<R1, R2, -1, TPL, true>(my, t, act, st_nat, WarpBarrier{});
            __syncthreads();
            if (sizeof(T) == 4 && tile + gridDim.x >= a.ntiles) pdl_trigger();
            constexpr int NH = N / 2 + 1;
            for (int it = tid; it < nqa * NH; it += nthr) {
                const int qq = it / NH;
                const int k = it - qq * NH;
                const T2 zk = lines[qq * LD + k], zn = lines[qq * LD + (k == 0 ? 0 : N - k)];
                const int L = 2 * qq, rl = L / 3, M = L + 1, rm = M / 3;
                const long long o = (k / KT) * a.kts + k % KT;
                spec[(L - 3 * rl) * a.nh + (r0 + rl) * KT + o] = cmk<T2>(zk.x + zn.x, zk.y - zn.y);
                if (M < nreal) spec[(M - 3 * rm) * a.nh + (r0 + rm) * KT + o] = cmk<T2>(zk.y + zn.y, zn.x - zk.x);
            }
        }
        __syncthreads();  // the lines are zeroed by the next tile
    }
}

// ---- P5: C2R x + gather + partial sums -------------------------------------------

// Persistent CTAs walk tiles of `rows` grid rows.  Bound by the latency of its
// loads (L1 at 56 % of its peak, DRAM at 40 %, 23 warps per SM).  Each thread reads
// its part of the two half spectra of a line straight from HBM (TPL neighbouring kx per
// load), so shared memory holds the lines of the exchange only and several
// CTAs per SM cover the latency of each other's loads.  Against the former
// form (raw rows staged by cp.async, Hermitian halves read from shared memory):
// 60 -> 35 M warp instructions at 256^3 FP32; 83.5 us under ncu with the last
// block's sum of 1216 partial rows, which was a kernel of its own beside 82.8 us.
template <typename T, int N, bool GROUP>
__global__ void __launch_bounds__(kMaxXThreads) k_fx_inv(const __grid_constant__ FastArgs a0) {
    pdl_wait();
    __shared__ ArgSlot<GROUP> slot;
    const FastArgs& a = member_args<GROUP>(a0, blockIdx.y, slot);
    if (a.skip && *a.skip) return;
    using T2 = c_t<T>;
    constexpr int R1 = Split<N>::R1, R2 = Split<N>::R2, TPL = Split<N>::TPL;
    constexpr int KT = kx_tile<N>();
    static_assert(32 % TPL == 0, "the threads of a line share a warp");
    constexpr int LD = x_ld<N, T>();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ double red[4 * 32];
    const int RB = a.rows;
    const int tid = threadIdx.x;
    const int nthr = blockDim.x;
    const int q = tid / TPL;
    const int t = tid - q * TPL;
    const T2* tw = tw_of<T>(a, 0);
    const T2* spec = reinterpret_cast<const T2*>(a.spec);
    T2* lines = reinterpret_cast<T2*>(smem_raw);
    const T scale = (T)(0.5 * a.scale);  // the forward pass stores twice the spectra
    T acc[4] = {(T)0, (T)0, (T)0, (T)0};
    // complex line q carries real lines 2q (A) and 2q + 1 (B)
    const int La = 2 * q, rla = La / 3, ca = La - 3 * rla;
    const int Lb = La + 1, rlb = Lb / 3, cb = Lb - 3 * rlb;

    for (long long tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
        const long long r0 = tile * RB;
        const int rows = (int)min((long long)RB, a.nrows - r0);
        const int nreal = 3 * rows;
        const int nqa = (nreal + 1) / 2;
        const bool act = q < nqa;
        T2* my = lines + (act ? q : 0) * LD;
        {
            const T2* pa = spec + ca * a.nh + (r0 + rla) * KT;
            const T2* pb = spec + cb * a.nh + (r0 + rlb) * KT;
            const bool hasb = act && Lb < nreal;
            auto ld = [&](int k, T2& A, T2& B) {
                const long long o = (k / KT) * a.kts + k % KT;
                A = act ? pa[o] : T2{};
                B = hasb ? pb[o] : T2{};
            };
            if constexpr (mirrored<N>()) {
                T2 z[R1 / TPL][R2];
                join_lines<R1, R2, TPL>(z, t, ld);
                stage_a_regs<R2, R1, +1, TPL>(my, t, act, tw, z);
            } else {
                // Z = A + iB, above N/2 from the mirror image (read again, from L1)
                auto ld_herm = [&](int k) {
                    const bool lo = 2 * k <= N;
                    T2 A, B;
                    ld(lo ? k : N - k, A, B);
                    if (k == 0 || 2 * k == N) A.y = B.y = (T)0;
                    return lo ? cmk<T2>(A.x - B.y, A.y + B.x) : cmk<T2>(A.x + B.y, B.x - A.y);
                };
                stage_a<R2, R1, +1, TPL, false>(my, t, act, tw, ld_herm);
            }
        }
        __syncwarp();
        {
            auto st_nat = [&](int pos, T2 v) { my[pos] = v; };
            stage_b<R2, R1, +1, TPL, true>(my, t, act, st_nat, WarpBarrier{});
        }
        __syncthreads();
        // gather to the support with the 1/N scale, partial sums
        {
            const int s0 = a.row_ptr[r0];
            const int s1 = a.row_ptr[r0 + rows];
            for (int s = s0 + tid; s < s1; s += nthr) {
                const int idx = a.support[s];
                const int row = idx / N;
                const int x = idx - row * N;
                const int rl = row - (int)r0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int L = 3 * rl + c;
                    const T2 zv = lines[(L >> 1) * LD + x];
                    const T val = ((L & 1) ? zv.y : zv.x) * scale;
                    a.dst[3LL * s + c] = (double)val;
                    acc[c] += val;
                    if (a.dot_with) acc[3] += (T)a.dot_with[3LL * s + c] * val;
                }
            }
        }
        __syncthreads();  // the lines are rewritten by the next tile
    }
    double accd[4] = {(double)acc[0], (double)acc[1], (double)acc[2], (double)acc[3]};
    double out[4];
    block_sum<4>(accd, red, out);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) a.partials[4LL * blockIdx.x + i] = out[i];
    }
    if (a.alpha_sc) {
        if (last_block(a.alpha_ticket, gridDim.x))
            alpha_body(a.alpha_sc, a.partials, (int)gridDim.x, a.inv_nb, red);
    } else if (a.sum_out && last_block(a.alpha_ticket, gridDim.x)) {
        sum_rows<4, 4>(a.partials, (int)gridDim.x, red, out);
        if (threadIdx.x == 0)
            for (int i = 0; i < 4; ++i) a.sum_out[i] = out[i];
    }
}

// ---- P2 / P4: y pass -------------------------------------------------------------

// One CTA: TX kx columns of one z plane for one component (blockIdx.z, or
// blockIdx.z mod 3 of member blockIdx.z / 3 in a group).
template <typename T, int N, int S, int TX, bool GROUP>
__global__ void __launch_bounds__(TX * Split<N>::TPL) k_fcol_y(const __grid_constant__ FastArgs a0) {
    pdl_wait();
    __shared__ ArgSlot<GROUP> slot;
    const FastArgs& a = member_args<GROUP>(a0, blockIdx.z / 3, slot);
    const int comp = GROUP ? (int)(blockIdx.z % 3) : (int)blockIdx.z;
    if (a.skip && *a.skip) return;
    using T2 = c_t<T>;
    constexpr int R1 = Split<N>::R1, R2 = Split<N>::R2, TPL = Split<N>::TPL;
    constexpr int LD = col_ld<N, T, TX>();
    __shared__ __align__(16) T2 lines[TX * LD];
    const int c = threadIdx.x % TX;
    const int t = threadIdx.x / TX;
    const int k0 = blockIdx.x * TX;
    const bool act = k0 + c < a.nxh;
    const T2* tw = tw_of<T>(a, 1);
    const int kx = k0 + (act ? c : 0);
    T2* base = reinterpret_cast<T2*>(a.spec) + comp * a.nh + (kx >> a.ktl) * a.kts +
               (((long long)blockIdx.y * N) << a.ktl) + (kx & ((1 << a.ktl) - 1));
    const int es = 1 << a.ktl;
    T2* my = lines + c * LD;
    auto ld_g = [&](int pos) { return base[pos * es]; };
    auto st_g = [&](int pos, T2 v) { base[pos * es] = v; };
    if (S < 0) {
        stage_a<R1, R2, -1, TPL, false>(my, t, act, tw, ld_g);
        __syncthreads();
        if (sizeof(T) == 4) pdl_trigger();
        stage_b<R1, R2, -1, TPL, false>(my, t, act, st_g);
    } else {
        stage_a<R2, R1, +1, TPL, false>(my, t, act, tw, ld_g);
        __syncthreads();
        if (sizeof(T) == 4) pdl_trigger();
        stage_b<R2, R1, +1, TPL, false>(my, t, act, st_g);
    }
}

// ---- P3: z forward + Green + z inverse -------------------------------------------

// Component stride (elements) of the spectral tile in shared memory: the
// padded lines of one component, rounded up so that each component block
// starts 128-byte aligned (a TMA destination) and the blocks never overlap.
template <typename T, int N, int TX>
__host__ __device__ constexpr int comp_stride() {
    return (int)(((size_t)TX * col_ld<N, T, TX>() * 2 * sizeof(T) + 127) / 128 * 128 /
                 (2 * sizeof(T)));
}
// Elements of one Green box [kz][TX], rounded up to whole 128 bytes as well.
template <typename T, int N, int TX>
__host__ __device__ constexpr int green_stride() {
    return (int)(((size_t)TX * N * sizeof(T) + 127) / 128 * 128 / sizeof(T));
}

// Shared memory of one pipeline stage of the z pass: the spectral tile (per
// component first raw [kz][TX] as the TMA box lands, then the padded lines
// [TX][LD] in the same block) and the Green tile [6][kz][TX].
template <typename T, int N, int TX>
__host__ __device__ constexpr size_t z_green_offset() {
    return (size_t)3 * comp_stride<T, N, TX>() * 2 * sizeof(T);
}
template <typename T, int N, int TX>
__host__ __device__ constexpr size_t z_stage_bytes() {
    return z_green_offset<T, N, TX>() + (size_t)6 * green_stride<T, N, TX>() * sizeof(T);
}

// Persistent CTAs walk the (kx tile, ky) tiles; thread = column + TX *
// (owner + TPL * comp).  One thread has the TMA engine bring the spectral
// tile (three boxes of {2 TX reals, 1, nz}) and the Green tile (six boxes of
// {TX, 1, nz}) into a stage, completing on that stage's mbarrier.  Past the
// last kx column the Green boxes read zeros and the spectral boxes the padding
// columns of the blocked layout, which nothing writes and only inactive threads
// would read.  With two stages the tiles of iteration
// i + 1 load while tile i is transformed (one CTA per SM); with one stage the
// next tile loads after the current one is done, and three CTAs per SM (at
// most 112 registers per thread) overlap one another instead.  The phases
// that touch one component only synchronise that component's threads (named
// barrier 1 + comp); the Green multiply reads all three.  Waits are bounded:
// on a timeout the CTA raises a.err and returns.
template <typename T, int N, int TX, int STAGES, bool GROUP>
__global__ void __launch_bounds__(3 * TX * Split<N>::TPL, STAGES == 1 ? 3 : 1)
    k_fz(const __grid_constant__ CUtensorMap spec_map, const __grid_constant__ CUtensorMap green_map,
         const __grid_constant__ FastArgs a0) {
    pdl_wait();
    // (the few fields read per tile are read through the table: a copy would
    // hold them in registers across the kernel)
    const FastArgs& a = GROUP ? a0.group[blockIdx.y] : a0;
    const CUtensorMap* smap = GROUP ? &a0.group_maps[2 * blockIdx.y] : &spec_map;
    const CUtensorMap* gmap = GROUP ? &a0.group_maps[2 * blockIdx.y + 1] : &green_map;
    if (a.skip && *a.skip) return;
    using T2 = c_t<T>;
    constexpr int R1 = Split<N>::R1, R2 = Split<N>::R2, TPL = Split<N>::TPL;
    constexpr int LD = col_ld<N, T, TX>();
    constexpr int CS = comp_stride<T, N, TX>();
    constexpr size_t STAGE = z_stage_bytes<T, N, TX>();
    constexpr size_t GOFF = z_green_offset<T, N, TX>();
    constexpr int GS = green_stride<T, N, TX>();
    constexpr uint32_t TILE_BYTES = (uint32_t)(3 * N * TX * sizeof(T2) + 6 * N * TX * sizeof(T));
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw);
    unsigned char* stage0 = smem_raw + 128;
    const int c = threadIdx.x % TX;
    const int t = (threadIdx.x / TX) % TPL;
    const int comp = threadIdx.x / (TX * TPL);
    // a named barrier per component needs whole warps per component
    using GBar = typename std::conditional<(TX * TPL) % 32 == 0, GroupBarrier, CtaBarrier>::type;
    GBar gbar = make_group_barrier<GBar>(1 + comp, TX * TPL);
    const int ntx = (a.nxh + TX - 1) / TX;
    const long long ntiles = (long long)ntx * a.ny;
    const T2* tw = tw_of<T>(a, 2);
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
        if (GROUP) {
            fence_tensormap_acquire(smap);
            fence_tensormap_acquire(gmap);
        }
    }
    __syncthreads();

    auto issue = [&](long long tile, int st) {
        unsigned char* base = stage0 + st * STAGE;
        const int k0 = (int)(tile % ntx) * TX;
        const int ky = (int)(tile / ntx);
        mbar_arrive_expect_tx(&bars[st], TILE_BYTES);
        for (int cc = 0; cc < 3; ++cc)
            tma_load_4d(base + (size_t)cc * CS * sizeof(T2), smap, 2 * ((ky << a.ktl) + (k0 & ((1 << a.ktl) - 1))), 0,
                        k0 >> a.ktl, cc, &bars[st]);
        for (int gc = 0; gc < 6; ++gc)
            tma_load_4d(base + GOFF + (size_t)gc * GS * sizeof(T), gmap, k0, ky, 0, gc, &bars[st]);
    };

    long long tile = blockIdx.x;
    if (threadIdx.x == 0 && tile < ntiles) issue(tile, 0);
    for (int i = 0; tile < ntiles; tile += gridDim.x, ++i) {
        const int st = STAGES == 2 ? (i & 1) : 0;
        const long long next = tile + gridDim.x;
        if (STAGES == 2) {
            if (threadIdx.x == 0 && next < ntiles) {
                fence_proxy_async_smem();
                issue(next, st ^ 1);
            }
            if (!tma_pipeline_wait<T2>(bars, i, st, next < ntiles, a.err)) return;
        } else {
            const bool ok = mbar_wait_bounded(&bars[0], (uint32_t)(i & 1));
            if (__syncthreads_or(!ok)) {
                if (threadIdx.x == 0) atomicExch(a.err, 1);
                return;
            }
        }
        T2* blk = reinterpret_cast<T2*>(stage0 + st * STAGE);
        const T* gsm = reinterpret_cast<const T*>(stage0 + st * STAGE + GOFF);
        const int k0 = (int)(tile % ntx) * TX;
        const long long ky = tile / ntx;
        const bool act = k0 + c < a.nxh;
        T2* my = blk + comp * CS + c * LD;  // padded line in this component's block
        // forward stage A from the raw box; Y into the lines after the group barrier
        {
            const T2* rc = blk + comp * CS + c;
            auto ld_raw = [&](int pos) { return rc[pos * TX]; };
            stage_a<R1, R2, -1, TPL, true>(my, t, act, tw, ld_raw, gbar);
        }
        gbar();
        {
            auto st_nat = [&](int pos, T2 v) { my[pos] = v; };
            stage_b<R1, R2, -1, TPL, true>(my, t, act, st_nat, gbar);
        }
        __syncthreads();
        // Green multiply while loading the inverse stage A (owner k1 = same owner)
        {
            const T2* lx = blk + 0 * CS + c * LD;
            const T2* ly = blk + 1 * CS + c * LD;
            const T2* lz = blk + 2 * CS + c * LD;
            // row `comp` of the symmetric tensor (xx xy xz yy yz zz)
            const int g0 = comp == 0 ? 0 : (comp == 1 ? 1 : 2);
            const int g1 = comp == 0 ? 1 : (comp == 1 ? 3 : 4);
            const int g2 = comp == 0 ? 2 : (comp == 1 ? 4 : 5);
            auto ld_green = [&](int pos) {
                const T2 X = lx[pos], Y = ly[pos], Z = lz[pos];
                const T a0 = gsm[g0 * GS + pos * TX + c];
                const T a1 = gsm[g1 * GS + pos * TX + c];
                const T a2 = gsm[g2 * GS + pos * TX + c];
                return cmk<T2>(a0 * X.x + a1 * Y.x + a2 * Z.x, a0 * X.y + a1 * Y.y + a2 * Z.y);
            };
            stage_a<R2, R1, +1, TPL, true>(my, t, act, tw, ld_green);  // CTA barrier
        }
        gbar();
        if (sizeof(T) == 4 && next >= ntiles) pdl_trigger();
        {
            T2* base = reinterpret_cast<T2*>(a.spec) + comp * a.nh + (k0 >> a.ktl) * a.kts + (ky << a.ktl) +
                       ((k0 + c) & ((1 << a.ktl) - 1));
            const int es = a.ny << a.ktl;
            auto st_g = [&](int pos, T2 v) { base[pos * es] = v; };
            stage_b<R2, R1, +1, TPL, false>(my, t, act, st_g);
        }
        __syncthreads();  // this stage is refilled by the next issue
        if (STAGES == 1 && threadIdx.x == 0 && next < ntiles) {
            fence_proxy_async_smem();
            issue(next, 0);
        }
    }
}

// The z pass of a group whose members share one Green table (the three load
// cases of one cell, or cells of one grid and Green parameters): each CTA
// walks its (kx, ky) tiles and, per tile, the members one after another as
// pipeline items (tile, member).  The spectral boxes of item i + 1 load into
// the other stage while item i is transformed, as in k_fz; the Green tile is
// loaded once per tile, with the tile's first item, into one of two Green
// buffers (tile parity) and serves all members.  Per tile the HBM reads are
// G spectral tiles and one Green tile instead of G of each (the byte model
// of a G-field block apply).  Members whose solve is done are left out: the
// flags are read while the first item (tile 0, member 0, whatever its flag) loads,
// and the items after it are those of the `na` active members; that first item is
// waited for and not transformed when member 0 is done.  (With done
// members transformed to the end of their chunk, 20 iterations of three FP64 load
// cases at 100 x 200 x 200 took 226 ms, without 183; 100 at 128^3 289 and 278.)
// Waits are bounded: on a timeout member 0's error flag is raised.
constexpr int kActiveMembers = 64;  // larger groups transform every member
template <typename T, int N, int TX>
__global__ void __launch_bounds__(3 * TX * Split<N>::TPL, sizeof(T) == 4 ? 2 : 1)
    k_fz_shared(const __grid_constant__ FastArgs a0) {
    pdl_wait();
    using T2 = c_t<T>;
    constexpr int R1 = Split<N>::R1, R2 = Split<N>::R2, TPL = Split<N>::TPL;
    constexpr int LD = col_ld<N, T, TX>();
    constexpr int CS = comp_stride<T, N, TX>();
    constexpr size_t SPEC = z_green_offset<T, N, TX>();  // one spectral stage (128-byte multiple)
    constexpr int GS = green_stride<T, N, TX>();
    constexpr size_t GREEN = (size_t)6 * GS * sizeof(T);
    constexpr uint32_t SPEC_BYTES = (uint32_t)(3 * N * TX * sizeof(T2));
    constexpr uint32_t GREEN_BYTES = (uint32_t)(6 * N * TX * sizeof(T));
    static_assert(128 + 2 * SPEC + 2 * GREEN <= 128 + 2 * z_stage_bytes<T, N, TX>(), "shared memory");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw);
    unsigned char* spec0 = smem_raw + 128;
    unsigned char* green0 = spec0 + 2 * SPEC;
    __shared__ int active[kActiveMembers];
    __shared__ int nactive;
    const int G = a0.share;
    int* err = a0.group[0].err;
    const int c = threadIdx.x % TX;
    const int t = (threadIdx.x / TX) % TPL;
    const int comp = threadIdx.x / (TX * TPL);
    using GBar = typename std::conditional<(TX * TPL) % 32 == 0, GroupBarrier, CtaBarrier>::type;
    GBar gbar = make_group_barrier<GBar>(1 + comp, TX * TPL);
    const int ntx = (a0.nxh + TX - 1) / TX;
    const long long ntiles = (long long)ntx * a0.ny;
    const T2* tw = tw_of<T>(a0, 2);
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
        fence_tensormap_acquire(&a0.group_maps[1]);
        for (int m = 0; m < G; ++m) fence_tensormap_acquire(&a0.group_maps[2 * m]);
    }
    __syncthreads();
    const long long my_tiles = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;

    // item i = turn j of member m, with the Green tile when it is the turn's first
    auto issue = [&](int i, int j, int m, bool with_green) {
        const int st = i & 1;
        const long long tile = blockIdx.x + (long long)j * gridDim.x;
        const int k0 = (int)(tile % ntx) * TX;
        const int ky = (int)(tile / ntx);
        unsigned char* sb = spec0 + st * SPEC;
        mbar_arrive_expect_tx(&bars[st], SPEC_BYTES + (with_green ? GREEN_BYTES : 0u));
        for (int cc = 0; cc < 3; ++cc)
            tma_load_4d(sb + (size_t)cc * CS * sizeof(T2), &a0.group_maps[2 * m],
                        2 * ((ky << a0.ktl) + (k0 & ((1 << a0.ktl) - 1))), 0, k0 >> a0.ktl, cc, &bars[st]);
        if (with_green) {
            unsigned char* gb = green0 + (j & 1) * GREEN;
            for (int gc = 0; gc < 6; ++gc)
                tma_load_4d(gb + (size_t)gc * GS * sizeof(T), &a0.group_maps[1], k0, ky, 0, gc,
                            &bars[st]);
        }
    };

    if (threadIdx.x == 0 && my_tiles > 0) issue(0, 0, 0, true);
    if (threadIdx.x < 32) {
        int n = 0;
        for (int m0 = 0; G <= kActiveMembers && m0 < G; m0 += 32) {
            const int m = m0 + threadIdx.x;
            const int* skip = m < G ? a0.group[m].skip : nullptr;
            const bool on = m < G && !(skip && *skip);
            const unsigned mask = __ballot_sync(0xffffffffu, on);
            if (on) active[n + __popc(mask & ((1u << threadIdx.x) - 1u))] = m;
            n += __popc(mask);
        }
        if (threadIdx.x == 0) nactive = G <= kActiveMembers ? n : G;
    }
    __syncthreads();
    const int na = nactive;
    auto member = [&](int k) { return G <= kActiveMembers ? active[k] : k; };
    const int lead = na > 0 && member(0) == 0 ? 0 : 1;  // 1: item 0 belongs to a done member
    const int nitems = my_tiles > 0 ? (int)(my_tiles * na) + lead : 0;
    for (int i = 0; i < nitems; ++i) {
        const int st = i & 1;
        const int q = i - lead;  // item among those of the active members
        if (threadIdx.x == 0 && i + 1 < nitems) {
            fence_proxy_async_smem();
            issue(i + 1, (q + 1) / na, member((q + 1) % na), (q + 1) % na == 0 && q + 1 > 0);
        }
        if (!tma_pipeline_wait<T2>(bars, i, st, i + 1 < nitems, err)) return;
        if (q < 0) continue;
        const int j = q / na;
        const int m = member(q % na);
        const long long tile = blockIdx.x + (long long)j * gridDim.x;
        T2* blk = reinterpret_cast<T2*>(spec0 + st * SPEC);
        const T* gsm = reinterpret_cast<const T*>(green0 + (j & 1) * GREEN);
        const int k0 = (int)(tile % ntx) * TX;
        const long long ky = tile / ntx;
        const bool act = k0 + c < a0.nxh;
        T2* my = blk + comp * CS + c * LD;
        {
            const T2* rc = blk + comp * CS + c;
            auto ld_raw = [&](int pos) { return rc[pos * TX]; };
            stage_a<R1, R2, -1, TPL, true>(my, t, act, tw, ld_raw, gbar);
        }
        gbar();
        {
            auto st_nat = [&](int pos, T2 v) { my[pos] = v; };
            stage_b<R1, R2, -1, TPL, true>(my, t, act, st_nat, gbar);
        }
        __syncthreads();
        {
            const T2* lx = blk + 0 * CS + c * LD;
            const T2* ly = blk + 1 * CS + c * LD;
            const T2* lz = blk + 2 * CS + c * LD;
            const int g0 = comp == 0 ? 0 : (comp == 1 ? 1 : 2);
            const int g1 = comp == 0 ? 1 : (comp == 1 ? 3 : 4);
            const int g2 = comp == 0 ? 2 : (comp == 1 ? 4 : 5);
            auto ld_green = [&](int pos) {
                const T2 X = lx[pos], Y = ly[pos], Z = lz[pos];
                const T a0g = gsm[g0 * GS + pos * TX + c];
                const T a1g = gsm[g1 * GS + pos * TX + c];
                const T a2g = gsm[g2 * GS + pos * TX + c];
                return cmk<T2>(a0g * X.x + a1g * Y.x + a2g * Z.x, a0g * X.y + a1g * Y.y + a2g * Z.y);
            };
            stage_a<R2, R1, +1, TPL, true>(my, t, act, tw, ld_green);  // CTA barrier
        }
        gbar();
        if (sizeof(T) == 4 && i + 1 >= nitems) pdl_trigger();
        {
            T2* base = reinterpret_cast<T2*>(a0.group[m].spec) + comp * a0.nh + (k0 >> a0.ktl) * a0.kts +
                       (ky << a0.ktl) + ((k0 + c) & ((1 << a0.ktl) - 1));
            const int es = a0.ny << a0.ktl;
            auto st_g = [&](int pos, T2 v) { base[pos * es] = v; };
            stage_b<R2, R1, +1, TPL, false>(my, t, act, st_g);
        }
        __syncthreads();  // this stage and, after the tile's last member, this Green buffer are refilled
    }
}


}  // namespace fast

// Runs the five passes with the specialised kernels when the grid, the
// precision and the source/destination allow it; returns false (nothing
// launched) otherwise.  Defined in fast_dispatch.cu.
cudaError_t fast_apply(Problem& P, int precision, const ApplyArgs& aa, int* nparts);

// Group applies (one launch per pass for several problems of one grid and
// tiling).  fast_member_args fills one member's kernel arguments, its two
// tensor maps (spectral, Green) and the launch geometry the members of a
// group must share (kGroupGeometry values); fast_apply_group launches the five
// passes over `members` members whose arguments and maps the caller copied to
// device memory (d_args[members], d_maps[2 * members], 64-byte aligned).
// shared_green: every member's Green map is member 0's (k_fz_shared).
constexpr int kGroupGeometry = 12;
cudaError_t fast_member_args(Problem& P, int precision, const ApplyArgs& aa, fast::FastArgs* args,
                             CUtensorMap* maps, long long* geometry);
cudaError_t fast_apply_group(Problem& P0, int precision, int members, const fast::FastArgs* d_args,
                             const CUtensorMap* d_maps, bool shared_green, int* nparts);

}  // namespace fp

// ---- launch runners (fast32.cu / fast64.cu) -------------------------------------

namespace fp {
namespace fast {

// kx columns per CTA of the y pass: 64-byte row segments, and at least a warp
template <typename T, int N>
__host__ __device__ constexpr int col_tx() {
    constexpr int base = sizeof(T) == 4 ? 8 : 4, warp = 32 / Split<N>::TPL;
    return base > warp ? base : warp;
}
// kx columns per tile of the z pass
template <typename T, int N>
__host__ __device__ constexpr int z_tx() {
    return 4;
}

// grid edges with specialised kernels
#define FP_FAST_EDGES(CALL)                                                                      \
    CALL(32) CALL(48) CALL(64) CALL(80) CALL(96) CALL(128) CALL(160) CALL(256)                  \
    CALL(20) CALL(24) CALL(25) CALL(27) CALL(30) CALL(36) CALL(40) CALL(45) CALL(50) CALL(54)   \
    CALL(60) CALL(72) CALL(75) CALL(81) CALL(90) CALL(100) CALL(108) CALL(120)                  \
    CALL(135) CALL(144) CALL(150) CALL(162) CALL(180) CALL(192) CALL(200) CALL(216) CALL(225)   \
    CALL(240)

inline bool edge_supported(int n) {
#define FP_CASE(N) if (n == N) return true;
    FP_FAST_EDGES(FP_CASE)
#undef FP_CASE
    return false;
}

// the two radices of a specialised edge; false for other edges
inline bool split_of(int n, int* r1, int* r2) {
#define FP_CASE(N)             \
    if (n == N) {              \
        *r1 = Split<N>::R1;    \
        *r2 = Split<N>::R2;    \
        return true;           \
    }
    FP_FAST_EDGES(FP_CASE)
#undef FP_CASE
    return false;
}

// log2 of the kx tile width of the spectral layout
inline int kt_log2(int nx) {
#define FP_CASE(N) \
    if (n == N) return kx_tile<N>() >= 16 ? 4 : (kx_tile<N>() >= 8 ? 3 : 2);
    const int n = nx;
    FP_FAST_EDGES(FP_CASE)
#undef FP_CASE
    return 2;
}
// elements of one component of the blocked spectral field
inline long long spec_elems(int nx, int ny, int nz) {
    const int l = kt_log2(nx);
    return ((long long)((nx / 2 + 1 + (1 << l) - 1) >> l) << l) * ny * nz;
}

inline int x_tpl(int n) {
#define FP_CASE(N) if (n == N) return Split<N>::TPL;
    FP_FAST_EDGES(FP_CASE)
#undef FP_CASE
    return 0;
}

// grid rows per tile of the x passes: about 192 threads per CTA, 96 where
// the lines are long and served by 4 threads (shared memory)
inline int x_rows_for(int n) {
    switch (n) {
        case 32: return 32;
        case 48: return 32;
        case 64: return 16;
        case 80: return 32;
        case 96: return 16;
        case 128: return 16;
        case 160: return 16;
        case 256: return 8;
        default: break;
    }
    const int tpl = x_tpl(n);  // about 192 threads, 96 where a line is long for its threads
    return tpl >= 16 ? 8 : (tpl == 8 || n > 60 ? 16 : 32);
}
// grid rows per tile at most (even): the lines of kMaxXLines, and no more than
// kMaxXThreads threads serve (a line of an edge with 16 threads per line, 240 and
// 256, takes as many threads as four of 64: 16 rows there, 32 elsewhere)
inline int x_rows_max(int n) {
    const int lines = std::min(kMaxXLines, kMaxXThreads / x_tpl(n));
    return (2 * lines / 3) & ~1;
}
template <typename T>
int x_ld_rt(int n) {
#define FP_CASE(N) if (n == N) return x_ld<N, T>();
    FP_FAST_EDGES(FP_CASE)
#undef FP_CASE
    return 0;
}

// column tile widths of the y and z passes
template <typename T>
int y_tx_rt(int n) {
#define FP_CASE(N) if (n == N) return col_tx<T, N>();
    FP_FAST_EDGES(FP_CASE)
#undef FP_CASE
    return 0;
}
template <typename T>
int z_tx_rt(int n) {
#define FP_CASE(N) if (n == N) return z_tx<T, N>();
    FP_FAST_EDGES(FP_CASE)
#undef FP_CASE
    return 0;
}

// dynamic shared memory of the z pass: mbarriers + its pipeline stages
template <typename T>
size_t z_smem_rt(int n, int stages) {
#define FP_CASE(N) if (n == N) return 128 + stages * z_stage_bytes<T, N, z_tx<T, N>()>();
    FP_FAST_EDGES(FP_CASE)
#undef FP_CASE
    return 0;
}

// Launch runners of one edge, defined in fast_runners.cuh and instantiated
// per precision and edge group (fast32.cu, fast64.cu: powers of two;
// fast32n.cu, fast64n.cu: 48, 80, 96, 160; fast_{s,m,l}{32,64}.cu: the edges of
// fft_edges.cuh) so that they build in parallel.
// A set a.group selects the group kernels; the grid then carries the member
// index (grid.y for the x and z passes, grid.z = 3 x members for the y pass).
template <typename T, int N>
struct Passes {
    static cudaError_t xfwd(const FastArgs& a, dim3 grid, int threads, size_t smem, cudaStream_t s);
    static cudaError_t xinv(const FastArgs& a, dim3 grid, int threads, size_t smem, cudaStream_t s);
    static cudaError_t y(int dir, const FastArgs& a, dim3 grid, cudaStream_t s);
    static cudaError_t z(int stages, const CUtensorMap& spec_map, const CUtensorMap& green_map,
                         const FastArgs& a, dim3 grid, size_t smem, cudaStream_t s);
    // the group z pass with one shared Green table (a.share members)
    static cudaError_t z_shared(const FastArgs& a, int grid, size_t smem, cudaStream_t s);
    // blocks resident per SM at this shared-memory size
    static int z_per_sm(int stages, size_t smem);
    static int x_per_sm(bool inverse, int threads, size_t smem);
};

template <typename T>
cudaError_t run_xfwd(int n, const FastArgs& a, dim3 grid, int threads, size_t smem, cudaStream_t s);
template <typename T>
cudaError_t run_xinv(int n, const FastArgs& a, dim3 grid, int threads, size_t smem, cudaStream_t s);
template <typename T>
cudaError_t run_y(int n, int dir, const FastArgs& a, dim3 grid, cudaStream_t s);
template <typename T>
cudaError_t run_z(int n, int stages, const CUtensorMap& spec_map, const CUtensorMap& green_map,
                  const FastArgs& a, dim3 grid, size_t smem, cudaStream_t s);
template <typename T>
cudaError_t run_z_shared(int n, const FastArgs& a, int grid, size_t smem, cudaStream_t s);
// blocks of the z kernel resident per SM at this shared-memory size
template <typename T>
int z_blocks_per_sm(int n, int stages, size_t smem);

// blocks of the x kernels resident per SM at this shared-memory size
template <typename T>
int x_blocks_per_sm(int n, bool inverse, int threads, size_t smem);

}  // namespace fast
}  // namespace fp
