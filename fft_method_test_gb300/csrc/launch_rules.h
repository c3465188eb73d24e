// launch_rules.h -- host rules that a run on one healthy GPU does not show at
// work (a second device in the process, a device error): plain C++, so that a
// host program can run them against stand-ins for the CUDA calls.
#pragma once

#include <atomic>

namespace fp {

// Blocks per cluster of a kernel on device `dev`: 16 where the device lets the
// kernel exceed the portable 8 (`allow` sets the function attribute, which
// belongs to one device, and returns whether it took) and `fits` says that it can
// place such a cluster, else the largest of 8, 4, 2, 1 that it can place.  The
// answer is kept per device (0: not asked yet); two threads that ask at once get
// the same one.
constexpr int kClusterDevices = 64;
template <class Allow, class Fits>
int cluster_blocks(std::atomic<int> (&known)[kClusterDevices], int dev, Allow allow, Fits fits) {
    const bool keep = dev >= 0 && dev < kClusterDevices;
    if (keep)
        if (const int n = known[dev].load(std::memory_order_acquire)) return n;
    int n = allow() ? 16 : 8;
    while (n > 1 && !fits(n)) n /= 2;
    if (keep) known[dev].store(n, std::memory_order_release);
    return n;
}

// The lockstep solve, or where it could not get its memory the load cases one at
// a time.  Every other failure is the caller's to see: a wait that timed out or a
// launch that failed in the lockstep is not made good by a second solve.
template <class Lockstep, class OneByOne>
int lockstep_or_one_by_one(Lockstep lockstep, OneByOne one_by_one) {
    bool no_memory = false;
    const int rc = lockstep(&no_memory);
    return rc != 0 && no_memory ? one_by_one() : rc;
}

// FP64 operator applies that stay with the generic passes although their grid has
// specialised ones: z = 162 with y one of 162, 200, 216, and grids of these edges
// alone.  The FP64 pipe bounds the passes, an idle owner's lane costs its full share
// of it, and the two radices of these edges leave most of them idle (162 = 18 x 9:
// eight threads take 24 and 16 owner slots), in the z pass for three components at
// once.  FP64 apply, generic | specialised, us (x, y, z): 162^3 3186 | 3621, 64 x 162 x
// 162 1162 | 1331, 200 x 200 x 162 4499 | 4976, 200^3 5550 | 5741, 216^3 6220 | 6692; on
// the other side of the line 162 x 96 x 162 1847 | 1867, 100 x 216 x 216 3039 | 3004,
// 162 x 162 x 32 828 | 665, 162 x 162 x 240 4734 | 4182, 192^3 3953 | 3803.
inline bool fp64_generic_passes(int nx, int ny, int nz) {
    auto slow = [](int n) { return n == 162 || n == 200 || n == 216; };
    return slow(nz) && slow(ny) && (nz == 162 || slow(nx));
}

}  // namespace fp
