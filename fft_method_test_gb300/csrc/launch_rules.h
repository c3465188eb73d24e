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

}  // namespace fp
