// conv_rules.h -- which form of the 3x3x3 tensor-core convolution a call runs
// (learned_tc.cu): the tile form (k_conv_halo) or the per-tap form (k_conv_tc), the
// output channels of a CTA, and the per-tap form's shared-memory buffers.  Plain
// C++, so that a host program can run it.
//
// No single count decides.  The tile form copies 3 * (128 + 2 (nx + 3)) rows per 128
// padded positions and repeats them for every split of the output channels; the
// per-tap form copies 27 * 128 rows per 128 voxels.  Fewer output channels per CTA
// shorten a call that leaves SMs idle and lengthen every other; more buffers hide
// the gathers' latency and cost resident CTAs.  So the rule estimates the time of
// each candidate and takes the least.  The estimates are fits to measured times (us
// on 152 SMs, 50 shapes from one voxel to 96^3 and 300 x 20 x 300 by 19 channel
// pairs, all candidates each: within 10 % of most).  Against the measured best of
// a call the choice costs 0.8 % on average, against two buffers at most 16 %.  Measured, two buffers and all output
// channels per CTA | the tile form wherever it fits, else three or four buffers and
// 304 CTAs at least | this rule:
//   4 x 32^3    16 ->  32    81 |   35 |   35    1024 x 2^3       64 -> 128    50 | 269 |  38
//   4 x 16^3   128 -> 128    82 |  194 |   76    4096 x 1^3       64 ->  64    42 | 526 |  30
//   2 x 64^3    64 -> 128   930 | 1350 |  930    1000 x 16 x 16   16 ->  32   120 | 620 | 110
//   96^3        64 -> 128  1567 | 4750 | 1567    16 x (64,1,64)   64 -> 128   208 | 495 | 152
#pragma once

#include <algorithm>
#include <cstddef>

namespace fp {

constexpr int kConvTile = 128;               // voxels (positions) per CTA tile: the MMA's M
constexpr std::size_t kConvMaxSmem = 232448;  // dynamic shared memory a CTA may use

struct ConvCall {
    long long nx, ny, nz, samples;
    int dilation, cin, cout, sms;
};
struct ConvPlan {
    bool halo;
    int tile;    // output channels per CTA
    int stages;  // buffers of the per-tap form
};

// A CTA's shared memory: barriers and buffers, and at least its share of the SM for
// the TMEM columns it holds, so that the CTAs of an SM never ask for more than there
// are.
inline std::size_t conv_tmem_share(int tile) { return (std::size_t)233472 * (tile < 32 ? 32 : tile) / 512; }
inline std::size_t conv_tap_smem(int cin, int tile, int stages) {
    return std::max((std::size_t)1024 + (std::size_t)stages * (kConvTile + tile) * cin * 2, conv_tmem_share(tile));
}
// voxel rows of one plane of a tile's neighbourhood
inline long long conv_halo_rows(long long nx) { return kConvTile + 2 * (nx + 3); }
inline std::size_t conv_halo_smem(long long nx, int cin, int tile) {
    const std::size_t rows = (std::size_t)3 * (std::size_t)conv_halo_rows(nx) + (std::size_t)27 * tile;
    return std::max((std::size_t)1024 + rows * cin * 2, conv_tmem_share(tile));
}
// CTAs resident on an SM at this much shared memory
inline int conv_residents(std::size_t smem) {
    return (int)std::clamp<std::size_t>(kConvMaxSmem / (smem + 1024), 1, 16);
}
inline long long conv_positions(const ConvCall& c) { return (c.nx + 2) * (c.ny + 2) * c.nz; }
inline long long conv_halo_tiles(const ConvCall& c) {
    return (conv_positions(c) + kConvTile - 1) / kConvTile * c.samples;
}
// CTAs along x of the tile form's persistent grid
inline long long conv_halo_grid(const ConvCall& c, int tile) {
    const long long fit = conv_residents(conv_halo_smem(c.nx, c.cin, tile));
    return std::min(conv_halo_tiles(c), std::max(1LL, fit * c.sms / (c.cout / tile)));
}
// The tile form takes dilation 1, up to 64 input channels, a neighbourhood whose rows
// a 14-bit descriptor offset and shared memory hold, and samples that 32-bit
// positions cover.
inline bool conv_halo_ok(const ConvCall& c, int tile) {
    return c.dilation == 1 && c.cin <= 64 && conv_positions(c) < (1LL << 30) && c.samples < (1LL << 30) &&
           3 * conv_halo_rows(c.nx) <= 0x3FFF && conv_halo_smem(c.nx, c.cin, tile) <= 226 * 1024;
}

// Waves of CTAs: the latency of 27 taps plus what the resident CTAs copy.  The
// last CTAs of several waves do not spread evenly over the SMs.
inline double conv_tap_us(const ConvCall& c, int tile, int stages) {
    const long long total = c.nx * c.ny * c.nz * c.samples;
    const long long n = (total + kConvTile - 1) / kConvTile * (c.cout / tile);
    const double lat = stages == 2 ? 14.0 : (stages == 3 ? 11.0 : 10.5);
    const double cta = 0.0015 * (kConvTile + 1.4 * tile) * c.cin + 1.3;
    const long long fit = conv_residents(conv_tap_smem(c.cin, tile, stages));
    const long long waves = n / (c.sms * fit), rest = n % (c.sms * fit);
    double us = 5.5 + waves * (lat + cta * fit);
    if (rest) {
        double k = (double)((rest + c.sms - 1) / c.sms);
        if (waves) k += 0.35 * (fit - k);
        us += lat + cta * k;
    }
    return us;
}
// The weights once per CTA, then its tiles: their copies' latency plus what the
// resident CTAs copy and multiply.
inline double conv_halo_us(const ConvCall& c, int tile) {
    const long long tiles = conv_halo_tiles(c), gx = conv_halo_grid(c, tile);
    const double resident = (double)((gx * (c.cout / tile) + c.sms - 1) / c.sms);
    const double rows = 3.0 * conv_halo_rows(c.nx);
    const double work = 5e-4 * rows + 2.5e-4 * c.cin * (64 + tile);
    const double lat = 5.4 + 9e-5 * rows * c.cin;
    return 4.4 + 0.003 * tile * c.cin * resident + (double)((tiles + gx - 1) / gx) * (lat + work * resident);
}

inline ConvPlan conv_plan(const ConvCall& c) {
    ConvPlan best{false, c.cout, 3};
    double us = conv_tap_us(c, c.cout, 3);
    for (int tile = 16; tile <= c.cout; tile *= 2)
        // (two buffers lose at every size up to 32 input channels)
        for (int stages = c.cin <= 32 ? 3 : 2; stages <= 4; ++stages)
            if (conv_tap_smem(c.cin, tile, stages) <= kConvMaxSmem) {
                const double t = conv_tap_us(c, tile, stages);
                if (t < us) us = t, best = {false, tile, stages};
            }
    // a tile form estimated within 7 % is taken: its fit reads high more often
    us /= 0.93;
    for (int tile = 16; tile <= c.cout; tile *= 2)
        if (conv_halo_ok(c, tile)) {
            const double t = conv_halo_us(c, tile);
            if (t < us) us = t, best = {true, tile, 0};
        }
    return best;
}

}  // namespace fp
