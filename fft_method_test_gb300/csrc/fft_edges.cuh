// fft_edges.cuh -- splits of the specialised edges beyond the eight of
// fft_fast.cuh: every product of 2, 3 and 5 from 20 to 240 whose two radices
// are at most 20 (all but 125 and 250 and the powers of three above 81).
//
// FP_EDGE(N, R1, R2, TPL): N = R1 * R2, TPL threads per line.  TPL need not
// divide the radices: a thread owns ceil(R / TPL) butterflies of a stage and
// the last of them may be idle.  TPL divides 32 (the threads of an x line share
// a warp) and keeps at most 40 values per thread in flight; R1 a multiple of
// TPL with R2 even lets the x passes separate the two real lines in registers
// (fft_fast.cuh), so those splits are taken where the edge has one.
//
// The generic passes (fft_passes.cuh), which these edges used before, carry
// three components per thread at 255 registers and choose their radices at run
// time.  Measured per mixed apply, generic against specialised: 72^3 98 -> 23 us,
// 100 x 90 x 72 166 -> 39, 120^3 205 -> 63, 144^3 360 -> 94, 192^3 759 -> 220,
// 240^3 1079 -> 464; FP64 (bound by its pipe either way) 100^3 734 -> 674.
#pragma once

#define FP_EDGES_SMALL(E) \
    E(20, 5, 4, 4) E(24, 4, 6, 4) E(25, 5, 5, 4) E(27, 9, 3, 4) E(30, 6, 5, 4) E(36, 9, 4, 4) E(40, 4, 10, 4) \
    E(45, 9, 5, 4) E(50, 10, 5, 4) E(54, 9, 6, 4)
#define FP_EDGES_MIDDLE(E) \
    E(60, 12, 5, 4) E(72, 12, 6, 4) E(75, 15, 5, 4) E(81, 9, 9, 4) E(90, 10, 9, 4) E(100, 10, 10, 4) \
    E(108, 12, 9, 4) E(120, 12, 10, 4)
#define FP_EDGES_LARGE(E) \
    E(135, 15, 9, 8) E(144, 12, 12, 4) E(150, 15, 10, 8) E(162, 18, 9, 8) E(180, 15, 12, 8) E(192, 16, 12, 8) \
    E(200, 20, 10, 8) E(216, 18, 12, 8) E(225, 15, 15, 8) E(240, 16, 15, 16)
