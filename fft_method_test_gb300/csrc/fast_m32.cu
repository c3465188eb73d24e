// fast_m32.cu -- the specialised apply passes in FP32 for the middle edges of
// fft_edges.cuh.
#include "fast_runners.cuh"

namespace fp {
namespace fast {
#define FP_INSTANCE(N, R1, R2, TPL) template struct Passes<float, N>;
FP_EDGES_MIDDLE(FP_INSTANCE)
#undef FP_INSTANCE
}  // namespace fast
}  // namespace fp
