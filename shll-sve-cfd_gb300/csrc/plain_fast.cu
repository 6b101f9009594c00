// SHLL_PREC_F64: reference arithmetic in FP64 with fused multiply-add allowed (compiled with
// the default -fmad=true).
#define SHLL_PLAIN_NS plain_fast
#define SHLL_PLAIN_FMA 1   // products and sums may be fused
#include "plain_resident.cuh"

namespace plain_fast {
cudaError_t step(const PlainArgs& a) { return step_t<double>(a); }
cudaError_t run(const PlainArgs& a, long steps, unsigned* prog, int stall, int* swaps) {
    return run_t<double>(a, steps, prog, stall, swaps);
}
cudaError_t stage(const PlainArgs& a, int which) { return stage_t<double>(a, which); }
}
