// SHLL_PREC_F64_EXACT and SHLL_PREC_F32_EXACT: reference arithmetic with every multiply and add
// rounded separately (this file is compiled with -fmad=false), IEEE division and square root:
// bit-identical to the reference's gcc builds (which contain no fused multiply-add on x86-64).
#define SHLL_PLAIN_NS plain_exact
#define SHLL_PLAIN_FMA 0   // every product is rounded before it is added
#include "plain_resident.cuh"

namespace plain_exact {
cudaError_t step(const PlainArgs& a) { return a.real_bits == 32 ? step_t<float>(a) : step_t<double>(a); }
cudaError_t run(const PlainArgs& a, long steps, unsigned* prog, int stall, int* swaps) {
    return a.real_bits == 32 ? run_t<float>(a, steps, prog, stall, swaps) : run_t<double>(a, steps, prog, stall, swaps);
}
cudaError_t load_by_planes(const PlainArgs& a, const double* const* in, void* work) {
    return load_by_planes_t<float>(a, in, work);
}
cudaError_t dump_by_planes(const PlainArgs& a, double* const* out, void* work) {
    return dump_by_planes_t<float>(a, out, work);
}
cudaError_t stage(const PlainArgs& a, int which) {
    return a.real_bits == 32 ? stage_t<float>(a, which) : stage_t<double>(a, which);
}
}
