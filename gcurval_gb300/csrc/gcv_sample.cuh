// Launcher of the sampling kernels (k_sample, FP64; k_sample_ff, mixed),
// defined in gcv_sample_impl.cuh and instantiated per curve code in the
// gcv_codes_*.cu units.
#pragma once

#include "gcv_kernels.cuh"

namespace gcv {

// Smallest tolerance at which FP64 tables are sampled by k_sample_ff (the
// in-leaf Newton in float-float) rather than k_sample.  At 1e-12 a sample is
// placed to 1e-13 L and a float-float leaf integral is good to 2.8e-14 of the
// leaf; below, the margin is gone and the FP64 kernel, bound by the FP64 pipe
// and 6-8 times slower, takes over.
constexpr double PLAIN_SPLIT_RTOL = 1e-12;

// PREC 0: FP64 table (k_sample_ff<CODE, double>, or k_sample<CODE> below
// PLAIN_SPLIT_RTOL); PREC 1: k_sample_ff<CODE, float2> on the float-float
// coefficients coef_ff.  CODE -1 dispatches per sample.
template <int CODE, int PREC>
cudaError_t sample_launch(const SampleParams& P, const float2* coef_ff, cudaStream_t stream, int grid, int threads);

}  // namespace gcv
