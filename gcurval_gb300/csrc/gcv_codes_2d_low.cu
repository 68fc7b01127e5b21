// Length-pass and sampling instantiations: planar B-splines of degree 1 to 3.
#include "gcv_length_hw.cuh"
#include "gcv_sample_impl.cuh"
#include "gcv_walk.cuh"

namespace gcv {
GCV_LENGTH_INST(0, bs_code(1, 2), 0)
GCV_LENGTH_INST(0, bs_code(2, 2), 0)
GCV_LENGTH_INST(0, bs_code(3, 2), 0)
GCV_LENGTH_INST2(1, bs_code(3, 2))
GCV_LENGTH_INST2(2, bs_code(3, 2))
GCV_SAMPLE_INST2(bs_code(1, 2))
GCV_SAMPLE_INST2(bs_code(2, 2))
GCV_SAMPLE_INST2(bs_code(3, 2))
GCV_LENGTH_HW_INST(bs_code(1, 2))
GCV_LENGTH_HW_INST(bs_code(2, 2))
GCV_LENGTH_HW_INST(bs_code(3, 2))
GCV_WALK_INST(bs_code(1, 2))
GCV_WALK_INST(bs_code(2, 2))
GCV_WALK_INST(bs_code(3, 2))
}  // namespace gcv
