// fvb_stage64_rs.cu -- the FP64 UP7 stage kernel with carb_fv's solvers on the
// reconstructed states (1 HLL, 2 Roe).
#include "fvb_stage64.cuh"

namespace fvb {

StageKernel stage64_up7_rs(int shape, int rs)
{
    return rs == 1 ? pick64<7, 1>(shape) : rs == 2 ? pick64<7, 2>(shape) : StageKernel{};
}

}  // namespace fvb
