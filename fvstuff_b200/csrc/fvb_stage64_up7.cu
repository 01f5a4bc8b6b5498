// fvb_stage64_up7.cu -- the FP64 stage kernel for UP7 + HLLC (single grid and
// batched), and the choice among the FP64 kernels.
#include "fvb_stage64.cuh"

namespace fvb {

StageKernel stage64_up7(int shape) { return pick64<7, 0>(shape); }

StageKernel stage64_kernel_of(int order, int shape, int rs)
{
    if (rs != 0) return order == 7 ? stage64_up7_rs(shape, rs) : StageKernel{};
    return order == 7 ? stage64_up7(shape) : stage64_orders(order, shape);
}

}  // namespace fvb
