// fvb_stage64_orders.cu -- the FP64 stage kernel for UP3, UP5 and UP9.
#include "fvb_stage64.cuh"

namespace fvb {

StageKernel stage64_orders(int order, int shape)
{
    return order == 5 ? pick64<5, 0>(shape) : order == 3 ? pick64<3, 0>(shape) : order == 9 ? pick64<9, 0>(shape)
                                                                                           : StageKernel{};
}

}  // namespace fvb
