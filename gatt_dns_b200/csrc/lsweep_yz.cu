// The y and z instantiations of k_lsweep.
#include "lsweep.cuh"

namespace gatt {

void *line_kernel_yz(bool per, int nR, int LL)
{
    if (LL == 32) return per ? pick_line_kernel<false, true, 32>(nR) : pick_line_kernel<false, false, 32>(nR);
    if (LL == 4) return per ? pick_line_kernel<false, true, 4>(nR) : pick_line_kernel<false, false, 4>(nR);
    if (LL == 16) return per ? pick_line_kernel<false, true, 16>(nR) : pick_line_kernel<false, false, 16>(nR);
    return per ? pick_line_kernel<false, true, 8>(nR) : pick_line_kernel<false, false, 8>(nR);
}

}  // namespace gatt
