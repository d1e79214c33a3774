// The x instantiations of k_lsweep.
#include "lsweep.cuh"

namespace gatt {

void *line_kernel_x(bool per, int nR, int LL)
{
    if (LL == 32) return per ? pick_line_kernel<true, true, 32>(nR) : pick_line_kernel<true, false, 32>(nR);
    if (LL == 4) return per ? pick_line_kernel<true, true, 4>(nR) : pick_line_kernel<true, false, 4>(nR);
    if (LL == 16) return per ? pick_line_kernel<true, true, 16>(nR) : pick_line_kernel<true, false, 16>(nR);
    return per ? pick_line_kernel<true, true, 8>(nR) : pick_line_kernel<true, false, 8>(nR);
}

}  // namespace gatt
