// The instantiations of k_lsweep_xy.
#include "lsweep.cuh"

namespace gatt {

template <bool PERX, bool PERY>
static void *pick(int nR)
{
    switch (nR) {
    case 2: return (void *)k_lsweep_xy<PERX, PERY, 2>;
    case 3: return (void *)k_lsweep_xy<PERX, PERY, 3>;
    case 4: return (void *)k_lsweep_xy<PERX, PERY, 4>;
    case 5: return (void *)k_lsweep_xy<PERX, PERY, 5>;
    case 6: return (void *)k_lsweep_xy<PERX, PERY, 6>;
    case 7: return (void *)k_lsweep_xy<PERX, PERY, 7>;
    default: return nullptr;
    }
}

void *line_kernel_xy(bool perx, bool pery, int nR)
{
    if (perx) return pery ? pick<true, true>(nR) : pick<true, false>(nR);
    return pery ? pick<false, true>(nR) : pick<false, false>(nR);
}

}  // namespace gatt
