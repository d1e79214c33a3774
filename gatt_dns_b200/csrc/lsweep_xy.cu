// The instantiations of k_lsweep_xy.
#include "lsweep.cuh"

namespace gatt {

template <bool PERX, bool PERY, int LL>
static void *pick(int nR)
{
    switch (nR) {
    case 2: return (void *)k_lsweep_xy<PERX, PERY, 2, LL>;
    case 3: return (void *)k_lsweep_xy<PERX, PERY, 3, LL>;
    case 4: return (void *)k_lsweep_xy<PERX, PERY, 4, LL>;
    case 5: return (void *)k_lsweep_xy<PERX, PERY, 5, LL>;
    case 6: return (void *)k_lsweep_xy<PERX, PERY, 6, LL>;
    case 7: return (void *)k_lsweep_xy<PERX, PERY, 7, LL>;
    default: return nullptr;
    }
}

void *line_kernel_xy(bool perx, bool pery, int nR, int LL)
{
    if (LL == 32) {
        if (perx) return pery ? pick<true, true, 32>(nR) : pick<true, false, 32>(nR);
        return pery ? pick<false, true, 32>(nR) : pick<false, false, 32>(nR);
    }
    if (perx) return pery ? pick<true, true, 8>(nR) : pick<true, false, 8>(nR);
    return pery ? pick<false, true, 8>(nR) : pick<false, false, 8>(nR);
}

}  // namespace gatt
