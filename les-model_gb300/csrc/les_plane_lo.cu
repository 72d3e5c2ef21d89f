// les_plane_lo.cu -- plane-march pass B for one to three Chebyshev levels.
#include "les_plane.cuh"

namespace les {
KPB plane_pick_b_lo(int S, int form, bool first)
{
    return S == 1 ? plane_pick_b_s<1>(form, first)
                  : (S == 2 ? plane_pick_b_s<2>(form, first) : plane_pick_b_s<3>(form, first));
}
}  // namespace les
