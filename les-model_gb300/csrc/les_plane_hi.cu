// les_plane_hi.cu -- plane-march pass B for four to six Chebyshev levels.
#include "les_plane.cuh"

namespace les {
KPB plane_pick_b_hi(int S, int form, bool first)
{
    return S == 4 ? plane_pick_b_s<4>(form, first)
                  : (S == 5 ? plane_pick_b_s<5>(form, first) : plane_pick_b_s<6>(form, first));
}
}  // namespace les
