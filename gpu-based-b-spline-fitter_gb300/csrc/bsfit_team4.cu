// The 4-warp instantiations of the one-ROI-per-block fit kernels.
#include "bsfit_team.cuh"

namespace bsfit {

TeamKern team_kern4(int mode, bool multi, bool var) { return team_kern<4>(mode, multi, var); }

}  // namespace bsfit
