// One-ROI-per-block fit kernels of 4 warps, five or six blocks per SM.
#include "bsfit_team.cuh"

namespace bsfit {

TeamKern team_kern4_dense(int mode, int blocks, bool multi, bool var) {
  if (mode == 6 && blocks == 6) return team_kern<6, 4, 6>(multi, var);
  if (mode == 7 && blocks == 5) return team_kern<7, 4, 5>(multi, var);
  if (mode == 8 && blocks == 5) return team_kern<8, 4, 5>(multi, var);
  return nullptr;
}

}  // namespace bsfit
