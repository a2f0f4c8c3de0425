// One-ROI-per-block fit kernels of 4 warps, up to four blocks per SM.
#include "bsfit_team.cuh"

namespace bsfit {

TeamKern team_kern4(int mode, int blocks, bool multi, bool var) {
  if (mode == 8 && blocks == 3) return team_kern<8, 4, 3>(multi, var);
  if (blocks != 4) return nullptr;
  switch (mode) {
    case 6: return team_kern<6, 4, 4>(multi, var);
    case 7: return team_kern<7, 4, 4>(multi, var);
    case 8: return team_kern<8, 4, 4>(multi, var);
    default: return team_kern<kFit4Pi, 4, 4>(multi, var);
  }
}

}  // namespace bsfit
