// One-ROI-per-block fit kernels of 16 warps.
#include "bsfit_team.cuh"

namespace bsfit {

TeamKern team_kern16(int mode, bool multi, bool var) {
  if (mode == 8) return team_kern<8, 16, 1>(multi, var);
  if (mode == kFit4Pi) return team_kern<kFit4Pi, 16, 1>(multi, var);
  return nullptr;
}

}  // namespace bsfit
