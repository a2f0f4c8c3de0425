// Launches of the one-ROI-per-block fit kernels (bsfit_team.cuh): the 8-warp
// instantiations and the choice of the form. The 4- and 16-warp ones are
// compiled beside it (bsfit_team4.cu, bsfit_team16.cu).
#include <cstdint>

#include "bsfit_team.cuh"

namespace bsfit {

TeamKern team_kern8(int mode, bool multi, bool var) { return team_kern<8>(mode, multi, var); }

namespace {

// Largest number of ROIs fitted by blocks of 16, 8 and 4 warps, in ROIs per SM
// (0: not used), where that form was the fastest (GB300, 152 SMs; us per call,
// ROIs of 13 px for 3D and 4D, 17 px for 5D, 4 x 16 px for 4Pi):
//
//   ROIs               1     150     300     450     600     800    1000    1300
//   3D   one warp   54.3    99.6    99.5    99.6   101.1   101.7   104.9   109.5
//        8 warps    30.8    56.5    58.3    62.4    79.2    95.5   108.1   136.3
//        4 warps    42.0    76.1    77.2    79.2    87.9    91.4   101.3   133.7
//   4D   one warp  349.9   390.1   393.4   396.7   394.5   434.6   441.0   479.8
//        8 warps   175.2   180.7   209.2   330.4   398.8   504.2   593.2   736.8
//        4 warps   202.2   206.5   227.7   247.5   273.6   399.9   469.9   538.4
//   5D   one warp   1017    1050    1051    1077    1073    1334    1342    1699
//        16 warps    363     387     742       -    1409       -    2219       -
//        8 warps     436     446     551     960    1033    1425    1678    2059
//        4 warps     617     617     676     741     827    1384    1522    1802
//   4Pi  one warp  441.6   599.7   606.1   606.0   628.6   671.9   673.1   737.5
//        16 warps  105.7   144.4   275.5       -   468.2       -   724.1       -
//        8 warps   120.0   161.0   198.0   314.4   366.8   460.5   546.3   674.5
//        4 warps   162.9   216.7   248.4   263.6   410.0   466.7   552.1   666.8
//
// A call within one wave of 8-warp blocks ends with its slowest fit, so the most
// warps per ROI win; beyond it the 4-warp blocks fit in one wave twice as long;
// beyond that the one-warp form's better throughput counts. 16 warps pay for
// the models whose stage A is the longest part (5D) or whose four channels share
// the block (4Pi), with one block per SM.
struct TeamLimits {
  double w16, w8, w4;
};

TeamLimits team_limits(int mode) {
  switch (mode) {
    case 6: return {0.0, 4.0, 6.5};
    case 7: return {0.0, 2.0, 5.0};
    case 8: return {1.0, 2.0, 4.0};
    default: return {1.0, 2.0, 9.0};
  }
}

}  // namespace

cudaError_t launch_team(const FitArgs& a, bool* taken, cudaStream_t stream) {
  *taken = false;
  const bool var = a.var != nullptr, multi = a.n_starts > 1;
  const int mode = a.m.fittype;
  if (a.trace || a.flags || (var && multi) || (var && mode == kFit4Pi) || (multi && mode == 6))
    return cudaSuccess;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  // a configuration that was put in force for this size is kept
  TuneConfig tc{0, 0};
  if (tune_lookup(mode, a.s, dev, &tc)) return cudaSuccess;
  e = sm_count(dev, &sms);
  if (e != cudaSuccess) return e;
  const TeamLimits lim = team_limits(mode);
  const double n = (double)a.nfits / sms;
  if (n > lim.w4 && n > lim.w8) return cudaSuccess;
  for (int T : {16, 8, 4}) {
    if (n > (T == 16 ? lim.w16 : T == 8 ? lim.w8 : lim.w4)) continue;
    const TeamKern kern = T == 16  ? team_kern16(mode, multi, var)
                          : T == 8 ? team_kern8(mode, multi, var)
                                   : team_kern4(mode, multi, var);
    const int per_warp = ((make_team_layout(mode, a.s, var, T).total * 4 + T - 1) / T + 15) & ~15;
    if (!kern || per_warp * T > kTeamMaxShared) continue;
    int wpb = 0, bps = 0;
    e = pick_launch_wpb((const void*)kern, per_warp, T, &wpb, &bps, &sms);
    if (e != cudaSuccess) return e;
    // large ROIs: fewer blocks fit an SM than the limits above were taken with
    if (n > 1.5 * bps) continue;
    *taken = true;
    kern<<<(unsigned)a.nfits, 32 * T, per_warp * T, stream>>>(a);
    return cudaGetLastError();
  }
  return cudaSuccess;
}

}  // namespace bsfit
