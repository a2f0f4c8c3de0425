// Launches of the one-ROI-per-block fit kernels (bsfit_team.cuh): the 8-warp
// instantiations and the choice of the form. The 4- and 16-warp ones are
// compiled beside it (bsfit_team4.cu, bsfit_team4_dense.cu, bsfit_team16.cu).
#include <cstdint>

#include "bsfit_team.cuh"

namespace bsfit {

namespace {

TeamKern team_kern8(int mode, bool multi, bool var) {
  switch (mode) {
    case 6: return team_kern<6, 8, 2>(multi, var);
    case 7: return team_kern<7, 8, 2>(multi, var);
    case 8: return team_kern<8, 8, 2>(multi, var);
    default: return team_kern<kFit4Pi, 8, 2>(multi, var);
  }
}

// A form: warps per block, blocks per SM that it is compiled for, and the most ROIs
// per SM that it is used for. The first whose range holds the call is taken. Measured (GB300, 152
// SMs; us per call, ROIs of 13 px for 3D and 4D, 17 px for 5D, 4 x 16 px for 4Pi;
// warps/blocks):
//
//   ROIs            1    150    300    450    600    750/800   900/1000
//   3D   one warp  54     99     99     99    101     102        105
//        8/2       28     50     53     75     86     105        128
//        8/4       30     56     59     63     80      96        108
//        4/4       42     76     77     61     69      89         99
//        4/6        -      -     64     65     73      77         98
//        4/8       42     76     77     79     88      91        101
//   4D   one warp 350    390    393    397    395     435        441
//        8/2      175    181    209    330    399     504        593
//        4/4      202    207    228    246    273     389        467
//        4/5        -      -    271    277    305     352        485
//   5D   one warp 987   1041   1049   1077   1073    1334       1342
//        16/1     363    387    742      -   1409       -       2219
//        8/2      414    445    551    960   1033    1425       1678
//        4/3        -      -    625    647   1104    1200       1463
//        4/4      617    617    676    737    817    1276       1520
//        4/5        -      -    868    889    965    1105       1756
//   4Pi  one warp 435    597    604    606    627     672        672
//        16/1     106    144    276      -    468       -        724
//        8/2      118    161    198    314    368     461        545
//        4/4      163    217    249    261    404     449        549 (1300: 667 / 738)
//
// A call within one wave of blocks ends with its slowest fit, so the most warps per
// ROI, and the most registers per thread (128 against 64 for 3D, where 64 spill),
// win as long as one wave holds the call; beyond the last form the one-warp form's
// better throughput counts. 16 warps pay for the models whose stage A is the longest
// part (5D) or whose four channels share the block (4Pi).
struct Form {
  int mode, warps, blocks;
  double most;
};
constexpr Form kForms[] = {
    {6, 8, 2, 2.0},       {6, 4, 4, 4.0},       {6, 4, 6, 6.5},
    {7, 8, 2, 2.0},       {7, 4, 4, 4.0},       {7, 4, 5, 5.0},
    {8, 16, 1, 1.0},      {8, 8, 2, 2.0},       {8, 4, 3, 3.0}, {8, 4, 4, 4.0}, {8, 4, 5, 5.0},
    {kFit4Pi, 16, 1, 1.0}, {kFit4Pi, 8, 2, 2.0}, {kFit4Pi, 4, 4, 9.0},
};
constexpr double kMostWaves = 7.0;

}  // namespace

cudaError_t pick_team(int mode, int s, bool var, bool multi, int64_t nfits, TeamLaunch* t) {
  *t = TeamLaunch{nullptr, 0, 0};
  if ((var && multi) || (var && mode == kFit4Pi) || (multi && mode == 6)) return cudaSuccess;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = sm_count(dev, &sms);
  if (e != cudaSuccess) return e;
  const double n = (double)nfits / sms;
  if (n > 9.0) return cudaSuccess;  // past every form
  constexpr int kNumForms = (int)(sizeof(kForms) / sizeof(kForms[0]));
  int at = 0;
  while (at < kNumForms && (kForms[at].mode != mode || n > kForms[at].most)) ++at;
  if (at == kNumForms) return cudaSuccess;
  // Large ROIs: fewer blocks than a form is compiled for fit an SM's shared memory, and
  // unless they still hold the call in one wave, its registers are short for nothing:
  // the next sparser form takes its place, down to the first. Measured (us; one warp /
  // the form by count / this): 5D 27 px, 760 ROIs 2,440 / 3,400 / 2,300, 33 px, 684
  // 3,900 / 5,150 / 2,885; 4Pi 24 px, 530 5,200 / 5,200 / 3,100; 3D 51 px, 760 1,280 /
  // 1,290 / 733.
  int blocks = 0;
  for (; at >= 0 && kForms[at].mode == mode; --at) {
    const Form& f = kForms[at];
    const int T = f.warps;
    TeamKern kern = T == 16 ? team_kern16(mode, multi, var) : T == 8 ? team_kern8(mode, multi, var)
                                                                     : team_kern4(mode, f.blocks, multi, var);
    if (!kern) kern = team_kern4_dense(mode, f.blocks, multi, var);
    const int per_warp = ((make_team_layout(mode, s, var, T).total * 4 + T - 1) / T + 15) & ~15;
    if (!kern || per_warp * T > kTeamMaxShared) continue;
    int wpb = 0, bps = 0;
    e = pick_launch_wpb((const void*)kern, per_warp, T, &wpb, &bps, &sms);
    if (e != cudaSuccess) return e;
    *t = TeamLaunch{kern, 32 * T, per_warp * T};
    blocks = bps;
    if (bps >= f.blocks || n <= bps) break;
  }
  // Several waves win over one warp per ROI up to seven (4Pi, one block per SM, one warp
  // / team: 7 ROIs per SM 24 px 5,760 / 5,450, 22 px 5,250 / 5,180, but 8 5,250 / 5,820).
  if (n > kMostWaves * blocks) *t = TeamLaunch{nullptr, 0, 0};
  return cudaSuccess;
}

}  // namespace bsfit
