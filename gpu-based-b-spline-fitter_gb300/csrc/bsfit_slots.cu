// Launches of the fit kernels with several ROIs in flight per warp
// (bsfit_slots.cuh).
#include <cstdint>

#include "bsfit_slots.cuh"

namespace bsfit {

namespace {

template <int MODE>
FitKern slot_kern_of(bool multi, bool var) {
  constexpr int B = slot_min_blocks(MODE);
  if (var) return slot_kernel<MODE, false, true, B>;
  if constexpr (MODE != 6) {
    if (multi) return slot_kernel<MODE, true, false, B>;
  }
  return slot_kernel<MODE, false, false, B>;
}

FitKern slot_kern(int mode, bool multi, bool var) {
  return mode == 6   ? slot_kern_of<6>(false, var)
         : mode == 7 ? slot_kern_of<7>(multi, var)
         : mode == 8 ? slot_kern_of<8>(multi, var)
                     : nullptr;
}

// The slot form's place. Measured on GB300 (ms; one ROI per warp / slot form,
// W the warps that the first keeps resident):
//   3D    200,000 x 13 px 5.09 / 4.56    100,000 x 7 px 2.00 / 1.78
//         50,000 x 21 px 2.73 / 2.69     50,000 x 15 px sCMOS 1.65 / 1.53
//         batch of 1,000,000 x 11, 13, 17 px 26.9 / 25.0
//         20,000 x 13 px (5.5 W) 0.593 / 0.561     6,000 (1.6 W) 0.251 / 0.258
//         batch of 10,000 x 11, 13, 17 px (2.7 W) 0.345 / 0.388
//   4D    40,000 x 13 px 6.60 / 5.53     20,000 x 17 px 4.72 / 4.27
//         10,000 x 13 px (4.1 W) 1.87 / 1.75       8,000 x 15 px, 3 starts 5.61 / 5.39
//   5D    12,000 x 13 px 6.05 / 5.57     8,000 x 17 px 6.75 / 6.70
//         2,000 x 17 px (1.1 W) 2.16 / 2.34
// With fewer than three ROIs per warp the slots are seldom full, and the end of the
// work, several ROIs to a warp, costs more than they save.
constexpr int64_t kEnough = 3;
// A 3D batch shares its warps among ROI sizes in the order of their cost, and its
// slots (sized for the largest) are drained at each change. Measured, us, one ROI
// per warp / slots: 11, 13, 17 px 11,500 ROIs (3.2 W) 380 / 421, 20,000 619 / 657,
// 36,000 (9.9 W) 1,048 / 1,072, 45,000 (12.3 W) 1,313 / 1,319, 60,000 1,715 / 1,684;
// 13 px alone 15,000 444 / 457, 20,000 570 / 567, 30,000 806 / 793. A 4D or 5D batch of
// one segment does as its plain call (4D 13 px 4 W 1,752 / 1,699, 5D 13 px 3.1 W 3,219 /
// 3,242, 4 W 4,057 / 3,952), but several lose at each change until their number is small
// against the work: 4D 13, 15 px, two segments 4 W 1,893 / 1,914, 6 W 2,724 / 2,839, 8 W
// 3,558 / 3,528, four 5 W 2,320 / 2,630, 8 W 3,551 / 3,349; 5D 13 px, two 5 W 4,957 /
// 5,667, 6 W 5,866 / 6,371, 8 W 7,659 / 7,655, 12 W 11,236 / 10,587.
constexpr int64_t kEnoughBatch3D = 12, kEnoughSegments = 8;
// Warps stop taking further ROIs when two per warp are left: 0, 1, 2, 3 measured
// 7.54, 7.01, 6.68, 6.77 ms on 8,000 5D ROIs, 5.68, 5.64, 5.54, 5.60 ms on 40,000
// 4D ROIs, within 0.2% on 200,000 3D ROIs.
constexpr int64_t kSparePerWarp = 2;

// The most slots that pay. q->slots 0: not even two do. more: floats per warp besides the
// layout's. The slots' shared memory costs resident warps or L1, which 3D minds least:
// - 3D: as many warps as with one ROI per warp (to 5%), else 85% of them (21 px: 17 per SM
//   against 20, and still 1.5% faster);
// - 4D: a tenth more warps, which 96 registers allow against 128; with as many, one ROI
//   per warp is as fast or faster (ms, 60 ROIs per SM: 25 px 4.08 / 4.12, 24 px, 14 warps
//   against 16, 4.54 / 4.83; 21 px, 18 against 16, 3.04 / 2.97);
// - 5D: all of the warps, at least 7 (50 ROIs per SM: 25 px, 6 warps, 14.1 / 14.5, 33 px,
//   4, 27.8 / 29.1; 19 px, 9 against 10, 55 per SM, 8.67 / 9.08), and the gathers' L1:
//   past the 196 KB configuration of shared memory the SM takes its largest and leaves them
//   28 KB of 60 (KB of shared memory per SM, ms; 14 px, 36 per SM, one ROI per warp 169,
//   3.55, three slots 193, 3.50, four 201, 3.97; 15 px, 42 per SM, one ROI per warp 180,
//   4.41, two slots 195.9, 4.93).
constexpr int kMinWarps5D = 7;
constexpr int64_t kSharedL1 = 194 * 1024, kBlockReserve = 1024;  // bytes per SM, per block

cudaError_t most_slots(const void* kern, int mode, int s, bool var, bool multi, int more, int wpb,
                       int64_t warps, SlotLaunch* q) {
  constexpr int least[3][2] = {{95, 85}, {110, 110}, {100, 100}};  // % of the warps, tried in turn
  for (int pass = 0; pass < 2; ++pass)
    for (int r = kMaxSlots; r >= 2; --r) {
      SlotLaunch t{r, (make_slot_layout(mode, s, var, r, multi).total + more) * 4, 0, 0, 0};
      if (pick_launch_wpb(kern, t.per_warp, wpb, &t.wpb, &t.bps, &t.sms) != cudaSuccess) continue;
      if ((int64_t)t.wpb * t.bps * t.sms * 100 < least[mode - 6][pass] * warps) continue;
      if (mode == 8) {
        if (t.wpb * t.bps < kMinWarps5D) continue;
        const int64_t one = warps / t.sms;  // warps per SM with one ROI each, four per block
        const int64_t before = one * make_layout(mode, s, var).total() * 4 + (one + 3) / 4 * kBlockReserve;
        const int64_t now = t.bps * ((int64_t)t.per_warp * t.wpb + kBlockReserve);
        if (now > kSharedL1 && before <= kSharedL1) continue;
      }
      *q = t;
      return cudaSuccess;
    }
  return cudaSuccess;
}

}  // namespace

cudaError_t pick_slots(int mode, int s, bool var, bool multi, int64_t nfits, int wpb, int64_t warps,
                       SlotLaunch* q) {
  *q = SlotLaunch{};
  if (nfits < kEnough * warps) return cudaSuccess;
  const FitKern kern = slot_kern(mode, multi, var);
  return kern ? most_slots((const void*)kern, mode, s, var, multi, 0, wpb, warps, q) : cudaSuccess;
}

cudaError_t pick_slots_batch(int mode, int s_max, bool multi, int segments, int64_t total, int wpb, int64_t warps,
                             SlotLaunch* q) {
  *q = SlotLaunch{};
  if (total < (mode == 6 ? kEnoughBatch3D : segments > 1 ? kEnoughSegments : kEnough) * warps) return cudaSuccess;
  const BatchKern kern = slot_batch_kern(mode, multi);
  return kern ? most_slots((const void*)kern, mode, s_max, false, multi, kSegWords, wpb, warps, q) : cudaSuccess;
}

cudaError_t launch_slots(const FitArgs& a, const SlotLaunch& q, bool* taken, cudaStream_t stream) {
  FitArgs b = a;
  WorkCounter claim;
  b.slots = q.slots;
  b.claim = claim.get(stream);
  *taken = b.claim != nullptr;
  if (!*taken) return cudaSuccess;
  const int64_t grid = (int64_t)q.sms * q.bps;
  b.spare = kSparePerWarp * grid * q.wpb;
  slot_kern(a.m.fittype, a.n_starts > 1, a.var != nullptr)
      <<<(unsigned)grid, 32 * q.wpb, q.per_warp * q.wpb, stream>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_slots_batch(const BatchArgs& a, int mode, bool multi, const SlotLaunch& q, cudaStream_t stream) {
  BatchArgs b = a;
  b.slots = q.slots;
  const int64_t grid = (int64_t)q.sms * q.bps;
  b.spare = kSparePerWarp * grid * q.wpb;
  slot_batch_kern(mode, multi)<<<(unsigned)grid, 32 * q.wpb, q.per_warp * q.wpb, stream>>>(b);
  return cudaGetLastError();
}

}  // namespace bsfit
