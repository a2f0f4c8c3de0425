// The default kernels of the batched fit with one ROI per warp (launch_batch,
// bsfit_fit.cu).
#include "bsfit_fit_kernels.cuh"

namespace bsfit {

BatchKern batch_kern_default(int mode, bool multi, bool cap) {
  constexpr int M6 = BSFIT_MINBLOCKS(6), M7 = BSFIT_MINBLOCKS(7), M8 = BSFIT_MINBLOCKS(8);
  if (cap) {
    // the serving loop's priority launches
    if (mode == 6 && !multi) return batch_kernel<6, false, M6, 0, true>;
    if (mode == 7) return multi ? batch_kernel<7, true, M7, 0, true> : batch_kernel<7, false, M7, 0, true>;
    if (mode == 8) return multi ? batch_kernel<8, true, M8, 0, true> : batch_kernel<8, false, M8, 0, true>;
    return nullptr;
  }
  if (mode == 6 && !multi) return batch_kernel<6>;
  if (mode == 7) return multi ? batch_kernel<7, true> : batch_kernel<7>;
  if (mode == 8) return multi ? batch_kernel<8, true> : batch_kernel<8>;
  return nullptr;
}

}  // namespace bsfit
