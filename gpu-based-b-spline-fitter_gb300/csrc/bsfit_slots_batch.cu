// The batched kernels with several ROIs in flight per warp (launches in
// bsfit_slots.cu).
#include "bsfit_slots.cuh"

namespace bsfit {

BatchKern slot_batch_kern(int mode, bool multi) {
  constexpr int M6 = slot_min_blocks(6), M7 = slot_min_blocks(7), M8 = slot_min_blocks(8);
  if (mode == 6 && !multi) return slot_batch_kernel<6, false, M6>;
  if (mode == 7) return multi ? slot_batch_kernel<7, true, M7> : slot_batch_kernel<7, false, M7>;
  if (mode == 8) return multi ? slot_batch_kernel<8, true, M8> : slot_batch_kernel<8, false, M8>;
  return nullptr;
}

}  // namespace bsfit
