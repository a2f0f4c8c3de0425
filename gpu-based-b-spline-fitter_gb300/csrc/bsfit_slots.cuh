// Several ROIs in flight per warp: the "slot" form of the FP32 fit kernels of fit
// types 6, 7 and 8, for calls with many more ROIs than resident warps
// (bsfit_team.cuh fits the small calls, fit_kernel one ROI per warp those between).
//
// What bounds these kernels is instruction issue (3D: 3.2 of 4 per cycle), and a
// fifth of a fit's instructions are the LM step's, a 5 x 5 (6 x 6, 8 x 8) solve on
// one lane per parameter: 600 (750, 1100) warp instructions for 5 (6, 8) useful
// lanes. Here a warp holds up to four ROIs, one per group of eight lanes, which own
// the group's LM state as the lanes of fit_roi own theirs. The whole warp evaluates
// the ROIs one after the other, in one set of maps, and leaves each one's sums in
// shared memory; then one LM step serves all of them. A ROI that stops has its
// Fisher pass at once, on the maps of its last evaluation, and its slot takes the
// next ROI before the step, so the groups stay full; towards the end of the work the
// warps take fewer (see SlotSource).
//
// What it took: no LM state in registers through the evaluations (see SlotLayout),
// or the compiler recomputes addresses and reloads to stay within the budget: warp
// instructions per 3D evaluation, LM step included, 2,840 with the state and the
// work source in registers, 2,420 with the state in shared memory, 2,270 with the
// source there too, 2,520 in the one-ROI form.
//
// Results are bit-identical to fit_roi: the evaluation is the same code, the LM
// step and the CRLB are the same per-lane operations with the broadcasts taken
// within the group, and sums that fit_roi takes over zero lanes leave them out.
//
// Measured: bsfit_slots.cu.
#pragma once

#include "bsfit_fit_kernels.cuh"

namespace bsfit {

constexpr int kMaxSlots = 4;  // groups of eight lanes

// Minimum resident blocks of 4 warps per SM (the register budget): 80, 96 and 168
// registers for fit types 6, 7 and 8. Without LM state in registers the 4D kernel
// fits 96 (the one-ROI form runs at 128): 40,000 ROIs of 13 px 5.92 -> 5.81 ms.
constexpr int slot_min_blocks(int mode) { return mode == 6 ? 6 : mode == 7 ? 5 : 3; }

// What a slot keeps of its ROI, the same for all lanes of its group.
struct __align__(16) SlotState {
  int64_t roi;
  int code;    // kEmpty ..
  int start;   // several starts: the start that is being fitted
  float err_hi, err_lo, oerr_hi, oerr_lo;
  float lambda, olambda, sum_update;
  int turn;
  int kk;
  int best_iters;  // several starts: the best result's iterations and log-likelihood
  float best_ll;
  int pad;
};
constexpr int kSlotWords = sizeof(SlotState) / 4;

// What a warp keeps between evaluations, in shared memory (the evaluation is
// short of registers).
struct __align__(16) WarpState {
  int64_t left;   // ROIs left when this warp last took one
  int staged;     // the slot whose pixels are in shared memory
  unsigned busy;  // slots with a ROI
};
constexpr int kWarpWords = sizeof(WarpState) / 4;

// Per-lane LM state in rows of 8 lanes per slot: value, value before the last
// step, signs and clamps of the last two; with several starts the initial guess
// and the best result; for fit type 8 the value at the last evaluation.
enum { kPar, kOpar, kSg, kOsg, kCl, kOcl, kGuess, kBestPar, kBestCrlb };
constexpr int kLaneRows = 6, kLaneRowsMulti = 9;

// Shared memory of a warp (floats): the one-ROI layout, whose pixel planes hold
// the ROI that is being evaluated (the others' are fetched again, from L2, when
// their turn comes: four ROIs of 17 px would take the room of 8 of 24 warps),
// then per slot its sums as NV rows (Hessian row l, gradient entry l; `row` floats
// apart, read as vectors by the LM lanes), and the slots' and lanes' state. The
// state lives here and not in registers: only the LM step needs it.
struct SlotLayout {
  WarpLayout L;
  int row, sums, sums_size, slot, warp, lanes, total;
};

__host__ __device__ constexpr SlotLayout make_slot_layout(int mode, int s, bool var, int slots, bool multi) {
  SlotLayout t{};
  t.L = make_layout(mode, s, var);
  const int nv = mode == 6 ? 5 : mode == 7 ? 6 : 8;
  t.row = nv + 1 <= 8 ? 8 : 12;
  t.sums = t.L.total();
  t.sums_size = nv * t.row;
  t.slot = t.sums + slots * t.sums_size;
  t.warp = t.slot + slots * kSlotWords;
  t.lanes = t.warp + kWarpWords;
  t.total = t.lanes + ((multi ? kLaneRowsMulti : kLaneRows) + (mode == 8 ? 1 : 0)) * 8 * slots;
  return t;
}

// Index of the value that `lane` holds in slot i after reduce_scatter<C, 16>.
template <int C>
__device__ __forceinline__ int rs_value(int lane, int i) {
  int size[5] = {C, 0, 0, 0, 0};
#pragma unroll
  for (int l = 1; l < 5; ++l) size[l] = size[l - 1] / 2 + (size[l - 1] & 1);
#pragma unroll
  for (int l = 4; l >= 0; --l) {
    const int half = size[l] / 2;
    i = i < half ? i + ((lane & (16 >> l)) ? half : 0) : 2 * half;
  }
  return i;
}

// Where a warp's ROIs come from: a shared work counter. A warp with a ROI in
// flight only takes another while more than `spare` are left: a warp works off its
// ROIs together, so at the end of the work several of them in one warp would
// finish after the others have run dry.
struct SlotSource {
  unsigned long long* counter;
  int64_t n;      // ROIs behind the counter
  int64_t later;  // ROIs of the work that follows (further segments)
  int64_t spare;
};

// Fit every ROI that the warp takes from src, in up to `slots` slots. done:
// optional counter of finished ROIs.
template <int MODE, bool MULTI, bool VAR, class Args>
__device__ __forceinline__ void fit_slots(const Args& a, const SlotLayout& SL, float* ws, int lane,
                                          int slots, const SlotSource& src, unsigned long long* done) {
  using TR = ModeTraits<MODE>;
  constexpr int NV = TR::NV;
  constexpr int K = NV + NV * (NV + 1) / 2;
  constexpr int KP = (K + 31) / 32 * 32;
  static_assert(TR::NCH == 1 && NV <= 8, "one image channel, one lane of the group per parameter");
  // slot codes: no ROI; an evaluation is due (the first one, one of the fit, the
  // Fisher pass); a step is due, or due again after a failed solve
  enum { kEmpty, kFirst, kEval, kFisher, kStep, kRetry };
  constexpr int RW = NV + 1 <= 8 ? 8 : 12;  // SlotLayout::row
  constexpr int kParEval = MULTI ? kLaneRowsMulti : kLaneRows;
  const int lw = 8 * slots;  // lanes of a row
  const WarpLayout& L = SL.L;
  const int s = L.s, s2 = s * s;
  const int li = lane & 7, grp = lane >> 3;
  const int ns = (MULTI && a.n_starts > 0) ? a.n_starts : 1;  // 0: the model's initP alone
  SlotState* slot = reinterpret_cast<SlotState*>(ws + SL.slot);
  float* lanes = ws + SL.lanes;
  const unsigned walk = Stride2D(lane, s).pack();
  // where this lane's totals go: gradient entry l to (l, NV), Hessian entry
  // (l, m) to (l, m) and (m, l); two places per value, in halves of a word
  unsigned place[rs_slots(K)];
#pragma unroll
  for (int i = 0; i < rs_slots(K); ++i) {
    const int x = rs_value<K>(lane, i);
    int l = x, m = NV;
    if (x >= NV) {
      l = 0;
      for (m = x - NV; m >= NV - l; ++l) m -= NV - l;
      m += l;
    }
    place[i] = (unsigned)(l * RW + m) | (unsigned)(x < NV ? l * RW + m : m * RW + l) << 16;
  }
  WarpState* wst = reinterpret_cast<WarpState*>(ws + SL.warp);
  if (lane < slots) slot[lane].code = kEmpty;
  if (lane == 0) {
    wst->staged = -1;
    wst->busy = 0;
    wst->left = src.n;
  }
  __syncwarp();
  for (;;) {
    // (1) slot by slot: take a ROI, evaluate, and finish it when it stops
    bool maps = false;  // the maps are those of this slot's last evaluation
    for (int r = 0; r < slots;) {
      SlotState* me = slot + r;
      float* mine = lanes + 8 * r;
      int code = me->code;
      if (code == kEmpty) {
        const int64_t left = wst->left;
        if (left <= 0 || (wst->busy && left + src.later <= src.spare)) {
          ++r;
          continue;
        }
        unsigned long long taken = 0;
        if (lane == 0) taken = atomicAdd(src.counter, 1ull);
        const int64_t roi = (int64_t)__shfl_sync(kFull, taken, 0);
        if (lane == 0) wst->left = src.n - 1 - roi;
        __syncwarp();
        if (roi >= src.n) continue;
        load_roi<MODE, VAR>(a, L, ws, lane, roi);
        const float g = start_guess<MODE>(L, ws, lane);
        if (lane < 8) {
          mine[kPar * lw + lane] = start_params<MODE>(a, lane, roi, 0, g);
          if constexpr (MULTI) mine[kGuess * lw + lane] = g;
        }
        if (lane == 0) {
          me->roi = roi;
          me->start = 0;
          wst->staged = r;
          wst->busy |= 1u << r;
        }
        code = kFirst;
        __syncwarp();
      } else if (code >= kStep) {
        ++r;
        continue;
      } else if (wst->staged != r) {
        // this slot's pixels, in flight until stage C (channel_pass waits)
        cp_async_warp(ws, a.rois + me->roi * s2, s2, lane);
        if constexpr (VAR) cp_async_warp(ws + L.s2p, a.var + me->roi * s2, s2, lane);
        __syncwarp();
        if (lane == 0) wst->staged = r;
      }
      if (code == kFirst && lane < 8) {
        // CPUmleFit_LM.cpp:2425-2450
        float cl, fd;
        clamp_fade<MODE>(lane, cl, fd);
        mine[kSg * lw + lane] = mine[kOsg * lw + lane] = 0.0f;
        mine[kCl * lw + lane] = mine[kOcl * lw + lane] = cl;
        if (lane == 0) {
          me->oerr_hi = 1e13f;
          me->oerr_lo = 0.0f;
          me->lambda = me->olambda = 1.0f;
          me->sum_update = 1e10f;
          me->turn = 1;
          me->kk = 0;
        }
      }
      const bool fish = code == kFisher;
      // fit type 8's Fisher pass keeps the positions and g2 of the last
      // evaluation (CPUmleFit_LM.cpp:3568-3584)
      float th[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k)
        th[k] = mine[((MODE == 8 && fish && k != 2 && k != 3) ? kParEval : kPar) * lw + k];
      float* sums = ws + SL.sums + r * SL.sums_size;
      FPair e{0.0f, 0.0f};
      {
        float acc[KP];
#pragma unroll
        for (int k = 0; k < KP; ++k) acc[k] = 0.0f;
        channel_pass<MODE, KP, VAR, 0, 32, 0, true>(a, L, ws, ws, lane, th, MODE == 7 && code == kFirst, fish, e,
                                                    acc, e, acc, kFull, maps, nullptr, nullptr, 0, nullptr, walk);
        reduce_scatter<K, 16>(acc, lane);
#pragma unroll
        for (int i = 0; i < rs_slots(K); ++i) {
          sums[place[i] & 0xffffu] = acc[i];
          sums[place[i] >> 16] = acc[i];
        }
        e = warp_sum_pair(e);
      }
      if (!fish) {
        LmLane st;
        st.err = e;
        st.oerr = FPair{me->oerr_hi, me->oerr_lo};
        st.sum_update = me->sum_update;
        maps = me->kk >= a.iterations || lm_converged<MODE>(st);  // then the Fisher pass follows
        __syncwarp();
        if (MODE == 8 && lane < 8) mine[kParEval * lw + lane] = mine[kPar * lw + lane];
        if (lane == 0) {
          me->err_hi = e.hi;
          me->err_lo = e.lo;
          me->code = maps ? kFisher : kStep;
        }
        __syncwarp();
        if (!maps) ++r;
        continue;
      }
      // the Fisher pass has run: variances and result
      maps = false;
      __syncwarp();
      const int i = lane < NV ? lane : NV - 1;
      float hr[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) hr[k] = sums[i * RW + k];
      float crlb = fisher_crlb<NV>(lane, hr);
      float ll = e.hi + e.lo, par = mine[kPar * lw + i];
      int iters = me->kk;
      const int64_t roi = me->roi;
      if constexpr (MULTI) {
        // keep the better result (fit_and_store's rule), then the next start
        const int k = me->start;
        const float d = ll - me->best_ll;
        if (k == 0 || (a.strict ? (d > 1e-4f) : (d >= 1e-4f))) {
          __syncwarp();
          if (lane < NV) {
            mine[kBestPar * lw + lane] = par;
            mine[kBestCrlb * lw + lane] = crlb;
          }
          if (lane == 0) {
            me->best_ll = ll;
            me->best_iters = iters;
          }
        }
        __syncwarp();
        if (k + 1 < ns) {
          if (lane < 8) mine[kPar * lw + lane] = start_params<MODE>(a, lane, roi, k + 1, mine[kGuess * lw + lane]);
          if (lane == 0) {
            me->start = k + 1;
            me->code = kFirst;
          }
          __syncwarp();
          continue;
        }
        par = mine[kBestPar * lw + i];
        crlb = mine[kBestCrlb * lw + i];
        ll = me->best_ll;
        iters = me->best_iters;
      }
      const int64_t o = a.out_offset + roi;
      if (lane < NV) {
        a.P[lane * a.out_n + o] = par;
        a.CRLB[lane * a.out_n + o] = crlb;
      }
      __syncwarp();
      if (lane == 0) {
        a.P[NV * a.out_n + o] = (float)iters;
        a.LL[o] = ll;
        if (done) atomicAdd(done, 1ull);
        me->code = kEmpty;
        wst->busy &= ~(1u << r);
      }
      __syncwarp();
    }
    if (wst->busy == 0) return;

    // (2) one LM step of every group that has one to make; the other groups' lanes
    // run the solve on values that they do not keep
    SlotState* me = slot + (grp < slots ? grp : 0);
    float* own = lanes + (grp < slots ? lane : li);
    int code = grp < slots ? me->code : (int)kEmpty;
    LmLane st;
    st.par = own[kPar * lw];
    st.opar = own[kOpar * lw];
    st.sg = own[kSg * lw];
    st.osg = own[kOsg * lw];
    st.cl = own[kCl * lw];
    st.ocl = own[kOcl * lw];
    st.err = FPair{me->err_hi, me->err_lo};
    st.oerr = FPair{me->oerr_hi, me->oerr_lo};
    st.lambda = me->lambda;
    st.olambda = me->olambda;
    st.sum_update = me->sum_update;
    st.turn = me->turn;
    const int kk = me->kk;
    {
      float cl;
      clamp_fade<MODE>(li, cl, st.fd);
    }
    if (code == kRetry && (kk >= a.iterations || lm_converged<MODE>(st))) code = kFisher;
    const bool step = code >= kStep;
    if (step) lm_weigh(st);
    float* sums = ws + SL.sums + (grp < slots ? grp : 0) * SL.sums_size + (li < NV ? li : NV - 1) * RW;
    float hr[NV], gl;
    {
      float v[RW];
#pragma unroll
      for (int k = 0; k < RW; k += 4) {
        const float4 q = *reinterpret_cast<const float4*>(sums + k);
        v[k] = q.x;
        v[k + 1] = q.y;
        v[k + 2] = q.z;
        v[k + 3] = q.w;
      }
#pragma unroll
      for (int k = 0; k < NV; ++k) hr[k] = (li == k) ? v[k] * st.lambda : v[k];
      gl = v[NV];
    }
    bool ok;
    float upd = lm_solve_lanes<MODE, 8>(li, hr, gl, true, ok);
    const float dz = (MODE == 7) ? bcast<8>(upd, 4) : 0.0f;
    float made = 0.0f;
    if (step && ok)
      made = lm_apply<MODE>(st, a.m, li, upd, dz, [&](float p) { return lm_bounds<MODE>(p, a.m, s, li); });
    if (MODE == 8) {
      made = lm_step_sum<NV, 8>(li, made);
      if (step && ok) st.sum_update = made;
    }
    __syncwarp();
    if (step) {
      own[kPar * lw] = st.par;
      own[kOpar * lw] = st.opar;
      own[kSg * lw] = st.sg;
      own[kOsg * lw] = st.osg;
      own[kCl * lw] = st.cl;
      own[kOcl * lw] = st.ocl;
      if (!ok) {
        // the damping of a failed solve stays (cumulative, as in the reference)
        if (li < NV) sums[li] *= st.lambda;
        st.lambda = 10.0f * st.lambda;
      }
      if (li == 0) {
        me->err_hi = st.err.hi;
        me->err_lo = st.err.lo;
        me->oerr_hi = st.oerr.hi;
        me->oerr_lo = st.oerr.lo;
        me->lambda = st.lambda;
        me->olambda = st.olambda;
        me->sum_update = st.sum_update;
        me->turn = st.turn;
        me->kk = kk + 1;
      }
      code = ok ? kEval : kRetry;
    }
    if (li == 0 && grp < slots) me->code = code;
    __syncwarp();
  }
}

// Plain form; a.claim: the work counter.
template <int MODE, bool MULTI, bool VAR, int MINB>
__global__ void __launch_bounds__(128, MINB) slot_kernel(const __grid_constant__ FitArgs a) {
  extern __shared__ float4 smem4[];
  const SlotLayout SL = make_slot_layout(MODE, a.s, VAR, a.slots, MULTI);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float* ws = reinterpret_cast<float*>(smem4) + wib * SL.total;
  const SlotSource src{a.claim, a.nfits, 0, a.spare};
  fit_slots<MODE, MULTI, VAR>(a, SL, ws, lane, a.slots, src, nullptr);
}

// What the batched form needs of a warp's segment, in shared memory: kept in
// registers, or fetched from the parameters by the compiler's choice, it took
// registers from the evaluation.
struct __align__(16) SegArgs {
  ModelDev m;
  const float* rois;
  float *P, *CRLB, *LL;
  int64_t nfits, out_n, out_offset;
  int iterations, n_starts, strict;
  const float (*starts)[4];
  SlotSource source;
};
constexpr int kSegWords = sizeof(SegArgs) / 4;

// Batched form: the segments one after the other (the host sorts them by
// decreasing cost), each worked off by all warps from its own counter; the
// warp's shared memory is laid out for the largest ROI of the batch.
template <int MODE, bool MULTI, int MINB>
__global__ void __launch_bounds__(128, MINB) slot_batch_kernel(const __grid_constant__ BatchArgs a) {
  extern __shared__ float4 smem4[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int room = make_slot_layout(MODE, a.s_max, false, a.slots, MULTI).total;
  float* ws = reinterpret_cast<float*>(smem4) + wib * (room + kSegWords);
  SegArgs& fa = *reinterpret_cast<SegArgs*>(ws + room);
  for (int seg = 0; seg < a.nseg; ++seg) {
    const BatchSeg& g = a.seg[seg];
    if (lane == 0) {
      fa.m = g.m;
      fa.rois = g.rois;
      fa.nfits = fa.out_n = g.n;
      fa.out_offset = 0;
      fa.iterations = g.iterations;
      fa.P = g.P;
      fa.CRLB = g.CRLB;
      fa.LL = g.LL;
      fa.n_starts = MULTI ? g.n_starts : 0;
      fa.strict = g.strict;
      fa.starts = g.starts;
      fa.source = SlotSource{&a.next[g.slot], g.n, 0, a.spare};
      for (int k = seg + 1; k < a.nseg; ++k) fa.source.later += a.seg[k].n;
    }
    __syncwarp();
    fit_slots<MODE, MULTI, false>(fa, make_slot_layout(MODE, g.s, false, a.slots, MULTI), ws, lane, a.slots,
                                  fa.source, &a.done[g.slot]);
    __syncwarp();
  }
}

BatchKern slot_batch_kern(int mode, bool multi);

}  // namespace bsfit
