// One ROI per block: the "team" form of the FP32 fit kernels, for launches with
// too few ROIs to fill the GPU with one warp each.
//
// What bounds such a launch is the latency of one fit: a chain of LM
// iterations, each an evaluation and a small solve, that one warp works off at
// well under one instruction per cycle. Here the T warps of a block share every
// evaluation: stages A and B and the per-pixel part of stage C are spread over
// all threads (channel_pass with TW = T), each pixel's terms go to shared
// memory, and the sums over the pixels are shared out by sum: warps 0 .. T - 2
// take the gradient and Hessian sums, warp T - 1 the compensated deviance. Warp
// 0 then does the LM step, with the factorisation and the triangular solves on
// every lane at once (their chain has no shuffles in it), and the block goes on
// with the parameters that it leaves in shared memory. Five block barriers per
// iteration.
//
// Results are bit-identical to the one-warp form (fit_roi): nodes, items and
// pixel terms are the same operations; the warp that forms a sum takes lane l
// through pixels l, l + 32, l + 64, ... as the one-warp form does and ends with
// the same butterfly tree; the LM step is the lane-parallel one's operations in
// its order (lm_solve).
//
// Measured (GB300): one 13 px 3D ROI 28 us per call against 54 us with one warp, 300
// of them 53 against 99 us; where each form is used and what it measured there:
// bsfit_team.cu.
#pragma once

#include "bsfit_fit_kernels.cuh"

namespace bsfit {

// Shared memory of a team (floats): the one-warp layout with the map sets apart
// (alias off: all threads work on one stage at once) and stage C's records over
// the stage-A maps (free by then), one such set per image channel (`set` floats
// apart: 4Pi's channels are evaluated side by side, T / 4 warps each), one more
// knot and weight region per further warp, the K sums, the deviance pair, the
// parameters and the control words.
struct TeamLayout {
  WarpLayout L;
  int rec, set, kws, sums, theta, ctl, total;
};

constexpr int kTeamCtl = 4;  // go, fisher, maps_ready, first

__host__ __device__ constexpr int mode_nv(int mode) {
  return mode == 6 ? 5 : mode == 8 ? 8 : 6;
}

__host__ __device__ constexpr TeamLayout make_team_layout(int mode, int s, bool var, int warps) {
  TeamLayout t{};
  t.L = make_layout(mode, s, var);
  t.L.alias = false;
  const int nv = mode_nv(mode);
  const int a_floats = t.L.wp * t.L.as(), r_floats = (3 + nv) * t.L.s2p;
  t.rec = t.L.off_a();
  t.set = (t.rec - t.L.off_maps() + (a_floats > r_floats ? a_floats : r_floats) + 3) & ~3;
  t.kws = t.L.off_maps() + t.L.nch * t.set;
  const int small = t.L.off_dt() - t.L.off_kx();
  t.sums = t.kws + (warps - 1) * small;
  t.theta = t.sums + ((nv + nv * (nv + 1) / 2 + 2 + 3) & ~3);
  t.ctl = t.theta + 8;
  t.total = t.ctl + kTeamCtl;
  return t;
}

// What a thread keeps through a fit: its walk over the stage-B items and the
// pixels (rows of s; the nodes' rows change with the window) and, for
// warps 0 .. T - 2, the sums that its warp forms (sum warp + (T - 1) j: gradient
// entry m, or Hessian entry (l, m); l + 3 and m + 3 in lm[j]'s low and high half).
template <int MODE, int T>
struct TeamThread {
  static constexpr int NV = ModeTraits<MODE>::NV;
  static constexpr int K = NV + NV * (NV + 1) / 2;
  static constexpr int SPW = (K + T - 2) / (T - 1);  // sums per warp
  static constexpr int TC = T / ModeTraits<MODE>::NCH;  // warps per image channel
  Stride2D walk;
  unsigned lm[SPW];
  __device__ __forceinline__ TeamThread(int warp, int s) : walk(threadIdx.x % (32 * TC), s, 32 * TC) {
#pragma unroll
    for (int j = 0; j < SPW; ++j) {
      const int k = min(warp + (T - 1) * j, K - 1);
      int l = 0, m = k;
      if (k >= NV) {
        for (m = k - NV; m >= NV - l; ++l) m -= NV - l;
        m += l;
      }
      lm[j] = (unsigned)(l + 3) | (unsigned)(m + 3) << 16;
    }
  }
};

// One evaluation by the whole block: the K sums at ws[TL.sums + k] (gradient
// 0 .. NV - 1, packed upper triangle), the deviance or log-likelihood pair
// behind them. Ends before the barrier that publishes them.
template <int MODE, bool VAR, int T>
__device__ __forceinline__ void evaluate_team(const FitArgs& a, const TeamLayout& TL, float* ws,
                                              float* kws, int lane, int warp,
                                              const TeamThread<MODE, T>& me, const float* th,
                                              bool dup45, bool fisher, bool maps_ready) {
  using TR = ModeTraits<MODE>;
  using TT = TeamThread<MODE, T>;
  constexpr int NV = TR::NV;
  constexpr int K = TT::K;
  constexpr int KP = (K + 31) / 32 * 32;
  constexpr int SPW = TT::SPW, TC = TT::TC;
  const WarpLayout& L = TL.L;
  const int s2 = L.s * L.s, rs = L.s2p;
  {
    FPair none{0.0f, 0.0f};
    float unused[KP];
    if constexpr (TR::NCH == 1) {
      channel_pass<MODE, KP, VAR, 0, 32, T>(a, L, ws, ws, lane, th, dup45, fisher, none, unused, none,
                                            unused, kFull, maps_ready, kws, ws + TL.rec, threadIdx.x,
                                            &me.walk);
    } else {
      const int ch = warp / TC;
      const float* dts = ws + L.off_dt() + ch * NV;
      float thc[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) thc[k] = th[k] + dts[k];
      thc[5] = wrap_phase(thc[5] + a.m.shift[ch], a.m.n[3]);
      float* wc = ws + ch * TL.set;
      channel_pass<MODE, KP, VAR, 0, 32, TC>(a, L, wc, ws + ch * rs, lane, thc, false, fisher, none,
                                             unused, none, unused, kFull, false, kws, wc + TL.rec,
                                             threadIdx.x - ch * 32 * TC, &me.walk);
    }
  }
  __syncthreads();
  const float* rec = ws + TL.rec;
  if (warp == T - 1) {
    FPair err{0.0f, 0.0f};
    for (int ch = 0; ch < TR::NCH; ++ch) {
      const float* e = rec + ch * TL.set;
      for (int p = lane; p < s2; p += 32) err.add(e[p]);
    }
    err = warp_sum_pair(err);
    if (lane == 0) {
      ws[TL.sums + K] = err.hi;
      ws[TL.sums + K + 1] = err.lo;
    }
  } else {
    // This warp's sums: x = t1 and y = dudt[l] for gradient entry l, x = t2 *
    // dudt[l] and y = dudt[m] for Hessian entry (l, m).
    int ot[SPW], ol[SPW], om[SPW];
    float acc[SPW];
#pragma unroll
    for (int j = 0; j < SPW; ++j) {
      ot[j] = (warp + (T - 1) * j < NV ? 1 : 2) * rs + lane;
      ol[j] = (int)(me.lm[j] & 0xffffu) * rs + lane;
      om[j] = (int)(me.lm[j] >> 16) * rs + lane;
      acc[j] = 0.0f;
    }
    for (int ch = 0; ch < TR::NCH; ++ch) {
      const float* r = rec + ch * TL.set;
#pragma unroll 2
      for (int p = lane; p < s2; p += 32, r += 32) {
#pragma unroll
        for (int j = 0; j < SPW; ++j) {
          float x = r[ot[j]];
          const float tl = x * r[ol[j]];
          if (warp + (T - 1) * j >= NV) x = tl;
          acc[j] = fmaf(x, r[om[j]], acc[j]);
        }
      }
    }
    warp_sum_array<SPW>(acc);
#pragma unroll
    for (int j = 0; j < SPW; ++j)
      if (lane == 0 && warp + (T - 1) * j < K) ws[TL.sums + warp + (T - 1) * j] = acc[j];
  }
}

// (L L^T) x = b on every lane: lane_solve's operations in its order.
template <int NV>
__device__ __forceinline__ void chol_substitute(const float (&l)[NV][NV], const float (&invd)[NV],
                                                const float (&b)[NV], float (&x)[NV]) {
  float y[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) y[i] = b[i];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    y[k] = y[k] * invd[k];
#pragma unroll
    for (int i = k + 1; i < NV; ++i) y[i] = fmaf(-l[i][k], y[k], y[i]);
  }
#pragma unroll
  for (int k = NV - 1; k >= 0; --k) {
    y[k] = y[k] * invd[k];
#pragma unroll
    for (int i = 0; i < k; ++i) y[i] = fmaf(-l[k][i], y[k], y[i]);
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) x[i] = y[i];
}

// The LM step's solve on one warp, every lane holding the whole system: H x = g
// with the gradient and the Hessian (packed upper triangle) at S, its diagonal
// damped by lambda. The operations of fit_roi's lane-parallel Cholesky, solves
// and refinement in their order; only the refinement's residual stays
// lane-parallel (lane i: row i, whose entries are at S[row[k]]). Returns whether
// the factorisation succeeded.
template <int NV>
__device__ __forceinline__ bool lm_solve(const float* S, int lane, const int (&row)[NV], float lambda,
                                         float (&x)[NV]) {
  float am[NV][NV], b[NV], ar[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    b[i] = S[i];
#pragma unroll
    for (int k = 0; k <= i; ++k) am[i][k] = S[NV + hidx<NV>(k, i)];
    ar[i] = S[row[i]];
  }
  float rhs = S[lane < NV ? lane : NV - 1];
  if (lambda != 1.0f) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      am[i][i] *= lambda;
      if (lane == i) ar[i] *= lambda;
    }
  }
  bool frz = false;
#pragma unroll
  for (int i = 0; i < NV; ++i) frz |= (am[i][i] == 0.0f);
  if (frz) {
    // parameters with an exactly zero Hessian row are held (fit_roi)
    unsigned fm = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (am[i][i] == 0.0f) fm |= 1u << i;
    const bool mine = (fm >> lane) & 1u;
    if (mine) rhs = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const bool fi = (fm >> i) & 1u;
      if (fi) b[i] = 0.0f;
#pragma unroll
      for (int k = 0; k <= i; ++k)
        if (fi || ((fm >> k) & 1u)) am[i][k] = (i == k) ? 1.0f : 0.0f;
      if (fi) ar[i] = 0.0f;
      if (mine) ar[i] = (i == lane) ? 1.0f : 0.0f;
    }
  }
  float l[NV][NV], invd[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const float ajj = am[j][j];
    if (!(ajj >= 0.0f)) return false;
    invd[j] = rsqrtf(ajj);
#pragma unroll
    for (int i = j + 1; i < NV; ++i) l[i][j] = am[i][j] * invd[j];
#pragma unroll
    for (int i = j + 1; i < NV; ++i)
#pragma unroll
      for (int k = j + 1; k <= i; ++k) am[i][k] = fmaf(-l[i][j], l[k][j], am[i][k]);
  }
  chol_substitute<NV>(l, invd, b, x);
  float sh = rhs, sl = 0.0f;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    float p_, pe_, t_, te_;
    two_prod(ar[k], x[k], p_, pe_);
    two_sum(sh, -p_, t_, te_);
    sh = t_;
    sl += te_ - pe_;
  }
  const float r = sh + sl;
  float rb[NV], dx[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) rb[i] = bcast(r, i);
  chol_substitute<NV>(l, invd, rb, dx);
  // (rounded apart: contracted with dx[0]'s product it differs from the lanes' sum)
#pragma unroll
  for (int i = 0; i < NV; ++i) x[i] = __fadd_rn(x[i], dx[i]);
  return true;
}

// lm_bounds with the limits of this lane's parameter made once per fit.
template <int MODE>
struct TeamBounds {
  float lo, hi;
  bool closed;  // an interval [lo, hi]
  int nw;
  __device__ __forceinline__ TeamBounds(const ModelDev& m, int s, int lane) {
    closed = lane >= 2 && lane <= 4;
    lo = lane == 2 ? 1.0f : lane == 3 ? 0.01f : 0.0f;
    hi = __int_as_float(0x7f800000);
    if (lane == 4) hi = (MODE == 6) ? (float)(m.n[2] - 4) : (float)m.n[2] - 0.5f;
    if (MODE == 7 && lane == 5) {
      closed = true;
      hi = (float)m.n[3] - 0.5f;
    }
    if (MODE == 8 && lane < 2) {
      closed = true;
      lo = (float)(s - 1) / 2.0f - (float)s / 4.0f;
      hi = (float)(s - 1) / 2.0f + (float)s / 4.0f;
    }
    if (MODE == 8 && lane == 6) {
      closed = true;
      lo = 1.0f;
      hi = (float)m.n[4] - 0.5f;
    }
    nw = m.n[3];
  }
  __device__ __forceinline__ float operator()(float par, int lane) const {
    if (closed) {
      par = (par > lo) ? par : lo;
      par = (par < hi) ? par : hi;
    }
    if (MODE == kFit4Pi && lane == 5) par = wrap_phase(par, nw);
    if (MODE == 8 && lane == 5) {
      if (par <= 1.0f)
        par = (float)(nw - 2) + par;
      else if (par > (float)(nw - 1))
        par = (2.0f + par) - (float)nw;
    }
    if (MODE == 8 && lane == 7) {
      par = (par < 1.0f) ? par : 1.0f;
      par = (par > 0.0f) ? par : 0.0f;
    }
    return par;
  }
};

// Fit of the ROI staged in ws by the whole block from one start; warp 0 returns
// the result (the other warps' is unspecified). g0: the initial x, y, N, bg on
// lanes 0 .. 3 of warp 0.
template <int MODE, bool VAR, int T>
__device__ __forceinline__ RoiResult fit_team(const FitArgs& a, const TeamLayout& TL, float* ws,
                                              float* kws, int lane, int warp,
                                              const TeamThread<MODE, T>& me, int64_t roi, int start,
                                              float g0) {
  using TR = ModeTraits<MODE>;
  constexpr int NV = TR::NV;
  constexpr int K = NV + NV * (NV + 1) / 2;
  float* S = ws + TL.sums;
  float* theta = ws + TL.theta;
  int4* ctl = reinterpret_cast<int4*>(ws + TL.ctl);

  // LM state of warp 0, as fit_roi: lane l < NV owns parameter l.
  float par = g0, cl = 1.0f, fd = 0.5f;
  if (warp == 0) {
    par = start_params<MODE>(a, lane, roi, start, g0);
    clamp_fade<MODE>(lane, cl, fd);
    if (lane < 8) theta[lane] = lane < NV ? par : 0.0f;
    if (lane == 0) *ctl = make_int4(1, 0, 0, 1);
  }
  LmLane st{par, par, 0.0f, 0.0f, cl, cl, fd, par, 1.0f, 1.0f, 1e10f, {1e12f, 0.0f}, {1e13f, 0.0f}, 1};
  const TeamBounds<MODE> bounds(a.m, TL.L.s, lane);
  int row[NV];  // entries of Hessian row `lane` in S
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = lane < NV ? lane : NV - 1;
    row[k] = NV + (i < k ? hidx<NV>(i, k) : hidx<NV>(k, i));
  }
  int kk = 0;
  bool fisher = false;
  RoiResult res{0.0f, 0.0f, 0.0f, 0};
  for (;;) {
    __syncthreads();
    const int4 c = *ctl;  // go, fisher, maps_ready, first
    if (!c.x) break;
    {
      const float4 t0 = reinterpret_cast<const float4*>(theta)[0];
      const float4 t1 = reinterpret_cast<const float4*>(theta)[1];
      const float th[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
      evaluate_team<MODE, VAR, T>(a, TL, ws, kws, lane, warp, me, th, MODE == 7 && c.w, c.y != 0,
                                  c.z != 0);
    }
    __syncthreads();
    if (warp != 0) continue;
    if (fisher) {
      float hr[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) hr[k] = S[row[k]];
      res.crlb = fisher_crlb<NV>(lane, hr);
      res.ll = S[K] + S[K + 1];
      res.par = st.par;
      res.kk = kk;
      if (lane == 0) *ctl = make_int4(0, 0, 0, 0);
      continue;
    }
    st.err = FPair{S[K], S[K + 1]};
    // LM steps until one succeeds (a failed solve needs no evaluation), or the
    // fit stops and its Fisher pass follows
    bool maps = false;
    for (;;) {
      if (kk >= a.iterations || lm_converged<MODE>(st)) {
        fisher = true;
        if (TR::NCH == 1) maps = lm_same_place<MODE>(st, lane);
        break;
      }
      lm_weigh(st);
      ++kk;
      float x[NV];
      bool ok = lm_solve<NV>(S, lane, row, st.lambda, x);
      if (ok) {
        float upd = x[0];
        bool nan = (x[0] != x[0]);
#pragma unroll
        for (int k = 1; k < NV; ++k) {
          if (lane == k) upd = x[k];
          nan |= (x[k] != x[k]);
        }
        // CPUmleFit_LM.cpp:2943-2950: a NaN step counts as a failed solve
        if (MODE != 6 && nan) ok = false;
        if (ok) {
          const float made =
              lm_apply<MODE>(st, a.m, lane, upd, x[NV > 4 ? 4 : 0], [&](float p) { return bounds(p, lane); });
          if (MODE == 8) st.sum_update = lm_step_sum<NV>(lane, made);
          break;
        }
      }
      // the damping of a failed solve stays (cumulative, as in the reference)
      __syncwarp();
      if (lane < NV) S[NV + hidx<NV>(lane, lane)] *= st.lambda;
      __syncwarp();
      st.lambda = 10.0f * st.lambda;
    }
    // fit type 8's Fisher pass keeps the last evaluation's positions and g2
    // (CPUmleFit_LM.cpp:3568-3584)
    if (lane < NV)
      theta[lane] = (MODE == 8 && fisher && lane != 2 && lane != 3) ? st.par_eval : st.par;
    if (!fisher) st.par_eval = st.par;
    if (lane == 0) *ctl = make_int4(1, fisher, maps, 0);
  }
  return res;
}

// Stage one ROI with all threads of the block (load_roi).
template <int MODE, bool VAR>
__device__ __forceinline__ void load_roi_team(const FitArgs& a, const WarpLayout& L, float* ws,
                                              int64_t roi) {
  const int s2 = L.s * L.s;
  constexpr int NCH = ModeTraits<MODE>::NCH;
  for (int ch = 0; ch < NCH; ++ch) {
    const float* src = a.rois + ((int64_t)ch * a.nfits + roi) * (int64_t)s2;
    for (int p = threadIdx.x; p < s2; p += blockDim.x) ws[ch * L.s2p + p] = __ldg(src + p);
    if constexpr (VAR) {
      const float* vsrc = a.var + ((int64_t)ch * a.nfits + roi) * (int64_t)s2;
      for (int p = threadIdx.x; p < s2; p += blockDim.x) ws[(NCH + ch) * L.s2p + p] = __ldg(vsrc + p);
    }
  }
  if constexpr (NCH > 1) {
    constexpr int ND = NCH * ModeTraits<MODE>::NV;
    if (threadIdx.x < ND) ws[L.off_dt() + threadIdx.x] = a.dT ? __ldg(a.dT + roi * ND + threadIdx.x) : 0.0f;
  }
  __syncthreads();
}

// Fit ROI `roi` by the whole block from every start and store the kept result
// (fit_and_store's rule).
template <int MODE, bool MULTI, bool VAR, int T>
__device__ __forceinline__ void fit_and_store_team(const FitArgs& a, const TeamLayout& TL, float* ws,
                                                   int64_t roi) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const WarpLayout& L = TL.L;
  // warp 0's knots and weights in the layout's own region, the others' behind
  // the records
  float* kws = warp == 0 ? ws : ws + TL.kws + (warp - 1) * (L.off_dt() - L.off_kx()) - L.off_kx();
  load_roi_team<MODE, VAR>(a, L, ws, roi);
  const TeamThread<MODE, T> me(warp, L.s);
  float g0 = 0.0f;
  if (warp == 0) g0 = start_guess<MODE>(L, ws, lane);
  RoiResult best{0.0f, 0.0f, 0.0f, 0};
  const int ns = (MULTI && a.n_starts > 0) ? a.n_starts : 1;  // 0: the model's initP alone
  for (int k = 0; k < ns; ++k) {
    const RoiResult r = fit_team<MODE, VAR, T>(a, TL, ws, kws, lane, warp, me, roi, k, g0);
    const float d = r.ll - best.ll;
    if (k == 0 || (a.strict ? (d > 1e-4f) : (d >= 1e-4f))) best = r;
    if (MULTI) __syncthreads();  // warp 0 writes the control words of the next start
  }
  if (warp == 0) store_result<MODE>(a, lane, roi, best);
}

// Plain form: block i fits ROI i (the block scheduler hands out the ROIs).
template <int MODE, bool MULTI, bool VAR, int T, int MINB>
__global__ void __launch_bounds__(32 * T, MINB) team_kernel(const __grid_constant__ FitArgs a) {
  extern __shared__ float4 smem4[];
  const TeamLayout TL = make_team_layout(MODE, a.s, VAR, T);
  fit_and_store_team<MODE, MULTI, VAR, T>(a, TL, reinterpret_cast<float*>(smem4), (int64_t)blockIdx.x);
}

// The kernel of T warps for a fit type, compiled for B resident blocks per SM.
using TeamKern = void (*)(const FitArgs);
constexpr int kTeamMaxShared = 227 * 1024;

template <int MODE, int T, int B>
TeamKern team_kern(bool multi, bool var) {
  if constexpr (MODE != kFit4Pi) {
    if (var) return team_kernel<MODE, false, true, T, B>;
  }
  if constexpr (MODE != 6) {
    if (multi) return team_kernel<MODE, true, false, T, B>;
  }
  return team_kernel<MODE, false, false, T, B>;
}

// The kernels are compiled in several files; each returns null for what it lacks.
TeamKern team_kern4(int mode, int blocks, bool multi, bool var);
TeamKern team_kern4_dense(int mode, int blocks, bool multi, bool var);
TeamKern team_kern16(int mode, bool multi, bool var);

}  // namespace bsfit
