// FP64 reference-precision fitter for fit types 6, 7 and 8.
//
// The FP32 kernels (bsfit_fit.cu) contract the spline separably and reorder
// every sum; the reference's LM then takes some discrete decisions (the 1e-6
// relative-deviance stop, update-sign clamp halving, accept / reject, the 4D
// "let it go" switch) differently from the reference run in double, as the
// reference's own float build does. This kernel instead computes what the
// reference computes with float promoted to double, in the reference's order
// of operations, so that its results follow the double-precision trajectory:
//   - per pixel, the 4^D-term tensor-product sums of VC/CPUmleFit_LM/
//     CPUsplineLib.cpp:1199-1288 (3D), :761-970 (4D), :43-475 (5D), with the
//     weights of :1129-1197 / :972-1126 / :477-758 and the basis of
//     :1289-1326 (float literals kept as float values), the two 5D index
//     quirks included (:313 and :420-421);
//   - the deviance, gradient and Hessian sums in pixel order (ii outer, jj
//     inner), VC/CPUmleFit_LM/CPUmleFit_LM.cpp:2537-2560;
//   - the LM control, unpivoted Cholesky and substitution
//     (CPUsplineLib.cpp:1363-1419), bounds and clamps of
//     CPUmleFit_LM.cpp:2411-2760 (type 6), :2763-3158 (type 7), :3163-3620
//     (type 8); the Fisher sums and the LU inverse of MatInvLib.h:17-77.
// The file is compiled without floating-point contraction (-fmad=false), as
// the double build it follows. The only other source of difference is the
// last bit of log().
//
// Layout: one block of four warps per ROI (TEAM; two or one for some counts,
// launch_mode): the sums' dependent adds let one warp use a quarter of the SM's FP64
// rate, and a call of few ROIs, or the last ones of a large call, lasts as long as one
// fit. Threads evaluate pixels 128 at a time and publish each pixel's terms in a shared row (its deviance term,
// t1 * dudt[l], and (t2 * dudt[l]) * dudt[m], the products the reference adds); the
// sums are owned one per thread and accumulated over the rows in pixel order, so
// every sum has the reference's order. The lead warp, another from ROI to ROI so that the
// four units share it, forms the sums (5D: 45, with the next one) and runs the LM control
// and the small dense solves, lane l on parameter or row l, on shared state: an FP64 instruction costs
// the same for one lane as for 32. Coefficients are a double copy of the model's table followed by
// one table per axis of the neighbour differences (-c[i]) + c[i + stride] the
// derivative terms use (computed once per model, the same double operation). ROIs are
// claimed from a work counter when there are more than resident blocks. Throughput
// is bounded by the FP64 pipe; this is the parity mode, the FP32 kernels are the
// production path.
//
// Measured (GB300, ms; one warp per ROI with the control on one lane / this): one
// 13 px 3D ROI 1.59 / 0.67, 150 of them 5.34 / 2.20, 3,000 of 11 px 8.93 / 6.63, 20,000
// of 13 px 64.9 / 55.3 (FP64 pipe 83% / about 82% busy with 16% fewer instructions),
// 500 4D ROIs of 13 px 40.0 / 34.2, 100 5D ROIs of 17 px 314 / 98 (its weight tables
// left three warps per SM room, now two blocks of four).
#include <climits>
#include <cmath>
#include <cstdint>
#include <mutex>

#include "bsfit_internal.h"

namespace bsfit {
namespace {

template <int MODE>
struct F64Traits;
template <>
struct F64Traits<6> {
  static constexpr int D = 3, NV = 5, NCH = 1;
};
template <>
struct F64Traits<7> {
  static constexpr int D = 4, NV = 6, NCH = 1;
};
template <>
struct F64Traits<8> {
  static constexpr int D = 5, NV = 8, NCH = 1;
};
// 4Pi (the restatement in the oracle, oracle/bsfit_oracle.cpp fit_4pi_roi):
// four channels of the 4D model at theta + dT[c], phase shifted by the
// channel's shift and wrapped, summed into one likelihood.
template <>
struct F64Traits<kFit4Pi> {
  static constexpr int D = 4, NV = 6, NCH = k4PiChannels;
};

// Float literals of the reference (VC/CPUmleFit_LM/definitions.h:15, :23-24).
constexpr float kPIf = 3.141592f;
constexpr float kTOLf = 1e-6f;
constexpr float kTOL1f = 1e-5f;

// LM state of one block, written by its lead warp (the owners of the sums write err / jac
// / hes / M / div between two block barriers).
struct LMState {
  double nt[8], ot[8], ns[8], os[8], nc[8], oc[8], fade[8], jac[8];
  double hes[64], M[64];
  double newErr, oldErr, newLambda, oldLambda, sumUpdate, div;
  double frame[8];  // yc, xc, off, zc, wc, uc, g2 of the last preparation
  unsigned long long claimed;
  int turn, action;
};
static_assert(sizeof(LMState) % 16 == 0, "LMState keeps the tables 16-byte aligned");
constexpr int kLMDoubles = (int)(sizeof(LMState) / sizeof(double));

template <int MODE, int TEAM>
struct F64Layout {
  using TR = F64Traits<MODE>;
  static constexpr int kThreads = 32 * TEAM;
  static constexpr int D = TR::D, NV = TR::NV;
  static constexpr int B = 1 << D, BB = B * B;
  static constexpr int WT = (D + 1) * BB;             // wf, then wd[0..D-1]
  static constexpr int WT3 = (MODE == 8) ? 4 * 64 : 0;  // fit type 8: the 3D tables
  static constexpr int AX = 40;                       // 1-D weights, 4 kinds x 5 axes x 2
  static constexpr int NE = 1 + NV + NV * (NV + 1) / 2;  // sums: deviance, gradient, Hessian
  static constexpr int RW = NE;                       // row: one term per sum
  static constexpr int ROWS = kThreads * RW;
  static constexpr int off_wt = kLMDoubles;
  static constexpr int off_wt3 = off_wt + WT;
  static constexpr int off_ax = off_wt3 + WT3;
  static constexpr int off_rows = off_ax + AX;
  static constexpr int total = off_rows + ROWS + (ROWS & 1);
};

// Phase position wrapped into [1, 1 + P), P = nw - 1, by one period.
__device__ __forceinline__ double wrap_phase64(double w, int nw) {
  const double P = (double)(nw - 1);
  if (w < 1.0) return w + P;
  if (w >= (double)nw) return w - P;
  return w;
}

__device__ __forceinline__ int floor_to_int64(double v) {
  const double f = floor(v);
  if (!(f >= -2147483648.0 && f < 2147483648.0)) return INT_MIN;
  return (int)f;
}

// Cardinal cubic and quadratic B-splines with the reference's float literals
// (CPUsplineLib.cpp:1289-1326), evaluated in double.
__device__ __forceinline__ double bspline3(double x) {
  constexpr float c43 = 4.0f / 3.0f, c16 = 1.0f / 6.0f, c23 = 2.0f / 3.0f;
  const double x2 = x * x, x3 = x2 * x;
  if (x >= 1.0 && x < 2.0) return (((double)c43 - 2.0 * x) + x2) - (double)c16 * x3;
  if (x >= 0.0 && x < 1.0) return ((double)c23 - x2) + 0.5 * x3;
  if (x >= -1.0 && x < 0.0) return ((double)c23 - x2) - 0.5 * x3;
  if (x >= -2.0 && x < -1.0) return (((double)c43 + 2.0 * x) + x2) + (double)c16 * x3;
  return 0.0;
}

__device__ __forceinline__ double bspline2(double x) {
  const double x2 = x * x;
  if (x >= 0.5 && x < 1.5) return (1.125 - 1.5 * x) + 0.5 * x2;
  if (x >= -0.5 && x < 0.5) return 0.75 - x2;
  if (x >= -1.5 && x < -0.5) return (1.125 + 1.5 * x) + 0.5 * x2;
  return 0.0;
}

// A model table: values c[0, total) followed by D difference tables,
// diff(d, i) = (-c[i]) + c[i + stride_d] (0 for a neighbour past the end: only
// the +1 neighbour of a position exactly on the last knot, whose weight is 0).
struct Coef {
  const double* c;
  int64_t total;
  __device__ __forceinline__ double val(int64_t i) const { return __ldg(c + i); }
  __device__ __forceinline__ double diff(int d, int64_t i) const {
    return __ldg(c + (int64_t)(d + 1) * total + i);
  }
};

// The 1-D weights of one axis (CPUsplineLib.cpp:1129-1197): kind 0 = B3(t+v-1),
// 1 = B3(t-v), 2 = B2(t-1+v-1/2), 3 = B2(t-1-v+1/2), v = 1, 2; stored at
// ax[(kind * 5 + axis) * 2 + v - 1].
__device__ __forceinline__ double axis_weight(double frac, int kind, int v) {
  const double dfrac = frac - 1.0;
  switch (kind) {
    case 0: return bspline3((frac + (double)v) - 1.0);
    case 1: return bspline3(frac - (double)v);
    case 2: return bspline2((dfrac + (double)v) - 0.5);
    default: return bspline2((dfrac - (double)v) + 0.5);
  }
}

// Tensor-product tables of D axes from ax[]: entry B*n + b, n the loop index
// (axis a at v = bit a of n, plus 1), b the side bits; the products run over
// the axes left to right.
template <int D, int THREADS>
__device__ __forceinline__ void build_tables(const double* ax, double* W) {
  constexpr int B = 1 << D, BB = B * B;
  for (int e = threadIdx.x; e < BB; e += THREADS) {
    const int n = e >> D, b = e & (B - 1);
    double val[D], der[D];
#pragma unroll
    for (int a = 0; a < D; ++a) {
      const int v = (n >> a) & 1;
      const bool side2 = (b >> a) & 1;
      val[a] = ax[((side2 ? 1 : 0) * 5 + a) * 2 + v];
      der[a] = ax[((side2 ? 3 : 2) * 5 + a) * 2 + v];
    }
    double p = val[0];
#pragma unroll
    for (int a = 1; a < D; ++a) p = p * val[a];
    W[e] = p;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      double q = (d == 0) ? der[0] : val[0];
#pragma unroll
      for (int a = 1; a < D; ++a) q = q * (a == d ? der[a] : val[a]);
      W[(1 + d) * BB + e] = q;
    }
  }
}

// Model value and derivatives at one pixel (CPUsplineLib.cpp:1199-1288 and
// the 4D / 5D copies). pos[a]: the pixel's position along axis a (Y, X, Z, W,
// U). Q5 adds the 5D model's two index quirks.
template <int D, bool Q5>
__device__ __forceinline__ void pixel_model(const Coef& c, const int* n, const int64_t* st,
                                            const double* pos, const double* W, double N, double bg,
                                            double* dudt, double* model) {
  constexpr int B = 1 << D, BB = B * B;
  int k[D];
#pragma unroll
  for (int a = 0; a < D; ++a) {
    int kc = floor_to_int64(pos[a]);
    kc = (kc > 1) ? kc : 1;
    kc = (kc < n[a] - 1) ? kc : n[a] - 1;
    if (pos[a] == (double)n[a]) kc = n[a];
    k[a] = kc + 1;
  }
  double f = 0.0;
  double dacc[D];
#pragma unroll
  for (int a = 0; a < D; ++a) dacc[a] = 0.0;
#pragma unroll 1
  for (int ni = 0; ni < B; ++ni) {
    int64_t lo[D], hi[D];
#pragma unroll
    for (int a = 0; a < D; ++a) {
      const int lv = ((ni >> a) & 1) + 1;
      lo[a] = (int64_t)(k[a] - lv) * st[a];
      hi[a] = (int64_t)(k[a] + lv - 1) * st[a];
    }
    const double* wf = W + B * ni;
    double s = 0.0, sd[D];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      int64_t node = 0;
#pragma unroll
      for (int a = 0; a < D; ++a) node += ((b >> a) & 1) ? hi[a] : lo[a];
      const double t = c.val(node) * wf[b];
      s = (b == 0) ? t : s + t;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        double w = W[(1 + d) * BB + B * ni + b];
        int64_t nd = node;
        if constexpr (Q5) {
          if (d == 2 && b == 27) {
            // CPUsplineLib.cpp:313 reads delta_dfz[32 * nIndex + 271]; past
            // the end of that array it reads the next one of the frame, the
            // W-derivative weights, which follow the Z table here as well.
            w = W[3 * BB + B * ni + 271];
          }
          if (d == 4 && b == 16) {
            // CPUsplineLib.cpp:420-421: the side-1 U node is differenced.
            nd = node - hi[4] + lo[4];
          }
        }
        const double term = c.diff(d, nd) * w;  // (-c[nd] + c[nd + stride]) * w
        sd[d] = (b == 0) ? term : sd[d] + term;
      }
    }
    f = f + s;
#pragma unroll
    for (int d = 0; d < D; ++d) dacc[d] = dacc[d] + sd[d];
  }
  dudt[0] = -N * dacc[1];
  dudt[1] = -N * dacc[0];
#pragma unroll
  for (int a = 2; a < D; ++a) dudt[a + 2] = N * dacc[a];
  dudt[2] = f;
  dudt[3] = 1.0;
  *model = bg + N * f;
}

struct Fit64Ctx {
  const Fit64Args* a;
  Coef c, c3;
  const float* data;  // channel 0's pixels; channel c at data + c * nfits * s * s
  const float* var;
  const float* dT;    // 4Pi: this ROI's [4][6] channel offsets
  int s;
};

template <int MODE, int TEAM>
struct Team64 {
  using L = F64Layout<MODE, TEAM>;
  static constexpr int kThreads = L::kThreads;
  static constexpr int D = L::D, NV = L::NV, RW = L::RW;
  LMState& st;
  double* wt;
  double* wt3;
  double* ax;
  double* rows;
  // The sum owned by this thread (entry `own`, also its index in a row): kind 0 =
  // deviance / log-likelihood, 1 = gradient l, 2 = Hessian / Fisher (l, m), m >= l;
  // -1 = none.
  int own = 0, kind = -1, el = 0, em = 0;

  __device__ explicit Team64(double* base)
      : st(*reinterpret_cast<LMState*>(base)),
        wt(base + L::off_wt),
        wt3(base + L::off_wt3),
        ax(base + L::off_ax),
        rows(base + L::off_rows) {}

  // The sums go to the threads from warp `lead` on.
  __device__ void assign(int lead) {
    static_assert(L::NE <= kThreads, "one sum per thread");
    const int t = (threadIdx.x - 32 * lead) & (kThreads - 1);
    own = t;
    kind = -1;
    if (t == 0) {
      kind = 0;
    } else if (t <= NV) {
      kind = 1;
      el = t - 1;
    } else {
      int p = t - 1 - NV;
      for (int l = 0; l < NV; ++l) {
        if (p < NV - l) {
          kind = 2;
          el = l;
          em = l + p;
          break;
        }
        p -= NV - l;
      }
    }
  }

  // Frame and weight tables at theta (the models' prepare(),
  // CPUmleFit_LM.cpp:2512-2523 and the 4D / 5D copies).
  __device__ void prepare(const Fit64Ctx& cx, const double* th) {
    const double half = (double)((cx.s + 1) / 2);
    const double xc = half - th[0], yc = half - th[1];
    const double zc = th[4];
    const double wc = (D >= 4) ? th[5] : 0.0;
    const double uc = (D >= 5) ? th[6] : 0.0;
    double fr[5] = {yc - floor(yc), xc - floor(xc), zc - floor(zc), wc - floor(wc), uc - floor(uc)};
    for (int t = threadIdx.x; t < 8 * D; t += kThreads) {
      const int kind = t / (2 * D), r = t - kind * 2 * D, axis = r >> 1, v = (r & 1) + 1;
      double f = fr[0];
#pragma unroll
      for (int q = 1; q < 5; ++q)
        if (axis == q) f = fr[q];
      ax[(kind * 5 + axis) * 2 + v - 1] = axis_weight(f, kind, v);
    }
    if (threadIdx.x == 0) {
      st.frame[0] = yc;
      st.frame[1] = xc;
      st.frame[3] = zc;
      st.frame[4] = wc;
      st.frame[5] = uc;
      st.frame[6] = (MODE == 8) ? th[7] : 0.0;
    }
    __syncthreads();
    build_tables<D, kThreads>(ax, wt);
    if constexpr (MODE == 8) build_tables<3, kThreads>(ax, wt3);
    __syncthreads();
  }

  // Value and derivative vector of pixel (ii, jj) with the prepared frame.
  __device__ void pixel(const Fit64Ctx& cx, int ii, int jj, double N, double bg, double* dudt,
                        double* model) const {
    const ModelDev& m = cx.a->m;
    double pos[5];
    pos[0] = (st.frame[0] + (double)ii) + st.frame[2];
    pos[1] = (st.frame[1] + (double)jj) + st.frame[2];
    pos[2] = st.frame[3];
    pos[3] = st.frame[4];
    pos[4] = st.frame[5];
    if constexpr (MODE == 8) {
      // Mixture (1 - g2) S3D + g2 S5D (CPUmleFit_LM.cpp:3280-3300).
      const double g2 = st.frame[6];
      double d3[5], m5, m3;
      pixel_model<5, true>(cx.c, m.n, m.st, pos, wt, N, bg, dudt, &m5);
      pixel_model<3, false>(cx.c3, m.n, m.st, pos, wt3, N, bg, d3, &m3);
#pragma unroll
      for (int l = 0; l < 5; ++l) dudt[l] = dudt[l] * g2 + (1.0 - g2) * d3[l];
      *model = m3 * (1.0 - g2) + m5 * g2;
      dudt[NV - 1] = m5 - m3;
    } else {
      pixel_model<D, false>(cx.c, m.n, m.st, pos, wt, N, bg, dudt, model);
    }
  }

  // The pixels of one plane, in the reference's order (ii outer, jj inner), one per
  // thread at a time: each thread publishes its pixel's terms in a row (the deviance
  // term, t1 * dudt[l] and (t2 * dudt[l]) * dudt[m]; or the log-likelihood term,
  // its use flag and (dudt[m] * dudt[l]) / model), then every owner adds its
  // entry of the rows in pixel order to acc.
  template <bool FISHER>
  __device__ void accumulate_plane(const Fit64Ctx& cx, const float* data, double N, double bg,
                                   bool dup45, double& acc) {
    const int s = cx.s, s2 = s * s, me = threadIdx.x;
    for (int r0 = 0; r0 < s2; r0 += kThreads) {
      const int q = r0 + me;
      if (q < s2) {
        const int ii = q / s, jj = q - ii * s;
        double dudt[NV], model;
        pixel(cx, ii, jj, N, bg, dudt, &model);
        const int di = s * jj + ii;
        double dval = (double)data[di];
        if (cx.var) {
          const double v = (double)cx.var[di];
          model += v;
          dval += v;
        }
        double* row = rows + me * RW;
        int k = 1 + NV;
        if constexpr (FISHER) {
          // CPUmleFit_LM.cpp:2730-2742
          double term = 0.0, use = 0.0;
          if (model > 0) {
            use = 1.0;
            term = (dval > 0) ? ((dval * log(model) - model) - dval * log(dval)) + dval : -model;
          }
          row[0] = term;
          row[1] = use;
#pragma unroll
          for (int l = 0; l < NV; ++l)
#pragma unroll
            for (int mm = l; mm < NV; ++mm, ++k) row[k] = (dudt[mm] * dudt[l]) / model;
        } else {
          // CPUmleFit_LM.cpp:2537-2560
          if (dup45) dudt[5] = dudt[4];
          double term;
          if (dval > 0) {
            term = 2.0 * ((model - dval) - dval * log(model / dval));
          } else {
            term = 2.0 * model;
            dval = 0.0;
          }
          const double t1 = 1.0 - dval / model;
          const double t2 = dval / (model * model);
          row[0] = term;
#pragma unroll
          for (int l = 0; l < NV; ++l) row[1 + l] = t1 * dudt[l];
#pragma unroll
          for (int l = 0; l < NV; ++l) {
            const double tl = t2 * dudt[l];
#pragma unroll
            for (int mm = l; mm < NV; ++mm, ++k) row[k] = tl * dudt[mm];
          }
        }
      }
      __syncthreads();
      const int cnt = (s2 - r0 < kThreads) ? s2 - r0 : kThreads;
      if (kind >= 0 && !(FISHER && kind == 1)) {
        double a = acc;
        if (FISHER && kind == 0) {
          for (int j = 0; j < cnt; ++j)
            if (rows[j * RW + 1] != 0.0) a = a + rows[j * RW];
        } else {
#pragma unroll 8
          for (int j = 0; j < cnt; ++j) a = a + rows[j * RW + own];
        }
        acc = a;
      }
      __syncthreads();
    }
  }

  // One pass over the ROI. FISHER = false: deviance, gradient and Hessian at
  // st.nt (CPUmleFit_LM.cpp:2530-2560) with the frame the caller prepared;
  // dup45 copies dudt[4] into dudt[5] (fit type 7's initial pass). FISHER =
  // true: Fisher matrix and log-likelihood at st.nt with the current frame
  // (:2714-2742). 4Pi: every channel at theta + dT[c], its phase shifted by the
  // channel's shift and wrapped, prepared here (Model4Pi of the restatement),
  // channel outer and pixel inner into the same sums.
  template <bool FISHER>
  __device__ void pass(const Fit64Ctx& cx, bool dup45) {
    constexpr int NCH = F64Traits<MODE>::NCH;
    double acc = 0.0;
    if constexpr (NCH == 1) {
      accumulate_plane<FISHER>(cx, cx.data, st.nt[2], st.nt[3], dup45, acc);
    } else {
      const int64_t plane = (int64_t)cx.a->nfits * cx.s * cx.s;
#pragma unroll 1
      for (int ch = 0; ch < NCH; ++ch) {
        double tc[NV];
#pragma unroll
        for (int t = 0; t < NV; ++t) tc[t] = st.nt[t] + (double)cx.dT[ch * NV + t];
        tc[5] = wrap_phase64(tc[5] + (double)cx.a->m.shift[ch], cx.a->m.n[3]);
        prepare(cx, tc);
        accumulate_plane<FISHER>(cx, cx.data + ch * plane, tc[2], tc[3], dup45, acc);
      }
    }
    if (kind == 0) {
      if (FISHER) st.div = acc;
      else st.newErr = acc;
    } else if (kind == 1) {
      if (!FISHER) st.jac[el] = acc;
    } else if (kind == 2) {
      double* Mx = FISHER ? st.M : st.hes;
      Mx[el * NV + em] = acc;
      Mx[em * NV + el] = acc;
    }
    __syncthreads();
  }
};

__device__ __forceinline__ double shfl64(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

// Unpivoted Cholesky (CPUsplineLib.cpp:1363-1390) and the substitutions
// (:1392-1419) of A x = b on one warp: lane i < NV holds row i of A in h and b_i.
// Every element is formed by the operations of the reference's loops in their order
// (the off-diagonal update multiplies by the reciprocal, as written); lanes past NV
// repeat row NV - 1. Returns 0, or 1 on a negative pivot; x on every lane.
template <int NV>
__device__ __forceinline__ int cholesky_solve64(int i, const double (&h)[NV], double b, double (&x)[NV]) {
  double u[NV], diag = 1.0;  // row i of the factor, U_ii
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < j; ++k) s = s + u[k] * shfl64(u[k], j);
    const double t = h[j] - s;
    const double piv = shfl64(t, j);
    if (!(piv >= 0)) return 1;
    const double ujj = sqrt(piv);
    u[j] = (1.0 / ujj) * t;
    if (i == j) diag = ujj;
  }
  double y = b;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const double yj = shfl64(y / diag, j);
    if (i == j) y = yj;
    else if (i > j) y = y - u[j] * yj;
  }
#pragma unroll
  for (int r = NV - 1; r >= 0; --r) {
    double t = shfl64(y, r);
#pragma unroll
    for (int j = r + 1; j < NV; ++j) t = t - shfl64(u[r], j) * x[j];
    x[r] = t / shfl64(diag, r);
  }
  return 0;
}

// LU inverse (MatInvLib.h:17-77, column-major) on one warp: lane c < SZ returns
// element (c, c). The factorisation column by column, its rows below the diagonal
// on the lanes; column c of the inverse by lane c.
template <int SZ>
__device__ double mat_inv64(double* M, int lane) {
  for (int jj = 0; jj < SZ; jj++) {
    if (lane == 0)
      for (int ii = 1; ii <= jj; ii++) {
        double t = 0.0;
        for (int kk = 0; kk <= ii - 1; kk++) t = t + M[ii + kk * SZ] * M[kk + jj * SZ];
        M[ii + jj * SZ] = M[ii + jj * SZ] - t;
      }
    __syncwarp();
    const int ii = lane;
    if (ii > jj && ii < SZ) {
      const double r = 1.0 / M[jj + jj * SZ];
      if (jj > 0) {
        double t = 0.0;
        for (int kk = 0; kk <= jj - 1; kk++) t = t + M[ii + kk * SZ] * M[kk + jj * SZ];
        M[ii + jj * SZ] = r * (M[ii + jj * SZ] - t);
      } else {
        M[ii + jj * SZ] = r * M[ii + jj * SZ];
      }
    }
    __syncwarp();
  }
  const int num = lane < SZ ? lane : SZ - 1;
  double yy[SZ], inv[SZ], own = 0.0;
  yy[0] = (num == 0) ? 1.0 : 0.0;
#pragma unroll
  for (int ii = 1; ii < SZ; ii++) {
    const double b = (ii == num) ? 1.0 : 0.0;
    double t = 0.0;
#pragma unroll
    for (int jj = 0; jj <= ii - 1; jj++) t = t + M[ii + jj * SZ] * yy[jj];
    yy[ii] = b - t;
  }
  inv[SZ - 1] = yy[SZ - 1] / M[(SZ - 1) + (SZ - 1) * SZ];
#pragma unroll
  for (int ii = SZ - 2; ii >= 0; ii--) {
    double t = 0.0;
#pragma unroll
    for (int jj = ii + 1; jj < SZ; jj++) t = t + M[ii + jj * SZ] * inv[jj];
    inv[ii] = (1.0 / M[ii + ii * SZ]) * (yy[ii] - t);
  }
#pragma unroll
  for (int ii = 0; ii < SZ; ii++)
    if (ii == num) own = inv[ii];
  return own;
}

// Initial guesses (CPUgaussLib.cpp:172-225, CPUmleFit_LM.cpp:2478-2482,
// :2839-2850, :3237-3256), lead warp.
// The single-channel rule on one plane: x, y, N, bg into t[0..3] on every lane. Lanes
// 0, 1, 2 sum the moments and the total, lanes 3 and 4 fold the maximum and minimum
// (of floats, which compare as their doubles do).
__device__ void guess_plane(const float* d, int s, int lane, double (&t)[4]) {
  double sum = 0.0;
  for (int ii = 0; ii < s; ii++)
    for (int jj = 0; jj < s; jj++) {
      const double v = (double)d[s * jj + ii];
      const double w = (lane == 0) ? (double)ii : (double)jj;
      const double p = v * w;
      sum = sum + ((lane < 2) ? p : v);
    }
  float fold = (lane == 3) ? 0.0f : 10e10f;
  for (int p = 0; p < s * s; p++) {
    const float v = d[p];
    if (lane == 3) fold = (fold > v) ? fold : v;
    else fold = (fold < v) ? fold : v;
  }
  const double ts = shfl64(sum, 2);
  const double maxn = (double)__shfl_sync(0xffffffffu, fold, 3), minbg = (double)__shfl_sync(0xffffffffu, fold, 4);
  t[0] = shfl64(sum, 0) / ts;
  t[1] = shfl64(sum, 1) / ts;
  const double n0 = ((((maxn - minbg) * 2.0) * (double)kPIf) * 1.5) * 1.5;
  t[2] = (0.0 > n0) ? 0.0 : n0;
  t[3] = (minbg > 0.01) ? minbg : 0.01;
}

// The first parameters into st.nt.
template <int MODE>
__device__ void initial_theta(const Fit64Ctx& cx, LMState& st, int64_t roi, int lane) {
  constexpr int NV = F64Traits<MODE>::NV;
  const int s = cx.s;
  double t[4];
  if constexpr (MODE == kFit4Pi) {
    // mean over the channels of the single-channel rule, lateral offsets
    // removed; z and phase per ROI (fit_4pi_roi of the restatement)
    double sx = 0.0, sy = 0.0, sn = 0.0, sb = 0.0;
    for (int c = 0; c < k4PiChannels; ++c) {
      guess_plane(cx.data + (int64_t)c * cx.a->nfits * s * s, s, lane, t);
      sx = sx + (t[0] - (double)cx.dT[c * NV + 0]);
      sy = sy + (t[1] - (double)cx.dT[c * NV + 1]);
      sn = sn + t[2];
      sb = sb + t[3];
    }
    if (lane == 0) {
      st.nt[0] = sx / 4.0;
      st.nt[1] = sy / 4.0;
      st.nt[2] = sn / 4.0;
      st.nt[3] = sb / 4.0;
      st.nt[4] = (double)cx.a->z0[roi];
      st.nt[5] = wrap_phase64((double)cx.a->w0[roi], cx.a->m.n[3]);
    }
    return;
  }
  guess_plane(cx.data, s, lane, t);
  if (lane != 0) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) st.nt[i] = t[i];
  const ModelDev& m = cx.a->m;
  if (MODE == 6) {
    st.nt[4] = (double)m.n[2] / 2.0;
  } else if (MODE == 7) {
    const bool use = m.init_p_len >= 2 && m.init_p[0] != 0.0f;
    st.nt[4] = use ? (double)m.init_p[0] : (double)m.n[2] / 2.0;
    st.nt[5] = use ? (double)m.init_p[1] : (double)m.n[3] / 2.0;
  } else {
    for (int i = 4; i < NV; i++) st.nt[i] = (double)m.init_p[i - 4];
  }
}

__device__ __forceinline__ double dmax(double a, double b) { return (a > b) ? a : b; }
__device__ __forceinline__ double dmin(double a, double b) { return (a < b) ? a : b; }

enum { kStop = 0, kEval = 1, kNoEval = 2 };

// One LM iteration up to the evaluation (CPUmleFit_LM.cpp:2569-2640 and the
// type 7 / 8 copies), lead warp, lane l < NV on parameter l (lanes past it repeat
// parameter NV - 1 and write nothing). Returns kStop on convergence, kEval with the
// new theta in st.nt, or kNoEval after a failed factorization.
template <int MODE>
__device__ int lm_control(LMState& st, const ModelDev& m, int s, int lane) {
  constexpr int NV = F64Traits<MODE>::NV;
  const int l = lane < NV ? lane : NV - 1;
  double newErr = st.newErr, oldErr = st.oldErr, newLambda = st.newLambda, oldLambda = st.oldLambda;
  bool conv = fabs((newErr - oldErr) / newErr) < (double)kTOLf;
  if (MODE == 8) conv = conv || (st.sumUpdate < (double)kTOL1f);
  if (conv) return kStop;
  double ns = st.ns[l], os = st.os[l], nc = st.nc[l], oc = st.oc[l], nt = st.nt[l], ot = st.ot[l];
  if (newErr > 1.5 * oldErr) {
    ns = os;
    nc = oc;
    nt = ot;
    newLambda = oldLambda;
    newErr = oldErr;
    newLambda = 10.0 * newLambda;
  } else if (newErr < oldErr) {
    if (newLambda > 1) newLambda = newLambda * 0.8;
    else if (newLambda < 1) newLambda = 1.0;
  }
  double h[NV], x[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    h[k] = st.hes[l * NV + k];
    if (k == l) h[k] = h[k] * newLambda;
  }
  const double b = st.jac[l];
  int turn = st.turn;
  __syncwarp();  // all reads of the state are done
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (lane == k) st.hes[k * NV + k] = h[k];
  int info = cholesky_solve64<NV>(l, h, b, x);
  if (info == 0 && MODE != 6) {
    // CPUmleFit_LM.cpp:2943-2950 / :3383-3390
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (isnan(x[k])) info = 1;
  }
  double sumUpdate = 0.0;
  if (info != 0) {
    newLambda = 10.0 * newLambda;
  } else {
    if (MODE == 7) x[NV - 1] = x[NV - 1] * 10.0;  // :2951
    os = ns;
    oc = nc;
    ot = nt;
    oldLambda = newLambda;
    oldErr = newErr;
    if (MODE == 7) {
      // "let it go", :2966-2971
      if (fabs(x[4]) < 0.005 && turn) {
        if (l == 5) nc = oc = (double)m.n[3] / 10.0;
        if (l == 4) nc = oc = 2.0;
        turn = 0;
      }
    }
    double u = x[0];
#pragma unroll
    for (int k = 1; k < NV; ++k)
      if (l == k) u = x[k];
    if (ns != 0) {
      const bool flip = (ns == 1 && u < 0) || (ns == -1 && u > 0);
      if (flip) nc = (MODE == 6) ? nc * 0.5 : nc * st.fade[l];
    }
    ns = (u > 0) ? 1.0 : -1.0;
    const double v = u / (1.0 + fabs(u / nc));
    nt = nt - v;
    if (MODE == 8) {
#pragma unroll
      for (int k = 0; k < NV; ++k) sumUpdate = sumUpdate + shfl64(fabs(v), k);
      if (l < 2) {
        // :3421-3445
        const double lo = ((double)s - 1.0) / 2.0 - (double)s / 4.0;
        const double hi = ((double)s - 1.0) / 2.0 + (double)s / 4.0;
        nt = dmin(dmax(nt, lo), hi);
      }
    }
    if (l == 2) nt = dmax(nt, 1.0);
    if (l == 3) nt = dmax(nt, 0.01);
    if (l == 4) nt = dmin(dmax(nt, 0.0), (MODE == 6) ? (double)(m.n[2] - 4) : (double)m.n[2] - 0.5);
    if (MODE == 7 && l == 5) nt = dmin(dmax(nt, 0.0), (double)m.n[3] - 0.5);
    if (MODE == kFit4Pi && l == 5) nt = wrap_phase64(nt, m.n[3]);
    if (MODE == 8) {
      if (l == 5) {
        if (nt <= 1) nt = (double)(m.n[3] - 2) + nt;
        else if (nt > (double)(m.n[3] - 1)) nt = (2.0 + nt) - (double)m.n[3];
      }
      if (l == 6) nt = dmin(dmax(nt, 1.0), (double)m.n[4] - 0.5);
      if (l == 7) nt = dmax(dmin(nt, 1.0), 0.0);
    }
  }
  if (lane < NV) {
    st.ns[l] = ns;
    st.os[l] = os;
    st.nc[l] = nc;
    st.oc[l] = oc;
    st.nt[l] = nt;
    st.ot[l] = ot;
  }
  if (lane == 0) {
    st.newErr = newErr;
    st.oldErr = oldErr;
    st.newLambda = newLambda;
    st.oldLambda = oldLambda;
    st.turn = turn;
    if (MODE == 8 && info == 0) st.sumUpdate = sumUpdate;
  }
  __syncwarp();
  return info != 0 ? kNoEval : kEval;
}

template <int MODE>
__device__ void init_state(LMState& st) {
  constexpr int NV = F64Traits<MODE>::NV;
  st.newLambda = st.oldLambda = 1.0;
  st.sumUpdate = 1e10;
  st.turn = 1;
  st.newErr = 1e12;
  st.oldErr = 1e13;
  for (int i = 0; i < 8; i++) {
    st.ns[i] = st.os[i] = 0.0;
    st.jac[i] = 0.0;
  }
  for (int i = 0; i < 64; i++) st.hes[i] = st.M[i] = 0.0;
  if (MODE == 6) {
    // :2434
    const double c[5] = {2.0, 2.0, 10000, 20, 20};
    for (int i = 0; i < NV; i++) st.nc[i] = st.oc[i] = c[i], st.fade[i] = 0.0;
  } else if (MODE == kFit4Pi) {
    const double c[6] = {1, 1, 10000, 20, 2, 2};
    for (int i = 0; i < NV; i++) st.nc[i] = st.oc[i] = c[i], st.fade[i] = 0.5;
  } else if (MODE == 7) {
    // :2786-2788
    const double c[6] = {1.0, 1.0, 10000, 20, 2, 0.00001};
    const double fd[6] = {0.5, 0.5, 0.4, 0.5, 0.7, 0.8};
    for (int i = 0; i < NV; i++) st.nc[i] = st.oc[i] = c[i], st.fade[i] = fd[i];
  } else {
    // :3191-3193
    const double c[8] = {1.0, 1.0, 10000, 20, 2, 2, 2, 0.1};
    for (int i = 0; i < NV; i++) st.nc[i] = c[i], st.fade[i] = 0.5;
  }
}

// BLOCKS: the resident blocks per SM that the registers are held to.
template <int MODE, int TEAM, int BLOCKS>
__global__ void __launch_bounds__(32 * TEAM, BLOCKS) fit64_kernel(const __grid_constant__ Fit64Args a) {
  using L = F64Layout<MODE, TEAM>;
  constexpr int NV = L::NV;
  extern __shared__ double smem64[];
  const int lane = threadIdx.x & 31;
  Team64<MODE, TEAM> w(smem64);
  LMState& st = w.st;
  Fit64Ctx cx;
  cx.a = &a;
  cx.c = Coef{a.c, a.total};
  cx.c3 = Coef{a.c3, a.total3};
  cx.s = a.s;
  const int64_t s2 = (int64_t)a.s * a.s;
  for (int64_t roi = blockIdx.x;; roi += gridDim.x) {
    if (a.claim) {
      if (threadIdx.x == 0) st.claimed = atomicAdd(a.claim, 1ull);
      __syncthreads();
      roi = (int64_t)st.claimed;
    }
    if (roi >= a.nfits) break;
    cx.data = a.rois + roi * s2;
    cx.var = a.var ? a.var + roi * s2 : nullptr;
    cx.dT = (MODE == kFit4Pi) ? a.dT + roi * (int64_t)(k4PiChannels * NV) : nullptr;
    // the warp that does the LM steps and forms the sums, another from ROI to ROI
    const int lead_warp = (int)(roi & (TEAM - 1));
    const bool lead = (int)(threadIdx.x >> 5) == lead_warp;
    w.assign(lead_warp);
    if (lead) {
      if (lane == 0) init_state<MODE>(st);
      initial_theta<MODE>(cx, st, roi, lane);
      if (lane == 0) {
        for (int i = 0; i < NV; i++) {
          st.ot[i] = st.nt[i];
          if (MODE == 8) st.oc[i] = st.nc[i];
        }
        st.frame[2] = (double)((float)(a.m.n[1] - a.s) / 2.0f);  // :2519, float arithmetic
      }
    }
    __syncthreads();
    // One LM step by the lead warp, its outcome for everyone.
    auto control = [&] {
      if (lead) {
        const int act = lm_control<MODE>(st, a.m, a.s, lane);
        if (lane == 0) st.action = act;
      }
      __syncthreads();
      const int act = st.action;
      __syncthreads();
      return act;
    };
    // Initial evaluation; fit type 7 copies dudt[4] into dudt[5] here only.
    // (4Pi prepares per channel inside the pass.)
    if (MODE != kFit4Pi) w.prepare(cx, st.nt);
    w.template pass<false>(cx, MODE == 7);
    if (MODE != kFit4Pi && a.handoff) {
      // Hand-off: the first LM steps in the reference's double arithmetic and
      // order, then the LM state for the double-float kernels. The step left
      // pending is the last one whose evaluation the double-float kernel makes.
      double te[8];
      if (threadIdx.x == 0)
        for (int i = 0; i < 8; i++) te[i] = st.nt[i];
      int kk = 0, state = Handoff::kCurrent;
      const int K = a.handoff_iters < a.iterations ? a.handoff_iters : a.iterations;
      while (kk < K) {
        const int act = control();
        if (act == kStop) {
          state = Handoff::kConverged;
          break;
        }
        ++kk;
        state = Handoff::kCurrent;
        if (act == kEval) {
          if (kk == K) {
            state = Handoff::kEvalPending;
            break;
          }
          w.prepare(cx, st.nt);
          w.template pass<false>(cx, false);
          if (threadIdx.x == 0)
            for (int i = 0; i < 8; i++) te[i] = st.nt[i];
        }
      }
      if (threadIdx.x == 0) {
        double* r = a.handoff + roi * (int64_t)kHandoffStride;
        for (int i = 0; i < 8; i++) {
          const bool in = i < NV;
          r[Handoff::nt + i] = in ? st.nt[i] : 0.0;
          r[Handoff::ot + i] = in ? st.ot[i] : 0.0;
          r[Handoff::ns + i] = in ? st.ns[i] : 0.0;
          r[Handoff::os + i] = in ? st.os[i] : 0.0;
          r[Handoff::nc + i] = in ? st.nc[i] : 0.0;
          r[Handoff::oc + i] = in ? st.oc[i] : 0.0;
          r[Handoff::te + i] = in ? te[i] : 0.0;
          r[Handoff::jac + i] = in ? st.jac[i] : 0.0;
        }
        for (int i = 0; i < NV * NV; i++) r[Handoff::hes + i] = st.hes[i];
        r[Handoff::new_lambda] = st.newLambda;
        r[Handoff::old_lambda] = st.oldLambda;
        r[Handoff::new_err] = st.newErr;
        r[Handoff::old_err] = st.oldErr;
        r[Handoff::sum_update] = st.sumUpdate;
        r[Handoff::turn] = (double)st.turn;
        r[Handoff::kk] = (double)kk;
        r[Handoff::state] = (double)state;
      }
      __syncthreads();
      continue;
    }
    int kk = 0;
    for (; kk < a.iterations; kk++) {
      const int act = control();
      if (act == kStop) break;
      if (act == kEval) {
        if (MODE != kFit4Pi) w.prepare(cx, st.nt);
        w.template pass<false>(cx, false);
      }
    }
    // CRLB and log-likelihood: types 6 and 7 re-prepare at the final theta;
    // type 8 keeps the frame, weights and g2 of its last evaluation
    // (CPUmleFit_LM.cpp:3568-3584).
    if (MODE != 8 && MODE != kFit4Pi) w.prepare(cx, st.nt);
    w.template pass<true>(cx, false);
    if (lead) {
      const double var = mat_inv64<NV>(st.M, lane);
      const int64_t n = a.nfits;
      if (lane < NV) {
        a.P[n * lane + roi] = st.nt[lane];
        a.CRLB[n * lane + roi] = var;
      }
      if (lane == 0) {
        a.P[n * NV + roi] = (double)kk;
        a.LL[roi] = st.div;
      }
    }
    __syncthreads();
  }
}

// dst = [c | diff_0 | ... | diff_{D-1}], each `total` long (see Coef).
struct Strides5 {
  int64_t st[5];
};

__global__ void widen_kernel(const float* __restrict__ src, double* __restrict__ dst,
                             int64_t total, int D, Strides5 st) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double c0 = (double)src[i];
    dst[i] = c0;
    for (int d = 0; d < D; ++d) {
      const int64_t j = i + st.st[d];
      const double c1 = (j < total) ? (double)src[j] : 0.0;
      dst[(int64_t)(d + 1) * total + i] = -c0 + c1;
    }
  }
}

// Blocks per SM and SM count of a kernel on a device, computed once (the kernel's
// shared-memory limit is set then), so later launches, including ones captured into a
// CUDA graph, make no attribute or occupancy calls.
struct Launch64 {
  int dev = -1, per_sm = 0, sms = 0;
};
std::mutex g_launch64_mu;

// Fits with TEAM warps per ROI. With `even`, only where the blocks hold all ROIs at
// once; *taken stays false otherwise.
template <int MODE, int TEAM, int BLOCKS>
cudaError_t launch64(const Fit64Args& a, bool even, bool* taken, cudaStream_t stream) {
  constexpr int threads = 32 * TEAM;
  const size_t smem = (size_t)F64Layout<MODE, TEAM>::total * sizeof(double);
  static Launch64 cache[8];  // per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 8) return cudaErrorInvalidDevice;
  int per_sm = 0, sms = 0;
  {
    std::lock_guard<std::mutex> lk(g_launch64_mu);
    Launch64& c = cache[dev];
    if (c.dev != dev) {
      e = cudaFuncSetAttribute(fit64_kernel<MODE, TEAM, BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem);
      if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c.sms, cudaDevAttrMultiProcessorCount, dev);
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c.per_sm, fit64_kernel<MODE, TEAM, BLOCKS>, threads,
                                                          smem);
      if (e != cudaSuccess) return e;
      c.dev = dev;
    }
    per_sm = c.per_sm;
    sms = c.sms;
  }
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  const int64_t cap = (int64_t)sms * per_sm;
  if (even && a.nfits > cap) return cudaSuccess;
  const int64_t grid = a.nfits < cap ? a.nfits : cap;
  // More ROIs than resident blocks: claimed one at a time, but from fixed shares in a
  // capture, which then records the launch alone (a graph with the counter's memory
  // nodes could not be a child of another, nor be cloned).
  Fit64Args b = a;
  WorkCounter claim;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (a.nfits > grid && cudaStreamIsCapturing(stream, &capture) == cudaSuccess &&
      capture == cudaStreamCaptureStatusNone)
    b.claim = claim.get(stream);
  *taken = true;
  fit64_kernel<MODE, TEAM, BLOCKS><<<(unsigned)grid, threads, smem, stream>>>(b);
  return cudaGetLastError();
}

// Four warps per ROI are the fastest for one ROI and for many, where the claims even the
// fits' lengths out. Fits of few iterations all make as many, so they run in waves: a
// call of a little more than a wave takes two, and one whose ROIs two warps or one (4D,
// 4Pi) hold at once is faster so. Measured (GB300, ms, the same number of iterations in
// all fits; one warp per ROI held to 140 registers / four warps / two / one):
//   4Pi 12 px  4 ROIs per SM, 6 iterations 17.5 / 26.7 / 16.7 / 17.3    10, 6: 42.0 / 53.3 / 48.0 / 41.3
//   4D  13 px  5, 6: 6.82 / 7.96 / 6.15 / 6.73    9, 6: 11.6 / 12.3 / 11.8 / 11.3
//   3D  17 px  5, 6: 4.42 / 3.80 / 2.70           7 px, 8, 1: 0.439 / 0.462 / 0.395
//   5D  13 px  3, 6: 24.5 / 23.9 / 18.0
// With more iterations than most fits need the four warps win by the longest fits; the
// line lies about where they do (cap of iterations, four warps / two): 3D 11 px, 7.5 per
// SM, 9 2.39 / 2.37, 13 2.61 / 2.70; 4D 13 px, 6 per SM, 45 47.7 / 43.0, 60 54.1 / 56.8;
// 5D 13 px, 2.2 per SM, 30 77.6 / 70.9, 45 100 / 104; 4Pi 12 px, 4 per SM, 60 160 / 127,
// 100 182 / 174, 3.3 per SM, 100 148 / 163.
template <int MODE>
cudaError_t launch_mode(const Fit64Args& a, cudaStream_t stream) {
  const int steps = a.handoff && a.handoff_iters < a.iterations ? a.handoff_iters : a.iterations;
  const bool alike = steps <= (MODE == 6 ? 10 : MODE == 7 ? 50 : MODE == 8 ? 30 : 80);
  bool taken = false;
  cudaError_t e = cudaSuccess;
  if constexpr (MODE == 6) {
    if (alike) e = launch64<6, 4, 4>(a, true, &taken, stream);
    if (alike && !taken && e == cudaSuccess) e = launch64<6, 2, 8>(a, true, &taken, stream);
    if (!taken && e == cudaSuccess) e = launch64<6, 4, 4>(a, false, &taken, stream);
  } else if constexpr (MODE == 8) {
    if (alike) e = launch64<8, 4, 2>(a, true, &taken, stream);
    if (alike && !taken && e == cudaSuccess) e = launch64<8, 2, 4>(a, true, &taken, stream);
    if (!taken && e == cudaSuccess) e = launch64<8, 4, 2>(a, false, &taken, stream);
  } else {
    // 4D at four blocks spills 96 bytes; three blocks (162 registers, no spills) need a
    // second wave from 457 ROIs: 600 of 13 px, three iterations, 4.16 ms against 2.92
    constexpr int B = MODE == 7 ? 4 : 3;
    if (alike) e = launch64<MODE, 4, B>(a, true, &taken, stream);
    if (alike && !taken && e == cudaSuccess) e = launch64<MODE, 2, 8>(a, true, &taken, stream);
    if (alike && !taken && e == cudaSuccess) e = launch64<MODE, 1, 11>(a, true, &taken, stream);
    if (!taken && e == cudaSuccess) e = launch64<MODE, 4, B>(a, false, &taken, stream);
  }
  return e;
}

}  // namespace

int fit64_smem_bytes(int mode) {
  switch (mode) {
    case 6: return F64Layout<6, 4>::total * 8;
    case 7: return F64Layout<7, 4>::total * 8;
    case 8: return F64Layout<8, 4>::total * 8;
    case kFit4Pi: return F64Layout<kFit4Pi, 4>::total * 8;
    default: return 0;
  }
}

cudaError_t widen_to_f64(const float* src, double* dst, int64_t total, int naxes,
                         const int64_t* strides, cudaStream_t stream) {
  if (total <= 0) return cudaSuccess;
  if (naxes < 0 || naxes > 5) return cudaErrorInvalidValue;
  Strides5 st{};
  for (int d = 0; d < naxes; ++d) st.st[d] = strides[d];
  const int64_t blocks = (total + 255) / 256;
  widen_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, stream>>>(src, dst, total,
                                                                              naxes, st);
  return cudaGetLastError();
}

cudaError_t launch_fit64(const Fit64Args& a, cudaStream_t stream) {
  if (a.nfits <= 0) return cudaSuccess;
  switch (a.m.fittype) {
    case 6: return launch_mode<6>(a, stream);
    case 7: return launch_mode<7>(a, stream);
    case 8: return launch_mode<8>(a, stream);
    case kFit4Pi: return launch_mode<kFit4Pi>(a, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace bsfit
