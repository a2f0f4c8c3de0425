// Cubic B-spline coefficient builder on the device: the reference's bsarray
// for degree 3 without smoothing, which produces the fitter's coefficient input
// from a sampled PSF stack.
//
// Per axis (MultiD_bspline/bsarray/directFilter.m:200-282, symExpFilt.m:27-44,
// getBSplineFiltCoeffs.m:45-50), every 1-D line x[0..n-1] is filtered with the
// symmetric exponential filter of pole z = sqrt(3) - 2 and gain 6:
//   y[0]   = sum_{k < K0} z^k x[m(k)], m the whole-sample mirror sequence
//            0..n-1, n-2..1 repeated, K0 = ceil(log(eps) / log|z|);
//   y[k]   = x[k] + z y[k-1];
//   y[n-1] = (2 y[n-1] - x[n-1]) (-z / (1 - z^2));
//   y[k]   = (y[k+1] - y[k]) z, k = n-2 .. 0;  then y *= 6.
// Lines of length 1 are left unchanged. Then every axis is padded by one sample
// on each side by whole-sample mirroring (directFilter.m:286-298): c[-1] = c[1],
// c[n] = c[n-2] (c[0] for n = 1), so the coefficients are two larger than the
// samples along every axis. Arithmetic is double, as in the MATLAB builder; the
// fitter's input is the float copy.
#include <cmath>
#include <cstdint>
#include <cstring>

#include "../../include/bsfit.h"
#include "bsfit_internal.h"

namespace bsfit {
namespace {

constexpr int kMaxK0 = 64;

// What bounds the builder is the FP64 pipe (two lanes per cycle and SM): four
// operations per sample and axis, k0 = 28 per line for the initial sum and one
// conversion per coefficient. The passes keep that pipe fed: lines are staged in
// shared memory with all their loads in flight, the gain is applied as a value is
// written (instead of in a pass of its own), the two fastest axes share one pass
// over memory, and the last pass writes the padded output itself. Measured (GB300,
// 34 x 34 x 41 x 18 x 9 samples): 822 -> 513 us per call; the FP64 pipe is 75%
// busy in the plane pass (197 us for two axes; 298 us one axis at a time from
// global memory) and 76 to 84% in the line passes (84, 94 us; the last one
// 150 us with the output, 317 us as a pass and a padding kernel). 26 x 26 x 61
// samples, where the recursions' latency and the launches count: 93 -> 53 us.
//
// The filter's constants, a launch parameter.
struct FilterConst {
  double zpow[kMaxK0];
  double z, c0, gain;
  int k0;
};

// One line of n samples at x[k * step], filtered in place in shared memory; the
// result's element k goes to put(k, value). Each element takes four FP64
// operations besides the initial sum's k0 per line.
template <class Put>
__device__ __forceinline__ void filter_line(double* x, int n, int step, const FilterConst& fc, Put&& put) {
  // causal initial value from the original samples, mirror sequence of period 2n - 2
  const int period = 2 * n - 2;
  double y0 = 0.0;
  int m = 0;  // position in the mirror sequence
#pragma unroll 4
  for (int k = 0; k < fc.k0; ++k) {
    const int idx = (m < n) ? m : period - m;
    y0 = (k == 0) ? fc.zpow[0] * x[idx * step] : y0 + fc.zpow[k] * x[idx * step];
    if (++m == period) m = 0;
  }
  const double x_last = x[(n - 1) * step], z = fc.z;
  double y = y0;
  x[0] = y0;
#pragma unroll 4
  for (int k = 1; k < n - 1; ++k) {
    y = x[k * step] + z * y;
    x[k * step] = y;
  }
  y = x_last + z * y;
  y = (2.0 * y - x_last) * fc.c0;
  // each element is read one step ahead of its use: put may write to the line
  double next = x[(n - 2) * step];
  put(n - 1, y * fc.gain);
#pragma unroll 4
  for (int k = n - 2; k >= 0; --k) {
    const double c = next;
    if (k > 0) next = x[(k - 1) * step];
    y = (y - c) * z;
    put(k, y * fc.gain);
  }
}

// Sizes of the samples and where the padded coefficients go.
struct PadDims {
  int ndim;
  int64_t n[5];   // sample sizes
  int64_t ps[5];  // padded strides
  float* out32;   // null: not wanted
  double* out64;
};

// Padded positions of sample i along an axis of n samples: i + 1, and the mirror
// images c[-1] = c[1], c[n] = c[n-2] (n = 1: all three positions).
__device__ __forceinline__ int pad_images(int64_t i, int64_t n, int64_t (&p)[3]) {
  int c = 0;
  p[c++] = i + 1;
  if (n == 1 || i == 1) p[c++] = 0;
  if (n == 1 || i == n - 2) p[c++] = n + 1;
  return c;
}

// Offsets of a line's images in the padded array: the line's fixed coordinates
// are those of `pos` in the axes other than `axis` (pos counts the samples of
// these axes, the faster ones first). Calls put(offset) for each.
template <class Put>
__device__ __forceinline__ void for_images(const PadDims& d, int axis, int64_t pos, Put&& put) {
  int64_t im[5][3];
  int cnt[5];
#pragma unroll
  for (int a = 0; a < 5; ++a) {
    cnt[a] = 1;
    im[a][0] = 0;
    if (a < d.ndim && a != axis) {
      const int64_t q = pos / d.n[a];
      cnt[a] = pad_images(pos - q * d.n[a], d.n[a], im[a]);
      pos = q;
    }
  }
  for (int e = 0; e < cnt[4]; ++e)
    for (int w = 0; w < cnt[3]; ++w)
      for (int z = 0; z < cnt[2]; ++z)
        for (int x = 0; x < cnt[1]; ++x)
          for (int y = 0; y < cnt[0]; ++y)
            put(im[0][y] * d.ps[0] + im[1][x] * d.ps[1] + im[2][z] * d.ps[2] + im[3][w] * d.ps[3] +
                im[4][e] * d.ps[4]);
}

__device__ __forceinline__ void store_padded(const PadDims& d, int64_t o, double v, float f) {
  if (d.out32) d.out32[o] = f;
  if (d.out64) d.out64[o] = v;
}

// Planes of the two fastest axes (n0 x n1 samples), P per block, filtered along
// both in shared memory: src -> dst (both in the sample layout). Rows are padded
// to an odd pitch, so that a warp's lines lie on different banks along either
// axis.
__global__ void filter_planes(const double* src, double* dst, int n0, int n1, int64_t planes, int P,
                              const __grid_constant__ FilterConst fc) {
  extern __shared__ double sm[];
  const int pitch = n0 | 1, size = n1 * pitch;
  const int64_t first = (int64_t)blockIdx.x * P;
  const int np = (int)(planes - first < P ? planes - first : P);
  const int64_t base = first * n0 * n1;
  for (int i = threadIdx.x; i < np * n0 * n1; i += blockDim.x) {
    const int r = i / n0;
    sm[r * pitch + (i - r * n0)] = src[base + i];
  }
  __syncthreads();
  if (n0 > 1)
    for (int l = threadIdx.x; l < np * n1; l += blockDim.x) {
      double* x = sm + l * pitch;
      filter_line(x, n0, 1, fc, [&](int k, double v) { x[k] = v; });
    }
  __syncthreads();
  if (n1 > 1)
    for (int l = threadIdx.x; l < np * n0; l += blockDim.x) {
      const int p = l / n0;
      double* x = sm + p * size + (l - p * n0);
      filter_line(x, n1, pitch, fc, [&](int k, double v) { x[k * pitch] = v; });
    }
  __syncthreads();
  for (int i = threadIdx.x; i < np * n0 * n1; i += blockDim.x) {
    const int r = i / n0;
    dst[base + i] = sm[r * pitch + (i - r * n0)];
  }
}

// Lines along one axis (length n, stride `stride`), one thread each, staged in
// shared memory (element k of thread t at [k * blockDim + t]: no bank conflicts,
// and no synchronisation, since a thread only touches its own). Consecutive
// threads take consecutive lines, so the reads and writes are coalesced when
// stride > 1. PAD: the last axis; the result goes to its places in the padded
// output instead of back to data.
template <bool PAD>
__global__ void filter_lines(const double* src, double* dst, int n, int64_t stride, int64_t lines,
                             int axis, const __grid_constant__ PadDims pd,
                             const __grid_constant__ FilterConst fc) {
  extern __shared__ double sm[];
  const int64_t line = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (line >= lines) return;
  const int64_t outer = line / stride, inner = line - outer * stride;
  const int64_t base = outer * n * stride + inner;
  const int step = blockDim.x;
  double* x = sm + threadIdx.x;
#pragma unroll 8
  for (int k = 0; k < n; ++k) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(x + k * step);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src + base + k * stride)
                 : "memory");
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  if constexpr (!PAD) {
    if (n == 1) {
      dst[base] = x[0];
    } else {
      filter_line(x, n, step, fc, [&](int k, double v) { dst[base + k * stride] = v; });
    }
  } else {
    // the float coefficients are converted once per sample, over the doubles
    // where those are not wanted themselves (conversions share the FP64 pipe); by
    // memcpy, which keeps its order with the accesses of doubles to the same place
    const bool both = pd.out64 != nullptr;
    auto put = [&](int k, double v) {
      const float f = (float)v;
      if (both) x[k * step] = v;
      else memcpy(x + k * step, &f, sizeof(f));
    };
    if (n > 1) filter_line(x, n, step, fc, put);
    else put(0, x[0]);
    for_images(pd, axis, line, [&](int64_t o) {
      for (int k = 0; k < n; ++k) {
        const double v = both ? x[k * step] : 0.0;
        float f = (float)v;
        if (!both) memcpy(&f, x + k * step, sizeof(f));
        int64_t p[3];
        const int c = pad_images(k, n, p);
        for (int i = 0; i < c; ++i) store_padded(pd, o + p[i] * pd.ps[axis], v, f);
      }
    });
  }
}

// Lines too long for shared memory: one thread per line, in place in global
// memory.
__global__ void prefilter_axis(double* data, int64_t n, int64_t stride, int64_t lines,
                               const __grid_constant__ FilterConst fc) {
  const int64_t line = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (line >= lines) return;
  const int64_t outer = line / stride, inner = line - outer * stride;
  double* x = data + outer * n * stride + inner;
  const int64_t period = 2 * n - 2;
  double y0 = 0.0;
  int64_t m = 0;
  for (int k = 0; k < fc.k0; ++k) {
    const int64_t idx = (m < n) ? m : period - m;
    y0 = (k == 0) ? fc.zpow[0] * x[idx * stride] : y0 + fc.zpow[k] * x[idx * stride];
    if (++m == period) m = 0;
  }
  const double x_last = x[(n - 1) * stride], z = fc.z;
  double y = y0;
  x[0] = y0;
  for (int64_t k = 1; k < n; ++k) {
    y = x[k * stride] + z * y;
    x[k * stride] = y;
  }
  y = (2.0 * y - x_last) * fc.c0;
  x[(n - 1) * stride] = y * fc.gain;
  for (int64_t k = n - 2; k >= 0; --k) {
    y = (y - x[k * stride]) * z;
    x[k * stride] = y * fc.gain;
  }
}

// The padded output from the filtered samples, one thread per padded element
// (where the last axis was filtered in global memory, or there is only one).
__global__ void mirror_pad(const double* y, const __grid_constant__ PadDims d, int64_t total) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  int64_t rem = i, src = 0, ss = 1;
  for (int a = 0; a < d.ndim; ++a) {
    const int64_t n = d.n[a];
    const int64_t p = rem % (n + 2);
    rem /= n + 2;
    int64_t s;
    if (n == 1) s = 0;
    else if (p == 0) s = 1;
    else if (p == n + 1) s = n - 2;
    else s = p - 1;
    src += s * ss;
    ss *= n;
  }
  const double v = y[src];
  store_padded(d, i, v, (float)v);
}

constexpr int kSharedMost = 200 * 1024;   // a block's shared memory at most
constexpr int kSharedGoal = 72 * 1024;    // three blocks on an SM

cudaError_t raise_shared(const void* kern) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedMost);
}

// Planes per block: as many as fill the threads of the line passes best within
// the shared-memory goal (0: not even one plane fits a block).
int planes_per_block(int64_t n0, int64_t n1) {
  const int64_t bytes = n1 * (n0 | 1) * 8;
  if (bytes > kSharedMost) return 0;
  int best = 1;
  double fill = 0.0;
  for (int p = 1; p == 1 || (p * bytes <= kSharedGoal && p * (n0 > n1 ? n0 : n1) <= 512); ++p) {
    const double f = (double)(p * n0 + p * n1) / (double)((p * n0 + 31) / 32 * 32 + (p * n1 + 31) / 32 * 32);
    if (f > fill + 0.02) {
      fill = f;
      best = p;
    }
  }
  return best;
}

// Threads per block of a line pass (0: a line does not fit): 128 if the lines'
// shared memory allows three blocks on an SM, fewer for long lines.
int line_threads(int64_t n, int64_t lines) {
  int t = 128;
  while (t > 32 && (t * n * 8 > kSharedGoal || lines < (int64_t)t * 152)) t >>= 1;
  return t * n * 8 <= kSharedMost ? t : 0;
}

}  // namespace
}  // namespace bsfit

extern "C" {

int bsfit_bsarray_coeffs_device(const double* d_samples, int32_t ndim, const int64_t* dims,
                                double* d_work, float* d_coeff, double* d_coeff64,
                                void* stream) {
  if (!d_samples || !dims || !d_work || (!d_coeff && !d_coeff64)) return BSFIT_E_INVALID;
  if (ndim < 1 || ndim > 5) return BSFIT_E_INVALID;
  int64_t total = 1, padded = 1;
  for (int a = 0; a < ndim; ++a) {
    if (dims[a] < 1 || dims[a] > (1 << 20)) return BSFIT_E_INVALID;
    total *= dims[a];
    padded *= dims[a] + 2;
  }
  if (total > ((int64_t)1 << 34)) return BSFIT_E_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  bsfit::FilterConst fc;
  const double z = std::sqrt(3.0) - 2.0;
  fc.k0 = (int)std::ceil(std::log(2.220446049250313e-16) / std::log(std::fabs(z)));
  if (fc.k0 > bsfit::kMaxK0) return BSFIT_E_INVALID;
  for (int k = 0; k < fc.k0; ++k) fc.zpow[k] = std::pow(z, (double)k);
  fc.z = z;
  fc.c0 = -z / (1.0 - z * z);
  fc.gain = 6.0;
  bsfit::PadDims pd;
  std::memset(&pd, 0, sizeof(pd));
  pd.ndim = ndim;
  pd.out32 = d_coeff;
  pd.out64 = d_coeff64;
  int64_t ps = 1;
  for (int a = 0; a < ndim; ++a) {
    pd.n[a] = dims[a];
    pd.ps[a] = ps;
    ps *= dims[a] + 2;
  }
  // The two fastest axes plane by plane, then one pass per further axis, the last
  // of which writes the padded output. What does not fit shared memory (planes
  // or lines of thousands of samples) is filtered line by line in global memory.
  cudaError_t e = cudaSuccess;
  const double* src = d_samples;
  int64_t stride = 1;
  bool padded_out = false;
  for (int a = 0; a < ndim && e == cudaSuccess; ++a) {
    const int64_t n = dims[a], lines = total / n;
    if (a == 0 && ndim > 1) {
      const int P = bsfit::planes_per_block(dims[0], dims[1]);
      if (P > 0) {
        const int64_t planes = total / (dims[0] * dims[1]);
        const int64_t most = P * (dims[0] > dims[1] ? dims[0] : dims[1]);
        const int threads = (int)(most >= 512 ? 512 : (most + 31) / 32 * 32);
        e = bsfit::raise_shared((const void*)bsfit::filter_planes);
        if (e == cudaSuccess) {
          bsfit::filter_planes<<<(unsigned)((planes + P - 1) / P), threads,
                                 (size_t)P * dims[1] * (dims[0] | 1) * 8, st>>>(
              src, d_work, (int)dims[0], (int)dims[1], planes, P, fc);
          e = cudaGetLastError();
        }
        src = d_work;
        stride *= n * dims[1];
        ++a;
        continue;
      }
    }
    const int threads = bsfit::line_threads(n, lines);
    const bool last = a == ndim - 1;
    if (threads > 0 && (a > 0 || ndim == 1)) {
      const unsigned blocks = (unsigned)((lines + threads - 1) / threads);
      const size_t smem = (size_t)threads * n * 8;
      e = bsfit::raise_shared(last ? (const void*)bsfit::filter_lines<true>
                                   : (const void*)bsfit::filter_lines<false>);
      if (e == cudaSuccess) {
        if (last)
          bsfit::filter_lines<true><<<blocks, threads, smem, st>>>(src, d_work, (int)n, stride, lines, a, pd, fc);
        else
          bsfit::filter_lines<false><<<blocks, threads, smem, st>>>(src, d_work, (int)n, stride, lines, a, pd, fc);
        e = cudaGetLastError();
      }
      padded_out = last;
    } else {
      if (src != d_work)
        e = cudaMemcpyAsync(d_work, src, (size_t)total * sizeof(double), cudaMemcpyDeviceToDevice, st);
      if (e == cudaSuccess && n > 1) {
        bsfit::prefilter_axis<<<(unsigned)((lines + 127) / 128), 128, 0, st>>>(d_work, n, stride, lines, fc);
        e = cudaGetLastError();
      }
    }
    src = d_work;
    stride *= n;
  }
  if (e == cudaSuccess && !padded_out) {
    const int64_t blocks = (padded + 255) / 256;
    bsfit::mirror_pad<<<(unsigned)blocks, 256, 0, st>>>(d_work, pd, padded);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) return BSFIT_OK;
  return e == cudaErrorMemoryAllocation ? BSFIT_E_NOT_ENOUGH_MEMORY : BSFIT_E_CUDA;
}

int bsfit_bsarray_coeffs(const double* samples, int32_t ndim, const int64_t* dims, float* coeff) {
  if (!samples || !dims || !coeff || ndim < 1 || ndim > 5) return BSFIT_E_INVALID;
  int64_t total = 1, padded = 1;
  for (int a = 0; a < ndim; ++a) {
    if (dims[a] < 1 || dims[a] > (1 << 20)) return BSFIT_E_INVALID;
    total *= dims[a];
    padded *= dims[a] + 2;
  }
  cudaStream_t st = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  double *d_in = nullptr, *d_work = nullptr;
  float* d_out = nullptr;
  if (e == cudaSuccess) e = cudaMallocAsync(&d_in, (size_t)total * sizeof(double), st);
  if (e == cudaSuccess) e = cudaMallocAsync(&d_work, (size_t)total * sizeof(double), st);
  if (e == cudaSuccess) e = cudaMallocAsync(&d_out, (size_t)padded * sizeof(float), st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_in, samples, (size_t)total * sizeof(double), cudaMemcpyHostToDevice, st);
  int rc = BSFIT_OK;
  if (e == cudaSuccess) rc = bsfit_bsarray_coeffs_device(d_in, ndim, dims, d_work, d_out, nullptr, st);
  if (e == cudaSuccess && rc == BSFIT_OK)
    e = cudaMemcpyAsync(coeff, d_out, (size_t)padded * sizeof(float), cudaMemcpyDeviceToHost, st);
  if (d_in) cudaFreeAsync(d_in, st);
  if (d_work) cudaFreeAsync(d_work, st);
  if (d_out) cudaFreeAsync(d_out, st);
  cudaError_t e2 = st ? cudaStreamSynchronize(st) : cudaSuccess;
  if (st) cudaStreamDestroy(st);
  if (rc != BSFIT_OK) return rc;
  if (e == cudaSuccess) e = e2;
  if (e == cudaSuccess) return BSFIT_OK;
  return e == cudaErrorMemoryAllocation ? BSFIT_E_NOT_ENOUGH_MEMORY : BSFIT_E_CUDA;
}

}  // extern "C"
