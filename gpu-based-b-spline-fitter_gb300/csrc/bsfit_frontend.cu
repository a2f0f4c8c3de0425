// Frame -> ROI front end on the device: the step before the fitter in the
// reference's acquisition loop (MultiD_fitter/simplefitter_cspline.m:197-319):
//   imphot = (frame - offset) * conversion                       (:226)
//   impf   = filter2(h, imphot [- min(imphot(:, 1))])            (:240-246)
//   strict 3x3 local maxima of impf in raster order, columns outer
//            (MultiD_fitter/shared/maximumfind2.c:18-66)
//   keep value > cutoff, dx < x <= W - dx, dx < y <= H - dx      (:249-251)
//   ROI k = imphot(y-dx:y+dx, x-dx:x+dx), x reversed if mirrored  (:295-301)
// Frames are MATLAB [H, W, F] (y fastest). One kernel filters a tile of a frame
// and marks its maxima in bit masks, the filtered image staying in shared memory
// unless the caller asks for it; a prefix sum over the tile columns' counts
// orders them, and one kernel writes coordinates and ROIs in the reference's
// scan order, so the ROI list is deterministic and equal to the reference's.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <utility>

#include "../../include/bsfit.h"
#include "bsfit_internal.h"

namespace bsfit {
namespace {

constexpr int kMaxKernel = 31;

// A block filters kFY x kFX pixels (rows x columns) of a frame; the maxima are
// taken in the kTY x kTX pixels inside its rim.
constexpr int kFY = 64, kFX = 32, kTY = kFY - 2, kTX = kFX - 2;
constexpr int kGroups = 4, kCols = kFX / kGroups;  // column groups of a block, columns of each

struct FrontArgs {
  const float* frames;
  int64_t nframes, H, W;
  int ytiles, xtiles;  // tiles along a column, along a row
  float offset, conversion;
  int k;              // kernel size
  int sub_min;        // subtract the first column's minimum before filtering
  float cutoff;       // a float c exceeds the caller's double cutoff exactly when c > cutoff
  int dx, s, mirror;
  float* impf;        // [F][W][H], or null
  float* colmin;      // [F]
  int* counts;        // [F * xtiles]: maxima kept per frame and tile column
  long long* offsets; // [F * xtiles + 1]
  unsigned* masks;    // [F][W][ytiles][2]: bit r of word w marks row 32 w + r of the tile
  float* coords;      // [capacity * 3]: x, y, frame (1-based), column-major
  float* rois;        // [capacity][s][s]
  int64_t capacity;
};

// The filter h(u, v) at [u + k v], twice, as the operand of a paired FMA; a
// launch parameter, so that calls on several streams keep to their own.
struct Filter {
  float2 h[kMaxKernel * kMaxKernel];
};

__device__ __forceinline__ float imphot(const FrontArgs& a, int64_t f, int64_t x, int64_t y) {
  return (__ldg(a.frames + (f * a.W + x) * a.H + y) - a.offset) * a.conversion;
}

// Per frame: the minimum over the first column (x = 0) of imphot, and its
// counts set to zero. One block per frame.
__global__ void prepare_frames(FrontArgs a) {
  __shared__ float red[32];
  const int64_t f = blockIdx.x;
  for (int i = threadIdx.x; i < a.xtiles; i += blockDim.x) a.counts[f * a.xtiles + i] = 0;
  if (!a.sub_min) return;
  float m = INFINITY;
  for (int64_t y = threadIdx.x; y < a.H; y += blockDim.x) m = fminf(m, imphot(a, f, 0, y));
  for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : INFINITY;
    for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) a.colmin[f] = m;
  }
}

// Filter and maxima of one tile. 'same'-size correlation with zero padding:
// Y(y, x) = sum_{u,v} h(u, v) X(y + u - o, x + v - o), o = (k - 1) / 2, summed
// over v, then u, with FMAs. Then the strict 3x3 maxima above the cutoff and off
// the border, one ballot per column and 32 rows.
//
// The filter is bound by its multiply-adds (49 per pixel for a 7 x 7 kernel):
// each thread takes rows r and r + 32 in the halves of paired FMAs and kCols
// neighbouring columns, reads a column's k row pairs into registers once for all
// of them (k (kCols + k - 1) shared loads for kCols k^2 paired FMAs), for which the
// size has to be known: a loop over any size, its columns read again for every term, took
// up to twice the time of a call (us, loop / this: 31 x 31 kernel, 30 frames of 100 x 100
// 200 / 106, 64 of 512 x 512 2,190 / 1,240; 14 x 14, 64 of 512 x 512 513 / 287). A pixel's
// neighbours are only read where it is above the cutoff. Keeping the filtered tile on chip leaves one read of the
// frames. 64 frames of 512 x 512, 7 x 7 kernel: 73 us (92 us with scalar FMAs)
// against 282 us for a filter with its sums in rows and 143 us for a counting and
// a writing pass over the filtered image; the whole call 605 -> 195 us.
template <int K>
__global__ void __launch_bounds__(32 * kGroups)
    filter_maxima(const __grid_constant__ FrontArgs a, const __grid_constant__ Filter flt) {
  extern __shared__ float2 tile2[];  // [kFX + k - 1][32 + k - 1]: rows q and q + 32
  float* tile = reinterpret_cast<float*>(tile2);  // then the filtered [kFX][kFY]
  constexpr int k = K, o = (k - 1) / 2;
  constexpr int ty = kFY + k - 1, tx = kFX + k - 1, py = 32 + k - 1;
  const int64_t f = blockIdx.z;
  const int64_t y0 = (int64_t)blockIdx.x * kTY - 1, x0 = (int64_t)blockIdx.y * kTX - 1;
  const int row = threadIdx.x, grp = threadIdx.y;
  const float sub = a.sub_min ? a.colmin[f] : 0.0f;
  {
    // tile element (cx, cy) is pixel (x0 - o + cx, y0 - o + cy): rows `row` and
    // row + 32 of a column by one warp, the k - 1 rows past 64 spread over all
    const int64_t gx0 = x0 - o, gy0 = y0 - o;
    const float* img = a.frames + (f * a.W + gx0) * a.H + gy0;
    const int cx0 = gx0 < 0 ? (int)-gx0 : 0;  // columns and rows inside the frame
    const int cx1 = (int)(a.W - gx0 < tx ? a.W - gx0 : tx);
    const int cy0 = gy0 < 0 ? (int)-gy0 : 0;
    const int cy1 = (int)(a.H - gy0 < ty ? a.H - gy0 : ty);
    auto pixel = [&](const float* p) { return (__ldg(p) - a.offset) * a.conversion - sub; };
    const bool in_a = row >= cy0 && row < cy1, in_b = row + 32 >= cy0 && row + 32 < cy1;
    const bool twice = row < k - 1;
    const float* p = img + grp * a.H + row;
    float2* d = tile2 + grp * py + row;
#pragma unroll 4
    for (int cx = grp; cx < tx; cx += kGroups, p += kGroups * a.H, d += kGroups * py) {
      const bool in_x = cx >= cx0 && cx < cx1;
      float va = 0.0f, vb = 0.0f;
      if (in_a && in_x) va = pixel(p);
      if (in_b && in_x) vb = pixel(p + 32);
      *d = make_float2(va, vb);
      if (twice) d[32].x = vb;
    }
    for (int i = grp * 32 + row; i < (k - 1) * tx; i += 32 * kGroups) {
      const int cx = i / (k > 1 ? k - 1 : 1), e = i - cx * (k - 1);
      float v = 0.0f;
      if (cx >= cx0 && cx < cx1 && kFY + e < cy1) v = pixel(img + cx * a.H + kFY + e);
      tile2[cx * py + 32 + e].y = v;
    }
  }
  __syncthreads();
  float2 acc[kCols];
#pragma unroll
  for (int i = 0; i < kCols; ++i) acc[i] = make_float2(0.0f, 0.0f);
  const float2* col = tile2 + grp * kCols * py + row;
#pragma unroll
  for (int c = 0; c < kCols + k - 1; ++c) {
    float2 x[k];
#pragma unroll
    for (int u = 0; u < k; ++u) x[u] = col[c * py + u];
#pragma unroll
    for (int i = 0; i < kCols; ++i) {
      const int v = c - i;
      if (v >= 0 && v < k) {
#pragma unroll
        for (int u = 0; u < k; ++u) acc[i] = __ffma2_rn(flt.h[u + k * v], x[u], acc[i]);
      }
    }
  }
  __syncthreads();  // the tile is read; the filtered one goes over it
#pragma unroll
  for (int i = 0; i < kCols; ++i) {
    tile[(grp * kCols + i) * kFY + row] = acc[i].x;
    tile[(grp * kCols + i) * kFY + row + 32] = acc[i].y;
  }
  const int c_end = (int)(a.W - x0 - 1 < kTX ? a.W - x0 - 1 : kTX);
  if (a.impf) {
#pragma unroll
    for (int i = 0; i < kCols; ++i) {
      const int c = grp * kCols + i;
      if (c < 1 || c > c_end) continue;
      float* out = a.impf + (f * a.W + x0 + c) * a.H + y0;
      if (row >= 1 && y0 + row < a.H) out[row] = acc[i].x;
      if (row < 31 && y0 + row + 32 < a.H) out[row + 32] = acc[i].y;
    }
  }
  __syncthreads();
  // rows and columns whose maxima are kept: strictly inside the image, and the
  // reference's border rule on 1-based coordinates (dx < x <= W - dx)
  const int64_t edge = a.dx > 1 ? a.dx : 1, y = y0 + row;
  const bool ok_a = row >= 1 && y >= edge && y < a.H - edge;
  const bool ok_b = row < 31 && y + 32 >= edge && y + 32 < a.H - edge;
  const int c_lo = (int)(edge - x0 > 1 ? edge - x0 : 1);
  const int c_hi = (int)(a.W - edge - x0 - 1 < kTX ? a.W - edge - x0 - 1 : kTX);
  uint2* mask = reinterpret_cast<uint2*>(a.masks) + (f * a.W + x0 + grp * kCols) * a.ytiles + blockIdx.x;
  auto maximum = [&](const float* m, float v) {
    const float *l = m - kFY, *r = m + kFY;
    return v > l[-1] && v > l[0] && v > l[1] && v > m[-1] && v > m[1] && v > r[-1] && v > r[0] &&
           v > r[1];
  };
  int found = 0;
#pragma unroll
  for (int i = 0; i < kCols; ++i, mask += a.ytiles) {
    const int c = grp * kCols + i;
    if (c < 1 || c > c_end) continue;
    const bool in = c >= c_lo && c <= c_hi;
    const float* m = tile + c * kFY + row;
    bool ha = in && ok_a && acc[i].x > a.cutoff, hb = in && ok_b && acc[i].y > a.cutoff;
    if (ha) ha = maximum(m, acc[i].x);
    if (hb) hb = maximum(m + 32, acc[i].y);
    const unsigned wa = __ballot_sync(0xffffffffu, ha), wb = __ballot_sync(0xffffffffu, hb);
    if (row == 0) *mask = make_uint2(wa, wb);
    found += __popc(wa) + __popc(wb);
  }
  if (row == 0 && found) atomicAdd(a.counts + f * a.xtiles + blockIdx.y, found);
}

// Exclusive prefix sum of the per-tile-column counts (one block of 1024);
// offsets[n] = total.
__global__ void scan_counts(const int* counts, long long* offsets, int64_t n) {
  __shared__ long long part[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long carry = 0;
  for (int64_t b = 0; b < n; b += blockDim.x) {
    const int64_t i = b + threadIdx.x;
    const long long own = i < n ? counts[i] : 0;
    long long v = own;
    for (int o = 1; o < 32; o <<= 1) {
      const long long t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
    }
    if (lane == 31) part[warp] = v;
    __syncthreads();
    if (warp == 0) {
      long long p = part[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, p, o);
        if (lane >= o) p += t;
      }
      part[lane] = p;
    }
    __syncthreads();
    v += carry + (warp > 0 ? part[warp - 1] : 0);
    if (i < n) offsets[i] = v - own;
    carry += part[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) offsets[n] = carry;
}

// Coordinates and cut-outs of one tile column's maxima (kTX columns of a frame),
// blockIdx.y's share of them: the mask words in scan order (columns, then rows) are
// counted per thread and prefix-summed over the block, every thread writes the
// coordinates of its maxima in the share, then the warps cut the ROIs out.
//
// The shares fill the GPU where a movie has few tile columns: with one block per column
// the cut-out of a frame of many maxima is the work of 18 or 69 blocks (us per call,
// without / with shares: 512 x 512, 7 x 7 kernel, 23,700 maxima 210 / 110, 2048 x 2048,
// 254,000 690 / 241; 369 in 512 x 512 91 / 93, 64 frames with 24,000 168 / 170).
constexpr int kCutThreads = 256;
__global__ void __launch_bounds__(kCutThreads) write_rois(const __grid_constant__ FrontArgs a) {
  __shared__ int part[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t f = blockIdx.x / a.xtiles;
  const int xt = (int)(blockIdx.x - f * a.xtiles);
  const long long base = a.offsets[blockIdx.x], end = a.offsets[blockIdx.x + 1];
  int share = (int)((unsigned)(end - base) + gridDim.y - 1) / (int)gridDim.y;
  if (share < kCutThreads >> 5) share = kCutThreads >> 5;  // a ROI per warp at least
  const long long k0 = base + (long long)share * blockIdx.y, k1 = k0 + share < end ? k0 + share : end;
  if (k0 >= k1 || k0 >= a.capacity) return;
  const int64_t xb = (int64_t)xt * kTX;
  const int cols = (int)(a.W - xb < kTX ? a.W - xb : kTX);
  const int64_t words = (int64_t)cols * a.ytiles * 2;
  const unsigned* masks = a.masks + (f * a.W + xb) * a.ytiles * 2;
  const int64_t per = (words + blockDim.x - 1) / blockDim.x;
  const int64_t w0 = per * threadIdx.x, w1 = w0 + per < words ? w0 + per : words;
  int own = 0;
  for (int64_t w = w0; w < w1; ++w) own += __popc(masks[w]);
  int v = own;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) part[warp] = v;
  __syncthreads();
  long long idx = base + v - own;
  for (int i = 0; i < warp; ++i) idx += part[i];
  for (int64_t w = w0; w < w1 && own > 0; ++w) {
    unsigned m = masks[w];
    const int64_t column = w / (a.ytiles * 2), q = w - column * a.ytiles * 2;
    while (m) {
      const int r = __ffs(m) - 1;
      m &= m - 1;
      if (idx >= k0 && idx < k1 && idx < a.capacity) {
        a.coords[idx] = (float)(xb + column + 1);
        a.coords[a.capacity + idx] = (float)((q >> 1) * kTY - 1 + (q & 1) * 32 + r + 1);
        a.coords[2 * a.capacity + idx] = (float)(f + 1);
      }
      ++idx;
    }
  }
  __syncthreads();
  const long long n = k1 < a.capacity ? k1 : a.capacity;
  const int s = a.s, s2 = s * s, dx = a.dx;
  for (long long k = k0 + warp; k < n; k += blockDim.x >> 5) {
    const int64_t cx = (int64_t)a.coords[k] - 1, cy = (int64_t)a.coords[a.capacity + k] - 1;
    float* roi = a.rois + k * s2;
    for (int p = lane; p < s2; p += 32) {
      const int jj = p / s, ii = p - jj * s;
      const int64_t x = a.mirror ? cx + dx - jj : cx - dx + jj;
      roi[p] = imphot(a, f, x, cy - dx + ii);
    }
  }
}

using FilterKern = void (*)(const FrontArgs, const Filter);

template <int... I>
FilterKern filter_kern_of(int k, std::integer_sequence<int, I...>) {
  constexpr FilterKern kern[] = {filter_maxima<I + 1>...};
  return kern[k - 1];
}

// The kernel of a filter size, 1 to kMaxKernel.
FilterKern filter_kern(int k) { return filter_kern_of(k, std::make_integer_sequence<int, kMaxKernel>()); }

}  // namespace
}  // namespace bsfit

extern "C" {

int bsfit_peak_kernel(int32_t mode, double sigma, float* kernel, int32_t* ksize) {
  if (!kernel || !ksize || !(sigma > 0.0) || (mode != 0 && mode != 1)) return BSFIT_E_INVALID;
  auto gauss = [](int k, double sg, double* h) {
    const double half = (k - 1) / 2.0;
    double mx = 0.0, sum = 0.0;
    for (int v = 0; v < k; ++v)
      for (int u = 0; u < k; ++u) {
        const double x = v - half, y = u - half;
        h[u + k * v] = std::exp(-(x * x + y * y) / (2.0 * sg * sg));
        mx = h[u + k * v] > mx ? h[u + k * v] : mx;
      }
    for (int i = 0; i < k * k; ++i) {
      if (h[i] < 2.220446049250313e-16 * mx) h[i] = 0.0;
      sum += h[i];
    }
    if (sum != 0.0)
      for (int i = 0; i < k * k; ++i) h[i] /= sum;
  };
  // fspecial('gaussian') kernels of simplefitter_cspline.m:197-211
  const int k = mode == 0 ? (int)std::fmax(3.0, std::ceil(3.0 * sigma + 1.0))
                          : (int)std::fmax(std::ceil(6.0 * sigma + 1.0), 3.0);
  if (k > bsfit::kMaxKernel) return BSFIT_E_INVALID;
  double h1[bsfit::kMaxKernel * bsfit::kMaxKernel], h2[bsfit::kMaxKernel * bsfit::kMaxKernel];
  gauss(k, sigma, h1);
  if (mode == 1) {
    gauss(k, std::fmax(1.0, 2.5 * sigma), h2);
    for (int i = 0; i < k * k; ++i) h1[i] -= h2[i];
  }
  for (int i = 0; i < k * k; ++i) kernel[i] = (float)h1[i];
  *ksize = k;
  return BSFIT_OK;
}

int64_t bsfit_find_rois_scratch_bytes(int64_t nframes, int64_t height, int64_t width) {
  if (nframes < 0 || height < 0 || width < 0) return 0;
  const int64_t cols = nframes * width;
  int64_t b = 0;
  b += (cols * 4 + 255) / 256 * 256;             // counts
  b += ((cols + 1) * 8 + 255) / 256 * 256;       // offsets and the total
  b += (nframes * 4 + 255) / 256 * 256;          // first-column minima
  b += (nframes * height * width * 4 + 255) / 256 * 256;  // filtered frames
  return b;
}

int bsfit_find_rois_device(const float* d_frames, int64_t nframes, int64_t height, int64_t width,
                           const bsfit_frontend* fe, float* d_rois, float* d_coords,
                           int64_t capacity, int64_t* n_found, float* d_filtered, void* d_scratch,
                           int64_t scratch_bytes, void* stream) {
  if (!fe || !n_found || nframes < 0 || capacity < 0) return BSFIT_E_INVALID;
  *n_found = 0;
  if (nframes == 0) return BSFIT_OK;
  if (!d_frames || !d_scratch || !fe->kernel) return BSFIT_E_INVALID;
  if (height < 3 || width < 3 || height > (1 << 20) || width > (1 << 20)) return BSFIT_E_INVALID;
  // launch limits of the filter grid (frames on z, column tiles on y)
  if (nframes > 65535 || (width + 7) / 8 > 65535) return BSFIT_E_INVALID;
  if (fe->ksize < 1 || fe->ksize > bsfit::kMaxKernel) return BSFIT_E_INVALID;
  if (fe->roi_size < 1 || fe->roi_size > 51 || fe->roi_size % 2 == 0) return BSFIT_E_SUBREGION_SIZE;
  if (capacity > 0 && (!d_rois || !d_coords)) return BSFIT_E_INVALID;
  if (scratch_bytes < bsfit_find_rois_scratch_bytes(nframes, height, width)) return BSFIT_E_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  bsfit::FrontArgs a;
  std::memset(&a, 0, sizeof(a));
  a.frames = d_frames;
  a.nframes = nframes;
  a.H = height;
  a.W = width;
  a.offset = fe->offset;
  a.conversion = fe->conversion;
  a.k = fe->ksize;
  a.sub_min = fe->subtract_first_column_min ? 1 : 0;
  // the largest float not above the cutoff: no float lies between the two
  a.cutoff = (float)fe->cutoff;
  if ((double)a.cutoff > fe->cutoff) a.cutoff = nextafterf(a.cutoff, -INFINITY);
  a.dx = fe->roi_size / 2;
  a.s = fe->roi_size;
  a.mirror = fe->mirror ? 1 : 0;
  a.capacity = capacity;
  a.coords = d_coords;
  a.rois = d_rois;
  char* p = (char*)d_scratch;
  const int64_t cols = nframes * width;
  a.counts = (int*)p;
  p += (cols * 4 + 255) / 256 * 256;
  a.offsets = (long long*)p;
  p += ((cols + 1) * 8 + 255) / 256 * 256;
  a.colmin = (float*)p;
  p += (nframes * 4 + 255) / 256 * 256;
  // the masks in the room of the filtered frames: 8 bytes per column and 62
  // rows, at most the 4 bytes per pixel (height >= 3)
  a.masks = (unsigned*)p;
  a.impf = d_filtered;
  a.ytiles = (int)((height + bsfit::kTY - 1) / bsfit::kTY);
  a.xtiles = (int)((width + bsfit::kTX - 1) / bsfit::kTX);
  bsfit::Filter flt;
  for (int i = 0; i < fe->ksize * fe->ksize; ++i) flt.h[i] = make_float2(fe->kernel[i], fe->kernel[i]);
  const int64_t tcols = nframes * a.xtiles;
  bsfit::prepare_frames<<<(unsigned)nframes, 256, 0, st>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) {
    const size_t smem = sizeof(float2) * (32 + a.k - 1) * (bsfit::kFX + a.k - 1);
    dim3 grid((unsigned)a.ytiles, (unsigned)a.xtiles, (unsigned)nframes);
    bsfit::filter_kern(a.k)<<<grid, dim3(32, bsfit::kGroups), smem, st>>>(a, flt);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    bsfit::scan_counts<<<1, 1024, 0, st>>>(a.counts, a.offsets, tcols);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && capacity > 0) {
    // no more blocks than are resident, eight on an SM: a second wave costs more than it
    // evens out (64 frames of 512 x 512, one / two shares 160 / 170 us); 16 shares leave a
    // warp few ROIs already
    int dev = 0, sms = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = bsfit::sm_count(dev, &sms);
    if (e == cudaSuccess) {
      const int64_t fit = 8 * (int64_t)sms / tcols, shares = fit < 1 ? 1 : fit < 16 ? fit : 16;
      bsfit::write_rois<<<dim3((unsigned)tcols, (unsigned)shares), bsfit::kCutThreads, 0, st>>>(a);
      e = cudaGetLastError();
    }
  }
  long long total = 0;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&total, a.offsets + tcols, sizeof(long long), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e == cudaErrorMemoryAllocation ? BSFIT_E_NOT_ENOUGH_MEMORY : BSFIT_E_CUDA;
  *n_found = total;
  return BSFIT_OK;
}

}  // extern "C"
