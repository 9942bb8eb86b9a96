// Matching-cost kernels: census, NCC, Sobel, SAD-on-Sobel, zero-mean SAD.
//
// Each kernel reproduces the reference's valid region, sentinel and
// arithmetic (cpp/matchers/matchers.cpp), so the float64 outputs equal the
// reference's bit for bit:
//   - census and SAD-on-Sobel are integer counts / sums;
//   - NCC's window sums are exact integers and the final
//     -(w^2 S - A_L A_R) * C_L * C_R is evaluated in float64 in the
//     reference's order (matchers.cpp:179);
//   - ZSAD accumulates fabs(L - muL - R + muR) in float64 in the reference's
//     wh-major order (matchers.cpp:499-505).
// Outputs are float32 or float64, in [H,W,D] or [D,H,W] layout.
//
// Thread mapping: for [H,W,D] outputs consecutive threads take consecutive
// d of a pixel (coalesced stores); for [D,H,W] they take consecutive x.
#include <type_traits>

#include "common.cuh"
#include "pipeline.cuh"

namespace cbmv {
namespace {

constexpr int kBlock = 128;

// Decodes the (y, x, d) a thread owns from a launch over (row-slab, y[, d]).
struct VolCoord {
  int64_t y, x;
  int d;
  bool in;
};

__device__ __forceinline__ VolCoord vol_coord(int layout, int64_t W, int D) {
  VolCoord c;
  c.y = blockIdx.y;
  if (layout == CBMV_HWD) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    c.in = idx < W * D;
    c.x = idx / D;
    c.d = (int)(idx - c.x * D);
  } else {
    c.x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    c.d = blockIdx.z;
    c.in = c.x < W;
  }
  return c;
}

inline dim3 vol_grid(int layout, int64_t H, int64_t W, int D) {
  if (layout == CBMV_HWD) return dim3((unsigned)((W * D + kBlock - 1) / kBlock), (unsigned)H, 1);
  return dim3((unsigned)((W + kBlock - 1) / kBlock), (unsigned)H, (unsigned)D);
}

// ---------------------------------------------------------------- census
// Descriptor of pixel (i+wc, j+wc), i < H-w, j < W-w: bit k set when the
// window's centre is below its k-th pixel in row-major order
// (_mm_cmplt_epi16(centre, neighbour), matchers.cpp:286-294).
__global__ void census_desc_kernel(const uint8_t* __restrict__ img, int64_t H, int64_t W, int w,
                                   ulonglong2* __restrict__ desc) {
  const int64_t n = (H - w) * (W - w);
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / (W - w), j = t - i * (W - w);
    const int wc = w / 2;
    const int c = img[(i + wc) * W + j + wc];
    unsigned long long b0 = 0, b1 = 0;
    int k = 0;
    for (int wh = 0; wh < w; wh++) {
      const uint8_t* row = img + (i + wh) * W + j;
      for (int ww = 0; ww < w; ww++, k++) {
        const unsigned long long bit = c < row[ww] ? 1ull : 0ull;
        if (k < 64) b0 |= bit << k;
        else b1 |= bit << (k - 64);
      }
    }
    desc[(i + wc) * W + j + wc] = make_ulonglong2(b0, b1);
  }
}

// ------------------------------------------------------------------- NCC
// Window sum A and 1/sqrt(w^2 B - A^2) (matchers.cpp:115-131); B is exact.
__global__ void ncc_stats_kernel(const uint8_t* __restrict__ img, int64_t H, int64_t W, int w,
                                 uint32_t* __restrict__ A, double* __restrict__ C) {
  const int64_t n = (H - w) * (W - w);
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / (W - w), j = t - i * (W - w);
    const int wc = w / 2;
    unsigned long long a = 0, b = 0;
    for (int wh = 0; wh < w; wh++)
      for (int ww = 0; ww < w; ww++) {
        const unsigned long long v = img[(i + wh) * W + j + ww];
        a += v;
        b += v * v;
      }
    const int64_t p = (i + wc) * W + j + wc;
    A[p] = (uint32_t)a;
    C[p] = 1.0 / sqrt((double)((unsigned long long)(w * w) * b) - (double)a * (double)a);
  }
}

template <class T>
__global__ void ncc_cost_kernel(const uint8_t* __restrict__ L, const uint8_t* __restrict__ R,
                                const uint32_t* __restrict__ Al, const uint32_t* __restrict__ Ar,
                                const double* __restrict__ Cl, const double* __restrict__ Cr,
                                int64_t H, int64_t W, int D, int w, int layout,
                                T* __restrict__ out) {
  const VolCoord c = vol_coord(layout, W, D);
  if (!c.in) return;
  const int wc = w / 2;
  const int64_t i = c.y - wc, j = c.x - wc;
  double v = kRandMax;
  // matchers.cpp:168-172: rows i < H-w, cols d <= j < W-w
  if (i >= 0 && i < H - w && j >= c.d && j < W - w) {
    unsigned long long s = 0;
    for (int wh = 0; wh < w; wh++) {
      const uint8_t* lr = L + (i + wh) * W + j;
      const uint8_t* rr = R + (i + wh) * W + j - c.d;
      for (int ww = 0; ww < w; ww++) s += (unsigned)lr[ww] * (unsigned)rr[ww];
    }
    const int64_t pl = c.y * W + c.x, pr = pl - c.d;
    const double cl = Cl[pl], cr = Cr[pr];
    if (isfinite(cl) && isfinite(cr)) {
      const double lD = (double)s;
      const unsigned long long aa = (unsigned long long)Al[pl] * (unsigned long long)Ar[pr];
      const double num = (double)(w * w) * lD - (double)aa;  // exact: integers < 2^53
      v = -num * cl * cr;                                      // matchers.cpp:179
    } else {
      v = 1.0;                                                 // matchers.cpp:181
    }
  }
  out[vol_index(layout, c.y, c.x, c.d, H, W, D)] = cvt_out<T>(v);
}

// ----------------------------------------------------------------- Sobel
template <class T>
__global__ void sobel_kernel(const uint8_t* __restrict__ img, int64_t H, int64_t W,
                             T* __restrict__ out) {
  const int64_t n = H * W;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t y = p / W, x = p - y * W;
    int v = 0;
    // matchers.cpp:539-548: written at (i+1, j+1) for i < H-3, j < W-3
    if (y >= 1 && y - 1 < H - 3 && x >= 1 && x - 1 < W - 3) {
      const uint8_t* a = img + (y - 1) * W + (x - 1);
      v = -(int)a[0] + (int)a[2] - 2 * (int)a[W] + 2 * (int)a[W + 2] - (int)a[2 * W] +
          (int)a[2 * W + 2];
    }
    out[p] = (T)v;
  }
}

template <class S>
__global__ void to_int_kernel(const S* __restrict__ in, int64_t n, int32_t* __restrict__ out) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
       p += (int64_t)gridDim.x * blockDim.x)
    out[p] = (int32_t)in[p];
}

// ---------------------------------------------------------- SAD on Sobel
template <class T>
__global__ void sadsob_cost_kernel(const int32_t* __restrict__ SL, const int32_t* __restrict__ SR,
                                   int64_t H, int64_t W, int D, int w, int layout,
                                   T* __restrict__ out) {
  const VolCoord c = vol_coord(layout, W, D);
  if (!c.in) return;
  const int wc = w / 2;
  const int64_t i = c.y - wc, j = c.x - wc;
  double v = kRandMax;
  // matchers.cpp:412-423: rows i < H-w, cols d <= j < W-w
  if (i >= 0 && i < H - w && j >= c.d && j < W - w) {
    int s = 0;
    for (int wh = 0; wh < w; wh++) {
      const int32_t* lr = SL + (i + wh) * W + j;
      const int32_t* rr = SR + (i + wh) * W + j - c.d;
      for (int ww = 0; ww < w; ww++) s += abs(lr[ww] - rr[ww]);
    }
    v = (double)s;
  }
  out[vol_index(layout, c.y, c.x, c.d, H, W, D)] = cvt_out<T>(v);
}

// ------------------------------------------------------------------ ZSAD
// Window means: exact integer sum, one float64 division (matchers.cpp:474-482).
__global__ void zsad_means_kernel(const uint8_t* __restrict__ img, int64_t H, int64_t W, int w,
                                  double* __restrict__ mean) {
  const int64_t n = (H - w) * (W - w);
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / (W - w), j = t - i * (W - w);
    const int wc = w / 2;
    int s = 0;
    for (int wh = 0; wh < w; wh++)
      for (int ww = 0; ww < w; ww++) s += img[(i + wh) * W + j + ww];
    mean[(i + wc) * W + j + wc] = (double)s / (double)(w * w);
  }
}

template <class T>
__global__ void zsad_cost_kernel(const uint8_t* __restrict__ L, const uint8_t* __restrict__ R,
                                 const double* __restrict__ ml, const double* __restrict__ mr,
                                 int64_t H, int64_t W, int D, int w, int layout,
                                 T* __restrict__ out) {
  const VolCoord c = vol_coord(layout, W, D);
  if (!c.in) return;
  const int wc = w / 2;
  const int64_t i = c.y - wc, j = c.x - wc;
  double v = kRandMax;
  // matchers.cpp:495-505: rows i < H-w, cols d <= j < W-w
  if (i >= 0 && i < H - w && j >= c.d && j < W - w) {
    const double mul = ml[c.y * W + c.x];
    const double mur = mr[c.y * W + c.x - c.d];
    double s = 0.0;
    for (int wh = 0; wh < w; wh++) {
      const uint8_t* lr = L + (i + wh) * W + j;
      const uint8_t* rr = R + (i + wh) * W + j - c.d;
      for (int ww = 0; ww < w; ww++) {
        // ((L - muL) - R) + muR, each step rounded as in the reference
        const double t = __dadd_rn(__dadd_rn(__dsub_rn((double)lr[ww], mul), -(double)rr[ww]), mur);
        s = __dadd_rn(s, fabs(t));
      }
    }
    v = s;
  }
  out[vol_index(layout, c.y, c.x, c.d, H, W, D)] = cvt_out<T>(v);
}

// ------------------------------------------------------ image terms
// The per-pixel terms of the default windows -- census descriptors (11),
// NCC sums (3), Sobel responses, ZSAD means (5) -- of one or two images
// (blockIdx.y) in one launch, from one shared-memory tile of the image; each
// array may be null.  The values and the regions written are those of the
// kernels above.  Bound by its 121 byte reads of shared memory per pixel, the
// tile's halo read from L2; both 694x554 images together 25 us (119 us in six
// launches that read every window from global memory), 96x64 5.2 us (29).
constexpr int kTermX = 32, kTermY = 16, kTermHalo = 5;

__global__ void __launch_bounds__(256) match_terms_kernel(MatchTerms t, int64_t H, int64_t W) {
  constexpr int SX = kTermX + 2 * kTermHalo, SY = kTermY + 2 * kTermHalo, P = 48;
  __shared__ uint8_t px[SY][P];
  const int im = blockIdx.y;
  const uint8_t* __restrict__ img = t.img[im];
  const int64_t ntx = (W + kTermX - 1) / kTermX;
  const int64_t X0 = blockIdx.x % ntx * kTermX, Y0 = blockIdx.x / ntx * kTermY;
  for (int q = threadIdx.x; q < SY * P; q += 256) {
    const int r = q / P, c = q % P;
    const int64_t y = Y0 - kTermHalo + r, x = X0 - kTermHalo + c;
    if (c < SX) px[r][c] = y >= 0 && y < H && x >= 0 && x < W ? __ldg(img + y * W + x) : 0;
  }
  __syncthreads();
  const int lx = threadIdx.x & 31;
  const int64_t x = X0 + lx;
  // pixel (i + r, j + r) of a w-wide window, r = w / 2, exists for i < H - w, j < W - w
  auto inside = [&](int64_t y, int w) { return y >= w / 2 && y < H - w + w / 2 && x >= w / 2 && x < W - w + w / 2; };
  for (int ly = threadIdx.x >> 5; ly < kTermY; ly += 8) {
    const int64_t y = Y0 + ly, p = y * W + x;
    if (y >= H || x >= W) continue;
    const uint8_t* c0 = &px[ly + kTermHalo][lx + kTermHalo];
    if (t.desc[im] && inside(y, 11)) {
      const int c = *c0;
      uint32_t b[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (int k = 0; k < 121; k++)
        if (c < (int)c0[(k / 11 - 5) * P + k % 11 - 5]) b[k >> 5] |= 1u << (k & 31);
      t.desc[im][p] = make_ulonglong2(b[0] | (unsigned long long)b[1] << 32, b[2] | (unsigned long long)b[3] << 32);
    }
    if (t.A[im] && inside(y, 3)) {
      unsigned a = 0, sq = 0;
#pragma unroll
      for (int k = 0; k < 9; k++) {
        const unsigned v = c0[(k / 3 - 1) * P + k % 3 - 1];
        a += v;
        sq += v * v;
      }
      t.A[im][p] = a;
      t.C[im][p] = 1.0 / sqrt((double)(9u * sq) - (double)a * (double)a);
    }
    if (t.mean[im] && inside(y, 5)) {
      int sum = 0;
#pragma unroll
      for (int k = 0; k < 25; k++) sum += c0[(k / 5 - 2) * P + k % 5 - 2];
      t.mean[im][p] = (double)sum / 25.0;
    }
    if (t.sob[im]) {
      // matchers.cpp:539-548: written at (i+1, j+1) for i < H-3, j < W-3
      const bool in = y >= 1 && y - 1 < H - 3 && x >= 1 && x - 1 < W - 3;
      t.sob[im][p] = in ? -(int)c0[-P - 1] + (int)c0[-P + 1] - 2 * (int)c0[-1] + 2 * (int)c0[1] - (int)c0[P - 1] + (int)c0[P + 1] : 0;
    }
  }
}

// ------------------------------------------------------- strip matchers
// The cost volumes of census (any window) and of the default windows of NCC
// (3), SAD-on-Sobel (5) and ZSAD (5), float32 or float64, either layout.  A
// warp owns 32 disparities (lane = d) of a strip of XS columns of one row
// and walks the strip, so a step adds one window column:
//   - the window columns the warp meets are staged once in its own shared
//     memory (XS + w - 1 left columns, 31 more right ones), clamped to the
//     image there, so a step is one or two shared-memory loads without
//     address arithmetic or bounds tests;
//   - NCC packs a column's three bytes in a word (one dp4a per column); SAD
//     and ZSAD in float32 keep a running window sum over a register ring of
//     columns; ZSAD in float64 follows the reference's order of operations
//     on a ring of doubles;
//   - [D,H,W] outputs are turned around in a shared-memory tile.
// Every window sum is an exact integer, so a float32 volume is the float32
// rounding of the reference's value (ZSAD: of the exact quotient; the
// reference's float64 chain differs from it by ~1e-15 relative).
// Bound by instruction issue (census: POPC; ZSAD float64: the FP64 pipe, 75
// additions per value, 0.21 ms of the 0.36).  At 694x554 D=128, us, before
// in brackets (thread per value, or a strip with its columns loaded from
// global memory at clamped 64-bit addresses):
//                  census     NCC        SAD-Sobel  ZSAD
//   float32 [H,W,D]  63 (93)    94 (199)   92 (282)   120 (369)
//   float64 [H,W,D]  67 (218)   99 (670)   98 (834)   359 (932)
//   float64 [D,H,W]             206        144        410
// against 31 / 61 us for writing the volume.
enum StripMode { kStripCensus, kStripNcc, kStripSadSob, kStripZsad };
constexpr int kStripWarps = 4;

struct StripArgs {
  const void *L, *R;            // census descriptors, uint8 images or int32 Sobel responses
  const uint32_t *Al, *Ar;      // NCC window sums and 1 / sqrt
  const double *Cl, *Cr;
  const double *ml, *mr;        // ZSAD window means (float64 volumes)
  int64_t H, W;
  int D, w;
};

// A column of a 5-pixel-high window of 8-bit pixels as packed 16-bit values
// scale * pixel + bias (rows 0..4, a sixth half zero) and the pixels' sum.
__device__ __forceinline__ uint4 zsad_column(const uint8_t* __restrict__ p, int64_t W, unsigned scale, unsigned bias) {
  const unsigned a = p[0], b = p[W], c = p[2 * W], d = p[3 * W], e = p[4 * W];
  return make_uint4((scale * a + bias) | (scale * b + bias) << 16, (scale * c + bias) | (scale * d + bias) << 16,
                    scale * e + bias, a + b + c + d + e);
}

template <int MODE, class T, int LAYOUT, int XS>
__global__ void __launch_bounds__(32 * kStripWarps) matcher_strip_kernel(StripArgs a, T* __restrict__ out) {
  constexpr bool kF64Zsad = MODE == kStripZsad && std::is_same<T, double>::value;
  constexpr int WIN = MODE == kStripCensus ? 1 : MODE == kStripNcc ? 3 : 5;  // window columns staged
  constexpr int r0 = WIN / 2, NL = XS + WIN - 1, NR = NL + 31;
  // shared memory per warp: left columns, right columns, [D,H,W] tile
  constexpr int kLBytes = kF64Zsad ? XS * 26 * 8 : NL * (MODE == kStripNcc ? 4 : MODE == kStripSadSob ? 32 : 16);
  constexpr int kRBytes = kF64Zsad ? 5 * NR * 8 : NR * (MODE == kStripNcc ? 4 : MODE == kStripSadSob ? 20 : 16);
  constexpr int kTile = LAYOUT == CBMV_DHW ? 32 * (XS + 1) * (int)sizeof(T) : 0;
  constexpr int kBytes = ((kLBytes + 15) / 16 + (kRBytes + 15) / 16 + (kTile + 15) / 16) * 16;
  __shared__ __align__(16) unsigned char smem[kStripWarps * kBytes];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* sl = smem + warp * kBytes;
  unsigned char* sr = sl + (kLBytes + 15) / 16 * 16;
  T* tile = reinterpret_cast<T*>(sr + (kRBytes + 15) / 16 * 16);
  const int64_t H = a.H, W = a.W, y = blockIdx.y;
  const int D = a.D, ndb = (D + 31) / 32;
  const int64_t unit = (int64_t)blockIdx.x * kStripWarps + warp;
  const int64_t x0 = unit / ndb * XS;
  const int d0 = (int)(unit % ndb) * 32, d = d0 + lane;
  if (x0 >= W) return;
  // the reference's valid region (matchers.cpp:168-172, 312-316, 412-423,
  // 495-505): rows and columns r .. size - w + r - 1, d <= column index - r
  const int r = a.w / 2;
  const bool row_ok = y >= r && y < H - a.w + r;
  const int64_t xend = W - a.w + r;
  if (row_ok) {
    const int64_t cl0 = x0 - r0, cr0 = x0 - r0 - d0 - 31, top = (y - r0) * W;
    auto col = [&](int64_t c) { return c < 0 ? (int64_t)0 : c >= W ? W - 1 : c; };
    if constexpr (MODE == kStripCensus) {
      const uint4 *L = static_cast<const uint4*>(a.L) + top, *R = static_cast<const uint4*>(a.R) + top;
      for (int i = lane; i < NL; i += 32) reinterpret_cast<uint4*>(sl)[i] = __ldg(L + col(cl0 + i));
      for (int i = lane; i < NR; i += 32) reinterpret_cast<uint4*>(sr)[i] = __ldg(R + col(cr0 + i));
    } else if constexpr (MODE == kStripNcc) {
      const uint8_t *L = static_cast<const uint8_t*>(a.L) + top, *R = static_cast<const uint8_t*>(a.R) + top;
      auto pack = [&](const uint8_t* p) { return (uint32_t)p[0] | (uint32_t)p[W] << 8 | (uint32_t)p[2 * W] << 16; };
      for (int i = lane; i < NL; i += 32) reinterpret_cast<uint32_t*>(sl)[i] = pack(L + col(cl0 + i));
      for (int i = lane; i < NR; i += 32) reinterpret_cast<uint32_t*>(sr)[i] = pack(R + col(cr0 + i));
    } else if constexpr (MODE == kStripSadSob) {
      const int32_t *L = static_cast<const int32_t*>(a.L) + top, *R = static_cast<const int32_t*>(a.R) + top;
      for (int i = lane; i < NL; i += 32) {
        const int32_t* p = L + col(cl0 + i);
        reinterpret_cast<int4*>(sl)[2 * i] = make_int4(p[0], p[W], p[2 * W], p[3 * W]);
        reinterpret_cast<int*>(sl)[8 * i + 4] = p[4 * W];
      }
      for (int i = lane; i < NR; i += 32) {
        const int32_t* p = R + col(cr0 + i);
#pragma unroll
        for (int k = 0; k < 5; k++) reinterpret_cast<int*>(sr)[k * NR + i] = p[k * W];
      }
    } else if constexpr (!kF64Zsad) {
      const uint8_t *L = static_cast<const uint8_t*>(a.L) + top, *R = static_cast<const uint8_t*>(a.R) + top;
      for (int i = lane; i < NL; i += 32) reinterpret_cast<uint4*>(sl)[i] = zsad_column(L + col(cl0 + i), W, 25u, 6375u);
      for (int i = lane; i < NR; i += 32) reinterpret_cast<uint4*>(sr)[i] = zsad_column(R + col(cr0 + i), W, 25u, 0u);
    } else {
      // L - mean of every window pixel, in the reference's order (row by row)
      const uint8_t *L = static_cast<const uint8_t*>(a.L) + top, *R = static_cast<const uint8_t*>(a.R) + top;
      for (int i = lane; i < XS * 25; i += 32) {
        const int s = i / 25, k = i - 25 * s;
        const int64_t x = x0 + s;
        if (x >= r && x < xend)
          reinterpret_cast<double*>(sl)[s * 26 + k] = __dsub_rn((double)L[(k / 5) * W + x - 2 + k % 5], a.ml[y * W + x]);
      }
      for (int i = lane; i < NR; i += 32) {
        const uint8_t* p = R + col(cr0 + i);
#pragma unroll
        for (int k = 0; k < 5; k++) reinterpret_cast<double*>(sr)[k * NR + i] = (double)p[k * W];
      }
    }
  }
  __syncwarp();
  // right column of this lane at left column index i: i + 31 - lane
  const int ro = 31 - lane;
  T* o = out + (y * W + x0) * D + d;
  // window columns of the ring: the sum over the column's rows, ZSAD's
  // packed 25 (L - R) + 6375 per row, ZSAD float64's right pixels
  int ring[WIN] = {}, sum = 0;
  uint32_t zr[MODE == kStripZsad && !kF64Zsad ? 15 : 1];
  double rr[kF64Zsad ? 25 : 1];
  auto push = [&](int i, int slot) {  // staged column i enters the window
    if constexpr (MODE == kStripNcc) {
      const int c = (int)__dp4a(reinterpret_cast<const uint32_t*>(sl)[i], reinterpret_cast<const uint32_t*>(sr)[i + ro], 0u);
      sum += c - ring[slot];
      ring[slot] = c;
    } else if constexpr (MODE == kStripSadSob) {
      const int4 l = reinterpret_cast<const int4*>(sl)[2 * i];
      const int l4 = reinterpret_cast<const int*>(sl)[8 * i + 4];
      const int* q = reinterpret_cast<const int*>(sr) + i + ro;
      const int c = abs(l.x - q[0]) + abs(l.y - q[NR]) + abs(l.z - q[2 * NR]) + abs(l.w - q[3 * NR]) + abs(l4 - q[4 * NR]);
      sum += c - ring[slot];
      ring[slot] = c;
    } else if constexpr (MODE == kStripZsad && !kF64Zsad) {
      const uint4 l = reinterpret_cast<const uint4*>(sl)[i], q = reinterpret_cast<const uint4*>(sr)[i + ro];
      zr[3 * slot] = l.x - q.x;  // 6375 + 25 (L - R) >= 0 in either half: no borrow between them
      zr[3 * slot + 1] = l.y - q.y;
      zr[3 * slot + 2] = l.z - q.z;
      const int c = (int)(l.w - q.w);
      sum += c - ring[slot];
      ring[slot] = c;
    } else if constexpr (kF64Zsad) {
#pragma unroll
      for (int k = 0; k < 5; k++) rr[slot * 5 + k] = reinterpret_cast<const double*>(sr)[k * NR + i + ro];
    }
  };
  if (row_ok && WIN > 1) {
#pragma unroll
    for (int i = 0; i < WIN - 1; i++) push(i, i);
  }
#pragma unroll
  for (int s = 0; s < XS; s++) {
    const int64_t x = x0 + s;
    if (x >= W) break;
    T v = (T)kRandMax;
    if (row_ok) {
      if constexpr (WIN > 1) push(s + WIN - 1, (s + WIN - 1) % WIN);
      if (x >= (int64_t)d + r && x < xend) {
        if constexpr (MODE == kStripCensus) {
          const uint4 l = reinterpret_cast<const uint4*>(sl)[s], q = reinterpret_cast<const uint4*>(sr)[s + ro];
          v = (T)(__popc(l.x ^ q.x) + __popc(l.y ^ q.y) + (__popc(l.z ^ q.z) + __popc(l.w ^ q.w)));
        } else if constexpr (MODE == kStripNcc) {
          const int64_t pl = y * W + x, pr = pl - d;
          const double cl = a.Cl[pl], cr = a.Cr[pr];
          // 9 S - A_L A_R exactly (both below 2^23), then the reference's product (matchers.cpp:179, 181)
          const double num = (double)(9 * sum - (int)(a.Al[pl] * a.Ar[pr]));
          v = isfinite(cl) && isfinite(cr) ? (T)(-num * cl * cr) : (T)1.0;
        } else if constexpr (MODE == kStripSadSob) {
          v = (T)sum;
        } else if constexpr (!kF64Zsad) {
          // sum |X - m| over the window's 25 values X = 25 (L - R), m = sum (L - R) = 25 x their mean difference,
          // as 2 sum max(X, m) - 50 m (the X sum to 25 m); offset by 6375 so that the packed halves are
          // unsigned, with the five unused sixth halves counting m' each: 2 S - 60 m'
          const unsigned m = (unsigned)(sum + 6375), m2 = m * 0x10001u;
          unsigned S = 0;
#pragma unroll
          for (int k = 0; k < 5; k++)  // at most 3 * 12750 per half of a column
            S = __dp2a_lo(__vmaxu2(zr[3 * k], m2) + __vmaxu2(zr[3 * k + 1], m2) + __vmaxu2(zr[3 * k + 2], m2), 0x0101u, S);
          // the correctly rounded quotient by 25 (Markstein's division with a correctly rounded reciprocal;
          // equal to IEEE division for every sum a window can have, 0 .. 318,750)
          const float acc = (float)(int)(2u * S - 60u * m);
          constexpr float inv = 1.0f / 25.0f;
          const float q = __fmul_rn(acc, inv);
          v = (T)fmaf(fmaf(-q, 25.0f, acc), inv, q);
        } else {
          const double mur = a.mr[y * W + x - d];
          const double* lm = reinterpret_cast<const double*>(sl) + s * 26;
          double acc = 0.0;
#pragma unroll
          for (int wh = 0; wh < 5; wh++)
#pragma unroll
            for (int ww = 0; ww < 5; ww++)  // ((L - muL) - R) + muR, each step rounded as in the reference
              acc = __dadd_rn(acc, fabs(__dadd_rn(__dsub_rn(lm[wh * 5 + ww], rr[(s + ww) % 5 * 5 + wh]), mur)));
          v = (T)acc;
        }
      }
    }
    if (LAYOUT == CBMV_DHW) {
      tile[lane * (XS + 1) + s] = v;
    } else {
      if (d < D) *o = v;
      o += D;
    }
  }
  if (LAYOUT == CBMV_DHW) {
    __syncwarp();
    constexpr int kRows = 32 / XS;  // disparities written per step
    const int64_t x = x0 + lane % XS;
    for (int k = lane / XS; k < 32 && d0 + k < D; k += kRows)
      if (x < W) out[((int64_t)(d0 + k) * H + y) * W + x] = tile[k * (XS + 1) + lane % XS];
  }
}

}  // namespace

// Argument checks shared by the matcher entry points (also cbmv_census_static).
int check_common(const void* a, const void* b, const void* out, int64_t H, int64_t W, int D, int w,
                 int dtype, int layout, int wmax) {
  CBMV_REQUIRE(a && b && out, CBMV_EINVAL, "null pointer argument");
  CBMV_REQUIRE(H > 0 && W > 0 && D > 0, CBMV_EINVAL, "bad size H=%lld W=%lld D=%d",
               (long long)H, (long long)W, D);
  CBMV_REQUIRE(H <= 65535, CBMV_ERANGE, "H=%lld exceeds 65535", (long long)H);
  CBMV_REQUIRE(D <= 65535, CBMV_ERANGE, "D=%d exceeds 65535", D);
  CBMV_REQUIRE(w >= 1 && (w & 1) && w <= wmax, CBMV_EINVAL, "window %d must be odd and <= %d", w,
               wmax);
  CBMV_REQUIRE(dtype == CBMV_F32 || dtype == CBMV_F64, CBMV_EINVAL, "bad dtype %d", dtype);
  CBMV_REQUIRE(layout == CBMV_HWD || layout == CBMV_DHW, CBMV_EINVAL, "bad layout %d", layout);
  return CBMV_OK;
}

namespace {

// Scratch allocation for the stand-alone matcher entry points (the fused
// pipeline keeps its scratch in its context instead).
struct Scratch {
  void* p = nullptr;
  ~Scratch() {
    if (p) cudaFree(p);
  }
};

}  // namespace

// Fills a volume with the sentinel where the valid region is empty.
template <class T>
__global__ void fill_kernel(T* out, int64_t n, T v) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
       p += (int64_t)gridDim.x * blockDim.x)
    out[p] = v;
}

int launch_match_terms(const MatchTerms& t, int64_t H, int64_t W, cudaStream_t st) {
  const int64_t tiles = ((W + kTermX - 1) / kTermX) * ((H + kTermY - 1) / kTermY);
  CBMV_REQUIRE(tiles < ((int64_t)1 << 31), CBMV_ERANGE, "image too large for the term grid");
  match_terms_kernel<<<dim3((unsigned)tiles, t.img[1] ? 2 : 1), 256, 0, st>>>(t, H, W);
  return check_launch("match_terms");
}

int launch_census_descs(const uint8_t* L, const uint8_t* R, int64_t H, int64_t W, int w, ulonglong2* dl,
                        ulonglong2* dr, cudaStream_t st) {
  if (w == 11) {
    MatchTerms t{{L, R}};
    t.desc[0] = dl, t.desc[1] = dr;
    return launch_match_terms(t, H, W, st);
  }
  if (H <= w || W <= w) return CBMV_OK;
  const int64_t n = (H - w) * (W - w);
  census_desc_kernel<<<grid_for(n, kBlock), kBlock, 0, st>>>(L, H, W, w, dl);
  census_desc_kernel<<<grid_for(n, kBlock), kBlock, 0, st>>>(R, H, W, w, dr);
  return check_launch("census_desc");
}

// The strip kernels' launch; W / XS * D / 32 warps per row.
static dim3 strip_grid(const StripArgs& a, int xs) {
  const int64_t units = ((a.W + xs - 1) / xs) * ((a.D + 31) / 32);
  return dim3((unsigned)((units + kStripWarps - 1) / kStripWarps), (unsigned)a.H);
}

// A strip's lanes are disparities: below 32 of them its time stays what it is
// at 32, and for a few the general kernels' thread per value is quicker; so it
// is for NCC volumes that fill neither.  us, general against strip, the last
// size of the general kernel and the next measured (census is quicker in
// strips from D = 1 on):
//   NCC        [H,W,D]  694x554 D=4   42 / 49     D=6   53 / 49
//   NCC        [D,H,W]  694x554 D=10  71 / 68-74  D=12  82 / 69-74
//   NCC                 320x240 D=6   22 / 24     D=8   25 / 24;  80x60 D=33 17 / 20
//   SAD-Sobel           694x554 D=3   38 / 38-42  D=4   44 / 38-43
//   ZSAD f64   [H,W,D]  694x554 D=10 100 / 114    D=12 116 / 114
//   ZSAD f64   [D,H,W]  694x554 D=12 114 / 120    D=14 129 / 120
static bool strip_is_quicker(int mode, int layout, int64_t H, int64_t W, int D) {
  const bool hwd = layout == CBMV_HWD;
  if (mode == kStripNcc && H * W * D <= 500000) return false;
  return D > (mode == kStripNcc ? (hwd ? 5 : 10) : mode == kStripSadSob ? 3 : mode == kStripZsad ? (hwd ? 11 : 13) : 0);
}

template <int MODE, class T, int XS>
static int launch_strip(const StripArgs& a, int layout, T* out, cudaStream_t st) {
  const dim3 grid = strip_grid(a, XS);
  if (layout == CBMV_HWD) matcher_strip_kernel<MODE, T, CBMV_HWD, XS><<<grid, 32 * kStripWarps, 0, st>>>(a, out);
  else matcher_strip_kernel<MODE, T, CBMV_DHW, XS><<<grid, 32 * kStripWarps, 0, st>>>(a, out);
  return check_launch("matcher_strip");
}

template <class T>
int launch_census_cost(const ulonglong2* dl, const ulonglong2* dr, int64_t H, int64_t W, int D,
                       int w, int layout, T* out, cudaStream_t st) {
  StripArgs a{};
  a.L = dl;
  a.R = dr;
  a.H = H;
  a.W = W;
  a.D = D;
  a.w = w;
  return launch_strip<kStripCensus, T, 32>(a, layout, out, st);
}

int launch_ncc_stats(const uint8_t* img, int64_t H, int64_t W, int w, uint32_t* A, double* C,
                     cudaStream_t st) {
  if (H <= w || W <= w) return CBMV_OK;
  const int64_t n = (H - w) * (W - w);
  ncc_stats_kernel<<<grid_for(n, kBlock), kBlock, 0, st>>>(img, H, W, w, A, C);
  return check_launch("ncc_stats");
}

template <class T>
int launch_ncc_cost(const uint8_t* L, const uint8_t* R, const uint32_t* Al, const uint32_t* Ar,
                    const double* Cl, const double* Cr, int64_t H, int64_t W, int D, int w,
                    int layout, T* out, cudaStream_t st) {
  if (w == 3 && strip_is_quicker(kStripNcc, layout, H, W, D)) {
    const StripArgs a{L, R, Al, Ar, Cl, Cr, nullptr, nullptr, H, W, D, w};
    return launch_strip<kStripNcc, T, 32>(a, layout, out, st);
  }
  ncc_cost_kernel<T><<<vol_grid(layout, H, W, D), kBlock, 0, st>>>(L, R, Al, Ar, Cl, Cr, H, W, D, w,
                                                                   layout, out);
  return check_launch("ncc_cost");
}

template <class T>
int launch_sadsob_cost(const int32_t* SL, const int32_t* SR, int64_t H, int64_t W, int D, int w,
                       int layout, T* out, cudaStream_t st) {
  if (w == 5 && strip_is_quicker(kStripSadSob, layout, H, W, D)) {
    const StripArgs a{SL, SR, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, H, W, D, w};
    return launch_strip<kStripSadSob, T, 32>(a, layout, out, st);
  }
  sadsob_cost_kernel<T><<<vol_grid(layout, H, W, D), kBlock, 0, st>>>(SL, SR, H, W, D, w, layout, out);
  return check_launch("sadsob_cost");
}

int launch_zsad_means(const uint8_t* img, int64_t H, int64_t W, int w, double* mean,
                      cudaStream_t st) {
  if (H <= w || W <= w) return CBMV_OK;
  const int64_t n = (H - w) * (W - w);
  zsad_means_kernel<<<grid_for(n, kBlock), kBlock, 0, st>>>(img, H, W, w, mean);
  return check_launch("zsad_means");
}

template <class T>
static int launch_zsad_general(const uint8_t* L, const uint8_t* R, const double* ml, const double* mr, int64_t H,
                               int64_t W, int D, int w, int layout, T* out, cudaStream_t st) {
  zsad_cost_kernel<T><<<vol_grid(layout, H, W, D), kBlock, 0, st>>>(L, R, ml, mr, H, W, D, w, layout,
                                                                    out);
  return check_launch("zsad_cost");
}

// The float32 volumes of the stand-alone entry point are the float32
// rounding of the reference's float64 chain; those of the learned path
// (launch_zsad_cost_f32) of the exact quotient.
template <class T>
int launch_zsad_cost(const uint8_t* L, const uint8_t* R, const double* ml, const double* mr,
                     int64_t H, int64_t W, int D, int w, int layout, T* out, cudaStream_t st) {
  if (w == 5 && std::is_same<T, double>::value && strip_is_quicker(kStripZsad, layout, H, W, D)) {
    const StripArgs a{L, R, nullptr, nullptr, nullptr, nullptr, ml, mr, H, W, D, w};
    return launch_strip<kStripZsad, double, 16>(a, layout, reinterpret_cast<double*>(out), st);
  }
  return launch_zsad_general<T>(L, R, ml, mr, H, W, D, w, layout, out, st);
}

int launch_zsad_cost_f32(const uint8_t* L, const uint8_t* R, const double* ml, const double* mr, int64_t H,
                         int64_t W, int D, int w, float* out, cudaStream_t st) {
  if (w == 5) {
    const StripArgs a{L, R, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, H, W, D, w};
    matcher_strip_kernel<kStripZsad, float, CBMV_HWD, 32><<<strip_grid(a, 32), 32 * kStripWarps, 0, st>>>(a, out);
    return check_launch("matcher_strip");
  }
  return launch_zsad_general<float>(L, R, ml, mr, H, W, D, w, CBMV_HWD, out, st);
}

template int launch_census_cost<double>(const ulonglong2*, const ulonglong2*, int64_t, int64_t, int,
                                        int, int, double*, cudaStream_t);
template int launch_census_cost<float>(const ulonglong2*, const ulonglong2*, int64_t, int64_t, int,
                                       int, int, float*, cudaStream_t);
template int launch_ncc_cost<double>(const uint8_t*, const uint8_t*, const uint32_t*,
                                     const uint32_t*, const double*, const double*, int64_t,
                                     int64_t, int, int, int, double*, cudaStream_t);
template int launch_sadsob_cost<double>(const int32_t*, const int32_t*, int64_t, int64_t, int, int,
                                        int, double*, cudaStream_t);
template int launch_zsad_cost<double>(const uint8_t*, const uint8_t*, const double*, const double*,
                                      int64_t, int64_t, int, int, int, double*, cudaStream_t);
template int launch_ncc_cost<float>(const uint8_t*, const uint8_t*, const uint32_t*, const uint32_t*,
                                    const double*, const double*, int64_t, int64_t, int, int, int, float*,
                                    cudaStream_t);
template int launch_sadsob_cost<float>(const int32_t*, const int32_t*, int64_t, int64_t, int, int, int,
                                       float*, cudaStream_t);
template int launch_zsad_cost<float>(const uint8_t*, const uint8_t*, const double*, const double*,
                                     int64_t, int64_t, int, int, int, float*, cudaStream_t);

}  // namespace cbmv

using namespace cbmv;

extern "C" int cbmv_census(const uint8_t* L, const uint8_t* R, int64_t H, int64_t W, int D,
                           int wsize, void* out, int dtype, int layout, void* stream) {
  int rc = check_common(L, R, out, H, W, D, wsize, dtype, layout, 11);
  if (rc) return rc;
  cudaStream_t st = as_stream(stream);
  Scratch s;
  CBMV_CUDA(cudaMallocAsync(&s.p, (size_t)H * W * sizeof(ulonglong2) * 2, st));
  ulonglong2* dl = (ulonglong2*)s.p;
  ulonglong2* dr = dl + H * W;
  if ((rc = launch_census_descs(L, R, H, W, wsize, dl, dr, st))) return rc;
  rc = dtype == CBMV_F64 ? launch_census_cost(dl, dr, H, W, D, wsize, layout, (double*)out, st)
                         : launch_census_cost(dl, dr, H, W, D, wsize, layout, (float*)out, st);
  CBMV_CUDA(cudaFreeAsync(s.p, st));
  s.p = nullptr;
  return rc;
}

extern "C" int cbmv_ncc(const uint8_t* L, const uint8_t* R, int64_t H, int64_t W, int D, int wsize,
                        void* out, int dtype, int layout, void* stream) {
  int rc = check_common(L, R, out, H, W, D, wsize, dtype, layout, 15);
  if (rc) return rc;
  cudaStream_t st = as_stream(stream);
  Scratch s;
  const size_t n = (size_t)H * W;
  CBMV_CUDA(cudaMallocAsync(&s.p, n * (2 * sizeof(uint32_t) + 2 * sizeof(double)), st));
  double* Cl = (double*)s.p;
  double* Cr = Cl + n;
  uint32_t* Al = (uint32_t*)(Cr + n);
  uint32_t* Ar = Al + n;
  if (wsize == 3 && strip_is_quicker(kStripNcc, layout, H, W, D)) {  // else two launches of the 9 values alone: 3 us less
    MatchTerms t{{L, R}};
    t.A[0] = Al, t.A[1] = Ar, t.C[0] = Cl, t.C[1] = Cr;
    rc = launch_match_terms(t, H, W, st);
  } else if (!(rc = launch_ncc_stats(L, H, W, wsize, Al, Cl, st))) {
    rc = launch_ncc_stats(R, H, W, wsize, Ar, Cr, st);
  }
  if (rc) return rc;
  rc = dtype == CBMV_F64
           ? launch_ncc_cost(L, R, Al, Ar, Cl, Cr, H, W, D, wsize, layout, (double*)out, st)
           : launch_ncc_cost(L, R, Al, Ar, Cl, Cr, H, W, D, wsize, layout, (float*)out, st);
  CBMV_CUDA(cudaFreeAsync(s.p, st));
  s.p = nullptr;
  return rc;
}

extern "C" int cbmv_sobel(const uint8_t* img, int64_t H, int64_t W, void* out, int dtype,
                          void* stream) {
  CBMV_REQUIRE(img && out, CBMV_EINVAL, "null pointer argument");
  CBMV_REQUIRE(H > 0 && W > 0, CBMV_EINVAL, "bad size");
  CBMV_REQUIRE(dtype == CBMV_F32 || dtype == CBMV_F64, CBMV_EINVAL, "bad dtype %d", dtype);
  cudaStream_t st = as_stream(stream);
  if (dtype == CBMV_F64)
    sobel_kernel<double><<<grid_for(H * W, kBlock), kBlock, 0, st>>>(img, H, W, (double*)out);
  else
    sobel_kernel<float><<<grid_for(H * W, kBlock), kBlock, 0, st>>>(img, H, W, (float*)out);
  return check_launch("sobel");
}

extern "C" int cbmv_sadsob(const void* SL, const void* SR, int sob_dtype, int64_t H, int64_t W,
                           int D, int wsize, void* out, int dtype, int layout, void* stream) {
  int rc = check_common(SL, SR, out, H, W, D, wsize, dtype, layout, 15);
  if (rc) return rc;
  CBMV_REQUIRE(sob_dtype == CBMV_F32 || sob_dtype == CBMV_F64, CBMV_EINVAL, "bad sobel dtype");
  cudaStream_t st = as_stream(stream);
  Scratch s;
  const int64_t n = H * W;
  CBMV_CUDA(cudaMallocAsync(&s.p, (size_t)n * 2 * sizeof(int32_t), st));
  int32_t* il = (int32_t*)s.p;
  int32_t* ir = il + n;
  if (sob_dtype == CBMV_F64) {
    to_int_kernel<double><<<grid_for(n, kBlock), kBlock, 0, st>>>((const double*)SL, n, il);
    to_int_kernel<double><<<grid_for(n, kBlock), kBlock, 0, st>>>((const double*)SR, n, ir);
  } else {
    to_int_kernel<float><<<grid_for(n, kBlock), kBlock, 0, st>>>((const float*)SL, n, il);
    to_int_kernel<float><<<grid_for(n, kBlock), kBlock, 0, st>>>((const float*)SR, n, ir);
  }
  if ((rc = check_launch("sadsob_convert"))) return rc;
  rc = dtype == CBMV_F64 ? launch_sadsob_cost(il, ir, H, W, D, wsize, layout, (double*)out, st)
                         : launch_sadsob_cost(il, ir, H, W, D, wsize, layout, (float*)out, st);
  CBMV_CUDA(cudaFreeAsync(s.p, st));
  s.p = nullptr;
  return rc;
}

extern "C" int cbmv_zsad(const uint8_t* L, const uint8_t* R, int64_t H, int64_t W, int D,
                         int wsize, void* out, int dtype, int layout, void* stream) {
  int rc = check_common(L, R, out, H, W, D, wsize, dtype, layout, 15);
  if (rc) return rc;
  cudaStream_t st = as_stream(stream);
  Scratch s;
  const size_t n = (size_t)H * W;
  CBMV_CUDA(cudaMallocAsync(&s.p, n * 2 * sizeof(double), st));
  double* ml = (double*)s.p;
  double* mr = ml + n;
  if (wsize == 5) {
    MatchTerms t{{L, R}};
    t.mean[0] = ml, t.mean[1] = mr;
    rc = launch_match_terms(t, H, W, st);
  } else if (!(rc = launch_zsad_means(L, H, W, wsize, ml, st))) {
    rc = launch_zsad_means(R, H, W, wsize, mr, st);
  }
  if (rc) return rc;
  rc = dtype == CBMV_F64
           ? launch_zsad_cost(L, R, ml, mr, H, W, D, wsize, layout, (double*)out, st)
           : launch_zsad_cost(L, R, ml, mr, H, W, D, wsize, layout, (float*)out, st);
  CBMV_CUDA(cudaFreeAsync(s.p, st));
  s.p = nullptr;
  return rc;
}
