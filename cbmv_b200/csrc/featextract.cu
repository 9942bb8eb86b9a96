// Feature extraction: the reference's layout helpers and confidence
// measures (cpp/featextract/featextract.cpp) and the fused 20-feature kernel
// that replaces Testing.__extract_features_lr (test.py:521-595).
//
// Every confidence is computed in float64 with the reference's operation
// order, so the features equal the reference's float64 values (and so their
// float32 roundings, which is what the random forest compares).  The one
// freedom taken is the order of the likelihood denominator's sum over d,
// which only moves it by an ulp of float64.
#include "common.cuh"
#include "features.cuh"

namespace cbmv {
namespace {

constexpr int kBlock = 256;

#define GRID_STRIDE(i, n) \
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// [rows, cols] -> [cols, rows] of float64 through 32 x 32 shared-memory
// tiles, both sides coalesced: bound by its traffic (787 MB for a 694x554
// D=128 volume).  Tiles are numbered along one grid axis: either side may be
// H*W.
__global__ void __launch_bounds__(256) transpose_f64_kernel(const double* __restrict__ in, int64_t rows, int64_t cols,
                                                            double* __restrict__ out) {
  __shared__ double tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t nc = (cols + 31) / 32, tiles = nc * ((rows + 31) / 32);
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int64_t r0 = t / nc * 32, c0 = t % nc * 32;
    __syncthreads();
#pragma unroll
    for (int k = ty; k < 32; k += 8)
      if (r0 + k < rows && c0 + tx < cols) tile[k][tx] = in[(r0 + k) * cols + c0 + tx];
    __syncthreads();
#pragma unroll
    for (int k = ty; k < 32; k += 8)
      if (c0 + k < cols && r0 + tx < rows) out[(c0 + k) * rows + r0 + tx] = tile[tx][k];
  }
}

// [D, H*W] -> [H*W, D] with the disparities of 32 pixels in one tile (64 of
// them where D has more), so that a run of `out` is written by one CTA: with
// D % 4 != 0 the runs of the 32 x 32 tiles share 32-byte sectors.
constexpr int kSwapD = 64;

__global__ void __launch_bounds__(256) swap_runs_kernel(const double* __restrict__ in, int64_t HW, int D, int dt,
                                                      double* __restrict__ out) {
  __shared__ double tile[kSwapD][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nd = (D + dt - 1) / dt;
  const int64_t tiles = (HW + 31) / 32 * nd;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int64_t p0 = t / nd * 32;
    const int d0 = (int)(t % nd) * dt, n = min(dt, D - d0), np = (int)min((int64_t)32, HW - p0);
    const double* src = in + (d0 + warp) * HW + p0 + lane;
    if (lane < np) {
#pragma unroll 8
      for (int d = warp; d < n; d += 8, src += 8 * HW) tile[d][lane] = __ldg(src);
    }
    __syncthreads();
    double* dst = out + (p0 + warp) * D + d0 + lane;
#pragma unroll 4
    for (int p = warp; p < np; p += 8, dst += 8 * (int64_t)D)
#pragma unroll
      for (int d = 0; d < kSwapD; d += 32)
        if (d + lane < n) dst[d] = tile[d + lane][p];
    __syncthreads();
  }
}

// A few disparities fill no tile: [D, H*W] -> [H*W, D] with a thread per value
// of `out`, and back with one per pixel.
__global__ void swap_few_kernel(const double* __restrict__ in, int64_t HW, int D, double* __restrict__ out) {
  GRID_STRIDE(t, D * HW) {
    const int64_t p = t / D, d = t - p * D;
    out[t] = in[d * HW + p];
  }
}
__global__ void swap_back_few_kernel(const double* __restrict__ in, int64_t HW, int D, double* __restrict__ out) {
  GRID_STRIDE(p, HW) {
#pragma unroll 4
    for (int d = 0; d < D; d++) out[d * HW + p] = __ldg(in + p * D + d);
  }
}

static unsigned tile_grid(int64_t tiles) { return (unsigned)(tiles < 1 << 30 ? tiles : 1 << 30); }

// us at 694x554: a few disparities' kernel, 32 x 32 tiles, whole runs
//   D     swap_axes          swap_axes_back
//     1     7 /  24            5 / 21
//    12    20 /  25           15 / 23
//    16    30 /  27
//    33    56 /  59 /  52
//    65   102 / 130 /  95
//    97   253 / 196 / 134
//   128   313 / 130 / 128
// Whole runs pay where the volume leaves L2 (450x375 D=50, 67 MB: 38 / 29 /
// 36; 1482x994 D=33, 389 MB: 307 / 230 / 179) and where the tiles' runs are
// unaligned (D=36 at 694x554: 56 with tiles).
int launch_swap_axes(const double* in, int64_t D, int64_t HW, double* out, cudaStream_t st) {
  if (D < 15) {
    swap_few_kernel<<<grid_for(D * HW, kBlock), kBlock, 0, st>>>(in, HW, (int)D, out);
  } else if (D % 4 != 0 && D > 32 && D < (1 << 20) && D * HW >= 12500000) {  // 100 MB
    const int64_t n = (D + kSwapD - 1) / kSwapD, dt = (D + n - 1) / n;
    swap_runs_kernel<<<tile_grid((HW + 31) / 32 * n), 256, 0, st>>>(in, HW, (int)D, (int)dt, out);
  } else {
    transpose_f64_kernel<<<tile_grid(((D + 31) / 32) * ((HW + 31) / 32)), 256, 0, st>>>(in, D, HW, out);
  }
  return check_launch("swap_axes");
}

int launch_swap_axes_back(const double* in, int64_t HW, int64_t D, double* out, cudaStream_t st) {
  if (D < 14) swap_back_few_kernel<<<grid_for(HW, kBlock), kBlock, 0, st>>>(in, HW, (int)D, out);
  else transpose_f64_kernel<<<tile_grid(((D + 31) / 32) * ((HW + 31) / 32)), 256, 0, st>>>(in, HW, D, out);
  return check_launch("swap_axes_back");
}

__global__ void get_cost_kernel(const double* __restrict__ in, int64_t n, int64_t K,
                                double* __restrict__ out) {
  GRID_STRIDE(t, n) out[t] = in[t * K];
}

// dir = +1: R[i,j,d] = C[i,j+d,d] for j < W-d (featextract.cpp:136-145)
// dir = -1: L[i,j,d] = R[i,j-d,d] for j >= d (featextract.cpp:473-481)
// otherwise the volume's first element (:130, :467).
__global__ void shift_kernel(const double* __restrict__ in, int64_t H, int64_t W, int64_t D,
                             int dir, double* __restrict__ out) {
  const double fill = in[0];
  GRID_STRIDE(t, H * W * D) {
    const int64_t d = t % D;
    const int64_t p = t / D;
    const int64_t j = p % W;
    const int64_t js = j + dir * d;
    out[t] = (js >= 0 && js < W) ? in[(p + dir * d) * D + d] : fill;
  }
}

// Row minimum as featextract.cpp:322-329 (start at RAND_MAX, strict <),
// one warp per row.
__device__ __forceinline__ double warp_row_min(const double* r, int64_t D) {
  double m = kRandMax;
  for (int64_t k = threadIdx.x & 31; k < D; k += 32) m = fmin(m, r[k]);
  for (int o = 16; o; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ double lik_term(double c, double m, double sigma) {
  const double num = c - m;
  return exp(-(num * num) / sigma);  // featextract.cpp:433-434
}

__global__ void ratio_kernel(const double* __restrict__ v, int64_t N, int64_t D, double e,
                             double* __restrict__ out) {
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; i < N; i += warps) {
    const double* r = v + i * D;
    const double m = warp_row_min(r, D);
    for (int64_t k = threadIdx.x & 31; k < D; k += 32)
      out[i * D + k] = (m == kRandMax) ? 0.0 : (m + e) / (r[k] + e);
  }
}

__global__ void likelihood_kernel(const double* __restrict__ v, int64_t N, int64_t D, double sigma,
                                  double* __restrict__ out) {
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; i < N; i += warps) {
    const double* r = v + i * D;
    const double m = warp_row_min(r, D);
    double den = 0.0;
    for (int64_t k = threadIdx.x & 31; k < D; k += 32) den += lik_term(r[k], m, sigma);
    den = warp_sum(den);
    for (int64_t k = threadIdx.x & 31; k < D; k += 32) {
      const double t = r[k] - m;
      out[i * D + k] = (m == kRandMax) ? 0.0 : exp(-((t * t) / sigma)) / den;
    }
  }
}

__global__ void ratio_samples_kernel(const double* __restrict__ v, int64_t N, int64_t D,
                                     const int32_t* __restrict__ s, double e,
                                     double* __restrict__ out) {
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; i < N; i += warps) {
    const double* r = v + i * D;
    const double m = warp_row_min(r, D);
    const int k = threadIdx.x & 31;
    if (k < 3) out[3 * i + k] = (m == kRandMax) ? 0.0 : (m + e) / (r[s[3 * i + k]] + e);
  }
}

__global__ void likelihood_samples_kernel(const double* __restrict__ v, int64_t N, int64_t D,
                                          const int32_t* __restrict__ s, double sigma,
                                          double* __restrict__ out) {
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; i < N; i += warps) {
    const double* r = v + i * D;
    const double m = warp_row_min(r, D);
    double den = 0.0;
    for (int64_t k = threadIdx.x & 31; k < D; k += 32) den += lik_term(r[k], m, sigma);
    den = warp_sum(den);
    const int k = threadIdx.x & 31;
    if (k < 3) {
      const double t = r[s[3 * i + k]] - m;
      out[3 * i + k] = (m == kRandMax) ? 0.0 : exp(-((t * t) / sigma)) / den;
    }
  }
}

__global__ void get_samples_kernel(const double* __restrict__ v, int64_t N, int64_t D,
                                   const int32_t* __restrict__ s, double* __restrict__ out) {
  GRID_STRIDE(t, 3 * N) out[t] = v[(t / 3) * D + s[t]];
}

__global__ void labels_kernel(int64_t N, int32_t* __restrict__ out) {
  GRID_STRIDE(t, 3 * N) out[t] = (t % 3) == 0 ? 1 : 0;
}

__device__ __forceinline__ uint32_t draw(uint64_t seed, int64_t s, int slot, uint32_t n) {
  uint64_t z = seed * 0x9E3779B97F4A7C15ull + (uint64_t)s * 3ull + (uint64_t)slot + 1;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (uint32_t)(z % n);
}

__global__ void d_indices_kernel(const int32_t* __restrict__ gt, int64_t N, int maxd, int thr,
                                 uint64_t seed, int32_t* __restrict__ out, int* __restrict__ bad) {
  GRID_STRIDE(s, N) {
    const int g = gt[s];
    const bool low = !(g - thr <= 0), high = !(g + thr >= maxd);
    const int lo_n = g - thr, hi_n = maxd - (g + thr + 1);
    int d1 = 0, d2 = 0;
    bool ok = g >= 0 && g <= maxd;
    if (low) d1 = (int)draw(seed, s, 0, (uint32_t)lo_n);
    else if (hi_n > 0) d1 = (int)draw(seed, s, 0, (uint32_t)hi_n) + (g + thr + 1);
    else ok = false;
    if (high && hi_n > 0) d2 = (int)draw(seed, s, 1, (uint32_t)hi_n) + (g + thr + 1);
    else if (!high && lo_n > 0) d2 = (int)draw(seed, s, 1, (uint32_t)lo_n);
    else ok = false;
    out[3 * s] = g;
    out[3 * s + 1] = d1;
    out[3 * s + 2] = d2;
    if (!ok) atomicExch(bad, 1);
  }
}

}  // namespace

// ------------------------------------------------------ fused features
// Per-pixel statistics of the matcher volumes for both reference views:
// stats[((m*2 + view)*HW + p)*2 + {0,1}] = {row minimum, likelihood
// denominator}; view 0 = left reference (row p of the volume), view 1 =
// right reference (right pixel p: entries C[p + d, d], the fill C[0,0,0]
// where x + d >= W, featextract.cpp:115-152).
// Bound by the FP64 pipe: 394 M exponentials of about 27 float64
// operations each at 694x554 D=128, 0.6 ms.  Left 571 us, right 835 us, all
// four matchers in a launch; 2351 us with one warp per (pixel, view) that
// read every row twice, the right view's diagonally, and a full division
// per term.  The right view through shared-memory tiles: 879 us.
struct VolsD {
  const double* v[4];
};

// view 0: one warp per pixel, its row in registers (KPL per lane; 0: D is
// beyond 32 KPL of any variant, the row is read twice)
template <int KPL>
__global__ void __launch_bounds__(kBlock) stats_left_kernel(VolsD vols, int64_t HW, int D, double* __restrict__ stats) {
  const int m = blockIdx.y, lane = threadIdx.x & 31;
  const double* __restrict__ vol = vols.v[m];
  double* __restrict__ o = stats + (int64_t)(2 * m) * HW * 2;
  const int64_t nwarps = (int64_t)gridDim.x * (kBlock / 32);
  for (int64_t p = ((int64_t)blockIdx.x * kBlock + threadIdx.x) >> 5; p < HW; p += nwarps) {
    const double* r = vol + p * D;
    double mn = kRandMax, den = 0.0;
    double v[KPL > 0 ? KPL : 1];
    if (KPL > 0) {
#pragma unroll
      for (int k = 0; k < KPL; k++) {
        v[k] = lane + 32 * k < D ? __ldg(r + lane + 32 * k) : kRandMax;
        mn = fmin(mn, v[k]);
      }
    } else {
      for (int d = lane; d < D; d += 32) mn = fmin(mn, r[d]);
    }
    for (int s = 16; s; s >>= 1) mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, s));
    if (KPL > 0) {
#pragma unroll
      for (int k = 0; k < KPL; k++)
        if (lane + 32 * k < D) den += lik_exp(v[k] - mn, m);
    } else {
      for (int d = lane; d < D; d += 32) den += lik_exp(r[d] - mn, m);
    }
    den = warp_sum(den);
    if (lane == 0) *reinterpret_cast<double2*>(o + 2 * p) = make_double2(mn, den);
  }
}

// view 1: a warp owns 32 right pixels of one row, lane l the pixel xr = X0 +
// 31 - l, whose costs are C[xr + d, d].  At step k the lane takes d = k + l
// (mod D): lanes that have not wrapped around read one row of the volume,
// x = X0 + 31 + k, at consecutive d, so every step is one or two coalesced
// runs and all lanes work in all D steps.  The second pass over the 32 x D
// values finds them in L1 or L2.
__global__ void __launch_bounds__(kBlock) stats_right_kernel(VolsD vols, int64_t H, int64_t W, int D,
                                                             double* __restrict__ stats) {
  const int m = blockIdx.y, lane = threadIdx.x & 31;
  const double* __restrict__ vol = vols.v[m];
  const double fill = __ldg(vol);
  const int64_t nxb = (W + 31) / 32, nwarps = (int64_t)gridDim.x * (kBlock / 32);
  for (int64_t u = ((int64_t)blockIdx.x * kBlock + threadIdx.x) >> 5; u < H * nxb; u += nwarps) {
    const int64_t y = u / nxb, xr = u % nxb * 32 + 31 - lane;
    const double* base = vol + (y * W + xr) * D;
    const int64_t left = W - xr;  // d < left lies inside the image (no d where the pixel does not)
    double mn = kRandMax, den = 0.0;
    int d = lane % D;
#pragma unroll 8
    for (int k = 0; k < D; k++) {
      mn = fmin(mn, d < left ? __ldg(base + (int64_t)d * (D + 1)) : fill);
      if (++d == D) d = 0;
    }
    // D steps on, d is where it began
#pragma unroll 4
    for (int k = 0; k < D; k++) {
      den += lik_exp((d < left ? __ldg(base + (int64_t)d * (D + 1)) : fill) - mn, m);
      if (++d == D) d = 0;
    }
    if (left > 0) *reinterpret_cast<double2*>(stats + ((int64_t)(2 * m + 1) * H * W + y * W + xr) * 2) = make_double2(mn, den);
  }
}

// One thread per (pixel, d), its 20 features as five 16-byte stores (VEC)
// where `out` allows them; I: the type the sample index is divided in.
template <class I, bool VEC>
__global__ void __launch_bounds__(kBlock) features_kernel(FeatVols fv, const double* __restrict__ stats, int64_t H,
                                                          int64_t W, int D, float* __restrict__ out) {
  const int64_t HW = H * W;
  GRID_STRIDE(t, HW * D) {
    const I p = (I)t / (I)D;
    float f[20];
    features_at(fv.v, stats, HW, W, D, (int64_t)p, (int64_t)(p % (I)W), (int)((I)t - p * (I)D), f);
    if (VEC) {
      float4* o = reinterpret_cast<float4*>(out + t * 20);
#pragma unroll
      for (int k = 0; k < 5; k++) o[k] = make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]);
    } else {
#pragma unroll
      for (int k = 0; k < 20; k++) out[t * 20 + k] = f[k];
    }
  }
}

__global__ void features_gather_kernel(FeatVols fv, const double* __restrict__ stats, int64_t H,
                                       int64_t W, int D, const int64_t* __restrict__ idx, int64_t n,
                                       float* __restrict__ out) {
  const int64_t HW = H * W, N = HW * D;
  GRID_STRIDE(i, n) {
    int64_t t = idx[i];
    t = t < 0 ? 0 : (t >= N ? N - 1 : t);  // indices are validated on the host; clamp anyway
    const int64_t p = t / D;
    const int d = (int)(t - p * D);
    features_store(fv.v, stats, HW, D, p, p % W, d, out + i * 20, 1);
  }
}

// The features of n chosen (p, d) with the statistics of their own rows only:
// a CTA takes eight (sample, matcher) pairs.  The left row is a warp's, as in
// stats_left_kernel; the right view's diagonal is read into shared memory, its
// exponentials are formed there by the warp and added by one thread per pair,
// from the disparity at which stats_right_kernel's lane begins, so every sum
// has its order.  Bound by the diagonals' sectors (8 of 32 bytes used) and the
// FP64 exponentials: 694x554 D=128, 100,000 samples 987 us against 1430 with
// the statistics of every pixel (32 pairs per CTA: 1409).
constexpr int kGatherThreads = 64, kGatherPairs = 8;  // small CTAs, so that some sum while others read
constexpr int kGatherBytes = kGatherPairs * 1025 * 8;  // of diagonals at D = 1024

__global__ void __launch_bounds__(kGatherThreads) features_gather_rows_kernel(FeatVols fv, int64_t H, int64_t W, int D,
                                                                              const int64_t* __restrict__ idx, int64_t n,
                                                                              float* __restrict__ out) {
  extern __shared__ double diag[];  // [kGatherPairs][D + 1]
  __shared__ double s_mn[kGatherPairs], s_den[kGatherPairs], s_rmn[kGatherPairs];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t N = H * W * D, pairs = 4 * n;
  for (int64_t q0 = (int64_t)blockIdx.x * kGatherPairs; q0 < pairs; q0 += (int64_t)gridDim.x * kGatherPairs) {
    const int count = (int)min((int64_t)kGatherPairs, pairs - q0);
    for (int c = warp; c < count; c += kGatherThreads / 32) {
      const int m = (int)((q0 + c) & 3);
      int64_t t = idx[(q0 + c) >> 2];
      t = t < 0 ? 0 : (t >= N ? N - 1 : t);  // indices are validated on the host; clamp anyway
      const int64_t p = t / D, y = p / W, x = p - y * W;
      const int d = (int)(t - p * D);
      const double* __restrict__ vol = fv.v[m];
      const double* r = vol + p * D;
      const bool both = x >= d;  // else the right view's confidences are 0
      const int64_t left = both ? W - x + d : 0;
      const double fill = __ldg(vol);
      const double* base = vol + (p - d) * D;  // right pixel x - d
      double* row = diag + c * (D + 1);
      double mn = kRandMax, den = 0.0, rmn = kRandMax;
#pragma unroll 4
      for (int k = lane; k < D; k += 32) {
        const double a = __ldg(r + k), b = k < left ? __ldg(base + (int64_t)k * (D + 1)) : fill;
        row[k] = b;
        mn = fmin(mn, a);
        rmn = fmin(rmn, b);
      }
      for (int o = 16; o; o >>= 1) {
        mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        rmn = fmin(rmn, __shfl_xor_sync(0xffffffffu, rmn, o));
      }
#pragma unroll 2
      for (int k = lane; k < D; k += 32) {
        den += lik_exp(__ldg(r + k) - mn, m);
        if (both) row[k] = lik_exp(row[k] - rmn, m);
      }
      den = warp_sum(den);
      if (lane == 0) s_mn[c] = mn, s_den[c] = den, s_rmn[c] = rmn;
    }
    __syncthreads();
    if (threadIdx.x < count) {
      const int c = threadIdx.x, m = (int)((q0 + c) & 3);
      const int64_t i = (q0 + c) >> 2;
      int64_t t = idx[i];
      t = t < 0 ? 0 : (t >= N ? N - 1 : t);
      const int64_t p = t / D, x = p % W;
      const int d = (int)(t - p * D);
      const double v = __ldg(fv.v[m] + t);
      float* f = out + i * 20 + m;
      f[0] = (float)v;
      confidences(v, s_mn[c], s_den[c], m, f + 4, f + 8);
      f[12] = f[16] = 0.0f;
      if (x >= d) {
        const double* row = diag + c * (D + 1);
        const int first = (int)(31 - (x - d) % 32) % D;
        double den = 0.0;
#pragma unroll 8
        for (int k = first; k < D; k++) den += row[k];
#pragma unroll 8
        for (int k = 0; k < first; k++) den += row[k];
        confidences(v, s_rmn[c], den, m, f + 12, f + 16);
      }
    }
    __syncthreads();
  }
}

// Up to a third of the pixels: the whole call at 694x554 D=128 with 0.001,
// 0.26, 0.40 and 0.49 samples per pixel takes 743, 1725, 2199 and 2507 us by their own
// rows, 2186 by the whole image's statistics; 1000x600 D=70 1768, 2245 and
// 2559 against 2366.
bool features_gather_rows(int64_t H, int64_t W, int64_t n) { return 3 * n <= H * W; }

// stats null: each sample's rows' own
int launch_features_gather(const double* const* vols, const double* stats, int64_t H, int64_t W,
                           int D, const int64_t* idx, int64_t n, float* out, cudaStream_t st) {
  FeatVols fv = {{vols[0], vols[1], vols[2], vols[3]}};
  if (!stats) {
    const size_t smem = (size_t)kGatherPairs * (D + 1) * sizeof(double);
    CBMV_CUDA(cudaFuncSetAttribute(features_gather_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGatherBytes));
    features_gather_rows_kernel<<<grid_for(4 * n, kGatherPairs), kGatherThreads, smem, st>>>(fv, H, W, D, idx, n, out);
  } else {
    features_gather_kernel<<<grid_for(n, kBlock), kBlock, 0, st>>>(fv, stats, H, W, D, idx, n, out);
  }
  return check_launch("features_gather");
}

// ---------------------------------------------- float32 row statistics
// The classifier network's row statistics (min, 1/den) in float32 from
// float32 volumes (the learned path never needs the float64 features):
// statsf[(m*2 + view)*HW + p], min = -e and 1/den = 0 where the row holds
// only sentinels.  All four matchers in one launch (blockIdx.y = matcher).
struct VolsF {
  const float* v[4];
};
static __constant__ float kInvSigmaF32[4] = {(float)(1.0 / (2.0 * 8 * 8)), (float)(1.0 / 0.02),
                                             (float)(1.0 / (2.0 * 100 * 100)), (float)(1.0 / (2.0 * 100 * 100))};

// of matcher m; a row of sentinels has min = -e, so that its ratio (min + e) / (c + e) is 0, and 1/den = 0
__device__ __forceinline__ float2 stats_pair(int m, float mn, float den) {
  return mn == kRandMaxF ? make_float2(-kEpsF[m], 0.0f) : make_float2(mn, 1.0f / den);
}

// view 0: one warp per pixel, the pixel's D costs are contiguous (rows too long
// for a warp's registers, and volumes that no vector load may take)
__global__ void stats_f32_left_kernel(VolsF vols, int64_t HW, int D, float2* __restrict__ statsf) {
  const int m = blockIdx.y;
  const float* __restrict__ vol = vols.v[m];
  const float inv_sigma = kInvSigmaF32[m];
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < HW; p += nw) {
    const float* r = vol + p * D;
    float mn = kRandMaxF, den = 0.0f;
    for (int d = lane; d < D; d += 32) mn = fminf(mn, __ldg(r + d));
    for (int o = 16; o; o >>= 1) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    for (int d = lane; d < D; d += 32) {
      const float t = __ldg(r + d) - mn;
      den += __expf(-(t * t) * inv_sigma);
    }
    for (int o = 16; o; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
    if (lane == 0) statsf[(int64_t)(m * 2) * HW + p] = stats_pair(m, mn, den);
  }
}

// view 0 for rows that a warp holds in registers: K vectors of V costs per
// lane, PX pixels at a time, so that their loads are in flight together; the
// minimum is a `redux`, and the sums of PX pixels are exchanged in one tree
// whose additions are those of stats_f32_left_kernel.  Bound by memory:
// 451x319 D=70 74 us (142 with one pixel per warp, its row read twice),
// 1482x994 D=256 1043 (1464).
template <int V, int K>
__global__ void __launch_bounds__(256) stats_f32_left_r_kernel(VolsF vols, int64_t HW, int D,
                                                               float2* __restrict__ statsf) {
  constexpr int PX = V * K <= 4 ? 4 : V * K <= 8 ? 2 : 1;
  const int m = blockIdx.y;
  const float* __restrict__ vol = vols.v[m];
  const float inv_sigma = kInvSigmaF32[m];
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t p0 = PX * (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); p0 < HW; p0 += PX * nw) {
    float v[PX][K][V], mn[PX], den[PX];
#pragma unroll
    for (int i = 0; i < PX; i++) {
      const float* r = vol + (p0 + i < HW ? p0 + i : p0) * D;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int d = V * (lane + 32 * k);
        if constexpr (V == 4) {
          const float4 q = d < D ? __ldg(reinterpret_cast<const float4*>(r + d))
                                 : make_float4(kRandMaxF, kRandMaxF, kRandMaxF, kRandMaxF);
          v[i][k][0] = q.x, v[i][k][1] = q.y, v[i][k][2] = q.z, v[i][k][3] = q.w;
        } else {
          v[i][k][0] = d < D ? __ldg(r + d) : kRandMaxF;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < PX; i++) {
      mn[i] = kRandMaxF;
#pragma unroll
      for (int k = 0; k < K; k++)
#pragma unroll
        for (int j = 0; j < V; j++) mn[i] = fminf(mn[i], v[i][k][j]);
      asm volatile("redux.sync.min.f32 %0, %0, 0xffffffff;" : "+f"(mn[i]));
      den[i] = 0.0f;
#pragma unroll
      for (int k = 0; k < K; k++) {
        if (V * (lane + 32 * k) < D) {
          float e[V];
#pragma unroll
          for (int j = 0; j < V; j++) {
            const float t = v[i][k][j] - mn[i];
            e[j] = __expf(-(t * t) * inv_sigma);
          }
          if constexpr (V == 4) den[i] += (e[0] + e[1]) + (e[2] + e[3]);
          else den[i] += e[0];
        }
      }
    }
    // lane l keeps the sum and minimum of pixel `mine`
    float sum = den[0], low = mn[0];
    int mine = 0, o = 16;
    if constexpr (PX == 4) {
      const bool up = lane & 16;
      const float a = (up ? den[2] : den[0]) + __shfl_xor_sync(0xffffffffu, up ? den[0] : den[2], 16);
      const float b = (up ? den[3] : den[1]) + __shfl_xor_sync(0xffffffffu, up ? den[1] : den[3], 16);
      const bool odd = lane & 8;
      sum = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
      mine = (up ? 2 : 0) + (odd ? 1 : 0);
      low = up ? (odd ? mn[3] : mn[2]) : (odd ? mn[1] : mn[0]);
      o = 4;
    } else if constexpr (PX == 2) {
      const bool up = lane & 16;
      sum = (up ? den[1] : den[0]) + __shfl_xor_sync(0xffffffffu, up ? den[0] : den[1], 16);
      mine = up ? 1 : 0;
      low = up ? mn[1] : mn[0];
      o = 8;
    }
    constexpr int kLanes = 32 / PX;
    for (; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane % kLanes == 0 && p0 + mine < HW) statsf[(int64_t)(m * 2) * HW + p0 + mine] = stats_pair(m, low, sum);
  }
}

// view 1: right pixel x' of row y sees C[y, x' + d, d] (the fill C[0,0,0]
// where x' + d >= W, featextract.cpp:115-152).  A CTA owns RS_PIX right
// pixels of one row; for each 32-wide disparity chunk it stages the
// (RS_PIX + 32) x 32 block of the volume the chunk's diagonals cross
// (coalesced along d) and each thread walks its diagonal in shared memory.
constexpr int RS_PIX = 256;

__global__ void __launch_bounds__(RS_PIX) stats_f32_right_kernel(VolsF vols, int64_t H, int64_t W, int D,
                                                                 float2* __restrict__ statsf) {
  __shared__ float tile[(RS_PIX + 32) * 33];
  const int m = blockIdx.y;
  const float* __restrict__ vol = vols.v[m];
  const float fill = __ldg(vol);
  const float inv_sigma = kInvSigmaF32[m];
  const int64_t nxb = (W + RS_PIX - 1) / RS_PIX;
  const int64_t y = blockIdx.x / nxb;
  const int64_t X0 = (blockIdx.x % nxb) * RS_PIX;
  const int tid = threadIdx.x;
  const int64_t xr = X0 + tid;
  float mn = kRandMaxF, den = 0.0f;
  for (int pass = 0; pass < 2; pass++) {
    for (int d0 = 0; d0 < D; d0 += 32) {
      __syncthreads();
      const int j = tid & 31, last = d0 + j < D ? (int)min(W - X0 - d0, (int64_t)RS_PIX + 32) : 0;
      const float* src = vol + (y * W + X0 + d0 + (tid >> 5)) * D + d0 + j;
#pragma unroll 9
      for (int i = tid >> 5; i < RS_PIX + 32; i += RS_PIX / 32, src += (RS_PIX / 32) * (int64_t)D)
        tile[i * 33 + j] = i < last ? __ldg(src) : fill;
      __syncthreads();
      if (xr < W) {
        const int nj = D - d0 < 32 ? D - d0 : 32;
        if (pass == 0) {
          for (int j = 0; j < nj; j++) mn = fminf(mn, tile[(tid + j) * 33 + j]);
        } else {
          for (int j = 0; j < nj; j++) {
            const float t = tile[(tid + j) * 33 + j] - mn;
            den += __expf(-(t * t) * inv_sigma);
          }
        }
      }
    }
  }
  if (xr < W) statsf[(int64_t)(m * 2 + 1) * H * W + y * W + xr] = stats_pair(m, mn, den);
}

// view 0 for D a multiple of 4 up to 128: a pixel's row is one float4 per
// lane, the minimum one `redux.sync.min.f32`, and each warp works on two
// pixels at a time; the per-lane sum and the shuffle tree are those of
// stats_f32_left_kernel, so the results are the same bit for bit.
__global__ void __launch_bounds__(256) stats_f32_left_q_kernel(VolsF vols, int64_t HW, int D,
                                                               float2* __restrict__ statsf) {
  const int m = blockIdx.y;
  const float inv_sigma = kInvSigmaF32[m];
  const int lane = threadIdx.x & 31;
  const int nq = D >> 2;  // float4s per row, <= 32
  const bool on = lane < nq;
  const float4* __restrict__ rows = reinterpret_cast<const float4*>(vols.v[m]) + lane;
  float2* __restrict__ out = statsf + (int64_t)(m * 2) * HW;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  const float4 big = make_float4(kRandMaxF, kRandMaxF, kRandMaxF, kRandMaxF);
  auto den4 = [&](float4 v, float mn) {
    const float tx = v.x - mn, ty = v.y - mn, tz = v.z - mn, tw = v.w - mn;
    return (__expf(-(tx * tx) * inv_sigma) + __expf(-(ty * ty) * inv_sigma)) +
           (__expf(-(tz * tz) * inv_sigma) + __expf(-(tw * tw) * inv_sigma));
  };
  for (int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < HW; p += 2 * nw) {
    const int64_t p2 = p + nw;
    const bool two = p2 < HW;
    const float4 va = on ? __ldg(rows + p * nq) : big;
    const float4 vb = on && two ? __ldg(rows + p2 * nq) : big;
    float ma = fminf(fminf(va.x, va.y), fminf(va.z, va.w));
    float mb = fminf(fminf(vb.x, vb.y), fminf(vb.z, vb.w));
    asm volatile("redux.sync.min.f32 %0, %0, 0xffffffff;" : "+f"(ma));
    asm volatile("redux.sync.min.f32 %0, %0, 0xffffffff;" : "+f"(mb));
    float da = on ? den4(va, ma) : 0.0f, db = on ? den4(vb, mb) : 0.0f;
    for (int o = 16; o; o >>= 1) {
      da += __shfl_xor_sync(0xffffffffu, da, o);
      db += __shfl_xor_sync(0xffffffffu, db, o);
    }
    if (lane == 0) out[p] = stats_pair(m, ma, da);
    if (lane == 1 && two) out[p2] = stats_pair(m, mb, db);
  }
}

// view 0 for D = 128 exactly (the headline's disparity count): eight lanes
// per pixel, four pixels per warp at a time, each lane four float4 of its
// pixel's row; the minimum and the denominator reduce over the eight lanes
// in three shuffle steps.  (Its denominator adds in another order than
// stats_f32_left_q_kernel: the same value to float32 rounding.)
__global__ void __launch_bounds__(256) stats_f32_left_g8_kernel(VolsF vols, int64_t HW,
                                                                float2* __restrict__ statsf) {
  const int m = blockIdx.y;
  const float inv_sigma = kInvSigmaF32[m];
  const int lane = threadIdx.x & 31, gi = lane >> 3, li = lane & 7;
  const float4* __restrict__ rows = reinterpret_cast<const float4*>(vols.v[m]);
  float2* __restrict__ out = statsf + (int64_t)(m * 2) * HW;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t p0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 4; p0 < HW; p0 += 4 * nw) {
    const int64_t p = p0 + gi;
    const bool on = p < HW;
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      v[k] = on ? __ldg(rows + p * 32 + li + 8 * k) : make_float4(kRandMaxF, kRandMaxF, kRandMaxF, kRandMaxF);
    float mn = kRandMaxF;
#pragma unroll
    for (int k = 0; k < 4; k++) mn = fminf(mn, fminf(fminf(v[k].x, v[k].y), fminf(v[k].z, v[k].w)));
#pragma unroll
    for (int o = 4; o; o >>= 1) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    float den = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float tx = v[k].x - mn, ty = v[k].y - mn, tz = v[k].z - mn, tw = v[k].w - mn;
      den += (__expf(-(tx * tx) * inv_sigma) + __expf(-(ty * ty) * inv_sigma)) +
             (__expf(-(tz * tz) * inv_sigma) + __expf(-(tw * tw) * inv_sigma));
    }
#pragma unroll
    for (int o = 4; o; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
    if (li == 0 && on) out[p] = stats_pair(m, mn, den);
  }
}

// view 1 for D a multiple of 4: as stats_f32_right_kernel, the staging
// loads one float4 (4 disparities) per thread and step with 32-bit row
// offsets; the diagonal walk, and so the order of the sums, is unchanged.
__global__ void __launch_bounds__(RS_PIX) stats_f32_right_q_kernel(VolsF vols, int64_t H, int64_t W, int D,
                                                                   float2* __restrict__ statsf) {
  __shared__ float tile[(RS_PIX + 32) * 33];
  const int m = blockIdx.y;
  const float* __restrict__ vol = vols.v[m];
  const float fill = __ldg(vol);
  const float inv_sigma = kInvSigmaF32[m];
  const int64_t nxb = (W + RS_PIX - 1) / RS_PIX;
  const int64_t y = blockIdx.x / nxb;
  const int X0 = (int)((blockIdx.x % nxb) * RS_PIX);
  const int Wi = (int)W;
  const float* __restrict__ rowp = vol + y * W * D;  // C[y, 0, 0]
  const int tid = threadIdx.x;
  const int xr = X0 + tid;
  float mn = kRandMaxF, den = 0.0f;
  for (int pass = 0; pass < 2; pass++) {
    for (int d0 = 0; d0 < D; d0 += 32) {
      __syncthreads();
#pragma unroll
      for (int it = 0; it < (RS_PIX + 32) * 8 / RS_PIX; it++) {
        const int q = tid + it * RS_PIX;
        const int i = q >> 3, j4 = (q & 7) * 4;
        const int x = X0 + d0 + i;
        float4 v = make_float4(fill, fill, fill, fill);
        if (x < Wi && d0 + j4 < D) v = __ldg(reinterpret_cast<const float4*>(rowp + (int64_t)x * D + d0 + j4));
        float* t = tile + i * 33 + j4;
        t[0] = v.x;
        t[1] = v.y;
        t[2] = v.z;
        t[3] = v.w;
      }
      __syncthreads();
      if (xr < Wi) {
        const int nj = D - d0 < 32 ? D - d0 : 32;
        if (pass == 0) {
          for (int j = 0; j < nj; j++) mn = fminf(mn, tile[(tid + j) * 33 + j]);
        } else {
          for (int j = 0; j < nj; j++) {
            const float t = tile[(tid + j) * 33 + j] - mn;
            den += __expf(-(t * t) * inv_sigma);
          }
        }
      }
    }
  }
  if (xr < Wi) statsf[(int64_t)(m * 2 + 1) * H * W + y * W + xr] = stats_pair(m, mn, den);
}

template <int V, int K>
static void launch_stats_left_r(const VolsF& v, int64_t HW, int D, float2* statsf, cudaStream_t st) {
  const int64_t blocks = (HW + 15) / 16;  // 8 warps per block, two pixels each (a warp of fewer or more strides)
  stats_f32_left_r_kernel<V, K><<<dim3((unsigned)(blocks < 65535 * 16 ? blocks : 65535 * 16), 4), 256, 0, st>>>(v, HW, D, statsf);
}

int launch_feature_stats_f32(const float* const* vols, int64_t H, int64_t W, int D, float2* statsf,
                             cudaStream_t st) {
  const VolsF v = {{vols[0], vols[1], vols[2], vols[3]}};
  const int64_t HW = H * W;
  const int64_t lblocks = (HW + 7) / 8;  // 8 warps per block, one pixel each
  const bool q = D % 4 == 0 && ((uintptr_t)vols[0] | (uintptr_t)vols[1] | (uintptr_t)vols[2] | (uintptr_t)vols[3]) % 16 == 0;
  if (q && D == 128) {
    const int64_t gblocks = (HW + 31) / 32;  // 8 warps per block, four pixels each
    stats_f32_left_g8_kernel<<<dim3((unsigned)(gblocks < 65535 * 16 ? gblocks : 65535 * 16), 4), 256, 0, st>>>(
        v, HW, statsf);
  } else if (q && D <= 128) {
    const int64_t qblocks = (HW + 15) / 16;  // 8 warps per block, two pixels each
    stats_f32_left_q_kernel<<<dim3((unsigned)(qblocks < 65535 * 16 ? qblocks : 65535 * 16), 4), 256, 0, st>>>(
        v, HW, D, statsf);
  } else if (q && D <= 512) {
    if (D <= 256) launch_stats_left_r<4, 2>(v, HW, D, statsf, st);
    else if (D <= 384) launch_stats_left_r<4, 3>(v, HW, D, statsf, st);
    else launch_stats_left_r<4, 4>(v, HW, D, statsf, st);
  } else if (D % 4 != 0 && D <= 256) {
#define LEFT_R(K) case K: launch_stats_left_r<1, K>(v, HW, D, statsf, st); break;
    switch ((D + 31) / 32) {
      LEFT_R(1) LEFT_R(2) LEFT_R(3) LEFT_R(4) LEFT_R(5) LEFT_R(6) LEFT_R(7) LEFT_R(8)
    }
#undef LEFT_R
  } else {
    stats_f32_left_kernel<<<dim3((unsigned)(lblocks < 65535 * 16 ? lblocks : 65535 * 16), 4), 256, 0, st>>>(
        v, HW, D, statsf);
  }
  const int64_t rblocks = H * ((W + RS_PIX - 1) / RS_PIX);
  CBMV_REQUIRE(rblocks < ((int64_t)1 << 31), CBMV_ERANGE, "image too large for the statistics grid");
  if (q && W < ((int64_t)1 << 30))
    stats_f32_right_q_kernel<<<dim3((unsigned)rblocks, 4), RS_PIX, 0, st>>>(v, H, W, D, statsf);
  else
    stats_f32_right_kernel<<<dim3((unsigned)rblocks, 4), RS_PIX, 0, st>>>(v, H, W, D, statsf);
  return check_launch("feature_stats_f32");
}

int launch_feature_stats(const double* const* vols, int64_t H, int64_t W, int D, double* stats, cudaStream_t st) {
  const VolsD v = {{vols[0], vols[1], vols[2], vols[3]}};
  const int64_t HW = H * W;
  const dim3 grid(grid_for(HW * 32, kBlock), 4);
  if (D <= 128) stats_left_kernel<4><<<grid, kBlock, 0, st>>>(v, HW, D, stats);
  else if (D <= 256) stats_left_kernel<8><<<grid, kBlock, 0, st>>>(v, HW, D, stats);
  else stats_left_kernel<0><<<grid, kBlock, 0, st>>>(v, HW, D, stats);
  stats_right_kernel<<<dim3(grid_for(H * ((W + 31) / 32) * 32, kBlock), 4), kBlock, 0, st>>>(v, H, W, D, stats);
  return check_launch("feature_stats");
}

}  // namespace cbmv

using namespace cbmv;

#define CHECK_VOL(p, q) CBMV_REQUIRE((p) && (q), CBMV_EINVAL, "null pointer argument")

extern "C" int cbmv_swap_axes(const double* in, int64_t D, int64_t H, int64_t W, double* out,
                              void* stream) {
  CHECK_VOL(in, out);
  CBMV_REQUIRE(D > 0 && H > 0 && W > 0, CBMV_EINVAL, "bad size");
  return launch_swap_axes(in, D, H * W, out, as_stream(stream));
}

extern "C" int cbmv_swap_axes_back(const double* in, int64_t H, int64_t W, int64_t D, double* out,
                                   void* stream) {
  CHECK_VOL(in, out);
  CBMV_REQUIRE(D > 0 && H > 0 && W > 0, CBMV_EINVAL, "bad size");
  return launch_swap_axes_back(in, H * W, D, out, as_stream(stream));
}

extern "C" int cbmv_get_cost(const double* in, int64_t H, int64_t W, int64_t D, int64_t K,
                             double* out, void* stream) {
  CHECK_VOL(in, out);
  CBMV_REQUIRE(D > 0 && H > 0 && W > 0 && K > 0, CBMV_EINVAL, "bad size");
  get_cost_kernel<<<grid_for(H * W * D, kBlock), kBlock, 0, as_stream(stream)>>>(in, H * W * D, K, out);
  return check_launch("get_cost");
}

extern "C" int cbmv_get_right_cost(const double* C, int64_t H, int64_t W, int64_t D, double* out,
                                   void* stream) {
  CHECK_VOL(C, out);
  CBMV_REQUIRE(D > 0 && H > 0 && W > 0 && C != out, CBMV_EINVAL, "bad size or in-place call");
  shift_kernel<<<grid_for(H * W * D, kBlock), kBlock, 0, as_stream(stream)>>>(C, H, W, D, 1, out);
  return check_launch("get_right_cost");
}

extern "C" int cbmv_get_left_cost(const double* Rv, int64_t H, int64_t W, int64_t D, double* out,
                                  void* stream) {
  CHECK_VOL(Rv, out);
  CBMV_REQUIRE(D > 0 && H > 0 && W > 0 && Rv != out, CBMV_EINVAL, "bad size or in-place call");
  shift_kernel<<<grid_for(H * W * D, kBlock), kBlock, 0, as_stream(stream)>>>(Rv, H, W, D, -1, out);
  return check_launch("get_left_cost");
}

extern "C" int cbmv_extract_ratio(const double* vol, int64_t N, int64_t D, double e, double* out,
                                  void* stream) {
  CHECK_VOL(vol, out);
  CBMV_REQUIRE(N > 0 && D > 0, CBMV_EINVAL, "bad size");
  ratio_kernel<<<grid_for(N * 32, kBlock), kBlock, 0, as_stream(stream)>>>(vol, N, D, e, out);
  return check_launch("extract_ratio");
}

extern "C" int cbmv_extract_likelihood(const double* vol, int64_t N, int64_t D, double sigma,
                                       double* out, void* stream) {
  CHECK_VOL(vol, out);
  CBMV_REQUIRE(N > 0 && D > 0 && sigma > 0, CBMV_EINVAL, "bad size or sigma");
  likelihood_kernel<<<grid_for(N * 32, kBlock), kBlock, 0, as_stream(stream)>>>(vol, N, D, sigma, out);
  return check_launch("extract_likelihood");
}

extern "C" int cbmv_extract_ratio_samples(const double* vol, int64_t N, int64_t D,
                                          const int32_t* samples, double e, double* out,
                                          void* stream) {
  CHECK_VOL(vol, out);
  CBMV_REQUIRE(samples && N > 0 && D > 0, CBMV_EINVAL, "bad argument");
  ratio_samples_kernel<<<grid_for(N * 32, kBlock), kBlock, 0, as_stream(stream)>>>(vol, N, D, samples,
                                                                                  e, out);
  return check_launch("extract_ratio_samples");
}

extern "C" int cbmv_extract_likelihood_samples(const double* vol, int64_t N, int64_t D,
                                               const int32_t* samples, double sigma, double* out,
                                               void* stream) {
  CHECK_VOL(vol, out);
  CBMV_REQUIRE(samples && N > 0 && D > 0 && sigma > 0, CBMV_EINVAL, "bad argument");
  likelihood_samples_kernel<<<grid_for(N * 32, kBlock), kBlock, 0, as_stream(stream)>>>(
      vol, N, D, samples, sigma, out);
  return check_launch("extract_likelihood_samples");
}

extern "C" int cbmv_get_samples(const double* vol, int64_t N, int64_t D, const int32_t* samples,
                                double* out, void* stream) {
  CHECK_VOL(vol, out);
  CBMV_REQUIRE(samples && N > 0 && D > 0, CBMV_EINVAL, "bad argument");
  get_samples_kernel<<<grid_for(3 * N, kBlock), kBlock, 0, as_stream(stream)>>>(vol, N, D, samples, out);
  return check_launch("get_samples");
}

extern "C" int cbmv_generate_labels(int64_t N, int32_t* out, void* stream) {
  CBMV_REQUIRE(out && N > 0, CBMV_EINVAL, "bad argument");
  labels_kernel<<<grid_for(3 * N, kBlock), kBlock, 0, as_stream(stream)>>>(N, out);
  return check_launch("generate_labels");
}

extern "C" int cbmv_generate_d_indices(const int32_t* gt, int64_t N, int maxd, int thr,
                                       uint64_t seed, int32_t* out, void* stream) {
  CBMV_REQUIRE(gt && out && N > 0 && maxd > 0 && thr >= 0, CBMV_EINVAL, "bad argument");
  cudaStream_t st = as_stream(stream);
  int* bad = nullptr;
  CBMV_CUDA(cudaMallocAsync(&bad, sizeof(int), st));
  CBMV_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), st));
  d_indices_kernel<<<grid_for(N, kBlock), kBlock, 0, st>>>(gt, N, maxd, thr, seed, out, bad);
  int rc = check_launch("generate_d_indices");
  int hbad = 0;
  CBMV_CUDA(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, st));
  CBMV_CUDA(cudaFreeAsync(bad, st));
  CBMV_CUDA(cudaStreamSynchronize(st));
  if (rc) return rc;
  CBMV_REQUIRE(!hbad, CBMV_EINVAL,
               "generate_d_indices: a ground-truth value is outside [0, maxd] or leaves an empty "
               "negative range (gt = maxd - thr - 1)");
  return CBMV_OK;
}

extern "C" int cbmv_features(const double* census, const double* ncc, const double* sob,
                             const double* sad, int64_t H, int64_t W, int D, float* out,
                             void* stream) {
  CBMV_REQUIRE(census && ncc && sob && sad && out, CBMV_EINVAL, "null pointer argument");
  CBMV_REQUIRE(H > 0 && W > 0 && D > 0, CBMV_EINVAL, "bad size");
  cudaStream_t st = as_stream(stream);
  double* stats = nullptr;
  CBMV_CUDA(cudaMallocAsync(&stats, sizeof(double) * 16 * H * W, st));
  const double* vols[4] = {census, ncc, sob, sad};
  int rc = launch_feature_stats(vols, H, W, D, stats, st);
  if (!rc) {
    FeatVols fv = {{census, ncc, sob, sad}};
    const unsigned grid = grid_for(H * W * D, kBlock);
    const bool vec = ((uintptr_t)out & 15) == 0, small = H * W * D < ((int64_t)1 << 32);
    if (small && vec) features_kernel<uint32_t, true><<<grid, kBlock, 0, st>>>(fv, stats, H, W, D, out);
    else if (small) features_kernel<uint32_t, false><<<grid, kBlock, 0, st>>>(fv, stats, H, W, D, out);
    else if (vec) features_kernel<int64_t, true><<<grid, kBlock, 0, st>>>(fv, stats, H, W, D, out);
    else features_kernel<int64_t, false><<<grid, kBlock, 0, st>>>(fv, stats, H, W, D, out);
    rc = check_launch("features");
  }
  CBMV_CUDA(cudaFreeAsync(stats, st));
  return rc;
}
