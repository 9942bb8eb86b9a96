// MC-CNN cost optimisation ("post", cpp/post/post.cu), float32 on the device.
//
// The reference keeps its volumes in float64 and does most arithmetic in
// float32; these kernels keep the volumes in float32 and do the same float32
// arithmetic as the reference kernels (comparisons, arm bounds, transition
// penalties, CBCA summation order, subpixel parabola, median, thresholded
// Gaussian).  Where the reference accumulates in float64 (the SGM path
// values and their sum over the four directions) the sums here are float32.
//
// SGM runs all four scan directions in one launch with one warp per scan line
// and the scan inside the kernel (the reference launches one kernel per scan
// step, 2(W+H) launches per call, post.cu:273-330); the lanes hold the path
// values in registers, the minimum over d is a warp reduction, and the next
// steps' costs are loaded ahead.
#include "common.cuh"
#include "post.cuh"

namespace cbmv {
namespace {

constexpr int kBlock = 128;

#define GRID_STRIDE(i, n) \
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

__device__ __forceinline__ void decode(int layout, int64_t t, int64_t H, int64_t W, int64_t D,
                                       int64_t* y, int64_t* x, int64_t* d) {
  if (layout == CBMV_HWD) {
    *d = t % D;
    const int64_t p = t / D;
    *x = p % W;
    *y = p / W;
  } else {
    *x = t % W;
    const int64_t q = t / W;
    *y = q % H;
    *d = q / H;
  }
}

// cross (post.cu:336-396)
__global__ void cross_kernel(const float* __restrict__ x0, int64_t H, int64_t W, int L1, float tau1,
                             float* __restrict__ out) {
  GRID_STRIDE(id, 4 * H * W) {
    const int64_t x = id % W, y = (id / W) % H;
    const int dir = (int)(id / (W * H));
    const int dx = dir == 0 ? -1 : dir == 1 ? 1 : 0;
    const int dy = dir == 2 ? -1 : dir == 3 ? 1 : 0;
    const float c = x0[y * W + x];
    int64_t xx = x + dx, yy = y + dy;
    for (;; xx += dx, yy += dy) {
      if (xx < 0 || xx >= W || yy < 0 || yy >= H) break;
      const int64_t dist = max(llabs(xx - x), llabs(yy - y));
      if (dist == 1) continue;
      if (fabsf(c - x0[yy * W + xx]) >= tau1) break;  // rule 1
      if (dist >= L1) break;                          // rule 2
    }
    out[id] = (float)(dir <= 1 ? xx : yy);
  }
}

// SGM's image terms (post.cu:230-248).  A step's penalties depend only on
// whether the left difference D1 and the right difference D2 of the scan
// direction's neighbouring pixels lie below or above tau_so, so the scan
// reads two bits per pixel, {D < tau, D > tau}, packed along the scan: 32
// pixels of a row for the horizontal directions, 32 rows of a column for the
// vertical ones (|a - b| == |b - a| in IEEE arithmetic: one difference per
// pair of neighbours serves both directions along it).  Where a right
// difference leaves the image D2 = 10.  A warp takes a 32 x 32 tile.
__global__ void __launch_bounds__(128) sgm_codes_kernel(const float* __restrict__ imL, const float* __restrict__ imR,
                                                      int H, int W, float tau, SgmCodes g) {
  const int lane = threadIdx.x & 31, gw = (W + 31) / 32, gh = (H + 31) / 32;
  const int64_t n = (int64_t)gridDim.x * 4;
  for (int64_t u = ((int64_t)blockIdx.x * 128 + threadIdx.x) >> 5; u < (int64_t)2 * gw * gh; u += n) {
    const bool right = u >= (int64_t)gw * gh;
    const int64_t t = u - (right ? (int64_t)gw * gh : 0);
    const int tw = (int)(t % gw), th = (int)(t / gw), x = 32 * tw + lane;
    const float* im = right ? imR : imL;
    const float none = right ? 10.0f : 0.0f;
    const bool xok = x < W;
    uint2 rows = make_uint2(0u, 0u), cols = make_uint2(0u, 0u);  // row 32 th + lane; column x
    float up = xok && th > 0 ? __ldg(im + ((int64_t)32 * th - 1) * W + x) : 0.0f;
    for (int r = 0; r < 32; r++) {
      const int y = 32 * th + r;
      if (y >= H) break;
      const float v = xok ? __ldg(im + (int64_t)y * W + x) : 0.0f;
      float before = __shfl_up_sync(0xffffffffu, v, 1);
      if (lane == 0 && x > 0) before = __ldg(im + (int64_t)y * W + x - 1);
      const float dh = xok && x > 0 ? fabsf(v - before) : none, dv = xok && y > 0 ? fabsf(v - up) : none;
      up = v;
      const uint32_t lo = __ballot_sync(0xffffffffu, dh < tau), hi = __ballot_sync(0xffffffffu, dh > tau);
      if (lane == r) rows = make_uint2(lo, hi);
      cols.x |= (uint32_t)(dv < tau) << r;
      cols.y |= (uint32_t)(dv > tau) << r;
    }
    if (32 * th + lane < H) (right ? g.right_h : g.left_h)[((int64_t)32 * th + lane) * gw + tw] = rows;
    if (xok) (right ? g.right_v : g.left_v)[(int64_t)th * W + x] = cols;
  }
}

// sgm2 (post.cu:178-261): one scan direction of one line.  A warp scans a
// line, lane l holding the KPL consecutive disparities KPL l .. KPL l + KPL-1
// of the path costs: the d-1 / d+1 neighbours are in the lane's own registers
// except at its two ends (two shuffles), the minimum over d is one
// `redux.sync.min.f32`.  Disparities beyond D hold +inf, which no minimum
// takes.  The four directions (2H + 2W lines) run in one launch through this
// one routine, the direction a run-time argument, each writing its own
// volume.
// A step's costs and classes do not depend on the recursion.  The warp copies
// the cost rows of the next PF steps into a shared-memory ring with
// asynchronous copies: loads into a register ring did not stay in flight
// (the warp's few scoreboards make the wait for the oldest one for the newest
// too).  Rows are copied and stored as VEC consecutive floats per lane, whole
// sectors per instruction, so with KPL != VEC a step's path costs pass
// through shared memory on their way out (two passes over every sector made
// 2.9 ms of 1482x994 D=256 where each lane copied its own 8).  The classes of 32 steps are
// loaded at once and folded into one word per disparity, whose bit says
// whether the pair agrees: with class loads in every step, even ones ahead,
// the scan waited for them (380 to 450 us per launch at 694x554 D=128
// against 240 without any).
// Per launch, us (before: loads in registers, float differences, lanes
// strided by 32 where D % 4 != 0): 694x554 D=128 240 (382), at 5.9 TB/s of
// its 1.42 GB; 451x319 D=70 98 (262); 901x600 D=192 558 (990); 1482x994
// D=256 1923 (2673).  A whole post with two of them, ms: 694x554 D=400 6.7
// (9.9), D=512 7.7 (11.2), D=694 10.7 (17.8), 1482x994 D=400 24.2 (36.6).  A ring of eight steps, blocks of 4 to 16 lines, and a
// cap on registers for more resident lines changed nothing; two steps lose
// 60 us at D=128.
template <int KPL>
constexpr int sgm_depth() { return KPL <= 12 ? 4 : 2; }
// Where float i of a row lies in shared memory: with 32 per lane, lanes would
// begin in one bank, so 4 floats stay free after every 32 (750x554 D=1000, a
// cbmv_sgm call: 7.01 -> 4.12 ms; 6.35 with lanes strided by 32).
template <int KPL>
__host__ __device__ constexpr int sgm_at(int i) { return KPL == 32 ? i + (i >> 5) * 4 : i; }
template <int KPL, int VEC>
constexpr int sgm_words() { return sgm_at<KPL>(32 * ((KPL + VEC - 1) / VEC) * VEC); }

template <int BYTES>
__device__ __forceinline__ void copy_async(uint32_t dst, const void* src, bool on) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(on ? BYTES : 0) : "memory");
}

template <int KPL, bool FULL, int VEC>
__global__ void __launch_bounds__(64) sgm_kernel(SgmCodes g, const float* __restrict__ in, int H, int W, int D,
                                               SgmParams sp, SgmOut o) {
  constexpr int PF = sgm_depth<KPL>(), NV = (KPL + VEC - 1) / VEC, WORDS = sgm_words<KPL, VEC>();
  constexpr bool kStaged = KPL != VEC;  // rows pass through shared memory between lanes
  extern __shared__ __align__(16) float sgm_ring[];
  const int lane = threadIdx.x & 31;
  int line = (int)(((int64_t)blockIdx.x * 64 + threadIdx.x) >> 5), dir;
  if (line < 2 * H) {
    dir = line >= H;
    line -= dir * H;
  } else {
    line -= 2 * H;
    if (line >= 2 * W) return;
    dir = 2 + (line >= W);
    line -= (dir - 2) * W;
  }
  float* __restrict__ out = dir == 0 ? o.dir[0] : dir == 1 ? o.dir[1] : dir == 2 ? o.dir[2] : o.dir[3];
  const float inf = __int_as_float(0x7f800000);
  const bool horizontal = dir <= 1;
  const int nsteps = horizontal ? W : H;
  // penalties of post.cu:239-248; the alpha1 split of :252/:255 applies to
  // the d-1 term in direction 2 and to the d+1 term in direction 3
  const float p1[3] = {sp.pi1, sp.pi1 / (sp.q1 * sp.q2), sp.pi1 / sp.q1};
  const float p2[3] = {sp.pi2, sp.pi2 / (sp.q1 * sp.q2), sp.pi2 / sp.q1};
  float p1lo[3], p1hi[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    p1lo[c] = dir == 2 ? p1[c] / sp.alpha1 : p1[c];
    p1hi[c] = dir == 3 ? p1[c] / sp.alpha1 : p1[c];
  }
  // step t visits pixel p0 + t * pstep; the difference to the step before
  // sits at the later (right or lower) of the two pixels
  const int64_t p0 = dir == 0 ? (int64_t)line * W
                   : dir == 1 ? (int64_t)line * W + W - 1
                   : dir == 2 ? (int64_t)line
                              : (int64_t)(H - 1) * W + line;
  const int64_t pstep = dir == 0 ? 1 : dir == 1 ? -1 : dir == 2 ? (int64_t)W : -(int64_t)W;
  const int s = sp.direction, d0 = KPL * lane;
  const float* lsrc = in + p0 * D + lane * VEC;  // this lane's vectors: floats (v * 32 + lane) * VEC of a row
  const int64_t vstride = pstep * D;
  // the class position of step t (the later, right or lower, pixel of the
  // pair): t forwards, nsteps - t backwards; agree[k] bit c & 31: at position
  // c the classes of disparity d0 + k agree (both below tau or both above),
  // low: the left one is below
  const int forward = dir == 0 || dir == 2 ? 1 : -1;
  int c = forward > 0 ? 1 : nsteps - 1;
  uint32_t agree[KPL], low = 0;
  const int gw = (W + 31) / 32;
  const uint2 outside = make_uint2(10.0f < sp.tau_so ? 0xFFFFFFFFu : 0u, 10.0f > sp.tau_so ? 0xFFFFFFFFu : 0u);
  auto load_classes = [&]() {
    const int group = c >> 5;
    const uint2 l = __ldg(horizontal ? g.left_h + (int64_t)line * gw + group : g.left_v + (int64_t)group * W + line);
    const uint2* __restrict__ row = horizontal ? g.right_h + (int64_t)line * gw : g.right_v + (int64_t)group * W;
#pragma unroll
    for (int k = 0; k < KPL; k++) {
      uint2 q = outside;
      if (horizontal) {
        const int p = 32 * group + (d0 + k) * s, w = p >> 5;  // right pixel of the group's first position
        const uint2 a = (unsigned)w < (unsigned)gw ? __ldg(row + w) : outside;
        const uint2 b = (unsigned)(w + 1) < (unsigned)gw ? __ldg(row + w + 1) : outside;
        q = make_uint2(__funnelshift_r(a.x, b.x, p), __funnelshift_r(a.y, b.y, p));
      } else {
        const int p = line + (d0 + k) * s;
        if ((unsigned)p < (unsigned)W) q = __ldg(row + p);
      }
      agree[k] = (l.x & q.x) | (l.y & q.y);
    }
    low = l.x;
  };
  auto vec_on = [&](int v) { return FULL ? (KPL % VEC == 0 || (v * 32 + lane) * VEC < D) : (v * 32 + lane) * VEC < D; };
  float* ring = sgm_ring + (threadIdx.x >> 5) * (PF + kStaged) * WORDS;
  float* stage = ring + PF * WORDS;
  const uint32_t ring_at = (uint32_t)__cvta_generic_to_shared(ring);
  auto load = [&](int slot) {  // the next step's costs
    const uint32_t at = ring_at + slot * (WORDS * 4);
#pragma unroll
    for (int v = 0; v < NV; v++)  // with VEC > 1, D % VEC == 0: all in or all out
      copy_async<4 * VEC>(at + sgm_at<KPL>((v * 32 + lane) * VEC) * 4, lsrc + v * 32 * VEC, vec_on(v));
    lsrc += vstride;
  };
  float* ldst = out + p0 * D + lane * VEC;
  const int at0 = sgm_at<KPL>(d0);
  // KPL floats between registers and their place in a row in shared memory
  auto get = [&](const float* at, float* f) {
    if constexpr (KPL % 4 == 0) {
#pragma unroll
      for (int k = 0; k < KPL; k += 4) *reinterpret_cast<float4*>(f + k) = *reinterpret_cast<const float4*>(at + at0 + k);
    } else if constexpr (KPL % 2 == 0) {
#pragma unroll
      for (int k = 0; k < KPL; k += 2) *reinterpret_cast<float2*>(f + k) = *reinterpret_cast<const float2*>(at + at0 + k);
    } else {
#pragma unroll
      for (int k = 0; k < KPL; k++) f[k] = at[at0 + k];
    }
  };
  auto put = [&](float* at, const float* f) {
    if constexpr (KPL % 4 == 0) {
#pragma unroll
      for (int k = 0; k < KPL; k += 4) *reinterpret_cast<float4*>(at + at0 + k) = *reinterpret_cast<const float4*>(f + k);
    } else if constexpr (KPL % 2 == 0) {
#pragma unroll
      for (int k = 0; k < KPL; k += 2) *reinterpret_cast<float2*>(at + at0 + k) = *reinterpret_cast<const float2*>(f + k);
    } else {
#pragma unroll
      for (int k = 0; k < KPL; k++) at[at0 + k] = f[k];
    }
  };
  auto store = [&](const float* L) {
    __align__(16) float f[NV * VEC];
    if constexpr (kStaged) {
      put(stage, L);
      __syncwarp();
#pragma unroll
      for (int v = 0; v < NV; v++)
#pragma unroll
        for (int k = 0; k < VEC; k++) f[v * VEC + k] = stage[sgm_at<KPL>((v * 32 + lane) * VEC) + k];
    } else {
#pragma unroll
      for (int k = 0; k < KPL; k++) f[k] = L[k];
    }
#pragma unroll
    for (int v = 0; v < NV; v++)
      if (vec_on(v)) {
        float* to = ldst + v * 32 * VEC;
        if constexpr (VEC == 4) *reinterpret_cast<float4*>(to) = make_float4(f[4 * v], f[4 * v + 1], f[4 * v + 2], f[4 * v + 3]);
        else if constexpr (VEC == 2) *reinterpret_cast<float2*>(to) = make_float2(f[2 * v], f[2 * v + 1]);
        else *to = f[v];
      }
    ldst += vstride;
  };
  float prev[KPL];
#pragma unroll
  for (int k = 0; k < KPL; k++)  // step 0: the path cost is the cost
    prev[k] = FULL || d0 + k < D ? __ldg(in + p0 * D + d0 + k) : inf;
  store(prev);
  lsrc += vstride;
  if (nsteps > 1) load_classes();
#pragma unroll
  for (int i = 0; i < PF; i++) {  // step 1 + i in slot i, one group per step
    if (1 + i < nsteps) load(i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  int slot = 0;
  for (int t = 1; t < nsteps; t++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(PF - 1) : "memory");
    if (kStaged) __syncwarp();  // the row's copies of every lane; the staged row of the step before is out
    __align__(16) float cost[KPL];
    get(ring + slot * WORDS, cost);
    const uint32_t bit = 1u << (c & 31);
    float m = prev[0];
#pragma unroll
    for (int k = 1; k < KPL; k++) m = fminf(m, prev[k]);
    float mn;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(mn) : "f"(m));
    // the neighbours across the lane's ends: d0 - 1 from the previous
    // lane's last register, d0 + KPL from the next lane's first
    float below = __shfl_up_sync(0xffffffffu, prev[KPL - 1], 1), above = __shfl_down_sync(0xffffffffu, prev[0], 1);
    if (lane == 0) below = inf;
    if (lane == 31) above = inf;
    // penalty class 0 (both below tau) or 1 (both above) where the classes agree, else 2
    const bool below_tau = low & bit;
    const float a2 = mn + (below_tau ? p2[0] : p2[1]), c2 = mn + p2[2];
    const float alo = below_tau ? p1lo[0] : p1lo[1], ahi = below_tau ? p1hi[0] : p1hi[1];
    __align__(16) float L[KPL];
#pragma unroll
    for (int k = 0; k < KPL; k++) {
      const bool same = agree[k] & bit;
      const float lo = (k > 0 ? prev[k > 0 ? k - 1 : 0] : below) + (same ? alo : p1lo[2]);
      const float hi = (k + 1 < KPL ? prev[k + 1 < KPL ? k + 1 : 0] : above) + (same ? ahi : p1hi[2]);
      const float best = fminf(fminf(fminf(prev[k], same ? a2 : c2), lo), hi);
      L[k] = FULL || d0 + k < D ? cost[k] + best - mn : inf;
    }
    store(L);
#pragma unroll
    for (int k = 0; k < KPL; k++) prev[k] = L[k];
    // every lane has read the slot (its values are in registers): refill it with step t + PF
    if (t + PF < nsteps) load(slot);
    asm volatile("cp.async.commit_group;" ::: "memory");
    slot = slot + 1 == PF ? 0 : slot + 1;
    c += forward;
    if ((c & 31) == (forward > 0 ? 0 : 31) && t + 1 < nsteps) load_classes();
  }
}

// out = base + (((L0 + L1) + L2) + L3) * scale over n elements (base may be
// out itself, or null for 0): the four directions summed as post.cu
// sgm_w adds them (directions in order 0..3).  V: float4 (n / 4 of them) or float.
__device__ __forceinline__ float sgm_sum(float a, float b, float c, float d) { return ((a + b) + c) + d; }
__device__ __forceinline__ float4 sgm_sum(float4 a, float4 b, float4 c, float4 d) {
  return make_float4(sgm_sum(a.x, b.x, c.x, d.x), sgm_sum(a.y, b.y, c.y, d.y), sgm_sum(a.z, b.z, c.z, d.z),
                     sgm_sum(a.w, b.w, c.w, d.w));
}
__device__ __forceinline__ float scaled(float s, float k) { return s * k; }
__device__ __forceinline__ float4 scaled(float4 s, float k) { return make_float4(s.x * k, s.y * k, s.z * k, s.w * k); }
__device__ __forceinline__ float added(float b, float s, float k) { return b + s * k; }
__device__ __forceinline__ float4 added(float4 b, float4 s, float k) {
  return make_float4(b.x + s.x * k, b.y + s.y * k, b.z + s.z * k, b.w + s.w * k);
}
template <class V>
__global__ void __launch_bounds__(256) sgm_combine_kernel(const V* __restrict__ l0, const V* __restrict__ l1,
                                                        const V* __restrict__ l2, const V* __restrict__ l3, int64_t n,
                                                        const V* base, float scale, V* out) {
  GRID_STRIDE(i, n) {
    const V s = sgm_sum(l0[i], l1[i], l2[i], l3[i]);
    out[i] = base ? added(base[i], s, scale) : scaled(s, scale);
  }
}

// cbca (post.cu:399-450) of one (y, x, d), any layout: the float sum over the
// support in the reference's order (rows ascending, then columns ascending,
// from 0) divided by its pixels; the input where the match is outside.
__device__ __forceinline__ float cbca_one(const float* __restrict__ lc, const float* __restrict__ rc,
                                          const float* __restrict__ in, int64_t H, int64_t W, int64_t D, int layout,
                                          int direction, int64_t y, int64_t x, int64_t d) {
  const int64_t xm = x + d * direction;
  if (xm < 0 || xm >= W) return in[vol_index(layout, y, x, d, H, W, D)];
  const int yy_s = (int)fmaxf(lc[(2 * H + y) * W + x], rc[(2 * H + y) * W + xm]);
  const int yy_t = (int)fminf(lc[(3 * H + y) * W + x], rc[(3 * H + y) * W + xm]);
  const float dd = (float)(d * direction);
  float sum = 0.0f;
  int cnt = 0;
  for (int yy = yy_s + 1; yy < yy_t; yy++) {
    const int xx_s = (int)fmaxf(lc[(0 * H + yy) * W + x], rc[(0 * H + yy) * W + xm] - dd);
    const int xx_t = (int)fminf(lc[(1 * H + yy) * W + x], rc[(1 * H + yy) * W + xm] - dd);
    for (int xx = xx_s + 1; xx < xx_t; xx++) {
      sum += in[vol_index(layout, yy, xx, d, H, W, D)];
      cnt++;
    }
  }
  return sum / (float)cnt;
}

__global__ void cbca_kernel(const float* __restrict__ lc, const float* __restrict__ rc,
                            const float* __restrict__ in, int64_t H, int64_t W, int64_t D,
                            int layout, int direction, float* __restrict__ out) {
  GRID_STRIDE(id, H * W * D) {
    int64_t y, x, d;
    decode(layout, id, H, W, D, &y, &x, &d);
    out[id] = cbca_one(lc, rc, in, H, W, D, layout, direction, y, x, d);
  }
}

// cbca on [H,W,D] volumes, tiled: a CTA owns CB_TY x CB_TX pixels x 32
// disparities.  Shared memory holds the input tile with a `halo`-pixel
// border (a pixel's support never reaches beyond its cross arms' interior,
// L1 - 1 pixels) and the tile's cross arms as int16: the left arms of the
// tile columns, and the right arms of every column x + d*direction the tile
// matches against.  Lane = disparity, so the running sums read consecutive
// banks.  Each output is the float sum over its support in the reference's
// order (rows ascending, then columns ascending, from 0; post.cu:415-429)
// divided by the count; a support row that reaches outside the staged tile
// (arms longer than the halo) is summed from global memory instead.
constexpr int CB_TX = 16, CB_TY = 16, CB_TD = 32;

__host__ __device__ constexpr int cbca_rw() { return CB_TX + CB_TD - 1; }

__host__ __device__ inline size_t cbca_smem_bytes(int halo) {
  const int SW = CB_TX + 2 * halo, SH = CB_TY + 2 * halo;
  return (size_t)SW * SH * CB_TD * sizeof(float) +
         (size_t)4 * SH * (CB_TX + cbca_rw()) * sizeof(int16_t);
}

__global__ void __launch_bounds__(256) cbca_hwd_tiled_kernel(
    const float* __restrict__ lc, const float* __restrict__ rc, const float* __restrict__ in,
    int H, int W, int D, int direction, int halo, float* __restrict__ out) {
  extern __shared__ float tile[];  // [SH*SW][CB_TD], then int16 arms
  const int SW = CB_TX + 2 * halo, SH = CB_TY + 2 * halo;
  const int RW = cbca_rw();
  int16_t* sl = reinterpret_cast<int16_t*>(tile + (size_t)SW * SH * CB_TD);  // [4][SH][CB_TX]
  int16_t* sr = sl + 4 * SH * CB_TX;                                         // [4][SH][RW]
  const int ntx = (W + CB_TX - 1) / CB_TX, nty = (H + CB_TY - 1) / CB_TY;
  const int ntd = (D + CB_TD - 1) / CB_TD;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int64_t HW = (int64_t)H * W;
  for (int64_t t = blockIdx.x; t < (int64_t)ntx * nty * ntd; t += gridDim.x) {
    const int td = (int)(t % ntd), tx = (int)((t / ntd) % ntx), ty = (int)(t / ((int64_t)ntd * ntx));
    const int X0 = tx * CB_TX, Y0 = ty * CB_TY, d0 = td * CB_TD;
    const int x0 = X0 - halo, y0 = Y0 - halo;
    // first matched column of the tile: x + d*direction over the tile
    const int xr0 = direction < 0 ? X0 - d0 - (CB_TD - 1) : X0 + d0;
    __syncthreads();
    for (int q = warp; q < SW * SH; q += nwarp) {
      const int yy = y0 + q / SW, xx = x0 + q % SW, d = d0 + lane;
      float v = 0.0f;
      if (yy >= 0 && yy < H && xx >= 0 && xx < W && d < D) v = __ldg(in + ((int64_t)yy * W + xx) * D + d);
      tile[q * CB_TD + lane] = v;
    }
    for (int q = threadIdx.x; q < 4 * SH * CB_TX; q += blockDim.x) {
      const int a = q / (SH * CB_TX), r = (q / CB_TX) % SH, c = q % CB_TX;
      const int yy = y0 + r, xx = X0 + c;
      sl[q] = (yy >= 0 && yy < H && xx < W) ? (int16_t)__ldg(lc + a * HW + (int64_t)yy * W + xx) : 0;
    }
    for (int q = threadIdx.x; q < 4 * SH * RW; q += blockDim.x) {
      const int a = q / (SH * RW), r = (q / RW) % SH, c = q % RW;
      const int yy = y0 + r, xx = xr0 + c;
      sr[q] = (yy >= 0 && yy < H && xx >= 0 && xx < W) ? (int16_t)__ldg(rc + a * HW + (int64_t)yy * W + xx) : 0;
    }
    __syncthreads();
    const int d = d0 + lane;
    const int dd = d * direction;
    for (int q = warp; q < CB_TX * CB_TY; q += nwarp) {
      const int cy = q / CB_TX, cx = q % CB_TX;
      const int y = Y0 + cy, x = X0 + cx;
      if (y >= H || x >= W || d >= D) continue;
      const int64_t id = ((int64_t)y * W + x) * D + d;
      const int xm = x + dd;
      if (xm < 0 || xm >= W) {
        out[id] = in[id];
        continue;
      }
      const int cm = xm - xr0;  // column of xm in the staged right arms
      const int ry = cy + halo;
      const int yy_s = max((int)sl[(2 * SH + ry) * CB_TX + cx], (int)sr[(2 * SH + ry) * RW + cm]);
      const int yy_t = min((int)sl[(3 * SH + ry) * CB_TX + cx], (int)sr[(3 * SH + ry) * RW + cm]);
      float sum = 0.0f;
      int cnt = 0;
      for (int yy = yy_s + 1; yy < yy_t; yy++) {
        const int r = yy - y0;
        int xx_s, xx_t;
        const bool row_in = r >= 0 && r < SH;
        if (row_in) {
          xx_s = max((int)sl[r * CB_TX + cx], (int)sr[r * RW + cm] - dd);
          xx_t = min((int)sl[(SH + r) * CB_TX + cx], (int)sr[(SH + r) * RW + cm] - dd);
        } else {
          xx_s = (int)fmaxf(lc[(int64_t)yy * W + x], rc[(int64_t)yy * W + xm] - (float)dd);
          xx_t = (int)fminf(lc[HW + (int64_t)yy * W + x], rc[HW + (int64_t)yy * W + xm] - (float)dd);
        }
        if (row_in && xx_s + 1 >= x0 && xx_t - 1 < x0 + SW) {
          const float* rowp = tile + ((size_t)r * SW - x0) * CB_TD + lane;
          for (int xx = xx_s + 1; xx < xx_t; xx++) sum += rowp[xx * CB_TD];
        } else {
          for (int xx = xx_s + 1; xx < xx_t; xx++) sum += in[((int64_t)yy * W + xx) * D + d];
        }
        cnt += max(xx_t - xx_s - 1, 0);
      }
      out[id] = sum / (float)cnt;
    }
  }
}

// cbca on [H,W,D] volumes in separable form, the row-then-column
// decomposition of integral-image aggregation: the support row of row yy
// for (x, d) is the same interval for every centre row y (it depends on the
// arms of (yy, x) and (yy, x + d*direction) only), so
//   R(yy, x, d) = sum of the support row,   C(yy, x, d) = its length,
//   out(y, x, d) = sum over the support rows yy of R / sum of C.
// A CTA owns CS_TY x CS_TX pixels x 32 disparities (lane = disparity): it
// forms R and C for its rows and HALO rows above and below into shared
// memory, then the column sums.  Both sums run over fixed 2*HALO+1 taps,
// masked to the support, in ascending order, from register windows (a tile
// row's inputs; a column's R and C); with arms of at most
// HALO = L1 - 1 pixels every support element is within the taps.  The
// result differs from the reference's single running float sum
// (post.cu:415-429) by rounding only.
constexpr int CS_TX = 8, CS_TD = 32;

template <int HALO, int CS_TY>
constexpr size_t cbca_sep_smem_bytes() {
  return (size_t)(CS_TY + 2 * HALO) * CS_TX * CS_TD * (sizeof(float) + sizeof(uint8_t));
}

template <int HALO, int CS_TY>
__global__ void __launch_bounds__(256, 4) cbca_hwd_sep_kernel(
    const float* __restrict__ lc, const float* __restrict__ rc, const float* __restrict__ in, int H, int W,
    int D, int direction, float* __restrict__ out) {
  constexpr int SR = CS_TY + 2 * HALO;   // rows of R: the tile's and HALO above and below
  constexpr int NV = CS_TX + 2 * HALO;   // input columns a tile row needs
  constexpr int G = 8;                   // output rows per column-sum window
  static_assert(CS_TX == 8 && CS_TY % G == 0, "one warp per tile column");
  extern __shared__ float sR[];                                       // [SR][CS_TX][CS_TD]
  uint8_t* sC = reinterpret_cast<uint8_t*>(sR + SR * CS_TX * CS_TD);  // [SR][CS_TX][CS_TD]
  const int ntd = (D + CS_TD - 1) / CS_TD, ntx = (W + CS_TX - 1) / CS_TX;
  const int64_t t = blockIdx.x;
  const int td = (int)(t % ntd), tx = (int)((t / ntd) % ntx), ty = (int)(t / ((int64_t)ntd * ntx));
  const int X0 = tx * CS_TX, Y0 = ty * CS_TY;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d = td * CS_TD + lane, dd = d * direction;
  const bool dok = d < D;
  const int64_t HW = (int64_t)H * W;
  // 1. row sums: warp w forms R and C of tile rows w, w + 8, ... for all CS_TX columns
  //    from the NV input values of its row, held in registers
  for (int r = warp; r < SR; r += 8) {
    const int yy = Y0 - HALO + r;
    const bool rok = yy >= 0 && yy < H && dok;
    float v[NV];
    const int64_t o = (int64_t)(rok ? yy : 0) * W;
    const float* row = in + o * D + d;
#pragma unroll
    for (int j = 0; j < NV; j++) {
      const int xx = X0 - HALO + j;
      v[j] = (rok && xx >= 0 && xx < W) ? __ldg(row + (int64_t)xx * D) : 0.0f;
    }
#pragma unroll
    for (int c = 0; c < CS_TX; c++) {
      const int x = X0 + c, xm = x + dd;
      float sum = 0.0f;
      int cnt = 0;
      if (rok && x < W && xm >= 0 && xm < W) {
        // support row of (yy, x, d) in tap coordinates: ks < k < kt
        const int ks = max((int)__ldg(lc + o + x), (int)__ldg(rc + o + xm) - dd) - x;
        const int kt = min((int)__ldg(lc + HW + o + x), (int)__ldg(rc + HW + o + xm) - dd) - x;
#pragma unroll
        for (int k = -HALO; k <= HALO; k++)
          if (k > ks && k < kt) sum += v[c + HALO + k];
        cnt = max(kt - ks - 1, 0);
      }
      sR[(r * CS_TX + c) * CS_TD + lane] = sum;
      sC[(r * CS_TX + c) * CS_TD + lane] = (uint8_t)cnt;
    }
  }
  __syncthreads();
  // 2. column sums: warp c owns tile column c; G output rows at a time from a
  //    register window of G + 2*HALO rows of R and C
  const int c = warp, x = X0 + c, xm = x + dd;
  if (x >= W || !dok) return;
  const bool xok = xm >= 0 && xm < W;
#pragma unroll 1
  for (int g0 = 0; g0 < CS_TY; g0 += G) {
    float wr[G + 2 * HALO];
    int wc[G + 2 * HALO];
#pragma unroll
    for (int j = 0; j < G + 2 * HALO; j++) {
      const int i = ((g0 + j) * CS_TX + c) * CS_TD + lane;
      wr[j] = sR[i];
      wc[j] = sC[i];
    }
#pragma unroll
    for (int cy = 0; cy < G; cy++) {
      const int y = Y0 + g0 + cy;
      if (y >= H) break;
      const int64_t o = (int64_t)y * W;
      const int64_t id = (o + x) * D + d;
      if (!xok) {
        out[id] = __ldg(in + id);
        continue;
      }
      const int ks = max((int)__ldg(lc + 2 * HW + o + x), (int)__ldg(rc + 2 * HW + o + xm)) - y;
      const int kt = min((int)__ldg(lc + 3 * HW + o + x), (int)__ldg(rc + 3 * HW + o + xm)) - y;
      float sum = 0.0f;
      int cnt = 0;
#pragma unroll
      for (int k = -HALO; k <= HALO; k++)
        if (k > ks && k < kt) {
          sum += wr[cy + HALO + k];
          cnt += wc[cy + HALO + k];
        }
      out[id] = sum / (float)cnt;
    }
  }
}

template <int HALO, int TY>
int launch_cbca_sep_ht(const float* lc, const float* rc, const float* in, int64_t H, int64_t W, int D,
                       int direction, float* out, cudaStream_t st) {
  constexpr size_t smem = cbca_sep_smem_bytes<HALO, TY>();
  CBMV_CUDA(cudaFuncSetAttribute(cbca_hwd_sep_kernel<HALO, TY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  const int64_t tiles = (int64_t)((W + CS_TX - 1) / CS_TX) * ((H + TY - 1) / TY) * ((D + CS_TD - 1) / CS_TD);
  cbca_hwd_sep_kernel<HALO, TY><<<(unsigned)tiles, 256, smem, st>>>(lc, rc, in, (int)H, (int)W, D, direction, out);
  return check_launch("cbca_sep");
}

// tile rows 16 or 32 (the results do not depend on them)
template <int HALO>
int launch_cbca_sep_h(const float* lc, const float* rc, const float* in, int64_t H, int64_t W, int D,
                      int direction, float* out, cudaStream_t st, int rows) {
  if (rows == 16) return launch_cbca_sep_ht<HALO, 16>(lc, rc, in, H, W, D, direction, out, st);
  return launch_cbca_sep_ht<HALO, 32>(lc, rc, in, H, W, D, direction, out, st);
}

// The separable CBCA with its supports precomputed: the support of every
// (y, x, d) depends on the cross arms only, so the cbca_i2 passes of one
// post share it.  One 32-bit word per (y, x, d), for arms of at most
// kMaskHalo pixels:
//   bits  0..10  taps k = -5..5 of its support row (bit k + 5),
//   bits 11..21  taps of its support column,
//   bits 22..28  the number of pixels in its support (at most 121),
//   bit  31      x + d*direction is outside the image (the input is copied).
// The passes then sum the same taps in the same ascending order as
// cbca_hwd_sep_kernel, so the results are bit-identical to it.
constexpr int kMaskHalo = kCbcaMaskMaxHalo;
constexpr uint32_t kMaskCopy = 1u << 31;

// A pixel's relative arms as four packed int8: arm a minus the pixel's x
// (arms 0, 1) or y (arms 2, 3), clamped.
__device__ __forceinline__ int clamp_i8(int v) { return min(max(v, -128), 127); }
template <int B>
__device__ __forceinline__ int rel_arm(uint32_t w) {
  return (int)((int32_t)(w << (24 - 8 * B)) >> 24);
}

// cbca on [D,H,W] volumes (the drop-in's layout) in the reference's order:
// a CTA owns 32 columns x 16 rows of eight disparities, one per warp (lane =
// column).  A support row's interval depends on its own row only, so a warp
// reads and masks each row of its tile once (eleven taps, those outside the
// interval as 0: adding 0 changes no sum) and adds the eleven values to the
// running sum of every one of four output rows whose support has the row --
// the rows ascend, so each sum runs in the reference's order.  Bound by
// instruction issue (the masks of a row are formed for every four outputs, 14
// rows; eight outputs at once need 79 registers: 613 us where four took 533).
// Now 694x320 D=128 458 us, 694x554 800; with a thread per output walking its
// support (cbca_kernel) 1380 and 2420.
// A tile whose arms may reach beyond the taps (cross arms of L1 > 6), or are
// no whole numbers, is left to cbca_dhw_left_kernel.
constexpr int CD_X = 32, CD_Y = 16, CD_D = 8, CD_G = 4, CD_HALO = 5;
constexpr int CD_LEFT = 24;  // at most, blocks of cbca_dhw_left_kernel per SM
constexpr uint32_t kCbcaLeft = 0x7FA5C3E1u;  // the mark of a run that is left, its first value: a NaN that no sum gives

// The relative arms of one pixel, packed without conversions (an arm below
// 2^22 is read off its sum with 1.5 * 2^23); *odd: one of them is no whole
// number, or too large for that, or reaches beyond the taps, or lies so far
// on the other side of its pixel that an interval of two such arms may lie
// beyond what a byte holds.
__device__ __forceinline__ uint32_t pack_whole_arms(const float* __restrict__ c, int64_t HW, int64_t o, int x, int y,
                                                    bool* odd) {
  constexpr float kMagic = 12582912.0f;
  uint32_t w = 0;
#pragma unroll
  for (int a = 0; a < 4; a++) {
    const float v = __ldg(c + a * HW + o), t = __fadd_rn(v, kMagic);
    const int rel = __float_as_int(t) - __float_as_int(kMagic) - (a < 2 ? x : y);
    *odd |= !(__fsub_rn(t, kMagic) == v && fabsf(v) < 4194304.0f) || (a & 1 ? rel < -120 || rel > CD_HALO + 1 : rel > 120 || rel < -CD_HALO - 1);
    w |= (uint32_t)(clamp_i8(rel) & 0xFF) << (8 * a);
  }
  return w;
}

// taps lo..hi (bit k + 5) of an interval, those within five pixels
__device__ __forceinline__ uint32_t tap_mask(int lo, int hi) {
  const int a = min(max(lo + CD_HALO, 0), 31), b = min(max(hi + CD_HALO + 1, 0), 31);
  return ((1u << b) - 1u) & ~((1u << a) - 1u);
}

__global__ void __launch_bounds__(32 * CD_D) cbca_dhw_kernel(const float* __restrict__ lc, const float* __restrict__ rc,
                                                               const float* __restrict__ in, int H, int W, int D,
                                                               int direction, float* __restrict__ out) {
  constexpr int SR = CD_Y + 2 * CD_HALO, SX = CD_X + 2 * CD_HALO, NXM = CD_X + CD_D - 1, NT = 2 * CD_HALO + 1;
  __shared__ uint32_t sAL[SR][CD_X];  // packed relative arms, left view at (yy, x)
  __shared__ uint32_t sAR[SR][NXM];   // right view at (yy, x + d * direction)
  __shared__ float tiles[CD_D][SR][SX];
  const int ntx = (W + CD_X - 1) / CD_X, nty = (H + CD_Y - 1) / CD_Y;
  const int64_t t = blockIdx.x;
  const int X0 = (int)(t % ntx) * CD_X, Y0 = (int)(t / ntx % nty) * CD_Y, D0 = (int)(t / ((int64_t)ntx * nty)) * CD_D;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t HW = (int64_t)H * W;
  const int xm_lo = direction > 0 ? X0 + D0 : X0 - (D0 + CD_D - 1);
  bool odd = false;
  auto leave = [&]() {  // whether the tile is cbca_dhw_left_kernel's; its runs are marked then
    if (!__syncthreads_or(odd)) return false;
    if (lane < CD_Y && Y0 + lane < H && D0 + warp < D)
      out[(int64_t)(D0 + warp) * HW + (int64_t)(Y0 + lane) * W + X0] = __uint_as_float(kCbcaLeft);
    return true;
  };
  for (int r = warp; r < SR; r += CD_D) {
    const int yy = Y0 - CD_HALO + r;
    const bool rok = yy >= 0 && yy < H;  // outside the image: an empty interval
    const int64_t o = (int64_t)yy * W;
    sAL[r][lane] = rok && X0 + lane < W ? pack_whole_arms(lc, HW, o + X0 + lane, X0 + lane, yy, &odd) : 0u;
  }
  if (leave()) return;
  for (int r = warp; r < SR; r += CD_D) {
    const int yy = Y0 - CD_HALO + r;
    const bool rok = yy >= 0 && yy < H;
    const int64_t o = (int64_t)yy * W;
    for (int j = lane; j < NXM; j += 32) {
      const int xm = xm_lo + j;
      sAR[r][j] = rok && xm >= 0 && xm < W ? pack_whole_arms(rc, HW, o + xm, xm, yy, &odd) : 0u;
    }
  }
  if (leave()) return;
  const int x = X0 + lane;
  float(*tile)[SX] = tiles[warp];
  const int xa = X0 - CD_HALO + lane, xb = xa + 32;
  const bool oka = xa >= 0 && xa < W, okb = lane < SX - 32 && xb < W;
  const int d = D0 + warp;
  if (d >= D) return;
  const float* src = in + (int64_t)d * HW + (int64_t)(Y0 - CD_HALO) * W + xa;
#pragma unroll
  for (int r = 0; r < SR; r++) {
    const bool rok = Y0 - CD_HALO + r >= 0 && Y0 - CD_HALO + r < H;
    tile[r][lane] = rok && oka ? __ldg(src) : 0.0f;
    if (lane < SX - 32) tile[r][lane + 32] = rok && okb ? __ldg(src + 32) : 0.0f;
    src += W;
  }
  __syncwarp();
  if (x >= W) return;
  const int xm = x + d * direction;
  const bool match = xm >= 0 && xm < W;
  const int jr = match ? xm - xm_lo : 0;
  float* dst = out + (int64_t)d * HW + x;
#pragma unroll 1
  for (int g = 0; g < CD_Y && Y0 + g < H; g += CD_G) {
    // the rows of every output's support as taps; its sum; its pixels
    uint32_t vm[CD_G];
    float sum[CD_G];
    int cnt[CD_G];
#pragma unroll
    for (int j = 0; j < CD_G; j++) {
      const uint32_t wl = sAL[g + j + CD_HALO][lane], wr = sAR[g + j + CD_HALO][jr];
      const int lo = max(rel_arm<2>(wl), rel_arm<2>(wr)) + 1, hi = min(rel_arm<3>(wl), rel_arm<3>(wr)) - 1;
      vm[j] = tap_mask(lo, hi);
      cnt[j] = 0;
      sum[j] = 0.0f;
    }
#pragma unroll
    for (int r = 0; r < CD_G + 2 * CD_HALO; r++) {
      const uint32_t wl = sAL[g + r][lane], wr = sAR[g + r][jr];
      const int lo = max(rel_arm<0>(wl), rel_arm<0>(wr)) + 1, hi = min(rel_arm<1>(wl), rel_arm<1>(wr)) - 1;
      const uint32_t hm = tap_mask(lo, hi);
      const int len = max(hi - lo + 1, 0);
      float v[NT];
#pragma unroll
      for (int k = 0; k < NT; k++) {
        v[k] = tile[g + r][lane + k];
        if (!(hm & (1u << k))) v[k] = 0.0f;
      }
#pragma unroll
      for (int j = r > 2 * CD_HALO ? r - 2 * CD_HALO : 0; j < CD_G && j <= r; j++)
        if (vm[j] & (1u << (r - j))) {
#pragma unroll
          for (int k = 0; k < NT; k++) sum[j] += v[k];
          cnt[j] += len;
        }
    }
#pragma unroll
    for (int j = 0; j < CD_G; j++) {
      const int y = Y0 + g + j;
      if (y >= H) break;
      dst[(int64_t)y * W] = match ? sum[j] / (float)cnt[j] : tile[g + j + CD_HALO][lane + CD_HALO];
    }
  }
}

// The runs of up to 32 outputs that cbca_dhw_kernel left, by cbca_one: a warp
// reads the marks of 32 runs at once and walks those that are marked.  A mark
// may also be the bits of a result: that run is formed again, to the same
// values.  Bound by the latency of the supports' loads, so what counts is
// that every output has a thread and runs of large supports are spread over
// the SMs: with the long supports summed by the tiles' own warps, 16 outputs
// one after the other, beside the taps of the others, L1=9 took at 694x554
// D=128 3390 us (cbca_kernel alone 2840, now 2440), at 320x240 D=16 262 (82,
// 91).  Launched beside the tiles' last wave (programmatic launch) its
// blocks keep the tiles' split of L1 and shared memory: 3570 us.  Where no run is
// marked the launch takes 2 us at 320x240 D=16 and 19 at 694x320 D=128, for
// the marks' sectors.
__global__ void __launch_bounds__(256) cbca_dhw_left_kernel(const float* __restrict__ lc, const float* __restrict__ rc,
                                                          const float* __restrict__ in, int H, int W, int D,
                                                          int direction, float* out) {
  const int ntx = (W + CD_X - 1) / CD_X, lane = threadIdx.x & 31;
  const int64_t runs = (int64_t)ntx * H * D, nw = (int64_t)gridDim.x * 8, w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  for (int64_t r0 = w; r0 < runs; r0 += 32 * nw) {
    const int64_t r = r0 + lane * nw, row = r / ntx;
    const bool left = r < runs && __float_as_uint(out[row * W + (r - row * ntx) * CD_X]) == kCbcaLeft;
    uint32_t marked = __ballot_sync(0xffffffffu, left);
    for (; marked; marked &= marked - 1) {
      const int64_t q = r0 + (__ffs(marked) - 1) * nw, qrow = q / ntx;  // row qrow % H of disparity qrow / H
      const int d = (int)(qrow / H), y = (int)(qrow - (int64_t)d * H), x = (int)(q - qrow * ntx) * CD_X + lane;
      if (x < W) out[qrow * W + x] = cbca_one(lc, rc, in, H, W, D, CBMV_DHW, direction, y, x, d);
    }
  }
}

// The cross arms of one pixel as the taps they allow: bits 0..10 of its row
// (tap k at bit k + 5), bits 11..21 of its column; from the reach (0..5
// pixels) to the left, right, up and down.
__device__ __forceinline__ uint32_t arm_word(int l, int r, int u, int d) {
  return ((1u << (l + r + 1)) - 1u) << (kMaskHalo - l) | ((1u << (u + d + 1)) - 1u) << (11 + kMaskHalo - u);
}

// *odd (zeroed by the caller) is set where an arm is none that cross_kernel
// gives: one that excludes its pixel, or is longer than a word's taps.
__global__ void arm_words_kernel(const float* __restrict__ lc, const float* __restrict__ rc, int64_t H, int64_t W,
                                 uint32_t* __restrict__ words, uint32_t* __restrict__ odd) {
  const int64_t n = H * W;
  const float* __restrict__ arms = blockIdx.y ? rc : lc;
  GRID_STRIDE(p, n) {
    const int y = (int)(p / W), x = (int)(p - y * W);
    bool ok = true;
    auto reach = [&](int v) {
      ok &= v >= 1 && v <= kMaskHalo + 1;
      return min(max(v - 1, 0), kMaskHalo);
    };
    words[blockIdx.y * n + p] = arm_word(reach(x - (int)arms[p]), reach((int)arms[n + p] - x),
                                         reach(y - (int)arms[2 * n + p]), reach((int)arms[3 * n + p] - y));
    if (!ok) *odd = 1u;
  }
}

// The support words of any arms, one thread per word, where *odd says that
// the arm words do not hold them: the taps of a support within five pixels
// and inside the image, and the pixels of its rows at their whole length.
__global__ void cbca_mask_any_kernel(const float* __restrict__ lc, const float* __restrict__ rc, int64_t H, int64_t W,
                                     int D, int direction, const uint32_t* __restrict__ odd, uint32_t* __restrict__ mask) {
  if (*odd == 0u) return;
  const int64_t n = H * W;
  GRID_STRIDE(id, n * D) {
    const int64_t p = id / D, y = p / W, x = p - y * W;
    const int64_t xm = x + (id - p * D) * direction;
    if (xm < 0 || xm >= W) {
      mask[id] = kMaskCopy;
      continue;
    }
    // taps lo..hi that arms a and a + 1 of row yy allow
    auto taps = [&](int a, int64_t yy, int* lo, int* hi) {
      const int64_t l = a * n + yy * W + x, r = a * n + yy * W + xm;
      const int ol = (int)(a < 2 ? x : yy), orr = (int)(a < 2 ? xm : yy);
      *lo = max(clamp_i8((int)lc[l] - ol), clamp_i8((int)rc[r] - orr)) + 1;
      *hi = min(clamp_i8((int)lc[l + n] - ol), clamp_i8((int)rc[r + n] - orr)) - 1;
    };
    int lo, hi;
    uint32_t w = 0, cnt = 0;
    taps(0, y, &lo, &hi);
    for (int k = max(lo, -kMaskHalo); k <= min(hi, kMaskHalo); k++)
      if (x + k >= 0 && x + k < W) w |= 1u << (k + kMaskHalo);
    taps(2, y, &lo, &hi);
    for (int k = max(lo, -kMaskHalo); k <= min(hi, kMaskHalo); k++)
      if (y + k >= 0 && y + k < H) {
        w |= 1u << (11 + k + kMaskHalo);
        int from, to;
        taps(0, y + k, &from, &to);
        cnt += (uint32_t)max(to - from + 1, 0);
      }
    mask[id] = w | (cnt & 0x7Fu) << 22;
  }
}

// The support words from the arm words of the volume's own view (wl) and of
// the matching view (wr): both arms allow a tap where both words do, so a
// support is one AND; a support row's length is its number of taps, and the
// count the difference of two prefix sums of those down the tile's column,
// which a warp walks once (column = warp, disparity = lane).  Bound by
// instruction issue, 4 B written per word: 694x554 D=128 89 us (238 from the
// arms' coordinates), 901x600 D=192 179 (481).
template <int CS_TY>
__global__ void __launch_bounds__(256) cbca_mask_build_kernel(const uint32_t* __restrict__ wl,
                                                              const uint32_t* __restrict__ wr, int H, int W, int D,
                                                              int direction, uint32_t* __restrict__ mask) {
  constexpr int HALO = kMaskHalo, SR = CS_TY + 2 * HALO;
  constexpr int NXM = CS_TX + CS_TD - 1;  // matching columns x + d * direction of the tile
  __shared__ uint16_t sP[SR + 1][CS_TX][CS_TD];  // taps of the rows above, per column and disparity
  __shared__ uint32_t sL[SR][CS_TX], sR[SR][NXM];
  const int ntd = (D + CS_TD - 1) / CS_TD, ntx = (W + CS_TX - 1) / CS_TX;
  const int64_t t = blockIdx.x;
  const int td = (int)(t % ntd), tx = (int)((t / ntd) % ntx), ty = (int)(t / ((int64_t)ntd * ntx));
  const int X0 = tx * CS_TX, Y0 = ty * CS_TY;
  const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;
  const int xm_lo = direction > 0 ? X0 + td * CS_TD : X0 - (td * CS_TD + CS_TD - 1);
  for (int q = threadIdx.x; q < SR * (CS_TX + NXM); q += blockDim.x) {
    const int r = q / (CS_TX + NXM), j = q - r * (CS_TX + NXM);
    const int yy = Y0 - HALO + r, xx = j < CS_TX ? X0 + j : xm_lo + j - CS_TX;
    const bool in = yy >= 0 && yy < H && xx >= 0 && xx < W;
    if (j < CS_TX) sL[r][j] = in ? __ldg(wl + (int64_t)yy * W + xx) : 0u;
    else sR[r][j - CS_TX] = in ? __ldg(wr + (int64_t)yy * W + xx) : 0u;
  }
  __syncthreads();
  const int d = td * CS_TD + lane, x = X0 + c, xm = x + d * direction;
  if (x >= W || d >= D) return;
  const int j = c + (direction > 0 ? lane : CS_TD - 1 - lane);
  const bool xok = xm >= 0 && xm < W;
  uint32_t run = 0;
  sP[0][c][lane] = 0;
  auto add_row = [&](int r) {
    run += __popc(sL[r][c] & sR[r][j] & 0x7FFu);
    sP[r + 1][c][lane] = (uint16_t)run;
  };
#pragma unroll
  for (int r = 0; r < 2 * HALO; r++) add_row(r);
  uint32_t* dst = mask + ((int64_t)Y0 * W + x) * D + d;
  const int n = min(CS_TY, H - Y0);
#pragma unroll 4
  for (int cy = 0; cy < n; cy++, dst += (int64_t)W * D) {
    add_row(cy + 2 * HALO);
    const int r = cy + HALO;
    const uint32_t w = sL[r][c] & sR[r][j];
    const int up = __popc(w & (0x1Fu << 11)), down = __popc(w & (0x1Fu << 17));
    const uint32_t cnt = (uint32_t)sP[r + down + 1][c][lane] - (uint32_t)sP[r - up][c][lane];
    *dst = xok ? w | cnt << 22 : kMaskCopy;
  }
}

// One CBCA pass from the precomputed supports (same tiling and summation
// order as cbca_hwd_sep_kernel<kMaskHalo>).  Bound by instruction issue (two
// per tap, 22 taps) with too few warps to cover its loads, so what stands
// between the loads is kept out: supports never leave the image, so columns
// are clamped and rows outside skipped instead of tested per value; the eight
// support words of a column step are read together; and the division is a
// multiplication by the count's reciprocal with one correction (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000",
// 1990), which rounds as the division does for every float32 significand and
// every count (all checked) while no exponent nears its limits; a step that
// holds any other value, or a copied one, is done again with the division.
// 694x554 D=128: 192 us per pass (240 before), 901x600 D=192 403 (499),
// 1482x994 D=256 1522 (1922).  Measured beside it: two disparities per lane
// 208-253 us, a ring of row sums down taller tiles 283, the next row's values
// loaded ahead 234.
template <int CS_TY>
__global__ void __launch_bounds__(256, 4) cbca_hwd_mask_kernel(const uint32_t* __restrict__ mask,
                                                               const float* __restrict__ in, int H, int W,
                                                               int D, float* __restrict__ out) {
  constexpr int HALO = kMaskHalo;
  constexpr int SR = CS_TY + 2 * HALO;
  constexpr int NV = CS_TX + 2 * HALO;
  constexpr int G = 8;
  static_assert(CS_TX == 8 && CS_TY % G == 0, "one warp per tile column");
  extern __shared__ float sR[];  // [SR][CS_TX][CS_TD]
  __shared__ float2 s_div[128];  // a count and its reciprocal
  const int ntd = (D + CS_TD - 1) / CS_TD, ntx = (W + CS_TX - 1) / CS_TX;
  const int64_t t = blockIdx.x;
  const int td = (int)(t % ntd), tx = (int)((t / ntd) % ntx), ty = (int)(t / ((int64_t)ntd * ntx));
  const int X0 = tx * CS_TX, Y0 = ty * CS_TY;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d = td * CS_TD + lane, dl = min(d, D - 1);  // a lane beyond D reads the last disparity
  const int64_t WD = (int64_t)W * D;
  if (threadIdx.x < 128) s_div[threadIdx.x] = make_float2((float)threadIdx.x, 1.0f / (float)threadIdx.x);
  // 1. row sums over each (yy, x, d)'s support-row taps; what clamped columns
  //    and skipped rows leave in the tile is never added below
  const bool interior = X0 >= HALO && X0 + CS_TX + HALO <= W;
  const int r1 = min(SR, H + HALO - Y0);
  for (int r = warp + (Y0 < HALO ? (HALO - Y0 - warp + 7) / 8 * 8 : 0); r < r1; r += 8) {
    const int64_t ro = (int64_t)(Y0 - HALO + r) * W * D + dl;
    const float* row = in + ro;
    float v[NV];
    if (interior) {
      row += (int64_t)(X0 - HALO) * D;
#pragma unroll
      for (int j = 0; j < NV; j++, row += D) v[j] = __ldg(row);
    } else {
#pragma unroll
      for (int j = 0; j < NV; j++) v[j] = __ldg(row + (int64_t)min(max(X0 - HALO + j, 0), W - 1) * D);
    }
    const uint32_t* m = mask + ro + (int64_t)X0 * D;
#pragma unroll
    for (int c = 0; c < CS_TX; c++) {
      const uint32_t hm = __ldg(m);
      float sum = 0.0f;
#pragma unroll
      for (int k = 0; k <= 2 * HALO; k++)
        if (hm & (1u << k)) sum += v[c + k];
      sR[(r * CS_TX + c) * CS_TD + lane] = sum;
      if (X0 + c + 1 < W) m += D;
    }
  }
  __syncthreads();
  // 2. column sums: warp c owns tile column c; G output rows at a time from
  //    a register window of G + 2*HALO row sums
  const int c = warp, x = X0 + c;
  if (x >= W || d >= D) return;
#pragma unroll 1
  for (int g0 = 0; g0 < CS_TY; g0 += G) {
    const int n = min(G, H - (Y0 + g0));
    if (n <= 0) break;
    const int64_t o = (Y0 + g0) * WD + (int64_t)x * D + d;
    uint32_t w[G];
    const uint32_t* m = mask + o;
#pragma unroll
    for (int cy = 0; cy < G; cy++) {
      w[cy] = __ldg(m);
      if (cy + 1 < n) m += WD;
    }
    float wr[G + 2 * HALO];
#pragma unroll
    for (int j = 0; j < G + 2 * HALO; j++) wr[j] = sR[((g0 + j) * CS_TX + c) * CS_TD + lane];
    auto column = [&](int cy) {
      float sum = 0.0f;
#pragma unroll
      for (int k = 0; k <= 2 * HALO; k++)
        if (w[cy] & (1u << (k + 11))) sum += wr[cy + k];
      return sum;
    };
    float* dst = out + o;
    bool again = false;
#pragma unroll
    for (int cy = 0; cy < G; cy++, dst += WD) {
      const float sum = column(cy);
      const float2 div = s_div[(w[cy] >> 22) & 0x7Fu];
      const float q = sum * div.y, res = fmaf(fmaf(-q, div.x, sum), div.y, q);
      again |= !(fabsf(res) <= 0x1p100f) || (fabsf(sum) < 0x1p-90f && sum != 0.0f) || (w[cy] & kMaskCopy);
      if (cy < n) *dst = res;
    }
    if (again) {
      dst = out + o;
#pragma unroll
      for (int cy = 0; cy < G; cy++, dst += WD) {
        if (cy >= n) break;
        *dst = w[cy] & kMaskCopy ? __ldg(in + o + cy * WD) : column(cy) / (float)((w[cy] >> 22) & 0x7Fu);
      }
    }
  }
}

template <int TY>
int launch_cbca_masked_t(const uint32_t* mask, const float* in, int64_t H, int64_t W, int D, float* out,
                         cudaStream_t st) {
  constexpr size_t smem = (size_t)(TY + 2 * kMaskHalo) * CS_TX * CS_TD * sizeof(float);
  const int64_t tiles = (int64_t)((W + CS_TX - 1) / CS_TX) * ((H + TY - 1) / TY) * ((D + CS_TD - 1) / CS_TD);
  cbca_hwd_mask_kernel<TY><<<(unsigned)tiles, 256, smem, st>>>(mask, in, (int)H, (int)W, D, out);
  return check_launch("cbca_masked");
}


// Winner-take-all (first minimum, as np.argmin) and the subpixel parabola
// (post.cu:453-483).  One warp per pixel on [H,W,D] volumes.
// A warp takes four pixels at a time, so that their loads are in flight
// together; lane l reads four consecutive disparities (V = 4, where D and the
// volume's alignment allow it) or N single ones 32 apart, as many as a row of
// up to 128 has.  Bound by memory.  us, one pixel at a time with single loads
// against this: 901x600 D=192 128 / 70; 694x554 D=128 58 / 36, D=127 45 / 37
// (50 with one single load per pixel), D=65 41 / 33, D=33 37 / 26.
template <int V, int N>
__global__ void __launch_bounds__(256) wta_subpixel_hwd_kernel(const float* __restrict__ c, int64_t HW, int D,
                                                               float* __restrict__ disp_int, float* __restrict__ disp) {
  constexpr int PX = 4;
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  const float inf = __int_as_float(0x7f800000);
  for (int64_t p0 = PX * (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); p0 < HW; p0 += PX * nw) {
    const int n = (int)min((int64_t)PX, HW - p0);
    // each lane's first minimum (NaN and +inf are never one) per pixel
    float bv[PX];
    int bd[PX];
#pragma unroll
    for (int k = 0; k < PX; k++) bv[k] = inf, bd[k] = 0x7fffffff;
    constexpr int S = V == 4 ? 1 : 32;  // between a lane's N disparities
    for (int d = V * lane; d < D; d += 32 * N) {
      float v[PX][N];
#pragma unroll
      for (int k = 0; k < PX; k++) {
        const float* r = c + (p0 + (k < n ? k : 0)) * D + d;
        if constexpr (V == 4) {
          const float4 q = __ldg(reinterpret_cast<const float4*>(r));
          v[k][0] = q.x, v[k][1] = q.y, v[k][2] = q.z, v[k][3] = q.w;
        } else {
#pragma unroll
          for (int i = 0; i < N; i++) v[k][i] = i == 0 || d + S * i < D ? __ldg(r + S * i) : inf;
        }
      }
#pragma unroll
      for (int k = 0; k < PX; k++)
#pragma unroll
        for (int i = 0; i < N; i++)
          if (v[k][i] < bv[k]) { bv[k] = v[k][i]; bd[k] = d + S * i; }
    }
    // the lowest d among the lanes that hold the warp's minimum; lane k keeps pixel k's
    int mine = 0;
#pragma unroll
    for (int k = 0; k < PX; k++) {
      float mn = bv[k];
      asm volatile("redux.sync.min.f32 %0, %0, 0xffffffff;" : "+f"(mn));
      const int first = (int)__reduce_min_sync(0xffffffffu, bv[k] == mn && mn < inf ? (unsigned)bd[k] : 0x7fffffffu);
      if (lane == k) mine = first == 0x7fffffff ? 0 : first;  // all NaN: np.argmin would return 0 for a NaN at 0
    }
    if (lane < n) {
      const int64_t p = p0 + lane;
      if (disp_int) disp_int[p] = (float)mine;
      if (disp) {
        const float* r = c + p * D;
        float o = (float)mine;
        if (1 <= mine && mine < D - 1) {
          const float cn = r[mine - 1], cz = r[mine], cp = r[mine + 1];
          const float denom = 2 * (cp + cn - 2 * cz);
          if (denom > 1e-5) {
            const double q = (double)((cp - cn) / denom);
            o = (float)(mine - fmin(1.0, fmax(-1.0, q)));
          }
        }
        disp[p] = o;
      }
    }
  }
}

__global__ void wta_dhw_kernel(const float* __restrict__ c, int64_t HW, int D,
                               float* __restrict__ disp) {
  GRID_STRIDE(p, HW) {
    float bv = c[p];
    int bd = 0;
    for (int d = 1; d < D; d++) {
      const float v = c[(int64_t)d * HW + p];
      if (v < bv) { bv = v; bd = d; }
    }
    disp[p] = (float)bd;
  }
}

__global__ void subpixel_kernel(const float* __restrict__ d0, const float* __restrict__ c,
                                int64_t H, int64_t W, int D, int layout, float* __restrict__ out) {
  GRID_STRIDE(id, H * W) {
    const int d = (int)d0[id];
    float o = (float)d;
    if (1 <= d && d < D - 1) {
      const int64_t y = id / W, x = id - y * W;
      const float cn = c[vol_index(layout, y, x, d - 1, H, W, D)];
      const float cz = c[vol_index(layout, y, x, d, H, W, D)];
      const float cp = c[vol_index(layout, y, x, d + 1, H, W, D)];
      const float denom = 2 * (cp + cn - 2 * cz);
      if (denom > 1e-5) {
        const double q = (double)((cp - cn) / denom);
        o = (float)(d - fmin(1.0, fmax(-1.0, q)));
      }
    }
    out[id] = o;
  }
}

__device__ void sort_small(float* x, int n) {
  for (int i = 0; i < n - 1; i++) {
    int mn = i;
    for (int j = i + 1; j < n; j++)
      if (x[j] < x[mn]) mn = j;
    const float t = x[mn];
    x[mn] = x[i];
    x[i] = t;
  }
}

// median2d (post.cu:486-518)
__global__ void median_kernel(const float* __restrict__ img, int64_t H, int64_t W, int r,
                              float* __restrict__ out) {
  GRID_STRIDE(id, H * W) {
    const int64_t x = id % W, y = id / W;
    float xs[11 * 11];
    int n = 0;
    for (int64_t xx = x - r; xx <= x + r; xx++)
      for (int64_t yy = y - r; yy <= y + r; yy++)
        if (0 <= xx && xx < W && 0 <= yy && yy < H) xs[n++] = img[yy * W + xx];
    sort_small(xs, n);
    out[id] = xs[n / 2];
  }
}

// mean2d (post.cu:520-566): kernel indexed xx-major as the reference.
__global__ void mean2d_kernel(const float* __restrict__ img, int64_t H, int64_t W,
                              const float* __restrict__ kernel, int r, float alpha2,
                              float* __restrict__ out) {
  GRID_STRIDE(id, H * W) {
    const int64_t x = id % W, y = id / W;
    const float c = img[id];
    float sum = 0.0f, cnt = 0.0f;
    int i = 0;
    for (int64_t xx = x - r; xx <= x + r; xx++)
      for (int64_t yy = y - r; yy <= y + r; yy++, i++)
        if (0 <= xx && xx < W && 0 <= yy && yy < H) {
          const float v = img[yy * W + xx];
          if (fabsf(v - c) < alpha2) {
            sum = fmaf(v, kernel[i], sum);
            cnt += kernel[i];
          }
        }
    out[id] = sum / cnt;
  }
}

// mean2d for kernels up to 15 x 15 (the pipeline's: blur_sigma <= 2.33):
// a 16 x 16 block of pixels stages its (16 + 2r)^2 window of the image in
// shared memory, pixels outside the image as NaN (so the |v - c| < alpha2
// test drops them, as mean2d_kernel's bounds test does), and the weights;
// the taps run in mean2d_kernel's order (xx outer, yy inner) with the same
// fused multiply-add, so the results are the same bit for bit.
constexpr int kMeanTile = 16, kMeanMaxR = 7;
__global__ void __launch_bounds__(kMeanTile * kMeanTile) mean2d_tiled_kernel(const float* __restrict__ img, int H,
                                                                           int W, const float* __restrict__ kernel,
                                                                           int r, float alpha2, float* __restrict__ out) {
  constexpr int TS = kMeanTile + 2 * kMeanMaxR;
  __shared__ float tile[TS][TS + 1];
  __shared__ float kw[(2 * kMeanMaxR + 1) * (2 * kMeanMaxR + 1)];
  const int ks = 2 * r + 1, span = kMeanTile + 2 * r;
  const int X0 = blockIdx.x * kMeanTile, Y0 = blockIdx.y * kMeanTile;
  const int tx = threadIdx.x % kMeanTile, ty = threadIdx.x / kMeanTile;
  for (int q = threadIdx.x; q < ks * ks; q += blockDim.x) kw[q] = kernel[q];
  const float nan = __int_as_float(0x7fc00000);
  for (int q = threadIdx.x; q < span * span; q += blockDim.x) {
    const int ry = q / span, rx = q - ry * span;
    const int yy = Y0 - r + ry, xx = X0 - r + rx;
    tile[ry][rx] = (yy >= 0 && yy < H && xx >= 0 && xx < W) ? img[(int64_t)yy * W + xx] : nan;
  }
  __syncthreads();
  const int x = X0 + tx, y = Y0 + ty;
  if (x >= W || y >= H) return;
  const float c = tile[ty + r][tx + r];
  float sum = 0.0f, cnt = 0.0f;
  int i = 0;
  for (int xo = 0; xo < ks; xo++)
    for (int yo = 0; yo < ks; yo++, i++) {
      const float v = tile[ty + yo][tx + xo];
      if (fabsf(v - c) < alpha2) {
        sum = fmaf(v, kw[i], sum);
        cnt += kw[i];
      }
    }
  out[(int64_t)y * W + x] = sum / cnt;
}

// outlier_detection (post.cu:717-754)
__global__ void outlier_kernel(const float* __restrict__ d0, const float* __restrict__ d1,
                               int64_t H, int64_t W, int disp_max, float* __restrict__ out) {
  GRID_STRIDE(id, H * W) {
    const int64_t x = id % W;
    const int d0i = (int)d0[id];
    float o;
    if (x - d0i < 0 || x - d0i >= W) {  // (>= W only for negative input, where the reference reads out of bounds)
      o = 1;
    } else if (fabsf(d0[id] - d1[id - d0i]) < 1.1) {
      o = 0;
    } else {
      o = 1;
      for (int d = 0; d < disp_max; d++)
        if (x - d >= 0 && fabsf((float)d - d1[id - d]) < 1.1) {
          o = 2;
          break;
        }
    }
    out[id] = o;
  }
}

// interpolate_mismatch (post.cu:757-827).  Where every direction leaves the
// image before meeting a non-mismatch pixel the reference asserts; here the
// pixel keeps its disparity.
__global__ void mismatch_kernel(const float* __restrict__ d0, const float* __restrict__ outlier,
                                int64_t H, int64_t W, float* __restrict__ out) {
  const float dir[32] = {0, 1, -0.5f, 1, -1, 1, -1, 0.5f, -1, 0, -1, -0.5f, -1, -1, -0.5f, -1,
                         0, -1, 0.5f, -1, 1, -1, 1, -0.5f, 1, 0, 1, 0.5f, 1, 1, 0.5f, 1};
  GRID_STRIDE(id, H * W) {
    if (outlier[id] != 2) {
      out[id] = d0[id];
      continue;
    }
    float vals[16];
    int n = 0;
    const int64_t x = id % W, y = id / W;
    for (int k = 0; k < 16; k++) {
      const float dx = dir[2 * k], dy = dir[2 * k + 1];
      float xx = (float)x, yy = (float)y;
      int64_t xi = (int64_t)roundf(xx), yi = (int64_t)roundf(yy);
      while (0 <= yi && yi < H && 0 <= xi && xi < W && outlier[yi * W + xi] == 2) {
        xx += dx;
        yy += dy;
        xi = (int64_t)roundf(xx);
        yi = (int64_t)roundf(yy);
      }
      if (0 <= yi && yi < H && 0 <= xi && xi < W) vals[n++] = d0[yi * W + xi];
    }
    if (n == 0) {
      out[id] = d0[id];
      continue;
    }
    sort_small(vals, n);
    out[id] = vals[n / 2];
  }
}

// interpolate_occlusion (post.cu:829-869)
__global__ void occlusion_kernel(const float* __restrict__ d0, const float* __restrict__ outlier,
                                 int64_t H, int64_t W, float* __restrict__ out) {
  GRID_STRIDE(id, H * W) {
    if (outlier[id] != 1) {
      out[id] = d0[id];
      continue;
    }
    const int64_t x = id % W;
    int64_t dx = 0;
    while (x + dx >= 0 && outlier[id + dx] != 0) dx--;
    if (x + dx < 0) {
      dx = 0;
      while (x + dx < W && outlier[id + dx] != 0) dx++;
    }
    out[id] = (x + dx < W) ? d0[id + dx] : d0[id];
  }
}

// [H*W, D] <-> [D, H*W] tiled transpose of float32.
__global__ void transpose_kernel(const float* __restrict__ in, int64_t rows, int64_t cols,
                                 float* __restrict__ out) {
  __shared__ float tile[32][33];
  const int64_t c0 = (int64_t)blockIdx.x * 32, r0 = (int64_t)blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int64_t r = r0 + k, c = c0 + threadIdx.x;
    if (r < rows && c < cols) tile[k][threadIdx.x] = in[r * cols + c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int64_t c = c0 + k, r = r0 + threadIdx.x;
    if (r < rows && c < cols) out[c * rows + r] = tile[threadIdx.x][k];
  }
}

__global__ void scale_kernel(float* a, int64_t n, float mul) {
  GRID_STRIDE(i, n) a[i] *= mul;
}

__global__ void f64_to_f32_kernel(const double* __restrict__ in, int64_t n, float* __restrict__ out) {
  GRID_STRIDE(i, n) out[i] = (float)in[i];
}

__global__ void f32_to_f64_kernel(const float* __restrict__ in, int64_t n, double* __restrict__ out) {
  GRID_STRIDE(i, n) out[i] = (double)in[i];
}

// Sum and sum of squares of two images (blockIdx.y) as exact 64-bit
// integers, so the result does not depend on the order of the additions:
// summed per block, then two integer atomics on the zeroed mom[2 * image].
// Bytes are read four at a time from the first aligned one on.  694x554: 6.7 us
// for both images (49 us with two atomics per warp and one byte per load).
__global__ void __launch_bounds__(256) moments_kernel(const uint8_t* __restrict__ L, const uint8_t* __restrict__ R,
                                                    int64_t n, unsigned long long* __restrict__ mom) {
  const uint8_t* __restrict__ img = blockIdx.y ? R : L;
  const int64_t head = min(n, (int64_t)(-(intptr_t)img & 3)), words = (n - head) / 4;
  unsigned long long a = 0, b = 0;
  GRID_STRIDE(i, words) {
    const uint32_t v = __ldg(reinterpret_cast<const uint32_t*>(img + head) + i);
    a += __dp4a(v, 0x01010101u, 0u);
    b += __dp4a(v, v, 0u);
  }
  if (blockIdx.x == 0) {
    const int64_t tail = head + 4 * words;
    for (int64_t i = threadIdx.x; i < head + (n - tail); i += 256) {
      const unsigned v = img[i < head ? i : tail + i - head];
      a += v;
      b += v * v;
    }
  }
  __shared__ unsigned long long s[2][8];
  for (int o = 16; o; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s[0][threadIdx.x >> 5] = a;
    s[1][threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    unsigned long long t = 0;
    for (int k = 0; k < 8; k++) t += s[threadIdx.x][k];
    atomicAdd(mom + 2 * blockIdx.y + threadIdx.x, t);
  }
}

// Two images (blockIdx.y): (I - mean) / std in float32 with float32 mean and
// population std, as test.py:489-492 does with numpy on the float32 image,
// and the cross arms of the result (cross_kernel's).  An 8-bit image has 256
// normalised values: each block divides them once, and a pixel's neighbours
// are looked up instead of read from the image the same launch writes.
// words (or null): both images' arm_word, for L1 - 1 <= kMaskHalo.  Bound
// by the arms' chain of dependent reads; both images of 694x554 24 us (77 us
// as four launches), 96x64 5.9 us (19).
__global__ void __launch_bounds__(256) normalise_cross_kernel(const uint8_t* __restrict__ L, const uint8_t* __restrict__ R,
                                                            int64_t H, int64_t W,
                                                            const unsigned long long* __restrict__ mom, int L1, float tau1,
                                                            float* __restrict__ imL, float* __restrict__ imR,
                                                            float* __restrict__ crossL, float* __restrict__ crossR,
                                                            uint32_t* __restrict__ words) {
  __shared__ float value[256];
  const int64_t n = H * W;
  const uint8_t* __restrict__ img = blockIdx.y ? R : L;
  float* __restrict__ out = blockIdx.y ? imR : imL;
  float* __restrict__ arms = blockIdx.y ? crossR : crossL;
  const double mean = (double)mom[2 * blockIdx.y] / (double)n;
  const double var = fmax((double)mom[2 * blockIdx.y + 1] / (double)n - mean * mean, 0.0);
  value[threadIdx.x] = ((float)threadIdx.x - (float)mean) / (float)sqrt(var);
  __syncthreads();
  GRID_STRIDE(p, n) {
    const int64_t y = p / W, x = p - y * W;
    const float c = value[img[p]];
    out[p] = c;
    int reach[4];
#pragma unroll
    for (int dir = 0; dir < 4; dir++) {
      // steps to the image's edge, and the pixel offset of one
      const int64_t room = dir == 0 ? x : dir == 1 ? W - 1 - x : dir == 2 ? y : H - 1 - y;
      const int64_t step = dir == 0 ? -1 : dir == 1 ? 1 : dir == 2 ? -W : W;
      int64_t k = 1;
      for (; k <= room; k++) {
        if (k == 1) continue;
        if (fabsf(c - value[__ldg(img + p + k * step)]) >= tau1) break;  // rule 1
        if (k >= L1) break;                                              // rule 2
      }
      arms[dir * n + p] = (float)((dir <= 1 ? x : y) + ((dir & 1) ? k : -k));
      reach[dir] = (int)k - 1;
    }
    if (words) words[blockIdx.y * n + p] = arm_word(reach[0], reach[1], reach[2], reach[3]);
  }
}

}  // namespace

int launch_cross(const float* img, int64_t H, int64_t W, int L1, float tau1, float* out,
                 cudaStream_t st) {
  cross_kernel<<<grid_for(4 * H * W, kBlock), kBlock, 0, st>>>(img, H, W, L1, tau1, out);
  return check_launch("cross");
}

int launch_sgm_codes(const float* imL, const float* imR, int64_t H, int64_t W, float tau, const SgmCodes& g,
                     cudaStream_t st) {
  sgm_codes_kernel<<<grid_for(2 * ((H + 31) / 32) * ((W + 31) / 32) * 32, 128), 128, 0, st>>>(imL, imR, (int)H, (int)W,
                                                                                              tau, g);
  return check_launch("sgm_codes");
}

template <int KPL, bool FULL, int VEC>
static int sgm_launch(const SgmCodes& g, const float* in, int H, int W, int D, const SgmParams& sp, const SgmOut& o,
                      cudaStream_t st) {
  constexpr int smem = 2 * (sgm_depth<KPL>() + (KPL != VEC)) * sgm_words<KPL, VEC>() * 4;
  static_assert(smem <= 48 * 1024, "no opt-in to more shared memory");
  sgm_kernel<KPL, FULL, VEC><<<(2 * H + 2 * W + 1) / 2, 64, smem, st>>>(g, in, H, W, D, sp, o);
  return check_launch("sgm4");
}

int launch_sgm4(const SgmCodes& g, const float* in, int64_t H, int64_t W, int D, const SgmParams& sp,
                const SgmOut& o, cudaStream_t st) {
  const int h = (int)H, w = (int)W;
  const uintptr_t at = (uintptr_t)in | (uintptr_t)o.dir[0] | (uintptr_t)o.dir[1] | (uintptr_t)o.dir[2] | (uintptr_t)o.dir[3];
  const int vec = D % 4 == 0 && at % 16 == 0 ? 4 : D % 2 == 0 && at % 8 == 0 ? 2 : 1;
  // the fewest disparities per lane that cover D in 32 lanes, rows in the
  // widest vectors that D and the volumes' alignment allow
#define SGM(KPL)                                                                                        \
  if (D <= 32 * KPL) {                                                                                  \
    if (vec == 4 && D == 32 * KPL) return sgm_launch<KPL, true, 4>(g, in, h, w, D, sp, o, st);          \
    if (vec == 4) return sgm_launch<KPL, false, 4>(g, in, h, w, D, sp, o, st);                          \
    if (vec == 2) return sgm_launch<KPL, false, 2>(g, in, h, w, D, sp, o, st);                          \
    return sgm_launch<KPL, false, 1>(g, in, h, w, D, sp, o, st);                                        \
  }
  SGM(1) SGM(2) SGM(3) SGM(4) SGM(5) SGM(6) SGM(7) SGM(8) SGM(10) SGM(12) SGM(16) SGM(24) SGM(32)
#undef SGM
  return set_error(CBMV_ERANGE, "D=%d beyond 1024", D);
}

int launch_sgm_combine(const SgmOut& o, int64_t n, const float* base, float scale, float* out,
                       cudaStream_t st) {
  const uintptr_t at = (uintptr_t)o.dir[0] | (uintptr_t)o.dir[1] | (uintptr_t)o.dir[2] | (uintptr_t)o.dir[3] |
                       (uintptr_t)base | (uintptr_t)out;
  if (n % 4 == 0 && at % 16 == 0) {
    auto f4 = [](const float* p) { return reinterpret_cast<const float4*>(p); };
    sgm_combine_kernel<<<grid_for(n / 4, 256), 256, 0, st>>>(f4(o.dir[0]), f4(o.dir[1]), f4(o.dir[2]), f4(o.dir[3]), n / 4,
                                                             f4(base), scale, reinterpret_cast<float4*>(out));
  } else {
    sgm_combine_kernel<float><<<grid_for(n, 256), 256, 0, st>>>(o.dir[0], o.dir[1], o.dir[2], o.dir[3], n, base, scale,
                                                                out);
  }
  return check_launch("sgm_combine");
}

int launch_cbca(const float* lc, const float* rc, const float* in, int64_t H, int64_t W, int D,
                int layout, int direction, float* out, cudaStream_t st, int halo) {
  if (layout == CBMV_HWD && halo >= 0 && halo <= 8 && H < 32767 && W < 32767) {
    const size_t smem = cbca_smem_bytes(halo);
    CBMV_CUDA(cudaFuncSetAttribute(cbca_hwd_tiled_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)cbca_smem_bytes(8)));
    const int64_t tiles = (int64_t)((W + CB_TX - 1) / CB_TX) * ((H + CB_TY - 1) / CB_TY) *
                          ((D + CB_TD - 1) / CB_TD);
    const unsigned grid = (unsigned)(tiles < (int64_t)1 << 30 ? tiles : (int64_t)1 << 30);
    cbca_hwd_tiled_kernel<<<grid, 256, smem, st>>>(lc, rc, in, (int)H, (int)W, D, direction, halo,
                                                   out);
    return check_launch("cbca_tiled");
  }
  const int64_t dhw_tiles = ((W + CD_X - 1) / CD_X) * ((H + CD_Y - 1) / CD_Y) * ((D + CD_D - 1) / CD_D);
  // A tile takes 30 us however few the tiles are, and its warps are
  // disparities.  us, a thread per output against tiles: 80x60 D=33 13 / 31;
  // 320x240 D=9 34 / 39, D=11 40 / 39, D=16 57 / 41; 694x554 D=3 57 / 63, D=4
  // 74 / 64; 1482x994 D=1 94 / 147, D=2 151 / 152.
  const bool few = H * W * D <= 800000 || (D <= 3 && H * W * D <= 1500000);
  if (layout == CBMV_DHW && !few && H < (1 << 30) && W < (1 << 30) && dhw_tiles < ((int64_t)1 << 31)) {
    cbca_dhw_kernel<<<(unsigned)dhw_tiles, 32 * CD_D, 0, st>>>(lc, rc, in, (int)H, (int)W, D, direction, out);
    if (const int rc_ = check_launch("cbca_dhw")) return rc_;
    int dev = 0, sms = 0;
    CBMV_CUDA(cudaGetDevice(&dev));
    CBMV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // two runs per warp at least: an empty launch costs by its blocks (320x240 D=16, a pass with
    // arms of L1 = 6 and 9: a run per warp 44.5 and 80 us, two 43.4 and 91, three 42.2 and 93)
    const int64_t need = ((W + CD_X - 1) / CD_X * H * D + 15) / 16, blocks = (int64_t)sms * CD_LEFT;
    cbca_dhw_left_kernel<<<(unsigned)(need < blocks ? need : blocks), 256, 0, st>>>(lc, rc, in, (int)H, (int)W, D, direction, out);
    return check_launch("cbca_dhw_left");
  }
  cbca_kernel<<<grid_for(H * W * D, kBlock), kBlock, 0, st>>>(lc, rc, in, H, W, D, layout, direction,
                                                             out);
  return check_launch("cbca");
}

int launch_cbca_sep(const float* lc, const float* rc, const float* in, int64_t H, int64_t W, int D,
                    int direction, float* out, cudaStream_t st, int halo, int rows) {
  CBMV_REQUIRE(H < (1 << 30) && W < (1 << 30) && (int64_t)((W + CS_TX - 1) / CS_TX) * ((H + 15) / 16) *
                   ((D + CS_TD - 1) / CS_TD) < ((int64_t)1 << 31),
               CBMV_ERANGE, "cbca: volume too large");
  switch (halo) {
    case 1: return launch_cbca_sep_h<1>(lc, rc, in, H, W, D, direction, out, st, rows);
    case 2: return launch_cbca_sep_h<2>(lc, rc, in, H, W, D, direction, out, st, rows);
    case 3: return launch_cbca_sep_h<3>(lc, rc, in, H, W, D, direction, out, st, rows);
    case 4: return launch_cbca_sep_h<4>(lc, rc, in, H, W, D, direction, out, st, rows);
    case 5: return launch_cbca_sep_h<5>(lc, rc, in, H, W, D, direction, out, st, rows);
    case 6: return launch_cbca_sep_h<6>(lc, rc, in, H, W, D, direction, out, st, rows);
    case 7: return launch_cbca_sep_h<7>(lc, rc, in, H, W, D, direction, out, st, rows);
    case 8: return launch_cbca_sep_h<8>(lc, rc, in, H, W, D, direction, out, st, rows);
    default: return launch_cbca(lc, rc, in, H, W, D, CBMV_HWD, direction, out, st, halo);
  }
}

// Tiles of the separable CBCA's kernels with `rows` rows each.  A tile's
// halo costs 10 rows, so 32 rows are the least work (a pass at 694x554 D=128:
// 192 us, 24 rows 205); below kCbcaFull tiles (two per SM) they leave SMs
// idle and each tile is a longer chain: a pass at 96x64 D=16 with 24 tiles of
// 32 rows 19.6 us, with 96 of 8 rows 5.3.
static unsigned cbca_tiles(int64_t H, int64_t W, int D, int rows) {
  return (unsigned)(((W + CS_TX - 1) / CS_TX) * ((H + rows - 1) / rows) * ((D + CS_TD - 1) / CS_TD));
}
constexpr unsigned kCbcaFull = 296;

int launch_cbca_mask_build(const uint32_t* wl, const uint32_t* wr, int64_t H, int64_t W, int D, int direction,
                           uint32_t* mask, cudaStream_t st) {
  CBMV_REQUIRE(H < (1 << 30) && W < (1 << 30) &&
                   (int64_t)((W + CS_TX - 1) / CS_TX) * ((H + 15) / 16) * ((D + CS_TD - 1) / CS_TD) <
                       ((int64_t)1 << 31),
               CBMV_ERANGE, "cbca: volume too large");
  const unsigned tiles32 = cbca_tiles(H, W, D, 32), tiles8 = cbca_tiles(H, W, D, 8);
  if (tiles32 >= kCbcaFull) cbca_mask_build_kernel<32><<<tiles32, 256, 0, st>>>(wl, wr, (int)H, (int)W, D, direction, mask);
  else cbca_mask_build_kernel<8><<<tiles8, 256, 0, st>>>(wl, wr, (int)H, (int)W, D, direction, mask);
  return check_launch("cbca_mask_build");
}

// at most 16 or 32 tile rows (0: 32), fewer where the volume is too small for
// them to fill the GPU (the results do not depend on them)
int launch_cbca_masked(const uint32_t* mask, const float* in, int64_t H, int64_t W, int D, float* out,
                       cudaStream_t st, int rows) {
  CBMV_REQUIRE(H < (1 << 30) && W < (1 << 30) &&
                   (int64_t)((W + CS_TX - 1) / CS_TX) * ((H + 15) / 16) * ((D + CS_TD - 1) / CS_TD) <
                       ((int64_t)1 << 31),
               CBMV_ERANGE, "cbca: volume too large");
  rows = rows != 16 && cbca_tiles(H, W, D, 32) >= kCbcaFull ? 32 : cbca_tiles(H, W, D, 16) >= kCbcaFull ? 16 : 8;
  if (rows == 8) return launch_cbca_masked_t<8>(mask, in, H, W, D, out, st);
  if (rows == 16) return launch_cbca_masked_t<16>(mask, in, H, W, D, out, st);
  return launch_cbca_masked_t<32>(mask, in, H, W, D, out, st);
}

int launch_wta_subpixel(const float* cost, int64_t H, int64_t W, int D, float* disp_int,
                        float* disp, cudaStream_t st) {
  const unsigned grid = grid_for((H * W + 3) / 4 * 32, 256);
  if (D % 4 == 0 && (uintptr_t)cost % 16 == 0) wta_subpixel_hwd_kernel<4, 4><<<grid, 256, 0, st>>>(cost, H * W, D, disp_int, disp);
  else if (D <= 32) wta_subpixel_hwd_kernel<1, 1><<<grid, 256, 0, st>>>(cost, H * W, D, disp_int, disp);
  else if (D <= 64) wta_subpixel_hwd_kernel<1, 2><<<grid, 256, 0, st>>>(cost, H * W, D, disp_int, disp);
  else wta_subpixel_hwd_kernel<1, 4><<<grid, 256, 0, st>>>(cost, H * W, D, disp_int, disp);
  return check_launch("wta_subpixel");
}

int launch_median(const float* in, int64_t H, int64_t W, int k, float* out, cudaStream_t st) {
  median_kernel<<<grid_for(H * W, kBlock), kBlock, 0, st>>>(in, H, W, k / 2, out);
  return check_launch("median2d");
}

int launch_mean2d(const float* in, int64_t H, int64_t W, const float* kernel, int ks, float alpha2,
                  float* out, cudaStream_t st) {
  if (ks / 2 <= kMeanMaxR && H < 65536 * kMeanTile && W < ((int64_t)1 << 30)) {
    const dim3 grid((unsigned)((W + kMeanTile - 1) / kMeanTile), (unsigned)((H + kMeanTile - 1) / kMeanTile));
    mean2d_tiled_kernel<<<grid, kMeanTile * kMeanTile, 0, st>>>(in, (int)H, (int)W, kernel, ks / 2, alpha2, out);
    return check_launch("mean2d");
  }
  mean2d_kernel<<<grid_for(H * W, kBlock), kBlock, 0, st>>>(in, H, W, kernel, ks / 2, alpha2, out);
  return check_launch("mean2d");
}

int launch_normalise_cross(const uint8_t* L, const uint8_t* R, int64_t H, int64_t W, double* mom, int L1, float tau1,
                           float* imL, float* imR, float* crossL, float* crossR, uint32_t* words, cudaStream_t st) {
  unsigned long long* m = reinterpret_cast<unsigned long long*>(mom);
  const int64_t n = H * W;
  CBMV_CUDA(cudaMemsetAsync(m, 0, 4 * sizeof(unsigned long long), st));
  moments_kernel<<<dim3(grid_for(n / 16 + 1, 256), 2), 256, 0, st>>>(L, R, n, m);
  normalise_cross_kernel<<<dim3(grid_for(n, 256), 2), 256, 0, st>>>(L, R, H, W, m, L1, tau1, imL, imR, crossL, crossR,
                                                                         L1 - 1 <= kMaskHalo ? words : nullptr);
  return check_launch("normalise_cross");
}

// get_right_cost (featextract.cpp:115-152) of a float32 [H,W,D] volume:
// R[y,x,d] = C[y,x+d,d] where x + d < W, else C[0,0,0] (test.py:154).  A CTA
// reads the columns that 64 pixels of 32 disparities need (95) in runs of 32
// disparities and writes the diagonals from shared memory.  Bound by memory;
// 901x600 D=192 237 us (418 reading the
// diagonals; 254 with 128 pixels).
constexpr int kRcX = 64;

__global__ void __launch_bounds__(256) right_cost_f32_kernel(const float* __restrict__ in, int H, int W, int D,
                                                             float* __restrict__ out) {
  __shared__ float tile[kRcX + 31][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ntd = (D + 31) / 32, ntx = (W + kRcX - 1) / kRcX;
  const int64_t t = blockIdx.x;
  const int d0 = (int)(t % ntd) * 32, x0 = (int)(t / ntd % ntx) * kRcX, y = (int)(t / ((int64_t)ntd * ntx));
  const int d = d0 + lane, X = x0 + d0;  // the tile's first source column
  const float fill = __ldg(in);
  if (d < D) {
    const float* row = in + ((int64_t)y * W + X) * D + d;
#pragma unroll 4
    for (int r = warp; r < kRcX + 31; r += 8)
      if (X + r < W) tile[r][lane] = __ldg(row + (int64_t)r * D);
  }
  __syncthreads();
  if (d >= D) return;
  float* dst = out + ((int64_t)y * W + x0) * D + d;
#pragma unroll
  for (int i = warp; i < kRcX; i += 8)
    if (x0 + i < W) dst[(int64_t)i * D] = x0 + i + d < W ? tile[i + lane][lane] : fill;
}

int launch_right_cost_f32(const float* in, int64_t H, int64_t W, int D, float* out, cudaStream_t st) {
  const int64_t tiles = H * ((W + kRcX - 1) / kRcX) * ((D + 31) / 32);
  CBMV_REQUIRE(tiles < ((int64_t)1 << 31) && W < (1 << 30), CBMV_ERANGE, "volume too large for the right view's grid");
  right_cost_f32_kernel<<<(unsigned)tiles, 256, 0, st>>>(in, (int)H, (int)W, D, out);
  return check_launch("right_cost_f32");
}

int launch_outlier(const float* d0, const float* d1, int64_t H, int64_t W, int disp_max, float* out,
                   cudaStream_t st) {
  outlier_kernel<<<grid_for(H * W, kBlock), kBlock, 0, st>>>(d0, d1, H, W, disp_max, out);
  return check_launch("outlier_detection");
}

int launch_mismatch(const float* d0, const float* o, int64_t H, int64_t W, float* out,
                    cudaStream_t st) {
  mismatch_kernel<<<grid_for(H * W, kBlock), kBlock, 0, st>>>(d0, o, H, W, out);
  return check_launch("interpolate_mismatch");
}

int launch_occlusion(const float* d0, const float* o, int64_t H, int64_t W, float* out,
                     cudaStream_t st) {
  occlusion_kernel<<<grid_for(H * W, kBlock), kBlock, 0, st>>>(d0, o, H, W, out);
  return check_launch("interpolate_occlusion");
}

}  // namespace cbmv

using namespace cbmv;

#define REQ_PTR(...) CBMV_REQUIRE(__VA_ARGS__, CBMV_EINVAL, "null pointer argument")
#define REQ_HW(H, W) \
  CBMV_REQUIRE((H) > 0 && (W) > 0 && (H) <= (1 << 30) && (W) <= (1 << 30), CBMV_EINVAL, "bad size")

extern "C" int cbmv_cross(const float* img, int64_t H, int64_t W, int L1, float tau1, float* out,
                          void* stream) {
  REQ_PTR(img && out);
  REQ_HW(H, W);
  return launch_cross(img, H, W, L1, tau1, out, as_stream(stream));
}

static int check_sgm(const float* imL, const float* imR, const float* in, int64_t H, int64_t W, int D, int direction,
                     const float* out) {
  REQ_PTR(imL && imR && in && out);
  REQ_HW(H, W);
  CBMV_REQUIRE(D > 0 && D <= 1024, CBMV_ERANGE, "D=%d not in 1..1024", D);
  CBMV_REQUIRE(in != out, CBMV_EINVAL, "sgm: in and out must differ");
  CBMV_REQUIRE(direction == 1 || direction == -1, CBMV_EINVAL, "direction must be +-1");
  return CBMV_OK;
}

// scratch: the direction volumes, then the image classes
static int run_sgm(const float* imL, const float* imR, const float* in, int64_t H, int64_t W, int D,
                   const SgmParams& sp, float* out, float* scratch, cudaStream_t st) {
  const int64_t V = H * W * D, S = (V + 3) / 4 * 4;  // every volume 16-byte aligned
  SgmOut o{{scratch, scratch + S, scratch + 2 * S, scratch + 3 * S}};
  const SgmCodes g = sgm_codes_at(scratch + 4 * S, H, W);
  int rc = launch_sgm_codes(imL, imR, H, W, sp.tau_so, g, st);
  if (!rc) rc = launch_sgm4(g, in, H, W, D, sp, o, st);
  if (!rc) rc = launch_sgm_combine(o, V, out, 1.0f, out, st);
  return rc;
}

extern "C" int64_t cbmv_sgm_scratch_bytes(int64_t H, int64_t W, int D) {
  if (H <= 0 || W <= 0 || H > (1 << 30) || W > (1 << 30) || D <= 0 || D > 1024) return -1;
  return (int64_t)sizeof(float) * 4 * ((H * W * D + 3) / 4 * 4) + sgm_codes_bytes(H, W);
}

extern "C" int cbmv_sgm_scratch(const float* imL, const float* imR, const float* in, int64_t H, int64_t W, int D,
                                float pi1, float pi2, float tau_so, float alpha1, float q1, float q2, int direction,
                                float* out, void* scratch, void* stream) {
  const int rc = check_sgm(imL, imR, in, H, W, D, direction, out);
  if (rc) return rc;
  REQ_PTR(scratch);
  CBMV_REQUIRE(((uintptr_t)scratch & 15) == 0, CBMV_EINVAL, "sgm: scratch must be 16-byte aligned");
  return run_sgm(imL, imR, in, H, W, D, SgmParams{pi1, pi2, tau_so, alpha1, q1, q2, direction}, out,
                 static_cast<float*>(scratch), as_stream(stream));
}

extern "C" int cbmv_sgm(const float* imL, const float* imR, const float* in, int64_t H, int64_t W,
                        int D, float pi1, float pi2, float tau_so, float alpha1, float q1, float q2,
                        int direction, float* out, void* stream) {
  int rc = check_sgm(imL, imR, in, H, W, D, direction, out);
  if (rc) return rc;
  cudaStream_t st = as_stream(stream);
  float* scratch = nullptr;
  CBMV_CUDA(cudaMallocAsync(&scratch, (size_t)cbmv_sgm_scratch_bytes(H, W, D), st));
  rc = run_sgm(imL, imR, in, H, W, D, SgmParams{pi1, pi2, tau_so, alpha1, q1, q2, direction}, out, scratch, st);
  CBMV_CUDA(cudaFreeAsync(scratch, st));
  return rc;
}

extern "C" int cbmv_cbca(const float* crossL, const float* crossR, const float* in, int64_t H,
                         int64_t W, int D, int layout, int direction, float* out, void* stream) {
  REQ_PTR(crossL && crossR && in && out);
  REQ_HW(H, W);
  CBMV_REQUIRE(D > 0, CBMV_EINVAL, "bad D");
  CBMV_REQUIRE(in != out, CBMV_EINVAL, "cbca: in and out must differ");
  CBMV_REQUIRE(direction == 1 || direction == -1, CBMV_EINVAL, "direction must be +-1");
  CBMV_REQUIRE(layout == CBMV_HWD || layout == CBMV_DHW, CBMV_EINVAL, "bad layout");
  return launch_cbca(crossL, crossR, in, H, W, D, layout, direction, out, as_stream(stream));
}

extern "C" int cbmv_cbca_separable(const float* crossL, const float* crossR, const float* in, int64_t H,
                                   int64_t W, int D, int L1, int direction, float* out, void* stream) {
  REQ_PTR(crossL && crossR && in && out);
  REQ_HW(H, W);
  CBMV_REQUIRE(D > 0, CBMV_EINVAL, "bad D");
  CBMV_REQUIRE(in != out, CBMV_EINVAL, "cbca: in and out must differ");
  CBMV_REQUIRE(direction == 1 || direction == -1, CBMV_EINVAL, "direction must be +-1");
  CBMV_REQUIRE(L1 >= 2 && L1 <= 9, CBMV_EINVAL, "cbca_separable: L1 must be in 2..9");
  cudaStream_t st = as_stream(stream);
  if (L1 - 1 > kCbcaMaskMaxHalo) return launch_cbca_sep(crossL, crossR, in, H, W, D, direction, out, st, L1 - 1);
  // the pipeline's form: supports precomputed into a stream-ordered scratch buffer
  uint32_t* mask = nullptr;
  CBMV_CUDA(cudaMallocAsync(&mask, sizeof(uint32_t) * (H * W * (D + 2) + 1), st));
  uint32_t *words = mask + H * W * D, *odd = words + 2 * H * W;
  cudaMemsetAsync(odd, 0, sizeof(uint32_t), st);
  arm_words_kernel<<<dim3(grid_for(H * W, kBlock), 2), kBlock, 0, st>>>(crossL, crossR, H, W, words, odd);
  int rc = check_launch("arm_words");
  if (rc == CBMV_OK) rc = launch_cbca_mask_build(words, words + H * W, H, W, D, direction, mask, st);
  if (rc == CBMV_OK) {
    cbca_mask_any_kernel<<<grid_for(H * W * D, kBlock), kBlock, 0, st>>>(crossL, crossR, H, W, D, direction, odd, mask);
    rc = check_launch("cbca_mask_any");
  }
  if (rc == CBMV_OK) rc = launch_cbca_masked(mask, in, H, W, D, out, st);
  CBMV_CUDA(cudaFreeAsync(mask, st));
  return rc;
}

extern "C" int cbmv_wta(const float* cost, int64_t H, int64_t W, int D, int layout, float* disp,
                        void* stream) {
  REQ_PTR(cost && disp);
  REQ_HW(H, W);
  CBMV_REQUIRE(D > 0, CBMV_EINVAL, "bad D");
  if (layout == CBMV_HWD) return launch_wta_subpixel(cost, H, W, D, disp, nullptr, as_stream(stream));
  wta_dhw_kernel<<<grid_for(H * W, kBlock), kBlock, 0, as_stream(stream)>>>(cost, H * W, D, disp);
  return check_launch("wta");
}

extern "C" int cbmv_subpixel(const float* disp, const float* cost, int64_t H, int64_t W, int D,
                             int layout, float* out, void* stream) {
  REQ_PTR(disp && cost && out);
  REQ_HW(H, W);
  CBMV_REQUIRE(D > 0, CBMV_EINVAL, "bad D");
  subpixel_kernel<<<grid_for(H * W, kBlock), kBlock, 0, as_stream(stream)>>>(disp, cost, H, W, D, layout,
                                                                            out);
  return check_launch("subpixel");
}

extern "C" int cbmv_median2d(const float* in, int64_t H, int64_t W, int k, float* out,
                             void* stream) {
  REQ_PTR(in && out);
  REQ_HW(H, W);
  CBMV_REQUIRE(k >= 1 && k <= 11 && (k & 1), CBMV_EINVAL, "median window %d must be odd <= 11", k);
  CBMV_REQUIRE(in != out, CBMV_EINVAL, "median2d: in and out must differ");
  return launch_median(in, H, W, k, out, as_stream(stream));
}

extern "C" int cbmv_mean2d(const float* in, int64_t H, int64_t W, const float* kernel, int ks,
                           float alpha2, float* out, void* stream) {
  REQ_PTR(in && out && kernel);
  REQ_HW(H, W);
  CBMV_REQUIRE(ks >= 1 && ks <= 31 && (ks & 1), CBMV_EINVAL, "kernel size %d must be odd <= 31", ks);
  CBMV_REQUIRE(in != out, CBMV_EINVAL, "mean2d: in and out must differ");
  return launch_mean2d(in, H, W, kernel, ks, alpha2, out, as_stream(stream));
}

extern "C" int cbmv_outlier_detection(const float* d0, const float* d1, int64_t H, int64_t W,
                                      int disp_max, float* out, void* stream) {
  REQ_PTR(d0 && d1 && out);
  REQ_HW(H, W);
  return launch_outlier(d0, d1, H, W, disp_max, out, as_stream(stream));
}

extern "C" int cbmv_interpolate_mismatch(const float* d0, const float* outlier, int64_t H,
                                         int64_t W, float* out, void* stream) {
  REQ_PTR(d0 && outlier && out);
  REQ_HW(H, W);
  CBMV_REQUIRE(d0 != out, CBMV_EINVAL, "in and out must differ");
  return launch_mismatch(d0, outlier, H, W, out, as_stream(stream));
}

extern "C" int cbmv_interpolate_occlusion(const float* d0, const float* outlier, int64_t H,
                                          int64_t W, float* out, void* stream) {
  REQ_PTR(d0 && outlier && out);
  REQ_HW(H, W);
  CBMV_REQUIRE(d0 != out, CBMV_EINVAL, "in and out must differ");
  return launch_occlusion(d0, outlier, H, W, out, as_stream(stream));
}

extern "C" int cbmv_transpose_f32(const float* in, int64_t H, int64_t W, int64_t D, int to_layout,
                                  float* out, void* stream) {
  REQ_PTR(in && out);
  CBMV_REQUIRE(H > 0 && W > 0 && D > 0 && in != out, CBMV_EINVAL, "bad argument");
  const int64_t rows = to_layout == CBMV_DHW ? H * W : D;
  const int64_t cols = to_layout == CBMV_DHW ? D : H * W;
  CBMV_REQUIRE((rows + 31) / 32 <= 65535, CBMV_ERANGE, "volume too large for the transpose grid");
  dim3 grid((unsigned)((cols + 31) / 32), (unsigned)((rows + 31) / 32));
  transpose_kernel<<<grid, dim3(32, 8), 0, as_stream(stream)>>>(in, rows, cols, out);
  return check_launch("transpose");
}

extern "C" int cbmv_scale_f32(float* a, int64_t n, float mul, void* stream) {
  REQ_PTR(a);
  CBMV_REQUIRE(n >= 0, CBMV_EINVAL, "bad size");
  if (n == 0) return CBMV_OK;
  scale_kernel<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(a, n, mul);
  return check_launch("scale");
}

extern "C" int cbmv_f64_to_f32(const double* in, int64_t n, float* out, void* stream) {
  REQ_PTR(in && out);
  if (n <= 0) return n == 0 ? CBMV_OK : set_error(CBMV_EINVAL, "bad size");
  f64_to_f32_kernel<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(in, n, out);
  return check_launch("f64_to_f32");
}

extern "C" int cbmv_f32_to_f64(const float* in, int64_t n, double* out, void* stream) {
  REQ_PTR(in && out);
  if (n <= 0) return n == 0 ? CBMV_OK : set_error(CBMV_EINVAL, "bad size");
  f32_to_f64_kernel<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(in, n, out);
  return check_launch("f32_to_f64");
}
