// BF16 tensor-core kernels of the learned matching-probability classifier
// (the MLP surrogate of the reference's random forest, test.py:603-620):
// a general C = A * B^T GEMM on tcgen05, and the trainer's two kernels.
//
// Every CTA computes a 128-row x N tile: the K dimension streams through
// shared memory in 64-wide, 128-byte-swizzled chunks (umma.cuh), one thread
// issues four 128xNx16 MMAs per chunk into a float32 accumulator in tensor
// memory, and the epilogue reads it back with tcgen05.ld (warp w owns rows
// 32w..32w+31).  Waits on the MMA-completion barrier are bounded: on a
// timeout the kernel records an error in `status` and returns.
#include <cuda_bf16.h>

#include <cooperative_groups.h>

#include "common.cuh"
#include "mlp_net.cuh"
#include "umma.cuh"

namespace cbmv {
namespace {

template <int NT>
__global__ void __launch_bounds__(128) gemm_bf16_kernel(const uint16_t* __restrict__ A,
                                                         const uint16_t* __restrict__ B,
                                                         float* __restrict__ C, int M, int N, int K,
                                                         int* __restrict__ status) {
  constexpr int kTmemCols = NT < 32 ? 32 : NT;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // 1024-byte aligned operand tiles: A 128x64, B NTx64 bf16
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sA = base;
  unsigned char* sB = base + 128 * 128;
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int m0 = blockIdx.x * 128;
  const int n0 = blockIdx.y * NT;

  if (warp == 0) umma::tmem_alloc(&tmem_base, kTmemCols);
  if (tid == 0) umma::mbar_init(&bar, 1);
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = tmem_base;
  const uint32_t idesc = umma::idesc_bf16(128, NT);
  bool ok = true;
  uint32_t phase = 0;

  for (int k0 = 0; k0 < K && ok; k0 += 64) {
    // stage A[m0:m0+128, k0:k0+64] and B[n0:n0+NT, k0:k0+64], 16 B per thread-step
    for (int q = tid; q < 128 * 8; q += 128) {
      const int r = q >> 3, c = q & 7;
      const uint4 v = *reinterpret_cast<const uint4*>(A + (size_t)(m0 + r) * K + k0 + c * 8);
      *reinterpret_cast<uint4*>(sA + umma::sw128_offset(128, r, c * 8)) = v;
    }
    for (int q = tid; q < NT * 8; q += 128) {
      const int r = q >> 3, c = q & 7;
      const uint4 v = *reinterpret_cast<const uint4*>(B + (size_t)(n0 + r) * K + k0 + c * 8);
      *reinterpret_cast<uint4*>(sB + umma::sw128_offset(NT, r, c * 8)) = v;
    }
    umma::fence_async_smem();
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    if (tid == 0) {
      const uint64_t da = umma::sw128_desc(umma::smem_u32(sA));
      const uint64_t db = umma::sw128_desc(umma::smem_u32(sB));
#pragma unroll
      for (int kk = 0; kk < 4; kk++)  // 16-wide K steps: +32 B = +2 in descriptor units
        umma::mma_bf16(tmem, da + 2 * kk, db + 2 * kk, idesc, k0 > 0 || kk > 0);
      umma::mma_commit(&bar);
    }
    ok = umma::mbar_wait(&bar, phase, kWaitLimit);
    phase ^= 1u;
    umma::tc_fence_after();
  }
  if (!ok) {
    if (tid == 0) atomicExch(status, 1);
    // let the MMAs still in flight finish (bounded) before freeing their memory
    umma::mbar_wait(&bar, phase ^ 1u, kWaitLimit);
  } else {
    // epilogue: warp w reads rows 32w..32w+31, 16 columns at a time
    const int row = m0 + warp * 32 + (tid & 31);
    for (int c0 = 0; c0 < NT; c0 += 16) {
      float v[16];
      umma::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + c0, v);
      float* dst = C + (size_t)row * N + n0 + c0;
#pragma unroll
      for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    }
  }
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, kTmemCols);
}

template <int NT>
int launch_gemm(const uint16_t* A, const uint16_t* B, float* C, int M, int N, int K, int* status,
                cudaStream_t st) {
  const size_t smem = 1024 + 128 * 128 + (size_t)NT * 128;
  CBMV_CUDA(cudaFuncSetAttribute(gemm_bf16_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  dim3 grid(M / 128, N / NT);
  gemm_bf16_kernel<NT><<<grid, 128, smem, st>>>(A, B, C, M, N, K, status);
  return check_launch("gemm_bf16");
}

}  // namespace

int launch_gemm_bf16(const uint16_t* A, const uint16_t* B, float* C, int M, int N, int K, int* status,
                     cudaStream_t st) {
  if (N % 128 == 0) return launch_gemm<128>(A, B, C, M, N, K, status, st);
  if (N % 64 == 0) return launch_gemm<64>(A, B, C, M, N, K, status, st);
  return launch_gemm<32>(A, B, C, M, N, K, status, st);
}

}  // namespace cbmv

using namespace cbmv;

extern "C" int cbmv_gemm_bf16(const uint16_t* A, const uint16_t* B, float* C, int64_t M, int64_t N,
                              int64_t K, int* status, void* stream) {
  CBMV_REQUIRE(A && B && C && status, CBMV_EINVAL, "null pointer argument");
  CBMV_REQUIRE(M > 0 && N > 0 && K > 0 && M % 128 == 0 && N % 32 == 0 && K % 64 == 0, CBMV_EINVAL,
               "gemm_bf16 needs M %% 128 == 0, N %% 32 == 0, K %% 64 == 0 (got %lld, %lld, %lld)",
               (long long)M, (long long)N, (long long)K);
  CBMV_REQUIRE(M < (1ll << 31) && N <= 65535 * 32 && K < (1 << 30), CBMV_ERANGE, "gemm too large");
  CBMV_REQUIRE(((uintptr_t)A & 15) == 0 && ((uintptr_t)B & 15) == 0 && ((uintptr_t)C & 15) == 0,
               CBMV_EINVAL, "gemm_bf16 operands must be 16-byte aligned");
  return launch_gemm_bf16(A, B, C, (int)M, (int)N, (int)K, status, as_stream(stream));
}

// ====================================================================
// Training: 20 -> 128 -> 128 -> 64 -> 1, GELU or ReLU, sigmoid output.
// Parameter vector (float32, host order):
//   cap[20] mu[20] inv_sd[20]        input transform x' = (min(x,cap)-mu)*inv_sd
//   W1[128x20] b1[128] W2[128x128] b2[128] W3[64x128] b3[64] w4[64] b4[1]
// float32 master weights (Adam), bfloat16 GEMM operands, float32
// accumulation.
//
// Two launches.  A batch of 8192 is 1.3 GFLOP on 0.7 MB of samples, so
// nothing but latency bounds it: as 24 launches with every intermediate in
// HBM it took 7.99 ms, 6.5 of it in the bias gradients (one block, one
// thread per column walking the whole batch) and 1.3 in GEMMs whose one or
// two CTAs staged the batch as their K dimension.
//
// mlp_train_kernel runs forward and backward of 128-sample tiles; the
// activations of a tile never leave the SM between layers:
//   shared memory  the bf16 weights (64 KB), the tile's X0, A1, A2 and dS3;
//                  dS2 and dS1 take the place of A2 and A1 once the MMAs that
//                  read those have completed
//   tensor memory  the accumulator [128 x 128] and the f16 arguments of the
//                  two 128-wide activations (what their derivatives need)
// The input gradients contract over a layer's outputs by reading the same
// K-major weight tiles as MN-major operands (umma.cuh, sw128_desc_mn).  The
// bias gradients are column sums of the float32 deltas, reduced over a
// warp's 32 rows by a 31-step exchange per 32 columns.
//
// Four threads take a row, 16 warps: with two threads and 8 warps a tile's
// chain of epilogues took 24.5 us, now 19.
//
// mlp_wgrad_kernel forms the weight gradients, contractions over the batch,
// from the operand tiles the first kernel stored as they were (bulk copies
// both ways, swizzle included): a CTA owns a 64 x 64 block of dW1, dW2 or
// dW3^T and streams the tiles through a ring of stages, bound by what one SM
// takes in, 32 KB per tile at 0.44 us.  From 8 to 64 tiles a cluster of four
// CTAs splits a block's tiles and adds the four sums through distributed
// shared memory (at 8192 samples 29 -> 13.5 us); fewer tiles are too short a
// chain, and above 64 a block stays one accumulator chain in sample order:
// the tensor core truncates, so split sums, though nearer to float64, move
// away from the single chain's (1.0e-5 relative at 8192, 6e-5 at 32768).  Its
// CTAs are set up while the first kernel runs (programmatic launch).
// Measured, forward and backward of one batch: 25 us at 128 samples, 33 us
// at 8192 (7.99 ms as 24 launches), 147 us at 32768.
// All sums have a fixed order, so a batch gives the same gradients every time.
// ====================================================================
namespace cbmv {
namespace {

constexpr int kTrainThreads = 512;  // four threads per tile row, each a quarter of the columns
// a CTA's share of the sums over the samples: db1, db2, db3, dw4, db4, loss
constexpr int kSums = kH1 + kH2 + 2 * kH3 + 2;

// shared memory: the operand tiles of one 128-sample tile, in the order
// they are stored for the weight gradients, then the weights
constexpr uint32_t kAtom = 128 * 128;  // one SW128 atom of 128 rows x 64 columns
constexpr uint32_t kTX0 = 0, kTA1 = kTX0 + kAtom, kTA2 = kTA1 + 2 * kAtom, kTD3 = kTA2 + 2 * kAtom,
                   kTW1 = kTD3 + kAtom, kTW2 = kTW1 + kAtom, kTW3 = kTW2 + 2 * kAtom, kTEnd = kTW3 + kAtom;
constexpr uint32_t kTScr = kTEnd;  // [32][128] floats of the output layer's dot products
constexpr size_t kSmTrain = 1024 + kTScr + 32 * 128 * 4;
// the stored image of a tile: X0, A1, A2, dS3, dS2, dS1
constexpr uint32_t kID2 = kTD3 + kAtom, kID1 = kID2 + 2 * kAtom, kImage = kID1 + 2 * kAtom;
// tensor-memory columns
constexpr uint32_t kCAcc = 0, kCS1 = 128, kCS2 = 192, kTrainCols = 256;

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 x = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&x);
}

// eight consecutive float32 weights -> one 16-byte chunk of a K-major tile
__device__ __forceinline__ void stage8(unsigned char* dst, const float* __restrict__ src) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(src)), b = __ldg(reinterpret_cast<const float4*>(src) + 1);
  *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
}

// The activation of two pre-activations as bf16, and in *s what its
// derivative needs, as two f16 values: the GELU's argument, the ReLU's 0/1.
template <int ACT>
__device__ __forceinline__ uint32_t train_act(float a, float b, uint32_t* s, float2* f = nullptr) {
  float2 v;
  __half2 arg;
  if (ACT == CBMV_ACT_GELU) {
    arg = gelu_arg(a, b);
    v = __half22float2(gelu_f16x2(arg));
  } else {
    v = make_float2(a > 0.0f ? a : 0.0f, b > 0.0f ? b : 0.0f);
    arg = __floats2half2_rn(a > 0.0f ? 1.0f : 0.0f, b > 0.0f ? 1.0f : 0.0f);
  }
  *s = *reinterpret_cast<const uint32_t*>(&arg);
  if (f) *f = v;
  return pack_bf16(v.x, v.y);
}

template <int ACT>
__device__ __forceinline__ float2 train_grad(uint32_t s) {
  const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&s));
  return ACT == CBMV_ACT_GELU ? make_float2(gelu_grad(x.x), gelu_grad(x.y)) : x;
}

// Sums over the warp's lanes of N values each (32 or 16): lane l receives the
// sum of v[l % N].  Every step exchanges one half of the remaining values (31
// shuffles); 16 values are first added across the half-warps.
template <int N>
__device__ __forceinline__ float warp_colsum(float (&v)[N], int lane) {
  if (N == 16)
#pragma unroll
    for (int i = 0; i < N; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i], 16);
#pragma unroll
  for (int o = N / 2; o; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; i++) {
      const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

template <int ACT>
__global__ void __launch_bounds__(kTrainThreads, 1)
    mlp_train_kernel(const float* __restrict__ X, const float* __restrict__ y, const float* __restrict__ P, int B,
                     unsigned char* __restrict__ images, float* __restrict__ sums, int* __restrict__ status) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ float s_nrm[kNormN], s_b1[kH1], s_b2[kH2], s_b3[kH3], s_w4[kH3];
  __shared__ float s_b4, s_z[128];
  __shared__ float s_red[4][kSums];
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, lane = tid & 31, quad = (tid >> 5) & 3, part = tid >> 7, row = tid & 127;

  // the weight gradients' CTAs may take free SMs and set up; they wait for this grid's end
  asm volatile("griddepcontrol.launch_dependents;");
  if (tid < 32) umma::tmem_alloc(&tmem_base, kTrainCols);
  if (tid == 0) umma::mbar_init(&bar, 1);
  // weights, K-major; columns of X0 and W1 beyond the 20 features are zero
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (int q = tid; q < kH1 * 4; q += kTrainThreads) {
    const int r = q >> 2, k = (q & 3) * 8;
    unsigned char* dst = base + kTW1 + umma::sw128_offset(128, r, k);
    if (k + 8 <= kF) {
      stage8(dst, P + kOffW1 + r * kF + k);
    } else {
      const float* w = P + kOffW1 + r * kF + k;
      *reinterpret_cast<uint4*>(dst) = k < kF ? make_uint4(pack_bf16(w[0], w[1]), pack_bf16(w[2], w[3]), 0u, 0u) : zero;
    }
  }
  for (int q = tid; q < kH2 * 16; q += kTrainThreads) {
    const int r = q >> 4, k = (q & 15) * 8;
    stage8(base + kTW2 + umma::sw128_offset(128, r, k), P + kOffW2 + r * kH1 + k);
  }
  for (int q = tid; q < kH3 * 16; q += kTrainThreads) {
    const int r = q >> 4, k = (q & 15) * 8;
    stage8(base + kTW3 + umma::sw128_offset(64, r, k), P + kOffW3 + r * kH2 + k);
  }
  *reinterpret_cast<uint4*>(base + kTX0 + umma::sw128_offset(128, row, 8 * (4 + part))) = zero;
  if (tid < kNormN) s_nrm[tid] = P[tid];
  if (tid < kH1) s_b1[tid] = P[kOffB1 + tid];
  if (tid < kH2) s_b2[tid] = P[kOffB2 + tid];
  if (tid < kH3) s_b3[tid] = P[kOffB3 + tid];
  if (tid < kH3) s_w4[tid] = P[kOffW4 + tid];
  if (tid == 0) s_b4 = P[kOffB4];
  umma::fence_async_smem();
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();

  const uint32_t tm = tmem_base, tlane = tm + ((uint32_t)(quad * 32) << 16);
  const uint32_t sb = umma::smem_u32(base);
  const int r7s = (row & 7) << 4;
  // 16-byte chunk holding columns c .. c+7 of this thread's row of a 128-row tile
  auto chunk = [&](uint32_t tile, int c) {
    return reinterpret_cast<uint4*>(base + tile + (c >> 6) * kAtom + (row >> 3) * 1024 + (row & 7) * 128 +
                                    ((((c & 63) >> 3) << 4) ^ r7s));
  };
  uint32_t phase = 0;
  bool ok = true;
  auto handoff = [&]() {  // the threads' shared- and tensor-memory accesses before the next MMAs
    umma::fence_async_smem();
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
  };
  // the leader waits for the MMAs, another warp's first thread for its stores
  // to have read the tiles that are overwritten next
  constexpr int kStorer = 32;
  auto wait = [&]() {
    if (tid == kStorer) umma::bulk_wait_read();
    const int r = __syncthreads_and(tid == 0 ? umma::mbar_wait(&bar, phase, kWaitLimit) : 1);
    phase ^= 1u;
    umma::tc_fence_after();
    return r != 0;
  };
  // column sums of this CTA's tiles (warp `quad` of each quarter): db1 and
  // db2 column 32*part + lane, db3 and dw4 column 16*part + lane % 16
  float db1 = 0.0f, db2 = 0.0f, db3 = 0.0f, dw4 = 0.0f, db4 = 0.0f, loss = 0.0f;

  // hidden layer: accumulator + bias -> activation (bf16 tile) and its argument (f16, tensor memory)
  auto forward = [&](const float* bias, uint32_t tile, uint32_t args) {
#pragma unroll
    for (int c0 = 0; c0 < 32; c0 += 16) {
      const int c = 32 * part + c0;
      uint32_t v[16], s[8], a[8];
      umma::tmem_ld16_issue(tlane + kCAcc + c, v);
      umma::tmem_ld16_wait(v);
#pragma unroll
      for (int i = 0; i < 8; i++)
        a[i] = train_act<ACT>(__uint_as_float(v[2 * i]) + bias[c + 2 * i], __uint_as_float(v[2 * i + 1]) + bias[c + 2 * i + 1], &s[i]);
      *chunk(tile, c) = make_uint4(a[0], a[1], a[2], a[3]);
      *chunk(tile, c + 8) = make_uint4(a[4], a[5], a[6], a[7]);
      umma::tmem_st8(tlane + args + c / 2, s);
    }
    umma::tmem_st_wait();
  };
  // dS = dA * act'(S) -> bf16 tile, and its column sums
  auto backward = [&](uint32_t tile, uint32_t args, float& db) {
    const int c = 32 * part;
    float d[32];
    {
      uint32_t v[32], s[16];
      umma::tmem_ld32_issue(tlane + kCAcc + c, v);
      umma::tmem_ld16_issue(tlane + args + c / 2, s);
      umma::tmem_ld32_wait(v);
      umma::tmem_ld16_wait(s);
#pragma unroll
      for (int i = 0; i < 16; i++) {
        const float2 g = train_grad<ACT>(s[i]);
        d[2 * i] = __uint_as_float(v[2 * i]) * g.x;
        d[2 * i + 1] = __uint_as_float(v[2 * i + 1]) * g.y;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
      *chunk(tile, c + 8 * i) = make_uint4(pack_bf16(d[8 * i], d[8 * i + 1]), pack_bf16(d[8 * i + 2], d[8 * i + 3]),
                                           pack_bf16(d[8 * i + 4], d[8 * i + 5]), pack_bf16(d[8 * i + 6], d[8 * i + 7]));
    db += warp_colsum(d, lane);
  };
  constexpr uint32_t id128 = umma::idesc_bf16(128, 128), id64 = umma::idesc_bf16(128, 64);

  const int tiles = B / 128;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    unsigned char* image = images + (size_t)tile * kImage;
    auto store = [&](uint32_t at, uint32_t smem, uint32_t bytes) {
      if (tid == kStorer) umma::bulk_store(image + at, sb + smem, bytes);
    };
    const int64_t b = (int64_t)tile * 128 + row;
    float x[8];
    const int k0 = 8 * part;
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = k0 + k < kF ? X[b * kF + k0 + k] : 0.0f;
    const float yy = y[b];
    // 1. normalised bf16 inputs
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (k0 + k < kF) x[k] = (fminf(x[k], s_nrm[k0 + k]) - s_nrm[kF + k0 + k]) * s_nrm[2 * kF + k0 + k];
    *chunk(kTX0, k0) = make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
    handoff();
    store(kTX0, kTX0, kAtom);
    // 2. layer 1 (K = 32)
    if (tid == 0) {
      const uint64_t da = umma::sw128_desc(sb + kTX0), dw = umma::sw128_desc(sb + kTW1);
      umma::mma_bf16(tm + kCAcc, da, dw, id128, false);
      umma::mma_bf16(tm + kCAcc, da + 2, dw + 2, id128, true);
      umma::mma_commit(&bar);
    }
    if (!(ok = wait())) break;
    forward(s_b1, kTA1, kCS1);
    handoff();
    store(kTA1, kTA1, 2 * kAtom);
    // 3. layer 2
    if (tid == 0) {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const uint32_t o = (k >> 2) * kAtom + (k & 3) * 32;
        umma::mma_bf16(tm + kCAcc, umma::sw128_desc(sb + kTA1 + o), umma::sw128_desc(sb + kTW2 + o), id128, k > 0);
      }
      umma::mma_commit(&bar);
    }
    if (!(ok = wait())) break;
    forward(s_b2, kTA2, kCS2);
    handoff();
    store(kTA2, kTA2, 2 * kAtom);
    // 4. layer 3
    if (tid == 0) {
#pragma unroll
      for (int k = 0; k < 8; k++)
        umma::mma_bf16(tm + kCAcc, umma::sw128_desc(sb + kTA2 + (k >> 2) * kAtom + (k & 3) * 32),
                       umma::sw128_desc(sb + kTW3 + (k >> 2) * 64 * 128 + (k & 3) * 32), id64, k > 0);
      umma::mma_commit(&bar);
    }
    if (!(ok = wait())) break;
    // 5. output layer, loss, dS3 = dz w4 act'(S3).  The row's dot product is
    //    summed in the order of a 32-lane exchange over
    //    fma(a[l], w[l], a[l+32] w[l+32]): the quarters 2 and 3 hand their
    //    products to 0 and 1, quarter 1 its sums to 0.
    {
      const int c = 16 * part;
      float a3[16];
      uint32_t s3[8];
      float* scr = reinterpret_cast<float*>(base + kTScr) + (part & 1) * 16 * 128 + row;
      {
        uint32_t v[16];
        umma::tmem_ld16_issue(tlane + kCAcc + c, v);
        umma::tmem_ld16_wait(v);
#pragma unroll
        for (int i = 0; i < 8; i++) {
          float2 f;
          train_act<ACT>(__uint_as_float(v[2 * i]) + s_b3[c + 2 * i], __uint_as_float(v[2 * i + 1]) + s_b3[c + 2 * i + 1], &s3[i], &f);
          a3[2 * i] = f.x;
          a3[2 * i + 1] = f.y;
        }
      }
      if (part >= 2)
#pragma unroll
        for (int i = 0; i < 16; i++) scr[i * 128] = a3[i] * s_w4[c + i];
      __syncthreads();
      float t[16];
      if (part < 2)
#pragma unroll
        for (int i = 0; i < 16; i++) t[i] = fmaf(a3[i], s_w4[c + i], scr[i * 128]);
      if (part == 1)
#pragma unroll
        for (int i = 0; i < 16; i++) scr[i * 128] = t[i];
      __syncthreads();
      if (part == 0) {
#pragma unroll
        for (int i = 0; i < 16; i++) t[i] += scr[(16 + i) * 128];
#pragma unroll
        for (int o = 8; o; o >>= 1)
#pragma unroll
          for (int i = 0; i < o; i++) t[i] += t[i + o];
        s_z[row] = t[0] + s_b4;
      }
      __syncthreads();
      const float z = s_z[row];
      const float prob = 1.0f / (1.0f + expf(-z));
      // BCE with logits, stable form
      const float l = fmaxf(z, 0.0f) - z * yy + log1pf(expf(-fabsf(z)));
      const float g = (prob - yy) / (float)B;
      loss += l / (float)B;
      db4 += g;
      float d[16];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float2 dg = train_grad<ACT>(s3[i]);
        d[2 * i] = g * s_w4[c + 2 * i] * dg.x;
        d[2 * i + 1] = g * s_w4[c + 2 * i + 1] * dg.y;
        a3[2 * i] *= g;
        a3[2 * i + 1] *= g;
      }
#pragma unroll
      for (int i = 0; i < 2; i++)
        *chunk(kTD3, c + 8 * i) =
            make_uint4(pack_bf16(d[8 * i], d[8 * i + 1]), pack_bf16(d[8 * i + 2], d[8 * i + 3]),
                       pack_bf16(d[8 * i + 4], d[8 * i + 5]), pack_bf16(d[8 * i + 6], d[8 * i + 7]));
      db3 += warp_colsum(d, lane);
      dw4 += warp_colsum(a3, lane);
    }
    handoff();
    store(kTD3, kTD3, kAtom);
    // 6. dA2 = dS3 W3; dS2 takes A2's place
    if (tid == 0) {
#pragma unroll
      for (int k = 0; k < 4; k++)
        umma::mma_bf16(tm + kCAcc, umma::sw128_desc(sb + kTD3 + 32 * k), umma::sw128_desc_mn(sb + kTW3 + 2048 * k, 64),
                       id128 | umma::kTransposeB, k > 0);
      umma::mma_commit(&bar);
    }
    if (!(ok = wait())) break;
    backward(kTA2, kCS2, db2);
    handoff();
    store(kID2, kTA2, 2 * kAtom);
    // 7. dA1 = dS2 W2; dS1 takes A1's place
    if (tid == 0) {
#pragma unroll
      for (int k = 0; k < 8; k++)
        umma::mma_bf16(tm + kCAcc, umma::sw128_desc(sb + kTA2 + (k >> 2) * kAtom + (k & 3) * 32),
                       umma::sw128_desc_mn(sb + kTW2 + 2048 * k, 128), id128 | umma::kTransposeB, k > 0);
      umma::mma_commit(&bar);
    }
    if (!(ok = wait())) break;
    backward(kTA1, kCS1, db1);
    handoff();
    store(kID1, kTA1, 2 * kAtom);
  }
  if (!ok && tid == 0) {
    // a wait gave up: record it and let the MMAs in flight finish (bounded)
    // before their memory is freed
    atomicExch(status, 1);
    umma::mbar_wait(&bar, phase ^ 1u, kWaitLimit);
  }
  // the four warps of a quarter cover the tile's rows: their column sums added in order
  s_red[quad][32 * part + lane] = db1;
  s_red[quad][kH1 + 32 * part + lane] = db2;
  if (lane < 16) {
    s_red[quad][kH1 + kH2 + 16 * part + lane] = db3;
    s_red[quad][kH1 + kH2 + kH3 + 16 * part + lane] = dw4;
  }
  if (part == 0) {
    for (int k = 16; k; k >>= 1) {
      db4 += __shfl_xor_sync(0xffffffffu, db4, k);
      loss += __shfl_xor_sync(0xffffffffu, loss, k);
    }
    if (lane == 0) {
      s_red[quad][kSums - 2] = db4;
      s_red[quad][kSums - 1] = loss;
    }
  }
  if (tid == kStorer) umma::bulk_wait();
  umma::tc_fence_before();
  __syncthreads();
  for (int i = tid; i < kSums; i += kTrainThreads)
    sums[(size_t)blockIdx.x * kSums + i] = ((s_red[0][i] + s_red[1][i]) + s_red[2][i]) + s_red[3][i];
  if (tid < 32) umma::tmem_dealloc(tm, kTrainCols);
}

struct AdamStep {
  float *P, *m, *v;
  float lr, b1, b2, eps, bc1, bc2, wd;
};

// What becomes of gradient g of parameter j (kNormN <= j < kNParams): Adam
// with decoupled weight decay (STEP) or a place in `grads`.
template <bool STEP>
__device__ __forceinline__ void finish_grad(const AdamStep& a, float* __restrict__ grads, int j, float g) {
  const int i = j - kNormN;
  if (!STEP) {
    grads[i] = g;
    return;
  }
  const float mi = a.b1 * a.m[i] + (1.0f - a.b1) * g;
  const float vi = a.b2 * a.v[i] + (1.0f - a.b2) * g * g;
  a.m[i] = mi;
  a.v[i] = vi;
  const bool is_weight = (j >= kOffW1 && j < kOffB1) || (j >= kOffW2 && j < kOffB2) ||
                         (j >= kOffW3 && j < kOffB3) || (j >= kOffW4 && j < kOffB4);
  float p = a.P[j];
  if (is_weight) p -= a.lr * a.wd * p;
  a.P[j] = p - a.lr * (mi / a.bc1) / (sqrtf(vi / a.bc2) + a.eps);
}

constexpr int kWgradThreads = 128, kWgradStages = 6, kWgradBlocks = 8;
constexpr int kSplitMin = 8, kSplitMax = 64;  // tiles of a batch whose chains are split
constexpr uint32_t kStageBytes = 2 * kAtom;
constexpr size_t kSmWgrad = 1024 + kWgradStages * kStageBytes;
constexpr int kSumBlocks = (kSums + kWgradThreads - 1) / kWgradThreads;

// Blocks 0..7: a 64 x 64 block of a weight gradient each, D[m][n] = sum over
// the samples of U[b][m] V[b][n] with U, V one 64-column atom of the stored
// operands; the further blocks: the sums over the training kernel's CTAs.
// The grid starts beside mlp_train_kernel's; what that stored is read, and the
// parameters are written, only after its end.
__device__ __forceinline__ void wait_for_train() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// SPLIT CTAs of a cluster take a quarter of the tiles of one block each; a
// quarter of the block's columns is then summed in each, in sample order.
template <bool STEP, int SPLIT>
__global__ void __launch_bounds__(kWgradThreads, 1)
    mlp_wgrad_kernel(const unsigned char* __restrict__ images, int tiles, const float* __restrict__ sums, int ctas,
                     AdamStep a, float* __restrict__ grads, float* __restrict__ loss, int* __restrict__ status) {
  const int r = blockIdx.x / SPLIT, part = blockIdx.x % SPLIT, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (r >= kWgradBlocks) {
    const int i = ((int)blockIdx.x - kWgradBlocks * SPLIT) * kWgradThreads + tid;
    if (i >= kSums) return;
    wait_for_train();
    float g = 0.0f;
#pragma unroll 8
    for (int c = 0; c < ctas; c++) g += sums[(size_t)c * kSums + i];
    if (i == kSums - 1) {
      if (loss) *loss = g;
      return;
    }
    finish_grad<STEP>(a, grads,
                      i < kH1               ? kOffB1 + i
                      : i < kH1 + kH2       ? kOffB2 + i - kH1
                      : i < kH1 + kH2 + kH3 ? kOffB3 + i - kH1 - kH2
                                            : kOffW4 + i - kH1 - kH2 - kH3,  // w4, then b4
                      g);
    return;
  }
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t sb = (umma::smem_u32(smem_raw) + 1023u) & ~1023u;
  __shared__ uint64_t full[kWgradStages], empty[kWgradStages], done;
  __shared__ uint32_t tmem_base;
  __shared__ int s_fail;
  if (tid < 32) umma::tmem_alloc(&tmem_base, 64);
  if (tid == 0) {
    for (int i = 0; i < kWgradStages; i++) {
      umma::mbar_init(&full[i], 1);
      umma::mbar_init(&empty[i], 1);
    }
    umma::mbar_init(&done, 1);
    s_fail = 0;
  }
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  wait_for_train();
  const uint32_t tm = tmem_base;
  const uint32_t u = r < 4 ? kID2 + (r & 1) * kAtom : r < 6 ? kTA2 + (r - 4) * kAtom : kID1 + (r - 6) * kAtom;
  const uint32_t v = r < 4 ? kTA1 + (r >> 1) * kAtom : r < 6 ? kTD3 : kTX0;
  const int t0 = (int)((int64_t)tiles * part / SPLIT), nt = (int)((int64_t)tiles * (part + 1) / SPLIT) - t0;
  if (tid == 0) {  // producer
    for (int t = 0; t < nt; t++) {
      const int s = t % kWgradStages, n = t / kWgradStages;
      if (n > 0 && !umma::mbar_wait(&empty[s], (uint32_t)(n - 1) & 1u, kWaitLimit)) {
        s_fail = 1;
        break;
      }
      const unsigned char* image = images + (size_t)(t0 + t) * kImage;
      umma::mbar_expect_tx(&full[s], kStageBytes);
      umma::bulk_load(sb + s * kStageBytes, image + u, kAtom, &full[s]);
      umma::bulk_load(sb + s * kStageBytes + kAtom, image + v, kAtom, &full[s]);
    }
  } else if (tid == 32) {  // MMAs, in sample order
    constexpr uint32_t id = umma::idesc_bf16(64, 64) | umma::kTransposeA | umma::kTransposeB;
    bool ok = true;
    for (int t = 0; t < nt && ok; t++) {
      const int s = t % kWgradStages, n = t / kWgradStages;
      ok = umma::mbar_wait(&full[s], (uint32_t)n & 1u, kWaitLimit);
      if (!ok) break;
      umma::tc_fence_after();
      const uint32_t at = sb + s * kStageBytes;
#pragma unroll
      for (int k = 0; k < 8; k++)
        umma::mma_bf16(tm, umma::sw128_desc_mn(at + 2048 * k, 128), umma::sw128_desc_mn(at + kAtom + 2048 * k, 128), id,
                       t > 0 || k > 0);
      umma::mma_commit(&empty[s]);
    }
    umma::mma_commit(&done);
    if (!umma::mbar_wait(&done, 0, kWaitLimit) || !ok) s_fail = 1;
  }
  __syncthreads();
  umma::tc_fence_after();
  if (s_fail) {
    // record it and let the copies in flight land (bounded) before the CTA ends
    if (tid == 0) {
      atomicExch(status, 1);
      for (int s = 0; s < kWgradStages && s < nt; s++)
        umma::mbar_wait(&full[s], (uint32_t)((nt - 1 - s) / kWgradStages) & 1u, kWaitLimit);
    }
  }
  auto finish = [&](int m, int n, float g) {
    if (r < 4) finish_grad<STEP>(a, grads, kOffW2 + (64 * (r & 1) + m) * kH1 + 64 * (r >> 1) + n, g);
    else if (r < 6) finish_grad<STEP>(a, grads, kOffW3 + n * kH2 + 64 * (r - 4) + m, g);
    else if (n < kF) finish_grad<STEP>(a, grads, kOffW1 + (64 * (r - 6) + m) * kF + n, g);
  };
  // row m of a 64-row accumulator: lane m % 16 of the tensor-memory quarter m / 16
  const int m = 16 * warp + lane;
  if (SPLIT > 1) {
    // this CTA's sums as [column][row], in the ring that every MMA has read
    float* own = reinterpret_cast<float*>(smem_raw + (sb - umma::smem_u32(smem_raw)));
    if (!s_fail)
      for (int c = 0; c < 64; c += 16) {
        float g[16];
        umma::tmem_ld16(tm + ((uint32_t)(warp * 32) << 16) + c, g);
        if (lane < 16)
#pragma unroll
          for (int i = 0; i < 16; i++) own[(c + i) * 64 + m] = g[i];
        __syncwarp();
      }
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    cl.sync();
    constexpr int kCols = 64 / SPLIT;
    bool failed = false;  // any of the four
#pragma unroll
    for (int q = 0; q < SPLIT; q++) failed |= *cl.map_shared_rank(&s_fail, q) != 0;
#pragma unroll
    for (int i = tid; i < kCols * 64 && !failed; i += kWgradThreads) {
      const int n = part * kCols + (i >> 6), k = i & 63;
      float g = 0.0f;
#pragma unroll
      for (int q = 0; q < SPLIT; q++) g += cl.map_shared_rank(own, q)[n * 64 + k];
      finish(k, n, g);
    }
    cl.sync();  // a CTA's shared memory is read by the others until here
  } else if (!s_fail) {
    for (int c = 0; c < 64; c += 16) {
      float g[16];
      umma::tmem_ld16(tm + ((uint32_t)(warp * 32) << 16) + c, g);
      if (lane < 16) {
#pragma unroll
        for (int i = 0; i < 16; i++) {
          finish(m, c + i, g[i]);
        }
      }
      __syncwarp();
    }
  }
  umma::tc_fence_before();
  __syncthreads();
  if (tid < 32) umma::tmem_dealloc(tm, 64);
}

size_t carve_mlp(cbmv_mlp* n, char* base) {
  size_t off = 0;
  auto take = [&](size_t bytes) -> void* {
    off = (off + 255) & ~(size_t)255;
    void* p = base ? base + off : nullptr;
    off += bytes;
    return p;
  };
  n->P = (float*)take(sizeof(float) * kNParams);
  n->m = (float*)take(sizeof(float) * kNParams);
  n->v = (float*)take(sizeof(float) * kNParams);
  n->sums = (float*)take(sizeof(float) * kSums * (size_t)n->ctas);
  n->images = (unsigned char*)take((size_t)kImage * (n->B / 128));
  n->status = (int*)take(4 * 4);
  return off + 256;
}

template <bool STEP, int SPLIT>
int launch_wgrad(const cbmv_mlp* n, const AdamStep& a, float* grads, float* loss, cudaStream_t st) {
  static_assert(kSumBlocks % SPLIT == 0 && 64 % SPLIT == 0, "whole clusters");
  CBMV_CUDA(cudaFuncSetAttribute(mlp_wgrad_kernel<STEP, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmWgrad));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kWgradBlocks * SPLIT + kSumBlocks);
  cfg.blockDim = dim3(kWgradThreads);
  cfg.dynamicSmemBytes = kSmWgrad;
  cfg.stream = st;
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = SPLIT;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  CBMV_CUDA(cudaLaunchKernelEx(&cfg, mlp_wgrad_kernel<STEP, SPLIT>, (const unsigned char*)n->images, n->B / 128,
                               (const float*)n->sums, n->ctas, a, grads, loss, n->status));
  return check_launch("mlp_wgrad");
}

// Forward and backward of one batch, then Adam (STEP) or the gradients.
template <int ACT, bool STEP>
int launch_train(const cbmv_mlp* n, const float* X, const float* y, const AdamStep& a, float* grads, float* loss,
                 cudaStream_t st) {
  CBMV_CUDA(cudaFuncSetAttribute(mlp_train_kernel<ACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmTrain));
  mlp_train_kernel<ACT><<<n->ctas, kTrainThreads, kSmTrain, st>>>(X, y, n->P, n->B, n->images, n->sums, n->status);
  int rc = check_launch("mlp_train");
  if (rc) return rc;
  const int tiles = n->B / 128;
  return tiles >= kSplitMin && tiles <= kSplitMax ? launch_wgrad<STEP, 4>(n, a, grads, loss, st)
                                                  : launch_wgrad<STEP, 1>(n, a, grads, loss, st);
}

template <bool STEP>
int mlp_batch(const cbmv_mlp* n, const float* X, const float* y, const AdamStep& a, float* grads, float* loss,
              cudaStream_t st) {
  return n->act == CBMV_ACT_GELU ? launch_train<CBMV_ACT_GELU, STEP>(n, X, y, a, grads, loss, st)
                                 : launch_train<CBMV_ACT_RELU, STEP>(n, X, y, a, grads, loss, st);
}

}  // namespace
}  // namespace cbmv

using namespace cbmv;

extern "C" int cbmv_mlp_num_params(void) { return kNParams; }

extern "C" int cbmv_mlp_create(int batch, cbmv_mlp** out) {
  CBMV_REQUIRE(out, CBMV_EINVAL, "null pointer argument");
  CBMV_REQUIRE(batch >= 128 && batch % 128 == 0 && batch <= (1 << 22), CBMV_EINVAL,
               "batch must be a multiple of 128 in [128, 4194304]");
  int dev = 0, sms = 0;
  CBMV_CUDA(cudaGetDevice(&dev));
  CBMV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  cbmv_mlp* n = new cbmv_mlp();
  n->B = batch;
  n->ctas = batch / 128 < sms ? batch / 128 : sms;
  const size_t bytes = carve_mlp(n, nullptr);
  cudaError_t e = cudaMalloc(&n->mem, bytes);
  if (e != cudaSuccess) {
    delete n;
    return set_error(CBMV_ENOMEM, "mlp workspace: %s", cudaGetErrorString(e));
  }
  carve_mlp(n, (char*)n->mem);
  if (cudaMemset(n->mem, 0, bytes) != cudaSuccess) {
    cudaFree(n->mem);
    delete n;
    return set_error(CBMV_ECUDA, "mlp workspace clear failed");
  }
  *out = n;
  return CBMV_OK;
}

extern "C" int cbmv_mlp_destroy(cbmv_mlp* n) {
  if (!n) return CBMV_OK;
  cudaDeviceSynchronize();
  cudaFree(n->mem);
  delete n;
  return CBMV_OK;
}

// Parameters in from / out to HOST memory (kNParams floats); setting them
// resets the optimiser state.
extern "C" int cbmv_mlp_set_params(cbmv_mlp* n, const float* host) {
  CBMV_REQUIRE(n && host, CBMV_EINVAL, "null pointer argument");
  CBMV_CUDA(cudaMemcpy(n->P, host, sizeof(float) * kNParams, cudaMemcpyHostToDevice));
  CBMV_CUDA(cudaMemset(n->m, 0, sizeof(float) * kNParams));
  CBMV_CUDA(cudaMemset(n->v, 0, sizeof(float) * kNParams));
  n->step = 0;
  CBMV_CUDA(cudaDeviceSynchronize());
  return CBMV_OK;
}

extern "C" int cbmv_mlp_get_params(const cbmv_mlp* n, float* host) {
  CBMV_REQUIRE(n && host, CBMV_EINVAL, "null pointer argument");
  CBMV_CUDA(cudaMemcpy(host, n->P, sizeof(float) * kNParams, cudaMemcpyDeviceToHost));
  return CBMV_OK;
}

// One Adam step on a batch of B samples: X float32 [B,20] raw CBMV features,
// y float32 [B] labels (1 = correct match), device memory.  loss (device,
// may be NULL) receives the batch's mean binary cross-entropy.
extern "C" int cbmv_mlp_train_step(cbmv_mlp* n, const float* X, const float* y, float lr,
                                   float weight_decay, float* loss, void* stream) {
  CBMV_REQUIRE(n && X && y, CBMV_EINVAL, "null pointer argument");
  const float b1 = 0.9f, b2 = 0.999f;
  const float step = (float)(n->step + 1);
  const AdamStep a{n->P, n->m, n->v, lr, b1, b2, 1e-8f, 1.0f - powf(b1, step), 1.0f - powf(b2, step), weight_decay};
  const int rc = mlp_batch<true>(n, X, y, a, nullptr, loss, as_stream(stream));
  if (rc == CBMV_OK) n->step++;
  return rc;
}

// Gradients of the batch loss without an update (for checking): grads
// float32 [num_params - 60] in parameter order (the input transform has no
// gradient), loss float32 [1]; both device memory.
extern "C" int cbmv_mlp_gradients(cbmv_mlp* n, const float* X, const float* y, float* grads, float* loss,
                                  void* stream) {
  CBMV_REQUIRE(n && X && y && grads, CBMV_EINVAL, "null pointer argument");
  return mlp_batch<false>(n, X, y, AdamStep{}, grads, loss, as_stream(stream));
}

extern "C" int cbmv_mlp_set_activation(cbmv_mlp* n, int act) {
  CBMV_REQUIRE(n, CBMV_EINVAL, "null pointer argument");
  CBMV_REQUIRE(act == CBMV_ACT_RELU || act == CBMV_ACT_GELU, CBMV_EINVAL, "unknown activation %d", act);
  n->act = act;
  return CBMV_OK;
}

extern "C" int cbmv_mlp_set_precision(cbmv_mlp* n, int prec) {
  CBMV_REQUIRE(n, CBMV_EINVAL, "null pointer argument");
  CBMV_REQUIRE(prec == CBMV_PREC_F16 || prec == CBMV_PREC_BF16, CBMV_EINVAL, "unknown precision %d", prec);
  n->prec = prec;
  return CBMV_OK;
}

extern "C" int cbmv_mlp_get_precision(const cbmv_mlp* n, int* prec) {
  CBMV_REQUIRE(n && prec, CBMV_EINVAL, "null pointer argument");
  *prec = n->prec;
  return CBMV_OK;
}

extern "C" int cbmv_mlp_get_activation(const cbmv_mlp* n, int* act) {
  CBMV_REQUIRE(n && act, CBMV_EINVAL, "null pointer argument");
  *act = n->act;
  return CBMV_OK;
}

// Status of the tensor-core waits since creation (0 = fine).
extern "C" int cbmv_mlp_status(const cbmv_mlp* n, int* status) {
  CBMV_REQUIRE(n && status, CBMV_EINVAL, "null pointer argument");
  CBMV_CUDA(cudaMemcpy(status, n->status, sizeof(int), cudaMemcpyDeviceToHost));
  return CBMV_OK;
}
