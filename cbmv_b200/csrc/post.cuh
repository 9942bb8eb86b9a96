// Launch helpers of the cost-optimisation kernels (post.cu), shared with the
// fused pipeline.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace cbmv {

struct SgmParams {
  float pi1, pi2, tau_so, alpha1, q1, q2;
  int direction;
};

int launch_cross(const float* img, int64_t H, int64_t W, int L1, float tau1, float* out,
                 cudaStream_t st);
// Classes of both normalised images' neighbour differences (see post.cu
// sgm_codes_kernel), 32 positions per word pair: rows [H][ceil(W / 32)] and
// columns [ceil(H / 32)][W] of each image, in 8-byte aligned memory.
struct SgmCodes {
  uint2 *left_h, *left_v, *right_h, *right_v;
};
inline int64_t sgm_codes_bytes(int64_t H, int64_t W) {
  return 2 * (H * ((W + 31) / 32) + (H + 31) / 32 * W) * (int64_t)sizeof(uint2);
}
inline SgmCodes sgm_codes_at(void* at, int64_t H, int64_t W) {
  uint2* c = static_cast<uint2*>(at);
  const int64_t nh = H * ((W + 31) / 32), nv = (H + 31) / 32 * W;
  return SgmCodes{c, c + nh, c + nh + nv, c + 2 * nh + nv};
}
int launch_sgm_codes(const float* imL, const float* imR, int64_t H, int64_t W, float tau, const SgmCodes& g,
                     cudaStream_t st);
// Path costs of the four scan directions, one volume each.
struct SgmOut {
  float* dir[4];
};
int launch_sgm4(const SgmCodes& g, const float* in, int64_t H, int64_t W, int D, const SgmParams& sp,
                const SgmOut& o, cudaStream_t st);
// out = base + (((L0 + L1) + L2) + L3) * scale; base may be null or out.
int launch_sgm_combine(const SgmOut& o, int64_t n, const float* base, float scale, float* out,
                       cudaStream_t st);
// halo: how far (pixels) the cross arms' interior reaches, L1 - 1; supports
// reaching further are still summed correctly, from global memory.
int launch_cbca(const float* lc, const float* rc, const float* in, int64_t H, int64_t W, int D,
                int layout, int direction, float* out, cudaStream_t st, int halo = 5);
// cbca on [H,W,D] in separable form (row sums, then column sums); arms of
// at most `halo` pixels (L1 - 1), halo 1..8 (larger: the reference-order kernel)
int launch_cbca_sep(const float* lc, const float* rc, const float* in, int64_t H, int64_t W, int D,
                    int direction, float* out, cudaStream_t st, int halo, int rows = 32);
// the separable cbca with its supports precomputed (arms of at most 5
// pixels, L1 <= 6): one 32-bit word per (p,d) in `mask`, built once per
// cross, then any number of passes; bit-identical to launch_cbca_sep
int launch_cbca_mask_build(const uint32_t* wl, const uint32_t* wr, int64_t H, int64_t W, int D, int direction,
                           uint32_t* mask, cudaStream_t st);
int launch_cbca_masked(const uint32_t* mask, const float* in, int64_t H, int64_t W, int D, float* out,
                       cudaStream_t st, int rows = 0);
constexpr int kCbcaMaskMaxHalo = 5;
int launch_wta_subpixel(const float* cost, int64_t H, int64_t W, int D, float* disp_int,
                        float* disp, cudaStream_t st);
int launch_median(const float* in, int64_t H, int64_t W, int k, float* out, cudaStream_t st);
int launch_mean2d(const float* in, int64_t H, int64_t W, const float* kernel, int ks, float alpha2,
                  float* out, cudaStream_t st);
// do_post's normalisation (test.py:485-504) of both images, their cross arms and (L1 - 1 <= kCbcaMaskMaxHalo) the
// arms as tap words, left view's [H, W] then right view's; mom: 4 doubles of scratch
int launch_normalise_cross(const uint8_t* L, const uint8_t* R, int64_t H, int64_t W, double* mom, int L1, float tau1,
                           float* imL, float* imR, float* crossL, float* crossR, uint32_t* words, cudaStream_t st);
// get_right_cost of a float32 [H,W,D] volume (the _interp post's right view)
int launch_right_cost_f32(const float* in, int64_t H, int64_t W, int D, float* out, cudaStream_t st);
int launch_outlier(const float* d0, const float* d1, int64_t H, int64_t W, int disp_max, float* out,
                   cudaStream_t st);
int launch_mismatch(const float* d0, const float* o, int64_t H, int64_t W, float* out,
                    cudaStream_t st);
int launch_occlusion(const float* d0, const float* o, int64_t H, int64_t W, float* out,
                     cudaStream_t st);

}  // namespace cbmv
