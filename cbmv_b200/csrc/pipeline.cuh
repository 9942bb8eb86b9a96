// Launch helpers shared by the fused pipeline (pipeline.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "rf.cuh"

namespace cbmv {

// Matcher arguments: non-null pointers, 0 < H <= 65535, 0 < D <= 65535
// (CBMV_ERANGE beyond), W > 0, window odd and <= wmax, dtype and layout.
int check_common(const void* a, const void* b, const void* out, int64_t H, int64_t W, int D, int w,
                 int dtype, int layout, int wmax);
// Per-pixel matcher terms of one or two images (img[1] null: one) at the
// default windows; null arrays are not formed.
struct MatchTerms {
  const uint8_t* img[2];
  ulonglong2* desc[2];  // census, 11 x 11
  uint32_t* A[2];       // NCC, 3 x 3: window sum and 1 / sqrt(9 B - A^2)
  double* C[2];
  double* mean[2];      // ZSAD, 5 x 5
  int32_t* sob[2];      // Sobel responses
};
int launch_match_terms(const MatchTerms& t, int64_t H, int64_t W, cudaStream_t st);
int launch_census_descs(const uint8_t* L, const uint8_t* R, int64_t H, int64_t W, int w, ulonglong2* dl,
                        ulonglong2* dr, cudaStream_t st);
template <class T>
int launch_census_cost(const ulonglong2* dl, const ulonglong2* dr, int64_t H, int64_t W, int D,
                       int w, int layout, T* out, cudaStream_t st);
int launch_ncc_stats(const uint8_t* img, int64_t H, int64_t W, int w, uint32_t* A, double* C,
                     cudaStream_t st);
template <class T>
int launch_ncc_cost(const uint8_t* L, const uint8_t* R, const uint32_t* Al, const uint32_t* Ar,
                    const double* Cl, const double* Cr, int64_t H, int64_t W, int D, int w,
                    int layout, T* out, cudaStream_t st);
template <class T>
int launch_sadsob_cost(const int32_t* SL, const int32_t* SR, int64_t H, int64_t W, int D, int w,
                       int layout, T* out, cudaStream_t st);
int launch_zsad_means(const uint8_t* img, int64_t H, int64_t W, int w, double* mean,
                      cudaStream_t st);
template <class T>
int launch_zsad_cost(const uint8_t* L, const uint8_t* R, const double* ml, const double* mr,
                     int64_t H, int64_t W, int D, int w, int layout, T* out, cudaStream_t st);
// the learned path's float32 [H,W,D] ZSAD (rounded from the exact quotient)
int launch_zsad_cost_f32(const uint8_t* L, const uint8_t* R, const double* ml, const double* mr, int64_t H,
                         int64_t W, int D, int w, float* out, cudaStream_t st);
int launch_feature_stats(const double* const* vols, int64_t H, int64_t W, int D, double* stats, cudaStream_t st);
// (min, 1/den) in float32 of float32 volumes, both views, the four matchers
int launch_feature_stats_f32(const float* const* vols, int64_t H, int64_t W, int D, float2* statsf,
                             cudaStream_t st);
int launch_features_mlp(const float* const* vols, const float2* statsf, int64_t H, int64_t W, int D,
                        const cbmv_mlp* m, float* prob0, cudaStream_t st, int max_ctas = 0);
// The learned path's float32 features of the samples idx[i] = (y*W + x)*D + d
// (the fused network kernel's own feature code), out [n, 20].
int launch_features_f32_gather(const float* const* vols, const float2* statsf, int64_t H, int64_t W, int D,
                               const int64_t* idx, int64_t n, float* out, cudaStream_t st);
// The 20 features (float32) of the samples idx[i] = (y*W + x)*D + d.
// n samples' features from the whole image's statistics, or (stats null) from
// those of their own rows; the second where features_gather_rows says so
bool features_gather_rows(int64_t H, int64_t W, int64_t n);
int launch_features_gather(const double* const* vols, const double* stats, int64_t H, int64_t W,
                           int D, const int64_t* idx, int64_t n, float* out, cudaStream_t st);
int launch_features_rf(const double* const* vols, const double* stats, int64_t H, int64_t W,
                       int D, const cbmv_forest* forest, float* prob0, cudaStream_t st);

}  // namespace cbmv
