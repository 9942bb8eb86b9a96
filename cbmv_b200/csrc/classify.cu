// Fused classifier kernels: the 20 CBMV features of every (pixel, d) built in
// shared memory and classified in place, so the [H*W*D, 20] feature matrix
// of the reference (test.py:541-595, handed to predict_proba at test.py:620)
// never exists in HBM.  Output: P(class 0), float32 [H,W,D], the matching
// cost the post-processing consumes (test.py:144-145).
//
// Random-forest walk (features_rf_tiled): bound by the L1 data stage, which
// serves four 32-byte sectors per clock (93 % busy in the same walk of
// rf_predict_kernel), so every choice is about sectors per step:
//  - a step reads one 16-byte entry and descends two tree levels (rf.cuh),
//    and the entry that ends a walk holds the leaf's value;
//  - a warp covers 4 x 2 pixels x 4 disparities: neighbouring samples have
//    similar features and walk similar paths, so a warp's requests touch
//    fewer distinct sectors than 32 disparities of one pixel;
//  - shared memory holds only the feature tile (40 KB per CTA), the rest of
//    the SM's 256 KB is L1 for the entries;
//  - 48 warps per SM with two trees each in flight hide the L2 latency of
//    the lower levels; the leaf values are added in tree order, as
//    predict_proba does.
// 694x554 D=128, 50 trees: 32.6 ms (67.3 ms with 32-byte blocks, 16 warps,
// four trees each).  Measured beside it: 32 warps 34.6-36.9 ms, one or four
// trees in flight 34.1-35.6, other warp shapes 32.8-34.1.
#include "common.cuh"
#include "features.cuh"
#include "pipeline.cuh"
#include "rf.cuh"

namespace cbmv {
namespace {

constexpr int kRfBlock = 512;  // threads per CTA
constexpr int kRfPerSm = 3;    // CTAs per SM
constexpr int kRfIlp = 2;      // trees walked at once
// samples of a warp (4 x 2 pixels x 4 disparities) and warps of a CTA (4 x 1 x 4)
constexpr int kWX = 4, kWY = 2, kWD = 32 / (kWX * kWY);
constexpr int kCX = 4, kCY = 1, kCD = kRfBlock / 32 / (kCX * kCY);
constexpr int kRfTileX = kWX * kCX, kRfTileY = kWY * kCY, kRfTileD = kWD * kCD;

template <int ILP>
__global__ void __launch_bounds__(kRfBlock, kRfPerSm)
    features_rf_tiled(FeatVols fv, const double* __restrict__ stats, int64_t H, int64_t W, int D,
                      RfView f, float* __restrict__ prob0) {
  extern __shared__ float xs[];  // [20][kRfBlock]: one feature column per thread
  const int T = f.n_trees;
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int lx = (warp % kCX) * kWX + lane % kWX, ly = (warp / kCX % kCY) * kWY + lane / kWX % kWY,
            ld = warp / (kCX * kCY) * kWD + lane / (kWX * kWY);
  const int64_t ntx = (W + kRfTileX - 1) / kRfTileX;
  const int64_t ntd = (D + kRfTileD - 1) / kRfTileD;
  const int64_t tiles = (H + kRfTileY - 1) / kRfTileY * ntx * ntd;
  const int64_t HW = H * W;
  float* col = xs + tid;

  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t td = tile % ntd;
    const int64_t tx = (tile / ntd) % ntx;
    const int64_t y = tile / (ntd * ntx) * kRfTileY + ly;
    const int64_t x = tx * kRfTileX + lx;
    const int d = (int)td * kRfTileD + ld;
    if (x >= W || d >= D || y >= H) continue;
    const int64_t p = y * W + x;
    features_store(fv.v, stats, HW, D, p, x, d, col, kRfBlock);

    double acc = 0.0;
    for (int t = 0; t < T; t += ILP) {
      uint4 v[ILP];
      rf_walk<ILP, kRfBlock>(f, t, col, v);
#pragma unroll
      for (int k = 0; k < ILP; k++)
        if (t + k < T) acc += rf_leaf_p0(v[k]);
    }
    prob0[p * D + d] = (float)(acc / T);
  }
}

}  // namespace

int launch_features_rf(const double* const* vols, const double* stats, int64_t H, int64_t W,
                       int D, const cbmv_forest* forest, float* prob0, cudaStream_t st) {
  const RfView& f = *forest_view(forest);
  CBMV_REQUIRE(f.n_features == 20, CBMV_EINVAL, "the forest must take the 20 CBMV features");
  int dev = 0, sms = 0;
  CBMV_CUDA(cudaGetDevice(&dev));
  CBMV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const size_t smem = (size_t)20 * kRfBlock * sizeof(float);
  FeatVols fv = {{vols[0], vols[1], vols[2], vols[3]}};
  features_rf_tiled<kRfIlp><<<sms * kRfPerSm, kRfBlock, smem, st>>>(fv, stats, H, W, D, f, prob0);
  return check_launch("features_rf_tiled");
}

}  // namespace cbmv
