// Random-forest classifier: sklearn's RandomForestClassifier.predict_proba
// (sklearn/ensemble/_forest.py; tree walk sklearn/tree/_tree.pyx
// Tree._apply_dense) over the device forest of rf.cuh.
// The class fractions of the leaves are summed in float64 in tree order and
// divided by the tree count, as predict_proba does with one job.
#include <string.h>

#include <new>
#include <unordered_map>
#include <vector>

#include "common.cuh"
#include "rf.cuh"

namespace cbmv {
namespace {

constexpr int kBlock = 256;
constexpr int kPerSm = 6;  // blocks per SM the registers allow for
constexpr int kIlp = 2;    // trees walked at once

// Bound by the L1 data stage like features_rf_tiled (classify.cu): 12.8 M
// rows of 50 trees 8.9 ms (13.6 ms over 32-byte blocks, one tree at a time).
__global__ void __launch_bounds__(kBlock, kPerSm)
    rf_predict_kernel(RfView f, const float* __restrict__ X, int64_t N, double* __restrict__ proba,
                      int32_t* __restrict__ leaves) {
  extern __shared__ float xs[];  // [F][kBlock]
  const int tid = threadIdx.x;
  for (int64_t n0 = (int64_t)blockIdx.x * kBlock; n0 < N; n0 += (int64_t)gridDim.x * kBlock) {
    const int64_t n = n0 + tid;
    __syncthreads();
    // stage the block's feature rows, coalesced, transposed to [F][block]
    for (int k = tid; k < f.n_features * kBlock; k += kBlock) {
      const int r = k / f.n_features, c = k - r * f.n_features;
      const int64_t row = n0 + r;
      xs[c * kBlock + r] = row < N ? X[row * f.n_features + c] : 0.0f;
    }
    __syncthreads();
    if (n >= N) continue;
    double p0 = 0.0, p1 = 0.0;
    for (int t = 0; t < f.n_trees; t += kIlp) {
      uint4 v[kIlp];
      rf_walk<kIlp, kBlock>(f, t, xs + tid, v);
#pragma unroll
      for (int k = 0; k < kIlp; k++) {
        if (t + k >= f.n_trees) break;
        p0 += rf_leaf_p0(v[k]);
        if (proba) p1 += __ldg(f.leaf_p1 + v[k].z);
        if (leaves) leaves[n * f.n_trees + t + k] = (int32_t)v[k].z;
      }
    }
    if (proba) {
      proba[2 * n] = p0 / f.n_trees;
      proba[2 * n + 1] = p1 / f.n_trees;
    }
  }
}

}  // namespace

// The device layout of rf.cuh from validated two-level blocks: one segment
// per tree, breadth-first; a group that its segment can no longer number
// starts a segment of its own, reached by a jump, and so does a block that
// several slots name as their child (laid out once, however many reach it).
// Every block begins at most one segment and forms at most one group, so
// there are at most 8 entries per block.
static void rf_entries(const uint32_t* blocks, int64_t n_blocks, const double* leaf_value, const int32_t* tree_offsets,
                       int n_trees, uint32_t max_group, std::vector<uint32_t>* entries, std::vector<uint32_t>* roots) {
  std::vector<uint32_t>& E = *entries;
  // the child block or leaf (kLeafFlag) in slot j of a block's child n
  auto child_of = [](const uint32_t* w, int n, int j) {
    return ((w[3] >> (8 * n)) & 0xFFu) == kLeafFeature ? w[2 + 2 * n] | kLeafFlag : w[2 + 2 * n + j];
  };
  auto leaf = [&](uint32_t at, uint32_t id) {
    memcpy(&E[4 * (size_t)at], &leaf_value[2 * (size_t)id], sizeof(double));
    E[4 * (size_t)at + 2] = id;
    E[4 * (size_t)at + 3] = kRfLeaf;
  };
  constexpr uint32_t kNone = 0xFFFFFFFFu;
  std::vector<uint8_t> named(n_blocks, 0);  // slots that name the block, at most 2
  for (int64_t k = 0; k < n_blocks; k++) {
    const uint32_t* w = blocks + 8 * (size_t)k;
    if ((w[3] & 0xFFu) == kLeafFeature) continue;
    for (int s = 0; s < 4; s++) {
      const uint32_t c = child_of(w, 1 + s / 2, s % 2);
      if (!(c & kLeafFlag) && named[c] < 2) named[c]++;
    }
  }
  std::unordered_map<uint32_t, uint32_t> shared;  // a block named twice -> its segment
  struct Item {
    uint32_t block, at;
  };
  for (int t = 0; t < n_trees; t++) {
    std::vector<Item> starts = {{(uint32_t)tree_offsets[t], kNone}};  // block, the jump leading to it
    for (size_t i = 0; i < starts.size(); i++) {
      const Item start = starts[i];
      uint32_t seg = (uint32_t)(E.size() / 4);
      bool laid = false;
      if (named[start.block] > 1) {
        const auto put = shared.emplace(start.block, seg);
        laid = !put.second;
        seg = put.first->second;
      }
      if (start.at == kNone) {
        roots->push_back(seg);
      } else {
        E[4 * (size_t)start.at] = seg;
        E[4 * (size_t)start.at + 3] = kRfJump;
      }
      if (laid) continue;
      E.resize(E.size() + 16, 0u);
      uint32_t group = 1;
      std::vector<Item> queue = {{start.block, seg}};
      for (size_t q = 0; q < queue.size(); q++) {
        const uint32_t at = queue[q].at;
        const uint32_t* w = blocks + 8 * (size_t)queue[q].block;
        const uint32_t f[3] = {w[3] & 0xFFu, (w[3] >> 8) & 0xFFu, (w[3] >> 16) & 0xFFu};
        if (f[0] == kLeafFeature) {
          leaf(at, w[4] & ~kLeafFlag);
          continue;
        }
        if (group > max_group) {
          starts.push_back(queue[q]);
          continue;
        }
        const uint32_t child = seg + 4 * group;
        E.resize(E.size() + 16, 0u);
        uint32_t* e = &E[4 * (size_t)at];
        for (int n = 0; n < 3; n++) e[n] = f[n] == kLeafFeature ? 0u : w[n];
        e[3] = group++ | f[0] << 17 | (f[1] == kLeafFeature ? 0u : f[1]) << 22 | (f[2] == kLeafFeature ? 0u : f[2]) << 27;
        for (int s = 0; s < 4; s++) {
          const uint32_t c = child_of(w, 1 + s / 2, s % 2), to = child + s;
          if (c & kLeafFlag) leaf(to, c & ~kLeafFlag);
          else (named[c] > 1 ? starts : queue).push_back({c, to});
        }
      }
    }
  }
}
}  // namespace cbmv

using namespace cbmv;

struct cbmv_forest {
  RfView view;
  void* mem;
};

extern "C" int cbmv_forest_create(const uint32_t* blocks, int64_t n_blocks, const double* leaf_value,
                                  int64_t n_leaves, const int32_t* tree_offsets, int n_trees,
                                  int n_features, cbmv_forest** out) {
  CBMV_REQUIRE(blocks && leaf_value && tree_offsets && out, CBMV_EINVAL, "null pointer argument");
  CBMV_REQUIRE(n_blocks > 0 && n_leaves > 0 && n_trees > 0, CBMV_EINVAL, "empty forest");
  CBMV_REQUIRE(n_features > 0 && n_features <= 32, CBMV_EINVAL, "n_features %d not in 1..32",
               n_features);
  CBMV_REQUIRE(n_blocks < (int64_t)kLeafFlag && n_leaves < (int64_t)kLeafFlag, CBMV_ERANGE,
               "forest too large for 31-bit indices");
  CBMV_REQUIRE(n_blocks + n_trees < (int64_t)1 << 29, CBMV_ERANGE, "forest too large for 32-bit entry indices");
  CBMV_REQUIRE(tree_offsets[0] == 0 && tree_offsets[n_trees] == n_blocks, CBMV_EINVAL,
               "tree offsets do not cover the block array");
  // Validate the structure on the host, so the device walk never reads
  // outside the arrays and always ends: every feature is in range, every
  // leaf index exists, every child block lies later in the same tree.
  for (int t = 0; t < n_trees; t++) {
    CBMV_REQUIRE(tree_offsets[t] < tree_offsets[t + 1], CBMV_EINVAL, "empty tree %d", t);
    for (int64_t k = tree_offsets[t]; k < tree_offsets[t + 1]; k++) {
      const uint32_t* w = blocks + 8 * k;
      const uint32_t f0 = w[3] & 0xFFu, f1 = (w[3] >> 8) & 0xFFu, f2 = (w[3] >> 16) & 0xFFu;
      auto leaf_ok = [&](uint32_t v) { return (int64_t)(v & ~kLeafFlag) < n_leaves; };
      auto feat_ok = [&](uint32_t f) { return f == kLeafFeature || (int)f < n_features; };
      CBMV_REQUIRE(feat_ok(f0) && feat_ok(f1) && feat_ok(f2), CBMV_EINVAL,
                   "block %lld: feature out of range", (long long)k);
      if (f0 == kLeafFeature) {
        CBMV_REQUIRE(leaf_ok(w[4]), CBMV_EINVAL, "block %lld: leaf index out of range", (long long)k);
        continue;
      }
      for (int n = 1; n <= 2; n++) {
        const uint32_t fn = n == 1 ? f1 : f2;
        const int slot = 4 + 2 * (n - 1);
        if (fn == kLeafFeature) {
          CBMV_REQUIRE(leaf_ok(w[slot]), CBMV_EINVAL, "block %lld: leaf index out of range",
                       (long long)k);
          continue;
        }
        for (int j = 0; j < 2; j++) {
          const uint32_t c = w[slot + j];
          if (c & kLeafFlag) {
            CBMV_REQUIRE(leaf_ok(c), CBMV_EINVAL, "block %lld: leaf index out of range",
                         (long long)k);
          } else {
            CBMV_REQUIRE((int64_t)c > k && (int64_t)c < tree_offsets[t + 1], CBMV_EINVAL,
                         "block %lld: child block outside its tree", (long long)k);
          }
        }
      }
    }
  }
  std::vector<uint32_t> entries, roots;
  std::vector<double> p1;
  cbmv_forest* f = nullptr;
  try {
    entries.reserve(16 * (size_t)(n_blocks + n_trees));
    rf_entries(blocks, n_blocks, leaf_value, tree_offsets, n_trees, kRfMaxGroup, &entries, &roots);
    p1.resize((size_t)n_leaves);
    f = new cbmv_forest();
  } catch (const std::bad_alloc&) {
    return set_error(CBMV_ENOMEM, "forest layout: out of host memory");
  }
  for (int64_t i = 0; i < n_leaves; i++) p1[i] = leaf_value[2 * i + 1];
  auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t eb = up(entries.size() * 4), lb = up((size_t)n_leaves * sizeof(double)), rb = roots.size() * 4;
  cudaError_t e = cudaMalloc(&f->mem, eb + lb + rb);
  if (e != cudaSuccess) {
    delete f;
    return set_error(CBMV_ENOMEM, "forest upload: %s", cudaGetErrorString(e));
  }
  char* base = (char*)f->mem;
  f->view.entries = (const uint4*)base;
  f->view.leaf_p1 = (const double*)(base + eb);
  f->view.roots = (const uint32_t*)(base + eb + lb);
  f->view.n_trees = n_trees;
  f->view.n_features = n_features;
  f->view.n_blocks = n_blocks;
  f->view.n_leaves = n_leaves;
  if (cudaMemcpy(base, entries.data(), entries.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(base + eb, p1.data(), p1.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(base + eb + lb, roots.data(), rb, cudaMemcpyHostToDevice) != cudaSuccess) {
    cudaFree(f->mem);
    delete f;
    return set_error(CBMV_ECUDA, "forest upload failed");
  }
  *out = f;
  return CBMV_OK;
}

namespace cbmv {
const RfView* forest_view(const cbmv_forest* f) { return &f->view; }
}  // namespace cbmv

extern "C" int cbmv_forest_info(const cbmv_forest* f, int* n_trees, int64_t* n_blocks,
                                int64_t* n_leaves) {
  CBMV_REQUIRE(f, CBMV_EINVAL, "null forest");
  if (n_trees) *n_trees = f->view.n_trees;
  if (n_blocks) *n_blocks = f->view.n_blocks;
  if (n_leaves) *n_leaves = f->view.n_leaves;
  return CBMV_OK;
}

extern "C" int cbmv_forest_destroy(cbmv_forest* f) {
  if (!f) return CBMV_OK;
  cudaDeviceSynchronize();
  cudaFree(f->mem);
  delete f;
  return CBMV_OK;
}

extern "C" int cbmv_forest_predict(const cbmv_forest* f, const float* X, int64_t N, double* proba,
                                   int32_t* leaves, void* stream) {
  CBMV_REQUIRE(f && X, CBMV_EINVAL, "null pointer argument");
  CBMV_REQUIRE(N > 0, CBMV_EINVAL, "N must be positive");
  const size_t smem = (size_t)f->view.n_features * kBlock * sizeof(float);
  rf_predict_kernel<<<grid_for(N, kBlock), kBlock, smem, as_stream(stream)>>>(f->view, X, N, proba,
                                                                             leaves);
  return check_launch("forest_predict");
}
