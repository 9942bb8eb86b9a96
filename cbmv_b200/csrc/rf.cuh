// Device view of a random forest and the tree walk shared by the classifier
// kernels.
//
// The forest arrives as two-level blocks of 32 bytes (cbmv_b200/forest.py,
// FlatForest.pack; include/cbmv.h cbmv_forest_create) and is laid out on the
// device as 16-byte entries, one load each, 16-byte aligned:
//   internal  words 0-2  float32 thresholds of a node and of its left and
//                        right child; t32 = the largest float32 <= sklearn's
//                        float64 threshold, so `x <= t32` branches as
//                        sklearn's `float32(x) <= threshold` does
//                        (sklearn/tree/_tree.pyx, Tree._apply_dense)
//             word 3     bits 17-31: the features of the three nodes, 5 bits
//                        each; bits 0-16: the group of the four grandchildren
//   leaf      words 0-1  the class-0 fraction (float64), word 2 the leaf's
//                        index, word 3 kRfLeaf
//   jump      word 0     the entry to go on from, word 3 kRfJump
// Four sibling entries form a 64-byte group, numbered from their segment's
// first entry; a child that is itself a leaf fills both of its slots.  A
// tree is one segment, its root the first entry; where it has more groups
// than 17 bits count, a jump leads to a subtree in a segment of its own, and
// so it does to a block that several slots name as their child.
//
// A walk step is one 16-byte load and descends two levels, and the leaf's
// value is in the entry that ends the walk.  (The 32-byte blocks took two
// loads per step and two more gathers for the leaf: with 16 warps per SM
// and four trees per thread 67.3 ms for the 694x554 D=128 volume.)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/cbmv.h"

namespace cbmv {

constexpr uint32_t kLeafFlag = 1u << 31;     // of a block's child word
constexpr uint32_t kLeafFeature = 0xFFu;     // of a block's feature byte
// Word 3 of a leaf and of a jump: features 0 (a walk step on them reads
// within the sample's columns) and a group that no internal entry has.
constexpr uint32_t kRfLeaf = 0u, kRfJump = (1u << 17) - 1;
constexpr uint32_t kRfMaxGroup = kRfJump - 1;

struct RfView {
  const uint4* entries;
  const uint32_t* roots;   // [n_trees] first entry of each tree
  const double* leaf_p1;   // class-1 fraction by leaf index
  int n_trees;
  int n_features;
  int64_t n_blocks;
  int64_t n_leaves;
};

const RfView* forest_view(const cbmv_forest* f);

// Walks trees t .. t+ILP-1 (those below n_trees) for the sample whose
// feature k is x[k * STRIDE] (STRIDE a power of two, 128..2048); v[k]
// receives the leaf entry of tree t + k.
template <int ILP, int STRIDE>
__device__ __forceinline__ void rf_walk(const RfView& f, int t, const float* x, uint4 (&v)[ILP]) {
  static_assert((STRIDE & (STRIDE - 1)) == 0 && STRIDE >= 128 && STRIDE <= 2048, "feature stride");
  // a feature's 5 bits shifted to the byte offset of its column
  constexpr uint32_t kMask = 31u * STRIDE * 4;
  constexpr int kLog = STRIDE == 128 ? 9 : STRIDE == 256 ? 10 : STRIDE == 512 ? 11 : STRIDE == 1024 ? 12 : 13;
  const char* xb = reinterpret_cast<const char*>(x);
  uint32_t seg[ILP];
#pragma unroll
  for (int k = 0; k < ILP; k++) {
    seg[k] = __ldg(f.roots + (t + k < f.n_trees ? t + k : t));
    v[k] = __ldg(f.entries + seg[k]);
  }
  for (;;) {
    bool live = false;
    uint32_t e[ILP];
#pragma unroll
    for (int k = 0; k < ILP; k++) {
      const uint32_t w = v[k].w;
      const bool right = !(*reinterpret_cast<const float*>(xb + ((w >> (17 - kLog)) & kMask)) <= __uint_as_float(v[k].x));
      const float thr = __uint_as_float(right ? v[k].z : v[k].y);
      const float xv = *reinterpret_cast<const float*>(xb + ((w >> (right ? 27 - kLog : 22 - kLog)) & kMask));
      e[k] = seg[k] + ((w & 0x1FFFFu) << 2) + (right ? 2u : 0u) + (xv <= thr ? 0u : 1u);
      if (w == kRfJump) e[k] = seg[k] = v[k].x;
      live |= w != kRfLeaf;
    }
    if (!live) break;
#pragma unroll
    for (int k = 0; k < ILP; k++)
      if (v[k].w != kRfLeaf) v[k] = __ldg(f.entries + e[k]);
  }
}

__device__ __forceinline__ double rf_leaf_p0(const uint4& v) { return __hiloint2double((int)v.y, (int)v.x); }

}  // namespace cbmv
