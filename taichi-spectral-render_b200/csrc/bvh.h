// Host-side BVH construction and conversion to the device layouts.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <string>
#include <thread>
#include <vector>

namespace ts {

// f(begin, end) over [0, n) in chunks, on up to 8 threads where there is enough to share
template <class F>
void parallel_chunks(int n, F f) {
  const int nt = std::min({8, (int)std::max(1u, std::thread::hardware_concurrency()), n / 16384});
  if (nt <= 1) {
    f(0, n);
    return;
  }
  std::vector<std::thread> th;
  th.reserve(nt);
  for (int k = 1; k < nt; ++k) {
    const int b = (int)((int64_t)n * k / nt), e = (int)((int64_t)n * (k + 1) / nt);
    try {
      th.emplace_back(f, b, e);
    } catch (...) {  // no thread to be had
      f(b, e);
    }
  }
  f(0, (int)((int64_t)n / nt));
  for (std::thread &x : th) x.join();
}

struct BvhParams {
  int bins = 32;          // SAH bins per axis
  float cost_trav = 1.0f; // SAH traversal cost (relative to one triangle test)
  float cost_tri = 1.0f;
  int leaf_max = 8;       // largest leaf the SAH may choose (hard cap 16)
  int sah_depth = 40;     // below this depth, object-median splits only (bounds the tree depth)
  int threads = 0;        // 0 = hardware concurrency
  int width = 2;          // node width of the device layout: 2, 4 or 8
  bool quantize = false;  // 4- / 8-wide: child boxes as 8-bit conservative offsets (64 / 96 B per node)
};

struct BvhOut {
  std::vector<int32_t> perm;   // slot -> original triangle index
  std::vector<float4> node2;   // nodes the device walks: 8 float4 each for full precision (four children)
  std::vector<float4> node_own;  // width 8: the layout's own nodes, 16 float4 each
  int width = 2;               // node width of the layout (a wide layout falls back to 2 if its stack bound is exceeded)
  int two_child_nodes = 0;     // inner nodes of the binary tree (1 for a lone leaf)
  bool quantized = false;      // node2 holds quantized wide nodes
  int stack_need = 0;          // deepest traversal stack the device layout can require
  std::vector<float> ref_min, ref_max;  // reference layout, [N][3]
  std::vector<int4> ref_link;           // (left, right, num_tris, tri_start); leaf: left = right = -1, or its halves
  int num_ref_nodes = 0;                // nodes of the tree; the halves of big leaves follow them (two-child layout)
  int max_depth = 0;
  int leaves = 0;
  double sah_cost = 0.0;
};

// Binned-SAH build over the triangles' bounding boxes and centroids.
bool build_bvh_binned(int T, const float *v0, const float *v1, const float *v2, const BvhParams &p, BvhOut &out,
                      std::string &err);

// float4s per node of a node array of this many children (quantized: child
// boxes as bytes relative to the node's origin -- 4 float4 for 4-wide, 6 for 8-wide).
inline int node_float4s(int width, bool quantized = false) {
  if (quantized) return width == 8 ? 6 : 4;
  return width == 8 ? 16 : 8;
}
// the device layout id: the node width, plus one for quantized child boxes (5, 9)
inline int layout_id(int width, bool quantized) { return quantized && width >= 4 ? width + 1 : width; }

// Adopt a tree given in the reference layout (e.g. produced by the reference's
// own build_bvh, main.py:437-507): perm[slot] = original triangle index.
bool bvh_from_reference(int T, const float *v0, const float *v1, const float *v2, int N, const float *nmin,
                        const float *nmax, const int32_t *left, const int32_t *right, const int32_t *ntris,
                        const int32_t *tstart, const int32_t *perm, BvhOut &out, std::string &err,
                        int width = 2, bool quantize = false);

}  // namespace ts
