// Plain single-scene renderer: one persistent megakernel per launch.
//
// Each lane owns one path (one pixel of cast_rays, main.py:1502-1590) and
// advances it one path vertex per loop iteration (mega_path.cuh).  Lanes whose
// path has ended fetch the next work item with one warp-aggregated atomic, so
// a warp stays full until the pool is exhausted (path regeneration) instead of
// idling behind its longest path.  A launch covers npass consecutive passes
// (a wavelength bundle): work item idx is pixel idx % npix of pass
// pass0 + idx / npix at band (band0 + idx / npix) mod B.  Bands of one launch
// are distinct; fluorescence can still move deposits into another pass's band,
// so multi-pass launches flush with atomics.
#include "mega_path.cuh"

namespace ts {

namespace {

// kCount: also count the work (for the roofline's algorithmic bytes):
// work[0..7] = paths, path vertices, traversals, node visits, triangle tests,
// surface hits resolved, film deposits, (unused).
// kMinBlocks: resident blocks of 128 threads per SM the compiler must allow
// (5: 96 registers; four children spill nothing, the layouts that hand ties to
// trace_plain(), two and eight children, 25 to 90 B, quantized nodes 10 to 210 B.
// 8: 64 registers with 250 B to 1.2 KB of spills -- more warps to hide the node-fetch
// latency, faster on large frames).
// kTogether: the block's warps take each vertex together (mega_vertex).
template <int W, bool kCount, int kMinBlocks = 5, bool kTogether = false>
__global__ void __launch_bounds__(128, kMinBlocks) k_render_mega(const __grid_constant__ DevScene s, const __grid_constant__ DevConfig c, uint32_t pass0, int npass, int band0,
                                                     Film f, int *__restrict__ counter, uint32_t *__restrict__ err,
                                                     unsigned long long *__restrict__ work) {
  const int lane = threadIdx.x & 31;
  MegaCounts cnt;
  const int npix = c.W * c.H;
  const int total = npix * npass;
  uint32_t errbits = 0;
  // Few paths: fewer lanes of each warp rather than fewer warps, whose lanes'
  // branches run one after the other.  us per pass, full warps / so: box 32^2
  // 513 / 193, 64^2 506 / 316; terrain 64^2 391 / 241; volume 32^2 3141 / 1081.
  const int warps = (int)min((int64_t)gridDim.x * (blockDim.x >> 5), (int64_t)kSMs * kMinBlocks * 4);  // what the device holds
  bool exhausted = lane >= max(1, (total - 1) / warps + 1);
  MegaLane L;
  L.pix = -1;
  for (;;) {
    const bool need = L.pix < 0 && !exhausted;
    const unsigned m = __ballot_sync(0xffffffffu, need);
    if (m) {
      const int leader = __ffs(m) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(counter, __popc(m));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (need) {
        const int idx = base + __popc(m & ((1u << lane) - 1u));
        if (idx < total) {
          const int po = idx / npix;
          int band = band0 + po;
          if (band >= c.B) band -= c.B;
          if (kCount) cnt.paths++;
          mega_start(s, c, L, pass0 + (uint32_t)po, band, idx - po * npix, idx);
        } else {
          exhausted = true;
        }
      }
    }
    if (kTogether ? __syncthreads_or(L.pix >= 0) == 0 : __ballot_sync(0xffffffffu, L.pix >= 0) == 0) break;
    mega_vertex<W, kCount, kTogether, false>(s, c, f, L, errbits, cnt, npass > 1);
  }
  if (errbits) atomicOr(err, errbits);
  if (kCount) {
    atomicAdd(work + 0, (unsigned long long)cnt.paths);
    atomicAdd(work + 1, (unsigned long long)cnt.vert);
    atomicAdd(work + 2, (unsigned long long)cnt.trace);
    atomicAdd(work + 3, (unsigned long long)cnt.tc.nodes);
    atomicAdd(work + 4, (unsigned long long)cnt.tc.tris);
    atomicAdd(work + 5, (unsigned long long)cnt.hit);
    atomicAdd(work + 6, (unsigned long long)cnt.dep);
  }
}

template <int W>
void launch_w(const DevScene &s, const DevConfig &c, uint32_t pass0, int npass, int band0, Film f, int *counter,
              uint32_t *err, int grid, int block, cudaStream_t st, unsigned long long *work, int occupancy) {
  // Together where shading, not the length of single traversals, takes the time:
  // small trees and enough paths.  us per pass apart / together: box (2,062
  // triangles) 64^2 306 / 316, 128^2 565 / 468, 192^2 737 / 584, 512^2 1570 / 1217,
  // volume (20,014) 128^2 3373 / 2640, 192^2 4183 / 3535.  By the size of the tree,
  // 256^2, 512^2 and a bundle of 25 at 256^2: terrain of 33,000 triangles 421 / 409, 630 /
  // 586, 2923 / 2493; 65,000 451 / 459, 658 / 635, 3058 / 2678; 130,000 482 / 504, 715 /
  // 696, 3253 / 2941; 647,258 570 / 590, 814 / 883, 3584 / 3559; volume of 60,000 5151 /
  // 4881, 12081 / 12092, 63878 / 57318; 200,000 5437 / 5381, 12806 / 13360, 67290 / 63059.
  const bool together = s.num_tris <= kTogetherTris && (int64_t)c.W * c.H * npass >= 16384;
  // Unless the caller chose, 64 registers where there are paths for the 8 blocks of
  // an SM that they allow, several for each lane; with fewer paths the spills cost
  // more than the warps hide.  us at 96 / 64 registers: bundles of 25 at 128^2
  // (409,600 paths) box 1857 / 1889, volume 17507 / 15320, terrain (20,000) 910 /
  // 835, (647,258) 1283 / 1263; at 256^2 (1.6M) 6131 / 5738, 64199 / 52926, 2745 /
  // 2349, 3957 / 3616; a pass at 512^2 (262,144) 1223 / 1245, 10952 / 9951, 540 / 572,
  // 797 / 890; at 256^2 (65,536) 669 / 845, 4433 / 5140, 365 / 375, 547 / 548.
  const bool narrow = occupancy >= 8 || (occupancy == 0 && (int64_t)c.W * c.H * npass >= (1 << 19));
  const auto k = work     ? k_render_mega<W, true>
                 : narrow ? (together ? k_render_mega<W, false, 8, true> : k_render_mega<W, false, 8>)
                          : (together ? k_render_mega<W, false, 5, true> : k_render_mega<W, false>);
  k<<<grid, block, 0, st>>>(s, c, pass0, npass, band0, f, counter, err, work);
}

}  // namespace

cudaError_t launch_render_mega(const DevScene &s, const DevConfig &c, uint32_t pass, int band, Film f,
                               int *counter, uint32_t *err, int grid, int block, cudaStream_t st,
                               unsigned long long *work, int npass, int occupancy) {
  cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  block = block > 128 ? 128 : block;  // the kernel is compiled for blocks of at most 128 threads
  if (s.node_width == 9) launch_w<9>(s, c, pass, npass, band, f, counter, err, grid, block, st, work, occupancy);
  else if (s.node_width == 5) launch_w<5>(s, c, pass, npass, band, f, counter, err, grid, block, st, work, occupancy);
  else if (s.node_width == 8) launch_w<8>(s, c, pass, npass, band, f, counter, err, grid, block, st, work, occupancy);
  else if (s.node_width == 4) launch_w<4>(s, c, pass, npass, band, f, counter, err, grid, block, st, work, occupancy);
  else launch_w<2>(s, c, pass, npass, band, f, counter, err, grid, block, st, work, occupancy);
  return cudaGetLastError();
}

}  // namespace ts
