// Batched renderer: many scenes (each a context with its own BVH, materials,
// camera, resolution, depth and film) in one persistent launch per step.
//
// A step renders one whole spectral block (B passes, one per band) of every
// active scene: the work pool is the concatenation of the scenes' B x W x H
// paths, so small frames no longer leave most of the 148 SMs idle and one
// scene's long paths overlap another's short ones.  Each lane finds the scene
// of its work item by binary search in a block-shared copy of the slot table
// and advances its path with the plain megakernel's vertex step
// (mega_path.cuh), so every scene gets exactly the paths ts_render_pass would
// give it.  Pass counters live in device memory and advance on the device,
// so the four kernels of a step (prepare, render, accumulate, advance) are
// captured once as a CUDA graph and replayed step after step.
#include "batch.cuh"
#include "mega_path.cuh"

namespace ts {

namespace {

// per step: work items of each active slot and the pool size; zero the pool counter
__global__ void k_batch_prepare(BatchSlot *slots, int n, BatchHeader *h, const int *__restrict__ active) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  int run = 0;
  for (int i = 0; i < n; ++i) {
    BatchSlot &sl = slots[i];
    sl.active = active[i];
    sl.npass = sl.active ? sl.c.B : 0;
    sl.item0 = run;
    sl.items = sl.npass * sl.c.W * sl.c.H;
    run += sl.items;
  }
  h->total = run;
  h->counter = 0;
}

// kTogether: the block's warps take each vertex together (mega_vertex)
template <int W, int kMinBlocks, bool kTogether>
__global__ void __launch_bounds__(128, kMinBlocks) k_render_batch(const BatchSlot *__restrict__ slots, int n,
                                                      BatchHeader *__restrict__ h, uint32_t *__restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BatchSlot *sh = reinterpret_cast<BatchSlot *>(smem_raw);
  {
    const int words = n * (int)(sizeof(BatchSlot) / 4);
    const uint32_t *src = reinterpret_cast<const uint32_t *>(slots);
    uint32_t *dst = reinterpret_cast<uint32_t *>(smem_raw);
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int total = h->total;
  uint32_t errbits = 0;
  bool exhausted = false;
  MegaCounts cnt;
  MegaLane L;
  L.pix = -1;
  int slot = 0;
  for (;;) {
    const bool need = L.pix < 0 && !exhausted;
    const unsigned m = __ballot_sync(0xffffffffu, need);
    if (m) {
      const int leader = __ffs(m) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(&h->counter, __popc(m));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (need) {
        const int idx = base + __popc(m & ((1u << lane) - 1u));
        if (idx < total) {
          slot = batch_find_slot(sh, n, idx);
          const BatchSlot &sl = sh[slot];
          const int npix = sl.c.W * sl.c.H;
          const int local = idx - sl.item0;
          const int po = local / npix;
          int band = sl.band0 + po;
          if (band >= sl.c.B) band -= sl.c.B;
          mega_start(sl.s, sl.c, L, sl.pass0 + (uint32_t)po, band, local - po * npix);
        } else {
          exhausted = true;
        }
      }
    }
    if (kTogether ? __syncthreads_or(L.pix >= 0) == 0 : __ballot_sync(0xffffffffu, L.pix >= 0) == 0) break;
    const BatchSlot &sl = sh[slot];
    mega_vertex<W, false, kTogether, true>(sl.s, sl.c, sl.f, L, errbits, cnt, true);
  }
  if (errbits) atomicOr(err, errbits);
}

// average_and_reset_block of every scene that rendered this step (grid.y = slot)
__global__ void k_batch_accumulate(const BatchSlot *__restrict__ slots) {
  const BatchSlot &sl = slots[blockIdx.y];
  if (!sl.npass) return;
  const Film f = sl.f;
  const size_t total = (size_t)f.W * f.H * f.B;
  const int n = sl.nblocks + 1;
  const double inv_n = 1.0 / (double)n;
  const double nm1 = (double)(n - 1);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const double b = f.block[i];
    f.mean[i] = (f.mean[i] * nm1 + b) * inv_n;
    f.m2[i] += b * b;
    f.block[i] = 0.0;
  }
}

__global__ void k_batch_advance(BatchSlot *slots, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !slots[i].npass) return;
  slots[i].pass0 += (uint32_t)slots[i].npass;
  slots[i].nblocks += 1;
}

}  // namespace

size_t batch_smem_bytes(int n) { return (size_t)n * sizeof(BatchSlot); }

namespace {
template <int W>
auto batch_kernel(int occupancy, bool together) {
  if (occupancy >= 8) return together ? k_render_batch<W, 8, true> : k_render_batch<W, 8, false>;
  return together ? k_render_batch<W, 5, true> : k_render_batch<W, 5, false>;
}
auto batch_kernel(int width, int occupancy, bool together) {
  return width == 9   ? batch_kernel<9>(occupancy, together)
         : width == 5 ? batch_kernel<5>(occupancy, together)
         : width == 8 ? batch_kernel<8>(occupancy, together)
         : width == 4 ? batch_kernel<4>(occupancy, together)
                      : batch_kernel<2>(occupancy, together);
}
}  // namespace

cudaError_t launch_batch_step(BatchSlot *slots, int n, BatchHeader *h, const int *active, uint32_t *err, int width,
                              int grid, int block, int acc_blocks, cudaStream_t st, int occupancy, bool together) {
  k_batch_prepare<<<1, 32, 0, st>>>(slots, n, h, active);
  const size_t smem = batch_smem_bytes(n);
  block = block > 128 ? 128 : block;
  batch_kernel(width, occupancy, together)<<<grid, block, smem, st>>>(slots, n, h, err);
  k_batch_accumulate<<<dim3(acc_blocks, n), 256, 0, st>>>(slots);
  k_batch_advance<<<(n + 127) / 128, 128, 0, st>>>(slots, n);
  return cudaGetLastError();
}

cudaError_t launch_batch_prepare(BatchSlot *slots, int n, BatchHeader *h, const int *active, cudaStream_t st) {
  k_batch_prepare<<<1, 32, 0, st>>>(slots, n, h, active);
  return cudaGetLastError();
}

cudaError_t launch_batch_finish(BatchSlot *slots, int n, int acc_blocks, cudaStream_t st) {
  k_batch_accumulate<<<dim3(acc_blocks, n), 256, 0, st>>>(slots);
  k_batch_advance<<<(n + 127) / 128, 128, 0, st>>>(slots, n);
  return cudaGetLastError();
}

// A function's limit is the process's: every batch sets the same one, so that a
// small batch does not lower it under a larger one.
cudaError_t batch_set_smem_limit(int width, int occupancy, bool together) {
  return cudaFuncSetAttribute(batch_kernel(width, occupancy, together), cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)batch_smem_bytes(kBatchMaxScenes));
}

}  // namespace ts
