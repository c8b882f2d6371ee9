// Film kernels (average_and_reset_block, color_rays, clear_pixel_space,
// visualize_normals of the reference, main.py:1592-1674) and the batched
// closest-hit query used by parity checks.
#include <algorithm>

#include "estimator.cuh"
#include "kernels.cuh"

namespace ts {

namespace {

constexpr int kThreads = 256;
constexpr int kTied = -2;               // tri_orig of a ray that k_trace_batch_ties decides

inline int grid_for(size_t n) {
  size_t g = (n + kThreads - 1) / kThreads;
  if (g > (1u << 20)) g = 1u << 20;
  return (int)(g ? g : 1);
}

// average_and_reset_block, main.py:1592-1607: running mean over blocks, and
// the per-cell sum of squared block values for the Monte Carlo error.
__global__ void k_accumulate(Film f, int n) {
  const size_t total = (size_t)f.W * f.H * f.B;
  const double inv_n = 1.0 / (double)n;
  const double nm1 = (double)(n - 1);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const double b = f.block[i];
    f.mean[i] = (f.mean[i] * nm1 + b) * inv_n;
    f.m2[i] += b * b;
    f.block[i] = 0.0;
  }
}

__global__ void k_clear(Film f) {
  const size_t total = (size_t)f.W * f.H * f.B;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    f.block[i] = 0.0;
    f.mean[i] = 0.0;
    f.m2[i] = 0.0;
  }
}

// The colour-matching functions as doubles, once per block: converting them at
// each pixel and band kept the conversion unit busier than the memory.
constexpr int kMaxBands = 64;
__device__ __forceinline__ void load_cmf(const float *__restrict__ cmf, int B, double *sh) {
  for (int i = threadIdx.x; i < 3 * B; i += blockDim.x) sh[i] = (double)cmf[i];
  __syncthreads();
}

// sum_k mean_k * cmf_k of one pixel, in band order
__device__ __forceinline__ void pixel_xyz(const Film &f, const double *cmf, int npix, int p, double scale, float &x,
                                          float &y, float &z) {
  double X = 0.0, Y = 0.0, Z = 0.0;
#pragma unroll 5
  for (int k = 0; k < f.B; ++k) {
    const double a = f.mean[(size_t)k * npix + p];
    X += a * cmf[3 * k + 0];
    Y += a * cmf[3 * k + 1];
    Z += a * cmf[3 * k + 2];
  }
  x = (float)(X * scale);
  y = (float)(Y * scale);
  z = (float)(Z * scale);
}

// XYZ half of color_rays (main.py:1617-1620): sum_k mean_k * cmf_k * scale,
// scale = step / normalisation.  Output [j][i][3] float32 at render resolution.
// HBM-bound: 200 B read and 12 B written per pixel.  Five bands' loads in flight
// per thread; 1024^2: 47 us with a band at a time, 34 us now (34 us at a copy's rate).
__global__ void k_resolve_xyz(const Film f, const float *__restrict__ cmf, double scale, float *__restrict__ xyz) {
  __shared__ double cmf64[3 * kMaxBands];
  load_cmf(cmf, f.B, cmf64);
  const int npix = f.W * f.H;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
    float x, y, z;
    pixel_xyz(f, cmf64, npix, p, scale, x, y, z);
    xyz[3 * (size_t)p + 0] = x;
    xyz[3 * (size_t)p + 1] = y;
    xyz[3 * (size_t)p + 2] = z;
  }
}

// XYZ -> RGB, Reinhard with exposure, gamma (main.py:1621-1629)
__device__ __forceinline__ void display_rgb(float x, float y, float z, const ColorMatrix &M, float exposure,
                                            float gamma, float *__restrict__ rgb) {
  for (int ch = 0; ch < 3; ++ch) {
    const float h = M.m[3 * ch + 0] * x + M.m[3 * ch + 1] * y + M.m[3 * ch + 2] * z;
    const float e = exposure * h;
    const float mapped = e / (e + 1.0f);
    rgb[ch] = powf(mapped, 1.0f / gamma);
  }
}

// source pixel of image pixel i of n (nearest neighbour, main.py:1613-1615)
__device__ __forceinline__ int source_of(int i, int n, int size) {
  return (int)((float)i / (float)n * (float)size);
}

// Whole color_rays (main.py:1609-1629), every image pixel by itself:
// nearest-neighbour, XYZ -> RGB, tone mapping.  Output [j][i][3].
__global__ void k_resolve_rgb(const Film f, const float *__restrict__ cmf, double scale, const __grid_constant__ ColorMatrix M,
                              float exposure, float gamma, int iw, int ih, float *__restrict__ rgb) {
  __shared__ double cmf64[3 * kMaxBands];
  load_cmf(cmf, f.B, cmf64);
  const int npix = f.W * f.H;
  const int n = iw * ih;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int i = p % iw, j = p / iw;
    float x, y, z;
    pixel_xyz(f, cmf64, npix, source_of(j, ih, f.H) * f.W + source_of(i, iw, f.W), scale, x, y, z);
    display_rgb(x, y, z, M, exposure, gamma, rgb + 3 * (size_t)p);
  }
}

// color_rays at render resolution: the colours that the image repeats
__global__ void k_frame_rgb(const Film f, const float *__restrict__ cmf, double scale, const __grid_constant__ ColorMatrix M,
                            float exposure, float gamma, float *__restrict__ rgb) {
  __shared__ double cmf64[3 * kMaxBands];
  load_cmf(cmf, f.B, cmf64);
  const int npix = f.W * f.H;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
    float x, y, z;
    pixel_xyz(f, cmf64, npix, p, scale, x, y, z);
    display_rgb(x, y, z, M, exposure, gamma, rgb + 3 * (size_t)p);
  }
}

// nearest-neighbour upscale, a row of the image per block row
__global__ void k_upscale(const float *__restrict__ src, int W, int H, int iw, int ih, float *__restrict__ dst) {
  for (int j = blockIdx.y; j < ih; j += gridDim.y) {
    const float *row = src + 3 * (size_t)source_of(j, ih, H) * W;
    float *out = dst + 3 * (size_t)j * iw;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < iw; i += gridDim.x * blockDim.x) {
      const float *s = row + 3 * (size_t)source_of(i, iw, W);
      const float r = s[0], g = s[1], b = s[2];
      float *o = out + 3 * (size_t)i;
      o[0] = r;
      o[1] = g;
      o[2] = b;
    }
  }
}

// visualize_normals, main.py:1631-1659 (render-resolution part)
template <int W>
__global__ void k_normals(const __grid_constant__ DevScene s, const __grid_constant__ DevConfig c, float *__restrict__ out, uint32_t *err) {
  const int npix = c.W * c.H;
  uint32_t eb = 0;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
    const int i = p % c.W, j = p / c.W;
    const float u = ((float)i + 0.5f) / (float)c.W;
    const float v = ((float)j + 0.5f) / (float)c.H;
    const float3 d = normalize(s.cam_u * ((u * 2.0f - 1.0f) * c.aspect * c.fov) +
                               s.cam_v * ((v * 2.0f - 1.0f) * c.fov) - s.cam_w * 2.0f);
    const Hit h = trace_closest<W>(s, s.cam_o, d, c.eps, eb);
    float3 col = f3(0.f, 0.f, 0.f);
    if (h.slot >= 0) col = surface_info(s, h, d).ns * 0.5f + f3(0.5f, 0.5f, 0.5f);
    out[3 * (size_t)p + 0] = col.x;
    out[3 * (size_t)p + 1] = col.y;
    out[3 * (size_t)p + 2] = col.z;
  }
  if (eb) atomicOr(err, eb);
}

// the reference-order query
__global__ void k_trace_batch(const __grid_constant__ DevScene s, float eps, const float *__restrict__ rays, int n,
                              int32_t *__restrict__ tri_orig, float *__restrict__ t, float *__restrict__ u,
                              float *__restrict__ v, uint32_t *err) {
  uint32_t eb = 0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const float *q = rays + 6 * (size_t)r;
    const Hit h = trace_reference_order(s, f3(q[0], q[1], q[2]), f3(q[3], q[4], q[5]), eps, eb);
    tri_orig[r] = h.slot >= 0 ? __float_as_int(__ldg(s.tri + 3 * (size_t)h.slot).w) : -1;
    t[r] = h.t;
    if (u) u[r] = h.u;
    if (v) v[r] = h.v;
  }
  if (eb) atomicOr(err, eb);
}

// The fast query with a ray per lane: a warp has `chunk` consecutive rays, and the
// lanes whose rays have ended take the next of them once 16 wait (one look every
// four phases), so that it does not idle behind its longest ray.
template <int W>
__global__ void __launch_bounds__(kThreads, 4) k_trace_batch_lanes(const __grid_constant__ DevScene s, float eps,
                                                                   const float *__restrict__ rays, int n, int chunk,
                                                                   int32_t *__restrict__ tri_orig,
                                                                   float *__restrict__ t, float *__restrict__ u,
                                                                   float *__restrict__ v, uint32_t *err) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t warp = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  int next = (int)min((int64_t)n, warp * chunk);
  const int end = (int)min((int64_t)n, (warp + 1) * chunk);
  uint32_t eb = 0;
  Traversal g;
  g.node = kTravDone;
  g.tie = 0;
  int2 stack[kWideStack];
  int r = -1;  // this lane's ray
  for (;;) {
    const bool done = g.node == kTravDone;
    const unsigned idle = __ballot_sync(kFull, done && (r >= 0 || next < end));
    if (__popc(idle) >= 16 || __ballot_sync(kFull, !done) == 0) {
      if (done && r >= 0) {
        tri_orig[r] = trav_tied<W>(g)    ? kTied
                      : g.h.slot >= 0 ? __float_as_int(__ldg(s.tri + 3 * (size_t)g.h.slot).w)
                                      : -1;
        t[r] = g.h.t;
        if (u) u[r] = g.h.u;
        if (v) v[r] = g.h.v;
        r = -1;
      }
      __syncwarp();
      const unsigned want = __ballot_sync(kFull, r < 0);
      const int mine = next + __popc(want & ((1u << lane) - 1u));
      if (r < 0 && mine < end) {
        r = mine;
        const float *q = rays + 6 * (size_t)r;
        trav_begin<W>(s, g, f3(q[0], q[1], q[2]), f3(q[3], q[4], q[5]), 1e9f);
      }
      next = min(end, next + __popc(want));
      if (__ballot_sync(kFull, r >= 0) == 0) break;
    }
#pragma unroll 1
    for (int i = 0; i < 4; ++i)
      if (!warp_phase<Nodes<W>::value>(s, g, stack, eps, eb)) break;
  }
  if (eb) atomicOr(err, eb);
}

// the rays whose hit a tie left open
template <int W>
__global__ void k_trace_batch_ties(const __grid_constant__ DevScene s, float eps, const float *__restrict__ rays, int n,
                                   int32_t *__restrict__ tri_orig, float *__restrict__ t, float *__restrict__ u,
                                   float *__restrict__ v, uint32_t *err) {
  uint32_t eb = 0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    if (tri_orig[r] != kTied) continue;
    const float *q = rays + 6 * (size_t)r;
    const Hit h = trace_plain<W>(s, f3(q[0], q[1], q[2]), f3(q[3], q[4], q[5]), eps, eb, 1e9f);
    tri_orig[r] = h.slot >= 0 ? __float_as_int(__ldg(s.tri + 3 * (size_t)h.slot).w) : -1;
    t[r] = h.t;
    if (u) u[r] = h.u;
    if (v) v[r] = h.v;
  }
  if (eb) atomicOr(err, eb);
}

// The fast query with a group of lanes per ray, `share` rays to a warp
template <int W>
__global__ void __launch_bounds__(kThreads, 2) k_trace_batch_groups(const __grid_constant__ DevScene s, float eps,
                                                                    const float *__restrict__ rays, int n, int share,
                                                                    int32_t *__restrict__ tri_orig,
                                                                    float *__restrict__ t, float *__restrict__ u,
                                                                    float *__restrict__ v, uint32_t *err) {
  constexpr int G = kGroupLanes;
  __shared__ int2 stacks[kGroupStack * (kThreads / G)];
  const int lane = threadIdx.x & 31, sub = lane & (G - 1), shift = lane & ~(G - 1);
  const int warp = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  const int64_t r = (int64_t)warp * share + lane / G;
  const bool active = lane / G < share && r < n;
  uint32_t eb = 0;
  GroupRay<G> g;
  float3 o = f3(0.f, 0.f, 0.f), d = o;
  if (active) {
    const float *q = rays + 6 * (size_t)r;
    o = f3(q[0], q[1], q[2]);
    d = f3(q[3], q[4], q[5]);
  }
  group_begin(s, g, o, d, 1e9f);
  if (!active) g.node = kTravDone;
  while (__any_sync(0xffffffffu, g.node != kTravDone))
    group_step(s, g, stacks + threadIdx.x / G, kThreads / G, sub, shift, eps);
  Hit h;
  const bool good = group_hit(g, shift, h);
  if (active && sub == 0) {
    if (!good) h = trace_plain<W>(s, o, d, eps, eb, 1e9f);
    tri_orig[r] = h.slot >= 0 ? __float_as_int(__ldg(s.tri + 3 * (size_t)h.slot).w) : -1;
    t[r] = h.t;
    if (u) u[r] = h.u;
    if (v) v[r] = h.v;
  }
  if (eb) atomicOr(err, eb);
}

}  // namespace

cudaError_t launch_accumulate_block(Film f, int n, cudaStream_t st) {
  k_accumulate<<<grid_for((size_t)f.W * f.H * f.B), kThreads, 0, st>>>(f, n);
  return cudaGetLastError();
}
cudaError_t launch_clear_film(Film f, cudaStream_t st) {
  k_clear<<<grid_for((size_t)f.W * f.H * f.B), kThreads, 0, st>>>(f);
  return cudaGetLastError();
}
cudaError_t launch_resolve_xyz(Film f, const float *cmf, double scale, float *xyz, cudaStream_t st) {
  k_resolve_xyz<<<grid_for((size_t)f.W * f.H), kThreads, 0, st>>>(f, cmf, scale, xyz);
  return cudaGetLastError();
}
bool resolve_rgb_by_frame(const Film &f, int iw, int ih) {
  // An image of more pixels than the frame repeats them: each is resolved and
  // tone-mapped once, then copied.  us, block average aside, every image pixel by
  // itself / by the frame: 1024^2 to 1600^2 111 / 86, 512^2 to 1024^2 44 / 28, 784x134
  // to 1568x268 28 / 26; but at the frame's size 1024^2 62 / 78, 700^2 31 / 46, and small
  // images are shorter than the second launch: 256^2 to 512^2 23 / 24.  In one kernel,
  // whose blocks kept the colours under a tile of the image in shared memory, 1600^2
  // took 138.
  return 2 * (int64_t)iw * ih >= 3 * (int64_t)f.W * f.H && (int64_t)iw * ih > (1 << 18);
}
cudaError_t launch_resolve_rgb(Film f, const float *cmf, double scale, float *frame_rgb, ColorMatrix M, float exposure,
                               float gamma, int iw, int ih, float *rgb, cudaStream_t st) {
  if (frame_rgb) {
    k_frame_rgb<<<grid_for((size_t)f.W * f.H), kThreads, 0, st>>>(f, cmf, scale, M, exposure, gamma, frame_rgb);
    const dim3 grid((unsigned)((iw - 1) / kThreads + 1), (unsigned)std::min(ih, 65535));
    k_upscale<<<grid, kThreads, 0, st>>>(frame_rgb, f.W, f.H, iw, ih, rgb);
  } else {
    k_resolve_rgb<<<grid_for((size_t)iw * ih), kThreads, 0, st>>>(f, cmf, scale, M, exposure, gamma, iw, ih, rgb);
  }
  return cudaGetLastError();
}
cudaError_t launch_render_normals(const DevScene &s, const DevConfig &c, float *out, uint32_t *err,
                                  cudaStream_t st) {
  const int g = grid_for((size_t)c.W * c.H);
  if (s.node_width == 9) k_normals<9><<<g, kThreads, 0, st>>>(s, c, out, err);
  else if (s.node_width == 5) k_normals<5><<<g, kThreads, 0, st>>>(s, c, out, err);
  else if (s.node_width == 8) k_normals<8><<<g, kThreads, 0, st>>>(s, c, out, err);
  else if (s.node_width == 4) k_normals<4><<<g, kThreads, 0, st>>>(s, c, out, err);
  else k_normals<2><<<g, kThreads, 0, st>>>(s, c, out, err);
  return cudaGetLastError();
}
cudaError_t launch_trace_batch(const DevScene &s, float eps, const float *rays, int n, int mode, int32_t *tri_orig,
                               float *t, float *u, float *v, uint32_t *err, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (mode != 0) {
    k_trace_batch<<<grid_for((size_t)n), kThreads, 0, st>>>(s, eps, rays, n, tri_orig, t, u, v, err);
    return cudaGetLastError();
  }
  // A group of lanes per ray while a ray per lane would leave the schedulers idle, or
  // wait for a large tree's nodes.  A ray per lane has a second launch for ties in the
  // two- and eight-child layouts; the eight-child one's groups have more ties to decide.
  // us, lanes / groups, layouts of two, four and eight children: 2,062 triangles 16k
  // rays 58 / 43, 52 / 40, 53 / 42; 64k 63 / 56, 54 / 50, 61 / 55; 80k 62 / 59, 58 / 60,
  // 58 / 64; 100k 65 / 63, 60 / 65, 64 / 70; 125k 68 / 71, 69 / 76, 64 / 79; 647,258
  // triangles 64k 121 / 104, 110 / 107, 125 / 111; 100k 134 / 128, 125 / 124 (another
  // 100k 158 / 133), 136 / 152; 150k 151 / 160, 154 / 163, 168 / 180.
  const bool large = s.num_tris > kTogetherTris;
  const int most = kSMs * (s.node_width == 8 ? 512 : large ? 1024 : s.node_width == 2 ? 768 : 512);
  if (n <= most && s.node_width != 5 && s.node_width != 9) {
    const int share = std::min(32 / kGroupLanes, std::max(1, n / (kSMs * 16)));
    const int warps = (n - 1) / share + 1;
    const auto k = s.node_width == 8   ? k_trace_batch_groups<8>
                   : s.node_width == 4 ? k_trace_batch_groups<4>
                                       : k_trace_batch_groups<2>;
    k<<<(warps - 1) / (kThreads / 32) + 1, kThreads, 0, st>>>(s, eps, rays, n, share, tri_orig, t, u, v, err);
    return cudaGetLastError();
  }
  const int blocks = std::min(kSMs * 4, (n - 1) / kThreads + 1);
  const int warps = blocks * (kThreads / 32);
  const auto k = s.node_width == 9   ? k_trace_batch_lanes<9>
                 : s.node_width == 5 ? k_trace_batch_lanes<5>
                 : s.node_width == 8 ? k_trace_batch_lanes<8>
                 : s.node_width == 4 ? k_trace_batch_lanes<4>
                                     : k_trace_batch_lanes<2>;
  k<<<blocks, kThreads, 0, st>>>(s, eps, rays, n, (n - 1) / warps + 1, tri_orig, t, u, v, err);
  const int tg = std::min(kSMs * 8, (n - 1) / kThreads + 1);
  if (s.node_width == 2) k_trace_batch_ties<2><<<tg, kThreads, 0, st>>>(s, eps, rays, n, tri_orig, t, u, v, err);
  if (s.node_width == 8) k_trace_batch_ties<8><<<tg, kThreads, 0, st>>>(s, eps, rays, n, tri_orig, t, u, v, err);
  return cudaGetLastError();
}

}  // namespace ts
