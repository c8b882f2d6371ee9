// Closest-hit BVH traversal on the device.
//
// Semantics follow trace() in main.py:831-864 of the reference: a triangle is
// accepted when its Moller-Trumbore distance t satisfies EPSILON < t < best
// (strict, so the first-visited of two exactly equal distances wins), a box
// is entered when t_enter < t_exit && t_exit > 0 (main.py:797-805), and the
// miss distance is 1e9.  Box and triangle tests use one IEEE rounding per
// operation (no FMA contraction) so that distances are bit-identical to the
// CPU oracle's.
//
// trace_closest() is the fast path: wide nodes, nearest child
// first, and boxes whose entry distance lies beyond the current best hit (by
// a relative margin of 2^-16, far larger than the rounding error of the box
// and triangle distances) are skipped.  The reference never skips boxes, so
// the closest hit differs only where two triangles' distances tie within the
// margin -- the "near tie" case the parity tests count.
//
// trace_reference_order() walks the reference-layout node table exactly like
// the reference: explicit 64-entry stack, left pushed before right (so right
// is popped first), no distance culling.
#pragma once
#include <climits>

#include "common.cuh"

namespace ts {

struct Hit {
  float t, u, v;
  int slot;  // triangle slot (BVH order); -1 on miss
};

// intersect_triangle (main.py:807-829): returns t, or -1 on miss.
TS_D float tri_hit(float3 o, float3 d, float4 A, float4 E1, float4 E2, float eps, float &u, float &v) {
  const float3 e1 = xyz(E1), e2 = xyz(E2);
  const float3 p = xcross(d, e2);
  const float det = xdot(e1, p);
  if (!(fabsf(det) > 1e-8f)) return -1.f;
  const float inv_det = __frcp_rn(det);
  const float3 tv = xsub3(o, xyz(A));
  const float uu = xmul(xdot(tv, p), inv_det);
  if (!(uu >= 0.f && uu <= 1.f)) return -1.f;
  const float3 q = xcross(tv, e1);
  const float vv = xmul(xdot(d, q), inv_det);
  if (!(vv >= 0.f && xadd(uu, vv) <= 1.f)) return -1.f;
  const float tt = xmul(xdot(e2, q), inv_det);
  if (!(tt > eps)) return -1.f;
  u = uu;
  v = vv;
  return tt;
}

// slab test for one box; returns entry/exit distances
TS_D void box_hit(float lox, float hix, float loy, float hiy, float loz, float hiz, float3 o, float3 inv,
                  float &te, float &tx) {
  const float ax = xmul(xsub(lox, o.x), inv.x), bx = xmul(xsub(hix, o.x), inv.x);
  const float ay = xmul(xsub(loy, o.y), inv.y), by = xmul(xsub(hiy, o.y), inv.y);
  const float az = xmul(xsub(loz, o.z), inv.z), bz = xmul(xsub(hiz, o.z), inv.z);
  te = fmaxf(fminf(ax, bx), fmaxf(fminf(ay, by), fminf(az, bz)));
  tx = fminf(fmaxf(ax, bx), fminf(fmaxf(ay, by), fmaxf(az, bz)));
}

TS_D float cull_bound(float best) { return best + best * (1.0f / 65536.0f); }

// Work counters of one traversal (compiled out unless a kernel asks for them).
struct TraceCount {
  uint32_t nodes = 0, tris = 0;
};

constexpr int kTravDone = -2147483647 - 1;  // never a leaf code: first slot < 2^27 - 1

// ------------------------------------------------------------ packed pairs
// Two float32 lanes in one register pair.  sm_100's packed add and multiply
// round each lane like the scalar instruction and take one issue slot.
typedef unsigned long long f32x2;
TS_D f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
TS_D void unpack2(f32x2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
TS_D f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
TS_D f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
TS_D float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
TS_D float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// A 32-byte record in one load.  A scattered load costs L1 one pass per sector
// and lane, so two 16-byte halves cost it twice.
struct Rec32 {
  f32x2 a, b, c, d;
};
TS_D Rec32 load32(const void *p) {
  Rec32 r;
  asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(r.a), "=l"(r.b), "=l"(r.c), "=l"(r.d) : "l"(p));
  return r;
}

// State of a traversal, in registers; the stack of (node, entry-distance bits)
// pairs is owned by the caller, so that a lane can stop between steps.
struct Traversal {
  f32x2 no[3], inv[3];  // per axis the negated origin and the reciprocal direction, in both lanes of a pair
  float3 d;
  float tcull;
  Hit h;
  int node, sp;
  int tie;              // another triangle lies at exactly h.t
};

// one triangle against the ray; keeps the first of equal distances
TS_D void trav_triangle(const DevScene &s, Traversal &t, float3 o, int slot, float eps) {
  const float4 *tp = s.tri + 3 * (size_t)slot;
  const float4 A = __ldg(tp + 0), E1 = __ldg(tp + 1), E2 = __ldg(tp + 2);
  float u, v;
  const float tt = tri_hit(o, t.d, A, E1, E2, eps, u, v);
  if (tt > eps && tt <= t.h.t) {
    if (tt == t.h.t) {
      t.tie = 1;
    } else {
      t.h.t = tt;
      t.h.u = u;
      t.h.v = v;
      t.h.slot = slot;
      t.tcull = fminf(t.tcull, cull_bound(tt));
      t.tie = 0;
    }
  }
}

TS_D float lane0(f32x2 v) {
  float a, b;
  unpack2(v, a, b);
  return a;
}

TS_D float3 trav_origin(const Traversal &t) {
  return f3(-lane0(t.no[0]), -lane0(t.no[1]), -lane0(t.no[2]));
}

// ---- wide nodes (4 or 8 children) ---------------------------------------
template <int W>
TS_D void cswap(float *k, int *r, int i, int j) {
  if (k[j] < k[i]) {
    const float tk = k[i];
    k[i] = k[j];
    k[j] = tk;
    const int tr = r[i];
    r[i] = r[j];
    r[j] = tr;
  }
}

// Sort W (entry distance, link) pairs ascending (misses carry +inf):
// 5-comparator network for 4, Batcher's 19-comparator network for 8.
template <int W>
TS_D void sort_children(float *k, int *r) {
  if (W == 4) {
    cswap<W>(k, r, 0, 1); cswap<W>(k, r, 2, 3); cswap<W>(k, r, 0, 2); cswap<W>(k, r, 1, 3); cswap<W>(k, r, 1, 2);
  } else {
    cswap<W>(k, r, 0, 1); cswap<W>(k, r, 2, 3); cswap<W>(k, r, 4, 5); cswap<W>(k, r, 6, 7);
    cswap<W>(k, r, 0, 2); cswap<W>(k, r, 1, 3); cswap<W>(k, r, 4, 6); cswap<W>(k, r, 5, 7);
    cswap<W>(k, r, 1, 2); cswap<W>(k, r, 5, 6);
    cswap<W>(k, r, 0, 4); cswap<W>(k, r, 1, 5); cswap<W>(k, r, 2, 6); cswap<W>(k, r, 3, 7);
    cswap<W>(k, r, 2, 4); cswap<W>(k, r, 3, 5);
    cswap<W>(k, r, 1, 2); cswap<W>(k, r, 3, 4); cswap<W>(k, r, 5, 6);
  }
}

// Slab test of one child record (lo.x hi.x lo.y hi.y | lo.z hi.z link -): the
// arithmetic of box_hit(), both planes of an axis in one packed operation.
TS_D void child_hit(const Rec32 &c, const f32x2 *no, const f32x2 *inv, float &te, float &tx) {
  float ax, bx, ay, by, az, bz;
  unpack2(mul2(add2(c.a, no[0]), inv[0]), ax, bx);
  unpack2(mul2(add2(c.b, no[1]), inv[1]), ay, by);
  unpack2(mul2(add2(c.c, no[2]), inv[2]), az, bz);
  te = max3(fminf(ax, bx), fminf(ay, by), fminf(az, bz));
  tx = min3(fmaxf(ax, bx), fmaxf(ay, by), fmaxf(az, bz));
}

// ---- quantized wide nodes (layout ids 5: 4 children in 64 B, 9: 8 children in 96 B)
// float4 0 = (origin.xyz, biased scale exponents x, y, z and the child count as
// bytes); then the child refs; then the child boxes as bytes q per plane
// (lo.x hi.x lo.y hi.y lo.z hi.z, one byte per child) with bound = origin + q *
// 2^e, decoded with one IEEE multiply (exact) and one add.  The host rounded
// every byte outwards against exactly this decode, so a decoded box contains
// the exact one: the slab test accepts at least the rays the exact box would,
// entry distances are no larger, and culling stays conservative -- the
// closest hit is the same as with full-precision boxes.
template <int WQ>
TS_D int node_children_q(const DevScene &s, const Traversal &t, float *key, int *ref) {
  constexpr int N = WQ == 9 ? 8 : 4;  // children per node
  constexpr int R = N / 4;            // float4s of refs (and 32-bit words per byte plane)
  constexpr int F = WQ == 9 ? 6 : 4;  // float4s per node
  const float3 o = trav_origin(t), inv = f3(lane0(t.inv[0]), lane0(t.inv[1]), lane0(t.inv[2]));
  const float4 *n = s.node + (size_t)F * t.node;
  const float4 h = __ldg(n);
  const uint32_t meta = __float_as_uint(h.w);
  const float sx = __uint_as_float((meta & 0xffu) << 23);
  const float sy = __uint_as_float(((meta >> 8) & 0xffu) << 23);
  const float sz = __uint_as_float(((meta >> 16) & 0xffu) << 23);
  const int nc = (int)(meta >> 24);
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int4 l = __ldg(reinterpret_cast<const int4 *>(n + 1 + q));
    ref[4 * q + 0] = l.x; ref[4 * q + 1] = l.y; ref[4 * q + 2] = l.z; ref[4 * q + 3] = l.w;
  }
  uint32_t wq[6 * R];  // plane r, children 4j..4j+3 in word r * R + j
  {
    const uint4 *b = reinterpret_cast<const uint4 *>(n + 1 + R);
#pragma unroll
    for (int i = 0; i < (6 * R + 3) / 4; ++i) {
      const uint4 v = __ldg(b + i);
      if (4 * i + 0 < 6 * R) wq[4 * i + 0] = v.x;
      if (4 * i + 1 < 6 * R) wq[4 * i + 1] = v.y;
      if (4 * i + 2 < 6 * R) wq[4 * i + 2] = v.z;
      if (4 * i + 3 < 6 * R) wq[4 * i + 3] = v.w;
    }
  }
  int nh = 0;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int j = k >> 2, sh = 8 * (k & 3);
    const float lox = xadd(h.x, xmul((float)((wq[0 * R + j] >> sh) & 0xffu), sx));
    const float hix = xadd(h.x, xmul((float)((wq[1 * R + j] >> sh) & 0xffu), sx));
    const float loy = xadd(h.y, xmul((float)((wq[2 * R + j] >> sh) & 0xffu), sy));
    const float hiy = xadd(h.y, xmul((float)((wq[3 * R + j] >> sh) & 0xffu), sy));
    const float loz = xadd(h.z, xmul((float)((wq[4 * R + j] >> sh) & 0xffu), sz));
    const float hiz = xadd(h.z, xmul((float)((wq[5 * R + j] >> sh) & 0xffu), sz));
    float te, tx;
    box_hit(lox, hix, loy, hiy, loz, hiz, o, inv, te, tx);
    const bool hit = k < nc && te < tx && tx > 0.f && te <= t.tcull;
    key[k] = hit ? te : INFINITY;
    nh += hit;
  }
  if (nh > 0) sort_children<N>(key, ref);
  return nh;
}

// The children of a wide node that the ray enters, as sorted (entry distance,
// link) pairs; returns how many.
// W: 4; 5 and 9 for quantized nodes.
template <int W>
TS_D int node_children(const DevScene &s, const Traversal &t, float *key, int *ref) {
  if (W == 5 || W == 9) return node_children_q<W>(s, t, key, ref);
  const float4 *n = s.node + (size_t)t.node * (2 * W);
  int nh = 0;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const Rec32 c = load32(n + 2 * k);
    float te, tx;
    child_hit(c, t.no, t.inv, te, tx);
    const bool h = te < tx && tx > 0.f && te <= t.tcull;
    key[k] = h ? te : INFINITY;
    ref[k] = (int)(uint32_t)c.d;
    nh += h;
  }
  if (nh > 0) sort_children<W>(key, ref);
  return nh;
}

// children per node of a layout
template <int W>
struct Children {
  static constexpr int value = W >= 8 ? 8 : 4;
};

TS_D void trav_pop(Traversal &t, const int2 *stack) {
  // the next box that is still closer than the cull bound
  for (;;) {
    if (t.sp == 0) {
      t.node = kTravDone;
      return;
    }
    const int2 e = stack[--t.sp];
    if (__int_as_float(e.y) <= t.tcull) {
      t.node = e.x;
      return;
    }
  }
}

// an inner node: the nearest child the ray enters is visited next, the others
// are pushed (farthest first) with their entry distances
template <int W>
TS_D void trav_inner(const DevScene &s, Traversal &t, int2 *stack, uint32_t &errbits) {
  constexpr int N = Children<W>::value;
  float key[N];
  int ref[N];
  const int nh = node_children<W>(s, t, key, ref);
  if (nh == 0) {
    trav_pop(t, stack);
    return;
  }
  if (t.sp + nh - 1 <= kWideStack) {
#pragma unroll
    for (int k = N - 1; k >= 1; --k)
      if (k < nh) stack[t.sp++] = make_int2(ref[k], __float_as_int(key[k]));
  } else {
    errbits |= kErrStackOverflow;
  }
  t.node = ref[0];
}

// One step of a traversal: an inner node, or a leaf and the pop that follows.
template <int W, bool kCount = false>
TS_D void trav_step(const DevScene &s, Traversal &t, int2 *stack, float eps, uint32_t &errbits,
                    TraceCount *tc = nullptr) {
  if (t.node >= 0) {
    if (kCount) tc->nodes++;
    trav_inner<W>(s, t, stack, errbits);
  } else {
    const int first = ~t.node >> 4, cnt = (~t.node & 15) + 1;
    if (kCount) tc->tris += cnt;
    const float3 o = trav_origin(t);
    for (int i = 0; i < cnt; ++i) trav_triangle(s, t, o, first + i, eps);
    trav_pop(t, stack);
  }
}

// A traversal by itself, to its end.
template <int W, bool kCount = false>
TS_D void trav_run(const DevScene &s, Traversal &t, int2 *stack, float eps, uint32_t &errbits,
                   TraceCount *tc = nullptr) {
  while (t.node != kTravDone) trav_step<W, kCount>(s, t, stack, eps, errbits, tc);
}

// One phase of a warp whose lanes step together: inner nodes, or one triangle of
// a leaf.  A lane at a leaf waits until kLeafLanes lanes are at one, or none has
// a node to test, so that both phases run with many lanes.  When every lane went
// on by itself (a budget of steps, leaves tested as a lane came to them), nodes
// ran with 16 to 19 lanes of 32, but triangles with 4 to 6 and the end of a ray
// with 2 to 4, and these were half of the instructions; in phases the same
// launches take 25 to 29 % fewer instructions.
// Returns false when no lane has anything left (node == kTravDone in all).
constexpr int kLeafLanes = 12;  // 8: 1 % slower, 16: the same, 20: 1 % slower (terrain, box, volume)

template <int W>
TS_D bool warp_phase(const DevScene &s, Traversal &t, int2 *stack, float eps, uint32_t &errbits,
                     unsigned mask = 0xffffffffu) {
  const bool at_leaf = t.node < 0 && t.node != kTravDone;
  const unsigned inner = __ballot_sync(mask, t.node >= 0);
  const unsigned leaf = __ballot_sync(mask, at_leaf);
  if (inner && __popc(leaf) < kLeafLanes) {
    if (t.node >= 0) trav_inner<W>(s, t, stack, errbits);
  } else if (leaf) {
    if (at_leaf) {
      const int code = ~t.node;
      trav_triangle(s, t, trav_origin(t), code >> 4, eps);
      if (code & 15) t.node = ~(code + 15);  // the leaf's next triangle: first + 1, count - 1
      else trav_pop(t, stack);
    }
  } else {
    return false;
  }
  __syncwarp(mask);
  return true;
}

// ---- the layouts' own visiting orders -------------------------------------
// Plain loops with box_hit() in the visiting order that defines a layout's
// results: which of two triangles at exactly the same distance wins.  They
// run for the rays that the fast loops hand over -- a tie, where those loops
// visit in another order -- and for the counting pass.

// two children per node, nearest first, over the reference-layout table; a leaf
// of more than kLeafMax triangles has two halves as its children
template <bool kCount = false>
TS_D Hit trace_two_child(const DevScene &s, float3 o, float3 d, float eps, uint32_t &errbits, TraceCount *tc,
                         float bound) {
  Hit h;
  h.t = 1e9f;
  h.u = h.v = 0.f;
  h.slot = -1;
  if (s.num_ref_nodes <= 0) return h;
  const float3 inv = f3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
  float tcull = cull_bound(fminf(bound, 1e9f));
  int2 stack[kStackDepth];
  int sp = 0;
  auto entry = [&](int ni, float &te) {
    const float *mn = s.ref_min + 3 * (size_t)ni, *mx = s.ref_max + 3 * (size_t)ni;
    float tx;
    box_hit(__ldg(mn), __ldg(mx), __ldg(mn + 1), __ldg(mx + 1), __ldg(mn + 2), __ldg(mx + 2), o, inv, te, tx);
    return te < tx && tx > 0.f && te <= tcull;
  };
  int ni = 0;
  int4 l = __ldg(s.ref_link);
  bool go = true;
  if (l.z > 0 && l.x < 0) {  // the root is a leaf: a node with one child
    float te;
    if (kCount) tc->nodes++;
    go = entry(0, te);
  }
  while (go) {
    bool down = false;
    if (l.z <= 0 || l.x >= 0) {
      float e0, e1;
      if (kCount) tc->nodes++;
      const bool h0 = entry(l.x, e0), h1 = entry(l.y, e1);
      if (h0 && h1) {
        const bool sw = e1 < e0;
        if (sp < kStackDepth) stack[sp++] = sw ? make_int2(l.x, __float_as_int(e0)) : make_int2(l.y, __float_as_int(e1));
        else errbits |= kErrStackOverflow;
        ni = sw ? l.y : l.x;
      } else {
        ni = h0 ? l.x : l.y;
      }
      down = h0 || h1;
    } else {
      if (kCount) tc->tris += l.z;
      for (int i = 0; i < l.z; ++i) {
        const int slot = l.w + i;
        const float4 *tp = s.tri + 3 * (size_t)slot;
        float u, v;
        const float tt = tri_hit(o, d, __ldg(tp), __ldg(tp + 1), __ldg(tp + 2), eps, u, v);
        if (tt > eps && tt < h.t) {
          h.t = tt;
          h.u = u;
          h.v = v;
          h.slot = slot;
          tcull = fminf(tcull, cull_bound(tt));
        }
      }
    }
    while (!down && sp > 0) {
      const int2 e = stack[--sp];
      if (__int_as_float(e.y) <= tcull) {
        ni = e.x;
        down = true;
      }
    }
    go = down;
    if (go) l = __ldg(s.ref_link + ni);
  }
  return h;
}

// 4 or 8 children per node, all that are entered sorted by distance
template <int W, bool kCount = false>
TS_D Hit trace_wide_plain(const DevScene &s, float3 o, float3 d, float eps, uint32_t &errbits, TraceCount *tc,
                          float bound) {
  Hit h;
  h.t = 1e9f;
  h.u = h.v = 0.f;
  h.slot = -1;
  if (s.num_tris <= 0) return h;
  const float3 inv = f3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
  float tcull = cull_bound(fminf(bound, 1e9f));
  int2 stack[kWideStack];
  int sp = 0, node = 0;
  for (;;) {
    if (node >= 0) {
      const float *n = reinterpret_cast<const float *>(s.node_own) + (size_t)(8 * W) * node;
      if (kCount) tc->nodes++;
      float key[W];
      int ref[W];
      int nh = 0;
#pragma unroll
      for (int k = 0; k < W; ++k) {
        float te, tx;
        const float *r = n + 8 * k;
        box_hit(__ldg(r), __ldg(r + 1), __ldg(r + 2), __ldg(r + 3), __ldg(r + 4), __ldg(r + 5), o, inv, te, tx);
        const bool hit = te < tx && tx > 0.f && te <= tcull;
        key[k] = hit ? te : INFINITY;
        ref[k] = __float_as_int(__ldg(r + 6));
        nh += hit;
      }
      if (nh > 0) {
        sort_children<W>(key, ref);
        if (sp + nh - 1 <= kWideStack) {
#pragma unroll
          for (int k = W - 1; k >= 1; --k)
            if (k < nh) stack[sp++] = make_int2(ref[k], __float_as_int(key[k]));
        } else {
          errbits |= kErrStackOverflow;
        }
        node = ref[0];
        continue;
      }
    } else {
      const int code = ~node;
      const int first = code >> 4;
      const int cnt = (code & 15) + 1;
      if (kCount) tc->tris += cnt;
      for (int i = 0; i < cnt; ++i) {
        const float4 *tp = s.tri + 3 * (size_t)(first + i);
        float u, v;
        const float tt = tri_hit(o, d, __ldg(tp), __ldg(tp + 1), __ldg(tp + 2), eps, u, v);
        if (tt > eps && tt < h.t) {
          h.t = tt;
          h.u = u;
          h.v = v;
          h.slot = first + i;
          tcull = fminf(tcull, cull_bound(tt));
        }
      }
    }
    for (;;) {
      if (sp == 0) return h;
      const int2 e = stack[--sp];
      if (__int_as_float(e.y) <= tcull) {
        node = e.x;
        break;
      }
    }
  }
}

// Not inlined: rare, and one copy per kernel.
template <int W>
__device__ __noinline__ Hit trace_plain(const DevScene &s, float3 o, float3 d, float eps, uint32_t &errbits,
                                        float bound) {
  if (W == 2) return trace_two_child(s, o, d, eps, errbits, nullptr, bound);
  return trace_wide_plain<W == 8 ? 8 : 4>(s, o, d, eps, errbits, nullptr, bound);
}

// ---- layouts ----------------------------------------------------------------
// A compile-time choice of each kernel instance.  W = 2 and 8: the fast loops walk
// the four-child nodes collapsed from the same tree (against two children half the
// steps of a ray; against eight a quarter of the sorting network: 17 % less time
// for the terrain's bundles); the boxes on the way to a leaf contain its own, so only a
// ray that meets two triangles at exactly the same distance can differ, and that ray
// is traced again in the layout's own order.  (A ray through the very edge of a box,
// entered and left at one distance, is rejected by it: four-child nodes have boxes that
// eight-child ones skip, and reject what the reference order rejects.  10 of 60,000
// rays made of zeros, ones and subnormals.)  W = 4; W = 5 / 9: quantized.
template <int W>
constexpr bool kWalkedAsFour = W == 2 || W == 8;

// bound: distance beyond which hits do not matter to the caller.  Boxes past
// it are skipped; a hit beyond it may still be returned (callers treat such a
// hit like a miss), so results are the same as with bound = 1e9.
template <int W>
TS_D void trav_begin(const DevScene &s, Traversal &t, float3 o, float3 d, float bound) {
  const float3 inv = f3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
  t.no[0] = pack2(-o.x, -o.x);
  t.no[1] = pack2(-o.y, -o.y);
  t.no[2] = pack2(-o.z, -o.z);
  t.inv[0] = pack2(inv.x, inv.x);
  t.inv[1] = pack2(inv.y, inv.y);
  t.inv[2] = pack2(inv.z, inv.z);
  t.d = d;
  t.h.t = 1e9f;
  t.h.u = t.h.v = 0.f;
  t.h.slot = -1;
  t.tcull = cull_bound(fminf(bound, 1e9f));
  t.node = s.num_nodes > 0 ? 0 : kTravDone;
  t.sp = 0;
  t.tie = kWalkedAsFour<W> && s.num_nodes <= 0;  // a tree too deep for the wide stack has no four-child nodes
}

// a finished traversal's hit does not stand: trace_plain() has to decide a tie
template <int W>
TS_D bool trav_tied(const Traversal &t) {
  return kWalkedAsFour<W> && t.tie;
}

// the node layout behind a layout id
template <int W>
struct Nodes {
  static constexpr int value = W == 2 || W == 8 ? 4 : W;
};

// Fast closest hit in one go (local-memory stack); slot kTiedSlot: a tie that
// trace_plain() decides.  errbits gets
// kErrStackOverflow if the tree is deeper than the stack (the builder bounds
// the depth below it, so this is a guard only).
// Not inlined: one copy of the traversal per kernel instead of one per call
// site keeps the megakernels' instruction footprint small (instruction-fetch
// stalls dominated them when inlined).
// kCount counts the layout's own node visits and triangle tests.
// kTogether: the lanes that arrive together step together (warp_phase): 9 % less
// time for the adjoint's replays and the batch kernel, 15 % for ray queries; a
// single pass of few paths waits more than it gains.
constexpr int kTiedSlot = -2;

template <int W, bool kCount, bool kTogether>
__device__ __noinline__ Hit trace_fast(const DevScene &s, float3 o, float3 d, float eps, uint32_t &errbits,
                                       TraceCount *tc, float bound) {
  if (kCount && W == 2) return trace_two_child<true>(s, o, d, eps, errbits, tc, bound);
  if (kCount && (W == 4 || W == 8)) return trace_wide_plain<W == 8 ? 8 : 4, true>(s, o, d, eps, errbits, tc, bound);
  Traversal t;
  int2 stack[kWideStack];
  trav_begin<W>(s, t, o, d, bound);
  if (kCount || !kTogether) {
    trav_run<Nodes<W>::value, kCount>(s, t, stack, eps, errbits, tc);
  } else {
    const unsigned mask = __activemask();
    while (warp_phase<Nodes<W>::value>(s, t, stack, eps, errbits, mask)) {}
  }
  if (trav_tied<W>(t)) t.h.slot = kTiedSlot;
  return t.h;
}

template <int W, bool kCount = false, bool kTogether = true>
TS_D Hit trace_closest(const DevScene &s, float3 o, float3 d, float eps, uint32_t &errbits, TraceCount *tc = nullptr,
                       float bound = 1e9f) {
  Hit h = trace_fast<W, kCount, kTogether>(s, o, d, eps, errbits, tc, bound);
  if (kWalkedAsFour<W> && h.slot == kTiedSlot) h = trace_plain<W>(s, o, d, eps, errbits, bound);
  return h;
}

// ---- group traversal ---------------------------------------------------------
// Four lanes (kGroupLanes, G below) walk one ray: lane k tests child k of a node
// and triangles k, k + G, ... of a leaf.  Against a ray per lane a step is a
// third of the instructions (one box, no sorting network, one triangle) and a
// node costs one or two contiguous loads of the warp instead of eight scattered
// ones per lane, and a warp serialises G times fewer rays.  All lanes of a warp run
// the same loop: its votes and shuffles take the whole warp.
constexpr int kGroupLanes = 4;
constexpr int kGroupStack = 32;  // entries per ray, in shared memory; a ray that needs more goes to trace_plain()

template <int G>
struct GroupRay {
  // the same in all lanes of the group
  f32x2 no[3], inv[3];
  float3 d;
  float tcull;
  int node, sp;
  bool over;   // stack overflow: the result does not stand
  // best of the triangles this lane tested
  Hit h;
  bool tie;
};

template <int G>
TS_D void group_begin(const DevScene &s, GroupRay<G> &r, float3 o, float3 d, float bound) {
  const float3 inv = f3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
  r.no[0] = pack2(-o.x, -o.x);
  r.no[1] = pack2(-o.y, -o.y);
  r.no[2] = pack2(-o.z, -o.z);
  r.inv[0] = pack2(inv.x, inv.x);
  r.inv[1] = pack2(inv.y, inv.y);
  r.inv[2] = pack2(inv.z, inv.z);
  r.d = d;
  r.tcull = cull_bound(fminf(bound, 1e9f));
  r.node = s.num_nodes > 0 ? 0 : kTravDone;
  r.sp = 0;
  r.over = s.num_nodes <= 0;
  r.h.t = 1e9f;
  r.h.u = r.h.v = 0.f;
  r.h.slot = -1;
  r.tie = false;
}

// One step of every group of the warp: an inner node, the leaf it may lead to
// and the pop that follows.  stack: shared, this group's column of [entry][stride].
template <int G>
TS_D void group_step(const DevScene &s, GroupRay<G> &r, int2 *stack, int stride, int sub, int shift, float eps) {
  constexpr unsigned kFull = 0xffffffffu, kBits = (1u << G) - 1u;
  bool pop = false;
  const bool inner = r.node >= 0;
  if (__any_sync(kFull, inner)) {
    bool hit = false;
    int key = 0x7fffffff, ref = 0;
    if (inner) {
      const Rec32 c = load32(s.node + (size_t)r.node * (2 * G) + 2 * sub);
      float te, tx;
      child_hit(c, r.no, r.inv, te, tx);
      hit = te < tx && tx > 0.f && te <= r.tcull;
      ref = (int)(uint32_t)c.d;
      // order by entry distance, then child: bits of a non-negative float with
      // the child in the lowest ones (rounded down: culling stays conservative)
      if (hit) key = (__float_as_int(fmaxf(te, 0.f)) & ~(G - 1)) | sub;
    }
    const unsigned gm = (__ballot_sync(kFull, hit) >> shift) & kBits;
    int rank = 0, best = key;
#pragma unroll
    for (int x = 1; x < G; ++x) {
      const int other = __shfl_xor_sync(kFull, key, x);
      rank += other < key;
      best = min(best, other);
    }
    const int near = __shfl_sync(kFull, ref, shift + (best & (G - 1)));
    if (inner) {
      const int far = __popc(gm) - 1;  // children to push
      if (far < 0) {
        pop = true;
      } else if (r.sp + far > kGroupStack) {
        r.over = true;
        r.node = kTravDone;
      } else {
        if (hit && rank > 0) stack[(r.sp + far - rank) * stride] = make_int2(ref, key & ~(G - 1));
        r.sp += far;
        r.node = near;
      }
    }
  }
  const bool leaf = r.node < 0 && r.node != kTravDone;
  if (__any_sync(kFull, leaf)) {
    int first = 0, cnt = 0;
    if (leaf) {
      first = ~r.node >> 4;
      cnt = (~r.node & 15) + 1;
      pop = true;
    }
    for (int i = sub; __any_sync(kFull, i - sub < cnt); i += G) {
      if (i < cnt) {
        const float4 *tp = s.tri + 3 * (size_t)(first + i);
        const float4 A = __ldg(tp + 0), E1 = __ldg(tp + 1), E2 = __ldg(tp + 2);
        const float3 o = f3(-lane0(r.no[0]), -lane0(r.no[1]), -lane0(r.no[2]));
        float u, v;
        const float tt = tri_hit(o, r.d, A, E1, E2, eps, u, v);
        if (tt > eps && tt <= r.h.t) {
          r.tie = tt == r.h.t;
          if (!r.tie) {
            r.h.t = tt;
            r.h.u = u;
            r.h.v = v;
            r.h.slot = first + i;
          }
        }
      }
    }
    float m = r.h.t;
#pragma unroll
    for (int x = 1; x < G; x <<= 1) m = fminf(m, __shfl_xor_sync(kFull, m, x));
    r.tcull = fminf(r.tcull, cull_bound(m));
  }
  __syncwarp();
  if (pop) {
    r.node = kTravDone;
    while (r.sp > 0) {
      const int2 e = stack[--r.sp * stride];
      if (__int_as_float(e.y) <= r.tcull) {
        r.node = e.x;
        break;
      }
    }
  }
  __syncwarp();
}

// The finished groups' hits, the same in all their lanes; false where the hit
// does not stand and trace_plain() has to be asked.  Run by the whole warp.
template <int G>
TS_D bool group_hit(const GroupRay<G> &r, int shift, Hit &h) {
  constexpr unsigned kFull = 0xffffffffu, kBits = (1u << G) - 1u;
  float m = r.h.t;
#pragma unroll
  for (int x = 1; x < G; x <<= 1) m = fminf(m, __shfl_xor_sync(kFull, m, x));
  const bool own = r.h.slot >= 0 && r.h.t == m;
  const unsigned owners = (__ballot_sync(kFull, own) >> shift) & kBits;
  const unsigned ties = (__ballot_sync(kFull, own && r.tie) >> shift) & kBits;
  const int src = shift + (owners ? __ffs(owners) - 1 : 0);
  h.t = m;
  h.u = __shfl_sync(kFull, r.h.u, src);
  h.v = __shfl_sync(kFull, r.h.v, src);
  h.slot = __shfl_sync(kFull, r.h.slot, src);
  return !r.over && !ties && (owners & (owners - 1)) == 0;
}

// Exact reference-order closest hit on the reference-layout table.
TS_D Hit trace_reference_order(const DevScene &s, float3 o, float3 d, float eps, uint32_t &errbits) {
  Hit h;
  h.t = 1e9f;
  h.u = h.v = 0.f;
  h.slot = -1;
  if (s.num_ref_nodes <= 0) return h;
  const float3 inv = f3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
  int stack[kStackDepth];
  int sp = 1;
  stack[0] = 0;
  while (sp > 0) {
    const int ni = stack[--sp];
    float te, tx;
    const float *mn = s.ref_min + 3 * (size_t)ni;
    const float *mx = s.ref_max + 3 * (size_t)ni;
    box_hit(mn[0], mx[0], mn[1], mx[1], mn[2], mx[2], o, inv, te, tx);
    if (!(te < tx && tx > 0.f)) continue;
    const int4 l = s.ref_link[ni];
    if (l.z > 0) {
      for (int i = 0; i < l.z; ++i) {
        const int slot = l.w + i;
        const float4 *tp = s.tri + 3 * (size_t)slot;
        float u, v;
        const float t = tri_hit(o, d, tp[0], tp[1], tp[2], eps, u, v);
        if (t > eps && t < h.t) {
          h.t = t;
          h.u = u;
          h.v = v;
          h.slot = slot;
        }
      }
    } else {
      if (sp + 2 > kStackDepth) {
        errbits |= kErrStackOverflow;
        continue;
      }
      stack[sp++] = l.x;
      stack[sp++] = l.y;
    }
  }
  return h;
}

// Hit-record completion (main.py:860-863): geometric normal, interpolated
// shading normal, front-face flag, material.
struct SurfaceInfo {
  float3 ng, ns;
  int front, mat;
};
TS_D SurfaceInfo surface_info(const DevScene &s, const Hit &h, float3 d) {
  SurfaceInfo r;
  const float4 s0 = __ldg(s.shade + 3 * (size_t)h.slot + 0);
  const float4 s1 = __ldg(s.shade + 3 * (size_t)h.slot + 1);
  const float4 s2 = __ldg(s.shade + 3 * (size_t)h.slot + 2);
  r.ng = f3(s0.w, s1.w, s2.w);
  const float w = 1.0f - h.u - h.v;
  r.ns = normalize(w * xyz(s0) + h.u * xyz(s1) + h.v * xyz(s2));
  r.front = dot(d, r.ng) < 0.f ? 1 : 0;
  r.mat = __float_as_int(__ldg(s.tri + 3 * (size_t)h.slot + 1).w);
  return r;
}

}  // namespace ts
