// trace.cu — closest-hit and any-hit ray traversal (RadixBVHBuilder::
// intersect / recursiveIntersect, radix_bvh.cpp:26-30,202-245, with the
// watertight Pluecker test of intersector.hpp:63-101).
//
// Layouts: BVH2 nodes carry both children's boxes (one 64-byte record per
// visit); 4-wide nodes hold their child boxes in 8 bits per plane (64 bytes);
// 8-wide nodes as structure of arrays in fp32 (224 bytes); triangles are
// gathered in sorted (leaf) order, 48 bytes each.
//
// Kernels:
//   k_trace4            4-wide: while-while traversal with parked leaves;
//                       persistent warps refill idle lanes from a global ray
//                       counter (work stealing across scenes of a batch);
//                       k_settle4 or k_trace_retry4 after it
//   k_trace_bvh2        one ray per thread over BVH2, leaf triangles tested
//                       directly as the reference does (no leaf box test)
//   k_trace_wide, k_trace_persistent, k_trace_ww   8-wide: one ray per thread,
//                       persistent warps, and these with parked leaves
//   k_trace_retry       rays whose short stack overflowed, with a deep stack
#include <algorithm>
#include <chrono>
#include <climits>
#include <cstring>
#include <mutex>
#include <string>

#include "common.cuh"
#include "internal.h"
#include "wide.cuh"

namespace flg {

struct RaySoA {
  const float *ox, *oy, *oz, *dx, *dy, *dz, *tmin, *tmax;
  float tmin_c, tmax_c;
};

struct Out {
  int32_t *prim;
  float *t, *u, *v;
  uint8_t *occ;
};

struct Scratch {
  int64_t *ovf;
  uint32_t *ovf_count;  // and above it the blocks that are done (clear_counters)
  int64_t ovf_cap;
  unsigned long long *work;
  uint32_t *err;
};

// Rays of a launch: their number, or the most there can be where it stands in
// device memory.
struct RayCount {
  int64_t most;
  const int32_t *at;
  __device__ __forceinline__ int64_t get() const { return at ? (int64_t)*at : most; }
};

constexpr int kRetryStack = 256;

__device__ __forceinline__ void load_ray(const RaySoA &R, int64_t i, float3 &o, float3 &d, float3 &inv,
                                         float &tmin, float &tmax) {
  o = make_float3(__ldg(R.ox + i), __ldg(R.oy + i), __ldg(R.oz + i));
  d = make_float3(__ldg(R.dx + i), __ldg(R.dy + i), __ldg(R.dz + i));
  inv = make_float3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
  tmin = R.tmin ? __ldg(R.tmin + i) : R.tmin_c;
  tmax = R.tmax ? __ldg(R.tmax + i) : R.tmax_c;
}

__device__ __forceinline__ int32_t scene_root(const int32_t *__restrict__ roots, const int64_t *__restrict__ ray_off,
                                              int n_scenes, int64_t i) {
  int s = ray_off ? find_segment(ray_off, n_scenes, i) : 0;
  return __ldg(roots + s);
}

// The same for a lane whose rays only grow (persistent kernels take them
// from one counter): `sc` holds the scene of the lane's previous ray (-1:
// none yet); one search, then a forward walk.
__device__ __forceinline__ int32_t scene_root_walk(const int32_t *__restrict__ roots,
                                                   const int64_t *__restrict__ ray_off, int n_scenes, int64_t i,
                                                   int &sc) {
  if (!ray_off) return __ldg(roots);
  if (sc < 0) {
    sc = find_segment(ray_off, n_scenes, i);
  } else {
    while (sc < n_scenes - 1 && __ldg(ray_off + sc + 1) <= i) ++sc;
  }
  return __ldg(roots + sc);
}

// Tests sorted triangle g; updates the closest hit.  Returns true on accept.
// MT selects the live renderer's Moller-Trumbore test and its strict
// t < tMax rule instead of the watertight Pluecker test.
template <bool MT = false>
__device__ __forceinline__ bool test_tri(const TriRec *__restrict__ tris, int64_t g, const float3 &o,
                                         const float3 &d, float tmin, float &best, bool &have, int32_t &prim) {
  const float4 *p = (const float4 *)(tris + g);
  float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  float t;
  const float3 pa = make_float3(a.x, a.y, a.z), pb = make_float3(b.x, b.y, b.z), pc = make_float3(c.x, c.y, c.z);
  if (MT) {
    if (!moller_t(pa, pb, pc, o, d, t)) return false;
    if (!(t >= tmin && t < best)) return false;
  } else {
    if (!pluecker_t(pa, pb, pc, o, d, t)) return false;
    if (!accept_closest(t, tmin, best, have)) return false;
  }
  best = t;
  have = true;
  prim = (int32_t)g;  // sorted position; write_result maps it to the original id
  return true;
}

// Any-hit variant: accepts t in [tmin, tmax] ([tmin, tmax) with MT).
template <bool MT = false>
__device__ __forceinline__ bool test_tri_any(const TriRec *__restrict__ tris, int64_t g, const float3 &o,
                                             const float3 &d, float tmin, float tmax) {
  const float4 *p = (const float4 *)(tris + g);
  float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  float t;
  const float3 pa = make_float3(a.x, a.y, a.z), pb = make_float3(b.x, b.y, b.z), pc = make_float3(c.x, c.y, c.z);
  if (MT) return moller_t(pa, pb, pc, o, d, t) && t >= tmin && t < tmax;
  if (!pluecker_t(pa, pb, pc, o, d, t)) return false;
  return t >= tmin && !(t > tmax);
}

__device__ __forceinline__ uint64_t stack_key(float t, int32_t ref) {
  return ((uint64_t)(__float_as_uint(t) & 0x7FFFFFFFu) << 32) | (uint32_t)ref;
}

// Writes one ray's result.  For closest hit, `prim` holds the sorted
// position of the winning triangle: its record gives the original id and the
// vertices for the float-float refinement of t, u, v.  The traversal keeps
// only t; the fp32 barycentrics (pluecker) are formed here, for the winner,
// and replaced by the refined ones unless the refinement finds den == 0.
// Result of a finished ray.  Closest hits store the sorted position of the
// triangle and the fp32 t; k_trace_finish turns them into the original id
// and the refined t, u, v afterwards.  Refining here cost several hundred
// instructions per ray, run whenever a ray retired, i.e. with few lanes of
// the warp active: about a fifth of the traversal kernel's issue slots.
__device__ __forceinline__ void write_result(const Out &O, int64_t i, bool any, bool have, int32_t prim,
                                             float best, float tmax) {
  if (any) {
    O.occ[i] = have ? 1 : 0;
  } else {
    O.prim[i] = have ? prim : -1;
    O.t[i] = have ? best : tmax;
    if (!have) {
      O.u[i] = 0.0f;
      O.v[i] = 0.0f;
    }
  }
}

// Hit values of every closest hit, one ray per thread after the traversal
// (same ray floats, same triangle record, same arithmetic as in the loop):
// barycentrics from the Pluecker quantities, then t, u, v recomputed in
// float-float and rounded once (refine_tuv); the sorted position becomes
// the caller's triangle id.
__global__ void __launch_bounds__(256, 4)
    k_trace_finish(RaySoA R, int64_t n, Out O, const TriRec *__restrict__ tris) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t g = O.prim[i];
    if (g < 0) continue;
    const float3 o = make_float3(__ldg(R.ox + i), __ldg(R.oy + i), __ldg(R.oz + i));
    const float3 d = make_float3(__ldg(R.dx + i), __ldg(R.dy + i), __ldg(R.dz + i));
    const float4 *p = (const float4 *)(tris + g);
    const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
    const float3 pa = make_float3(a.x, a.y, a.z), pb = make_float3(b.x, b.y, b.z), pc = make_float3(c.x, c.y, c.z);
    float best = O.t[i], u = 0.0f, v = 0.0f;
    if (!refine_tuv(pa, pb, pc, o, d, best, u, v)) {
      // N.D == 0: the fp32 barycentrics of the test stand (t stays the test's)
      float tf;
      pluecker(pa, pb, pc, o, d, tf, u, v);
    }
    O.prim[i] = __float_as_int(a.w);
    O.t[i] = best;
    O.u[i] = u;
    O.v[i] = v;
  }
}

__device__ __forceinline__ void record_overflow(const Scratch &S, int64_t ray) {
  uint32_t k = atomicAdd(S.ovf_count, 1u);
  if (k < S.ovf_cap) S.ovf[k] = ray;
  else atomicOr(S.err, kErrStack);
}

// ----------------------------------------------------------------------------
// BVH2 traversal (reference-faithful leaf handling).
// ----------------------------------------------------------------------------
template <bool ANY, int STACK, bool MT = false>
__device__ __forceinline__ bool trace_bvh2(const Node2 *__restrict__ nodes, const TriRec *__restrict__ tris,
                                           int32_t root, const float3 &o, const float3 &d, const float3 &inv,
                                           float tmin, float tmax, bool &have, int32_t &prim, float &best) {
  best = tmax;
  have = false;
  prim = -1;
  if (root == INT32_MIN) return true;
  if (root < 0) {
    if (ANY) have = test_tri_any<MT>(tris, ~(int64_t)root, o, d, tmin, tmax);
    else test_tri<MT>(tris, ~(int64_t)root, o, d, tmin, best, have, prim);
    return true;
  }
  uint64_t stk[STACK];
  int sp = 0;
  int32_t cur = root;
  const float miss = __int_as_float(0x7fffffff);  // NaN: never <= a limit
  while (true) {
    const float4 *np = (const float4 *)(nodes + cur);
    const float4 A = __ldg(np), B = __ldg(np + 1), C = __ldg(np + 2);
    const int4 Dd = __ldg((const int4 *)(np + 3));
    const int32_t c0 = Dd.x, c1 = Dd.y;
    if (c0 < 0) {
      if (ANY) {
        if (test_tri_any<MT>(tris, ~(int64_t)c0, o, d, tmin, tmax)) { have = true; return true; }
      } else {
        test_tri<MT>(tris, ~(int64_t)c0, o, d, tmin, best, have, prim);
      }
    }
    if (c1 < 0) {
      if (ANY) {
        if (test_tri_any<MT>(tris, ~(int64_t)c1, o, d, tmin, tmax)) { have = true; return true; }
      } else {
        test_tri<MT>(tris, ~(int64_t)c1, o, d, tmin, best, have, prim);
      }
    }
    const float lim = ANY ? tmax : best;
    float t0 = c0 >= 0 ? slab_tnear(A.x, A.y, A.z, A.w, C.x, C.y, o, inv) : miss;
    float t1 = c1 >= 0 ? slab_tnear(B.x, B.y, B.z, B.w, C.z, C.w, o, inv) : miss;
    const bool h0 = c0 >= 0 && t0 <= lim, h1 = c1 >= 0 && t1 <= lim;
    if (h0 && h1) {
      if (sp >= STACK) return false;
      const bool swap = t1 < t0;
      stk[sp++] = swap ? stack_key(t0, c0) : stack_key(t1, c1);
      cur = swap ? c1 : c0;
      continue;
    }
    if (h0) { cur = c0; continue; }
    if (h1) { cur = c1; continue; }
    bool found = false;
    while (sp > 0) {
      uint64_t e = stk[--sp];
      if (__uint_as_float((uint32_t)(e >> 32)) > (ANY ? tmax : best)) continue;
      cur = (int32_t)(uint32_t)e;
      found = true;
      break;
    }
    if (!found) return true;
  }
}

template <bool ANY, bool MT = false>
__global__ void __launch_bounds__(256)
    k_trace_bvh2(const Node2 *__restrict__ nodes, const TriRec *__restrict__ tris, const int32_t *__restrict__ roots,
                 const int64_t *__restrict__ ray_off, int n_scenes, RaySoA R, int64_t n, Out O, Scratch S) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float3 o, d, inv;
  float tmin, tmax;
  load_ray(R, i, o, d, inv, tmin, tmax);
  const int32_t root = scene_root(roots, ray_off, n_scenes, i);
  bool have;
  int32_t prim;
  float best;
  if (!trace_bvh2<ANY, 64, MT>(nodes, tris, root, o, d, inv, tmin, tmax, have, prim, best)) {
    record_overflow(S, i);
    return;
  }
  write_result(O, i, ANY, have, prim, best, tmax);
}

// ----------------------------------------------------------------------------
// Wide traversal as a resumable state machine (one node or leaf range per
// step) so the persistent kernel can swap rays between steps.
// ----------------------------------------------------------------------------
// Child keys for the nearest-first order: the bits of tnear (non-negative,
// so integer order is float order) with the child's slot in the low
// log2(W) bits.  Dropping those mantissa bits only rounds tnear down, which
// keeps the stack's culling test (entry tnear > best) conservative.
__device__ __forceinline__ void cas(uint32_t &a, uint32_t &b) {
  const uint32_t lo = min(a, b), hi = max(a, b);
  a = lo;
  b = hi;
}

template <int W>
__device__ __forceinline__ void sort_keys(uint32_t (&k)[W]) {
  if constexpr (W == 4) {
    cas(k[0], k[1]); cas(k[2], k[3]); cas(k[0], k[2]); cas(k[1], k[3]); cas(k[1], k[2]);
  } else {
    cas(k[0], k[1]); cas(k[2], k[3]); cas(k[4], k[5]); cas(k[6], k[7]);
    cas(k[0], k[2]); cas(k[1], k[3]); cas(k[4], k[6]); cas(k[5], k[7]);
    cas(k[1], k[2]); cas(k[5], k[6]);
    cas(k[0], k[4]); cas(k[1], k[5]); cas(k[2], k[6]); cas(k[3], k[7]);
    cas(k[2], k[4]); cas(k[3], k[5]);
    cas(k[1], k[2]); cas(k[3], k[4]); cas(k[5], k[6]);
  }
}

// The child ref a sorted key names (selects, no dynamic register index).
template <int W>
__device__ __forceinline__ int32_t key_ref(uint32_t key, const int32_t (&ref)[W]) {
  if constexpr (W == 4) {
    const int32_t a = (key & 1u) ? ref[1] : ref[0];
    const int32_t b = (key & 1u) ? ref[3] : ref[2];
    return (key & 2u) ? b : a;
  } else {
    const uint32_t slot = key & (uint32_t)(W - 1);
    int32_t r = ref[0];
#pragma unroll
    for (int m = 1; m < W; ++m) r = slot == (uint32_t)m ? ref[m] : r;
    return r;
  }
}

// Stack entry (tnear rounded down | ref) of a sorted key.
template <int W>
__device__ __forceinline__ uint64_t key_entry(uint32_t key, const int32_t (&ref)[W]) {
  return ((uint64_t)(key & ~(uint32_t)(W - 1)) << 32) | (uint32_t)key_ref<W>(key, ref);
}

// Tests the W children of a wide node (7 / 14 16-byte loads) with the
// reference's slab test (BoundIntersect, intersector.hpp:103-120).  The
// near and far plane arrays of each axis are picked by the sign of the
// ray's inverse direction when they are loaded, so the per-child swap of
// slab1 disappears; the products are the same roundings, so tnear and the
// hit decision equal slab_tnear's (a NaN slab, 0 * inf, constrains nothing
// in both).  Returns the number of children hit with tnear <= lim; their
// keys are in key[] (misses are ~0), the child refs in ref[] — loaded only
// when a child is hit (the kernel is bound by L1 throughput; skipping that
// 16-byte load on visits without hits gave +2.5 %).  Empty slots need no
// test of their ref: they hold +inf boxes, which no ray enters.
template <int W>
__device__ __forceinline__ int visit_node(const NodeW<W> *__restrict__ node, const float3 &o, const float3 &inv,
                                          float lim, uint32_t (&key)[W], int32_t (&ref)[W]) {
  constexpr int Q = W / 4;  // float4s per child array
  const float4 *np = (const float4 *)node;
  // Float4 offsets of the near arrays: lo (sign 0) or hi (sign 1) per axis.
  const int nx = (int)(__float_as_uint(inv.x) >> 31) * Q;
  const int ny = 2 * Q + (int)(__float_as_uint(inv.y) >> 31) * Q;
  const int nz = 4 * Q + (int)(__float_as_uint(inv.z) >> 31) * Q;
  float pn[3][W], pf[3][W];
#pragma unroll
  for (int h = 0; h < Q; ++h) {
    const float4 a = __ldg(np + nx + h), b = __ldg(np + (nx ^ Q) + h);
    const float4 c = __ldg(np + ny + h), e = __ldg(np + (ny ^ Q) + h);
    const float4 f = __ldg(np + nz + h), g = __ldg(np + (nz ^ Q) + h);
    const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
    const float cv[4] = {c.x, c.y, c.z, c.w}, ev[4] = {e.x, e.y, e.z, e.w};
    const float fv[4] = {f.x, f.y, f.z, f.w}, gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      pn[0][4 * h + k] = av[k]; pf[0][4 * h + k] = bv[k];
      pn[1][4 * h + k] = cv[k]; pf[1][4 * h + k] = ev[k];
      pn[2][4 * h + k] = fv[k]; pf[2][4 * h + k] = gv[k];
    }
  }
  const float t1c = fminf(lim, 3.402823466e+38f);
  int nh = 0;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const float tnx = (pn[0][k] - o.x) * inv.x, tfx = (pf[0][k] - o.x) * inv.x;
    const float tny = (pn[1][k] - o.y) * inv.y, tfy = (pf[1][k] - o.y) * inv.y;
    const float tnz = (pn[2][k] - o.z) * inv.z, tfz = (pf[2][k] - o.z) * inv.z;
    const float t0 = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, 0.0f));
    const float t1 = fminf(fminf(tfx, tfy), fminf(tfz, t1c));
    const bool ok = t0 <= t1;  // empty slots hold +inf boxes, which no ray enters
    key[k] = ok ? ((__float_as_uint(t0) & 0x7FFFFFFFu & ~(uint32_t)(W - 1)) | (uint32_t)k) : ~0u;
    nh += ok ? 1 : 0;
  }
  if (nh > 0) {
#pragma unroll
    for (int h = 0; h < Q; ++h) {
      const int4 r = __ldg((const int4 *)np + 6 * Q + h);
      ref[4 * h] = r.x; ref[4 * h + 1] = r.y; ref[4 * h + 2] = r.z; ref[4 * h + 3] = r.w;
    }
  }
  return nh;
}

template <int W, bool ANY, int STACK>
struct Tracer {
  float3 o, d, inv;
  float tmin, tmax, best;
  int32_t cur, prim;
  int sp;
  bool have, overflow;
  uint64_t stk[STACK];

  __device__ __forceinline__ void start(int32_t root) {
    best = tmax;
    have = false;
    overflow = false;
    prim = -1;
    sp = 0;
    cur = root;
  }

  __device__ __forceinline__ bool pop() {
    const float lim = ANY ? tmax : best;
    while (sp > 0) {
      uint64_t e = stk[--sp];
      if (__uint_as_float((uint32_t)(e >> 32)) > lim) continue;
      cur = (int32_t)(uint32_t)e;
      return true;
    }
    return false;
  }

  // Returns true when the ray is finished.
  __device__ __forceinline__ bool step(const NodeW<W> *__restrict__ nodes, const TriRec *__restrict__ tris) {
    if (cur == kEmptyChild || cur == INT32_MIN) return true;
    if (cur >= 0) {
      uint32_t key[W];
      int32_t ref[W];
      const int nh = visit_node<W>(nodes + cur, o, inv, ANY ? tmax : best, key, ref);
      if (nh == 0) return !pop();
      sort_keys<W>(key);
      if (sp + nh - 1 > STACK) {
        overflow = true;
        return true;
      }
#pragma unroll
      for (int k = W - 1; k >= 1; --k)
        if (k < nh) stk[sp++] = key_entry<W>(key[k], ref);
      cur = key_ref<W>(key[0], ref);
      return false;
    }
    const int32_t enc = ~cur;
    const int64_t first = (int64_t)((uint32_t)enc >> 3);
    const int count = (enc & 7) + 1;
    for (int j = 0; j < count; ++j) {
      if (ANY) {
        if (test_tri_any(tris, first + j, o, d, tmin, tmax)) {
          have = true;
          return true;
        }
      } else {
        test_tri(tris, first + j, o, d, tmin, best, have, prim);
      }
    }
    return !pop();
  }
};

template <int W, bool ANY, int STACK>
__global__ void __launch_bounds__(256)
    k_trace_wide(const NodeW<W> *__restrict__ nodes, const TriRec *__restrict__ tris, const int32_t *__restrict__ roots,
                 const int64_t *__restrict__ ray_off, int n_scenes, RaySoA R, int64_t n, Out O, Scratch S) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Tracer<W, ANY, STACK> tr;
  load_ray(R, i, tr.o, tr.d, tr.inv, tr.tmin, tr.tmax);
  tr.start(scene_root(roots, ray_off, n_scenes, i));
  while (!tr.step(nodes, tris)) {
  }
  if (tr.overflow) record_overflow(S, i);
  else write_result(O, i, ANY, tr.have, tr.prim, tr.best, tr.tmax);
}

template <int W, bool ANY, int STACK>
__global__ void __launch_bounds__(256)
    k_trace_persistent(const NodeW<W> *__restrict__ nodes, const TriRec *__restrict__ tris,
                       const int32_t *__restrict__ roots, const int64_t *__restrict__ ray_off, int n_scenes, RaySoA R,
                       int64_t n, Out O, Scratch S, int refill) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt = (1u << lane) - 1u;
  Tracer<W, ANY, STACK> tr;
  bool active = false, exhausted = false;
  int64_t ray = -1;
  int scene = -1;
  while (true) {
    const unsigned idle = __ballot_sync(0xFFFFFFFFu, !active);
    const int nidle = __popc(idle);
    if (!exhausted && nidle >= refill) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(S.work, (unsigned long long)nidle);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (!active) {
        const int64_t my = (int64_t)base + __popc(idle & lt);
        if (my < n) {
          ray = my;
          load_ray(R, ray, tr.o, tr.d, tr.inv, tr.tmin, tr.tmax);
          tr.start(scene_root_walk(roots, ray_off, n_scenes, ray, scene));
          active = true;
        }
      }
      if ((int64_t)base + nidle >= n) exhausted = true;
    }
    if (__ballot_sync(0xFFFFFFFFu, active) == 0u) {
      if (exhausted) break;
      continue;
    }
    if (active && tr.step(nodes, tris)) {
      if (tr.overflow) record_overflow(S, ray);
      else write_result(O, ray, ANY, tr.have, tr.prim, tr.best, tr.tmax);
      active = false;
    }
  }
}

// ----------------------------------------------------------------------------
// 4-wide traversal over quantised nodes (NodeQ).
//
// The results are those of a traversal over the exact child boxes (fp32, the
// reference's slab test, children nearest first, first found kept among equal
// t), although the boxes the traversal reads are a little larger:
//   * A quantised box contains the exact one with room for every rounding of
//     visit_q, so the leaves visited are a superset of the exact ones.  (A ray
//     whose direction leaves no such room is traced over the exact boxes: inv_q.)
//     The leaf ranges are the exact tree's: in smaller ones, which would be faster
//     (24 batched scenes in ranges of up to 1 / 2 / 3 / 4: 18.9 / 20.1 / 22.3 / 24.7 ms),
//     a ray that misses a triangle's own box by rounding, but not its range's,
//     would not test it.
//   * Closest hit: a finished ray's winner stands if its own box, which its
//     leaf range's and every ancestor's box contain, passes the exact slab
//     test with tnear <= t: then the exact traversal reaches it, whatever it
//     found before.  So it does if tnear > t by at most kNear (a matter of
//     rounding, for flat boxes) and neither another candidate tested nor tmax
//     lay within kNear.  Among equal t the first in the exact order of visits
//     wins.  The rays that this does not settle go on a list, and k_settle4
//     settles the equal pairs (first_of_two) and traces the others again over
//     the exact boxes (retrace4), of which those around the hit decide where only
//     rounding is in question: about one ray per million on random soups.
//   * A triangle's fp32 t may also lie outside of its own box: by rounding at
//     vertices and edges, the more the smaller the triangle is for its distance
//     or the direction along an axis, and without bound for a grazing one, as
//     N.D goes to 0.  The exact order may come to such a triangle before
//     another hit whose t lies between, so boxes up to kBeyond of t beyond the hit
//     are entered too.  Left open are triangles that lie further than that in front
//     of their box: none in 150 M rays at the vertices of spheres and soups from 3,
//     30 and 300 sizes away, 2 of 2 M where the direction has 1e-3 of its length
//     along x, 10 of 2 M where two of its components are 1 to 1e-7 of it, 35 of
//     131,072 rays through 16 slivers each, of 1e-7 to 1e-6 of the distance, none
//     with slivers ten times as wide; and in all of these no occlusion.
//   * Any hit: an accepted triangle counts if its own box passes the exact slab
//     test.  A ray that found only others is traced again over the exact boxes
//     (k_trace_retry4).
// ----------------------------------------------------------------------------
constexpr float kNear = 4.76837158203125e-07f;  // 2^-21
constexpr float kBeyond = 1.220703125e-04f;     // 2^-13: of 4.2 M rays at vertices 2^-20 left up to 37 open, 2^-14 one
constexpr float kAround = 9.765625e-04f;        // 2^-10: what retrace4 takes for the surroundings of a hit
// prim between k_trace4 and the kernels after it: a sorted position (< 2^28) with
// kPending, -1, or kListed for a listed ray.  A listed ray's u and v hold two
// positions at the same t; or v = kByWalk: candidates within kNear; or v = -1:
// trace it again.
constexpr int32_t kPending = 1 << 30;
constexpr int32_t kListed = INT32_MIN;
constexpr int32_t kByWalk = -2;
constexpr uint8_t kOccListed = 2;  // in occ: an any-hit ray on the list

__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Inverse directions with a component below kInvMin or from kInvMax on, for the
// quantised slab test.  False if the ray has to be traced over the exact boxes.
//
// An infinite component (of a direction's zero, or below 2^-128), or one so large
// that 2^16 steps times it overflow, would make plane distances of its axis NaN
// and drop the axis.  +-B takes its place, the largest power of two for which
// 2^16 steps of the scene's root, and so of every node, times B stay finite (2^90
// if the root's step is infinite).  The exact plane distances have the same signs
// and are larger or infinite; an origin between an exact plane and the quantised
// one is inside.  So no box is lost by its near planes.  But the far distance of
// a box is smaller now.  It is at least 1/128 step x B, what quantise adds less
// the rounding of the distance, and the step at least 2^-40 and at least 2^-30
// of the box's coordinates, which are at least half the origin's if the far plane
// is not half of that away.  Boxes nearer than that (`sure`), and than the 2^126
// of visit_q, are tested as the exact test tests them; and no box that the
// exact test accepts is farther (`far`) than tmax, or than the root's far plane on
// another axis.  (1 M rays along z with 1e-38 along x: 10.2 ms with that axis
// dropped, 0.67 with B.)
constexpr uint32_t kInvMin = (127u - 100u) << 23, kInvMax = (127u + 64u) << 23;  // 2^-100 (the step is at least 2^-40), 2^64
__device__ __forceinline__ uint32_t above_min(float inv) { return (__float_as_uint(inv) & 0x7FFFFFFFu) - kInvMin; }
__device__ __forceinline__ bool odd_inv(const float3 &inv) {
  return max(max(above_min(inv.x), above_min(inv.y)), above_min(inv.z)) >= kInvMax - kInvMin;
}
__device__ __forceinline__ bool is_finite(float x) { return fabsf(x) <= 3.402823466e+38f; }
__device__ __forceinline__ bool inv_q(const NodeQ *__restrict__ root, const float3 &o, const float3 &d, float tmax,
                                      float3 &inv) {
  const uint4 A = __ldg((const uint4 *)root);
  const float oo[3] = {o.x, o.y, o.z}, dd[3] = {d.x, d.y, d.z};
  const uint32_t org[3] = {A.x, A.y, A.z}, e[3] = {A.w >> 7 & 255u, A.w >> 23, A.w >> 15 & 255u};
  float *const ii[3] = {&inv.x, &inv.y, &inv.z};
  float far = tmax, sure = 8.507059173023462e+37f;  // 2^126
  bool hits = A.w != kLoneStep;  // one triangle, in a box that constrains nothing
  bool small = false;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float b = __uint_as_float((e[a] == 255u ? 217u : min(254u, 379u - e[a])) << 23);
    if (fabsf(*ii[a]) <= b) {
      // 256 steps cover the box
      far = fminf(far, (fabsf(__uint_as_float(org[a]) - oo[a]) + __uint_as_float(e[a] << 23) * 0.00390625f) * fabsf(*ii[a]));
      small |= (__float_as_uint(*ii[a]) & 0x7FFFFFFFu) < kInvMin;
    } else {
      *ii[a] = copysignf(b, *ii[a]);
      // half of it, for the roundings here
      sure = fminf(sure, fmaxf(3.5527136788005009e-15f, fabsf(oo[a]) * 3.637978807091713e-12f) * b);
    }
    hits &= is_finite(oo[a]) && dd[a] == dd[a];  // else the ray hits nothing
  }
  return !hits || (!small && far < sure);
}

// Two fp32 values in one 64-bit register: sm_103a's packed add, multiply and
// fused multiply-add do both in one issue slot, with the scalar roundings.
// The traversal is bound by issue slots once its loads are few.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Byte k of w as the float 1/2 + byte / 2^16: one byte permute puts it above the
// last mantissa byte of 1/2.  (As 2^15 + byte, with s smaller by 2^16, the offset
// 2^15 s would overflow before s itself, and planes at -inf reject the box
// that planes at NaN leave alone.)
template <int K>
__device__ __forceinline__ float byte_f(uint32_t w) {
  return __uint_as_float(__byte_perm(w, 0x3F000000u, 0x7604 | (K << 4)));
}

// Tests the children of a quantised node.  key[k]: tnear with child k's kind
// byte in place of its low byte (masked off again, i.e. rounded down, when a
// stack entry is culled); a miss is ~0.  Per axis the plane distance
// of byte q is fma(1/2 + q / 2^16, s, (origin - o) inv - s / 2) with s = 2^16 step inv.
// Its error is below 1/64 step (the boxes' slack) plus 2^-22 of itself, and the
// exact test's own below 2^-23: with tnear scaled by 1 - kBeyond the test passes
// whenever the exact one does (2^-20 would do).  For that s must not be subnormal (rays with
// an inverse below kInvMin are traced over the exact boxes).  Where s is infinite
// the distances are NaN and the axis constrains nothing.  Where s is finite and
// (origin - o) inv - s / 2 is not, the origin lies 2^15 steps or more outside and
// the distances have the exact ones' sign; those are beyond 2^126.
__device__ __forceinline__ void visit_q(const NodeQ *__restrict__ node, const float3 &o, const float3 &inv, float lim,
                                        uint32_t (&key)[4], int32_t &base) {
  const uint4 *np = (const uint4 *)node;
  const uint4 A = __ldg(np), B = __ldg(np + 1), C = __ldg(np + 2);
  base = (int32_t)C.z;
  const float ex = __uint_as_float((A.w << 16) & 0x7F800000u);
  const float ey = __uint_as_float(A.w & 0x7F800000u);
  const float ez = __uint_as_float((A.w << 8) & 0x7F800000u);
  const float sx = ex * inv.x, sy = ey * inv.y, sz = ez * inv.z;
  const float bx = fmaf(-0.5f, sx, (__uint_as_float(A.x) - o.x) * inv.x);
  const float by = fmaf(-0.5f, sy, (__uint_as_float(A.y) - o.y) * inv.y);
  const float bz = fmaf(-0.5f, sz, (__uint_as_float(A.z) - o.z) * inv.z);
  // (near, far) pairs, the near one scaled
  constexpr float k = 1.0f - kBeyond;
  const f32x2 sx2 = pack2(sx * k, sx), sy2 = pack2(sy * k, sy), sz2 = pack2(sz * k, sz);
  const f32x2 bx2 = pack2(bx * k, bx), by2 = pack2(by * k, by), bz2 = pack2(bz * k, bz);
  const bool gx = __float_as_int(inv.x) < 0, gy = __float_as_int(inv.y) < 0, gz = __float_as_int(inv.z) < 0;
  const uint32_t nx = gx ? B.w : B.x, fx = gx ? B.x : B.w;
  const uint32_t ny = gy ? C.x : B.y, fy = gy ? B.y : C.x;
  const uint32_t nz = gz ? C.y : B.z, fz = gz ? B.z : C.y;
  const float t1c = fminf(lim, 3.402823466e+38f);
  auto child = [&](auto kc) {
    constexpr int K = decltype(kc)::value;
    float ax, ay, az, cx, cy, cz;
    unpack2(fma2(pack2(byte_f<K>(nx), byte_f<K>(fx)), sx2, bx2), ax, cx);
    unpack2(fma2(pack2(byte_f<K>(ny), byte_f<K>(fy)), sy2, by2), ay, cy);
    unpack2(fma2(pack2(byte_f<K>(nz), byte_f<K>(fz)), sz2, bz2), az, cz);
    const float t0 = fmaxf(max3f(ax, ay, az), 0.0f);
    const float t1 = fminf(min3f(cx, cy, cz), t1c);
    key[K] = t0 <= t1 ? __byte_perm(__float_as_uint(t0), C.w, 0x3214 + K) : ~0u;
  };
  child(std::integral_constant<int, 0>{});
  child(std::integral_constant<int, 1>{});
  child(std::integral_constant<int, 2>{});
  child(std::integral_constant<int, 3>{});
}

// The child of node `cur` that a key names: an inner child's slot, or, with
// the sign bit set, 4 cur + its slot in the node for a leaf, whose range is
// read when it is tested.
__device__ __forceinline__ int32_t child_ref(uint32_t key, int32_t cur, int32_t base) {
  const uint32_t code = key & 0xFFu;
  const uint32_t from = code & 0x80u ? 0x7FFFFF80u + 4u * (uint32_t)cur : (uint32_t)base;
  return (int32_t)(from + code);
}

// pluecker_t with the U and V sides in packed arithmetic: the same operations
// in the same order.  ptxas contracts a packed multiplication and addition
// whatever their rounding modifiers and -fmad say, so sums of products are
// formed as fma(p, one, q) with a `one` that it cannot see through (the two
// are equal: p x 1 is exact), and differences as sums with a negated edge.
__device__ __forceinline__ bool pluecker_t2(float3 a, float3 b, float3 c, float3 O, float3 D, f32x2 one, float &t) {
  const float3 v0 = f3sub(a, O), v1 = f3sub(b, O), v2 = f3sub(c, O);
  // lower half: edge e0 = v2 - v0 with v2 + v0, upper half: e1 = v0 - v1 with v0 + v1
  const f32x2 px = pack2(v2.x, v0.x), py = pack2(v2.y, v0.y), pz = pack2(v2.z, v0.z);
  const f32x2 qx = pack2(v0.x, v1.x), qy = pack2(v0.y, v1.y), qz = pack2(v0.z, v1.z);
  const f32x2 ex = sub2(px, qx), ey = sub2(py, qy), ez = sub2(pz, qz);
  const f32x2 mx = sub2(qx, px), my = sub2(qy, py), mz = sub2(qz, pz);
  const f32x2 sx = add2(px, qx), sy = add2(py, qy), sz = add2(pz, qz);
  const f32x2 kx = fma2(mul2(mz, sy), one, mul2(ey, sz)), ky = fma2(mul2(mx, sz), one, mul2(ez, sx)),
              kz = fma2(mul2(my, sx), one, mul2(ex, sy));
  float U, V;
  unpack2(fma2(fma2(mul2(kx, pack2(D.x, D.x)), one, mul2(ky, pack2(D.y, D.y))), one, mul2(kz, pack2(D.z, D.z))), U, V);
  const float3 e2 = f3sub(v1, v2);
  const float W = f3dot(f3cross(e2, f3add(v1, v2)), D);
  const float UVW = U + V + W;
  const float eps = 1.1920928955078125e-07f * fabsf(UVW);
  if (!(min3f(U, V, W) >= -eps || max3f(U, V, W) <= eps)) return false;
  float3 e0, e1;
  unpack2(ex, e0.x, e1.x);
  unpack2(ey, e0.y, e1.y);
  unpack2(ez, e0.z, e1.z);
  return pluecker_dist(v0, e0, e1, e2, D, t);
}

// The exact slab test of a box against (o, inv), limit lim: tnear, or NaN on
// a miss — the same operations as the fp32 wide nodes' visit_node.  `reach`: where
// the ray leaves the box enlarged by `slack`.
__device__ __forceinline__ float slab_exact(const float *lo, const float *hi, const float3 &o, const float3 &inv,
                                            float lim, float slack, float &reach) {
  const float oo[3] = {o.x, o.y, o.z}, ii[3] = {inv.x, inv.y, inv.z};
  float t0 = 0.0f, t1 = fminf(lim, 3.402823466e+38f);
  reach = __int_as_float(0x7f800000);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const bool g = (__float_as_uint(ii[a]) >> 31) != 0u;
    const float tn = ((g ? hi[a] : lo[a]) - oo[a]) * ii[a], tf = ((g ? lo[a] : hi[a]) - oo[a]) * ii[a];
    t0 = fmaxf(tn, t0);
    t1 = fminf(tf, t1);
    reach = fminf(tf + slack * fabsf(ii[a]), reach);
  }
  return t0 <= t1 ? t0 : __int_as_float(0x7fffffff);
}
__device__ __forceinline__ float slab_exact(const float *lo, const float *hi, const float3 &o, const float3 &inv,
                                            float lim) {
  float reach;
  return slab_exact(lo, hi, o, inv, lim, 0.0f, reach);
}

// The exact-box tree of a 4-wide handle.
struct Exact4 {
  const Node2 *nodes2;
  const TriRec *tris;
  Ranges R;
  int32_t leaf_size;
  const int32_t *roots;  // BVH2 roots per scene
  const int64_t *ray_off;
  int32_t n_scenes;
  int64_t most;          // steps of a walk: each node and leaf range once, at most
};

__device__ __forceinline__ void tri_rec_box(const TriRec *__restrict__ tris, int64_t g, float *lo, float *hi) {
  const float4 *p = (const float4 *)(tris + g);
  const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  tri_box(make_float3(a.x, a.y, a.z), make_float3(b.x, b.y, b.z), make_float3(c.x, c.y, c.z), lo, hi);
}

// Ray `ray` over the exact boxes, in the exact order: the children of a wide
// node are formed from the BVH2 records as the collapse forms them, and
// visited nearest first with a deep stack.  Returns the sorted position and t
// of the closest hit (any hit: any position), or -1 and tmax.
//
// `near` >= 0: the t that the traversal found to be the closest.  What the exact
// order finds is decided by the candidates that lie within rounding of it, so the
// walk only enters boxes that the ray is in there, give or take kAround: about as
// many as the tree is deep.  (Should it find nothing, it starts again without `near`.)  1 M rays on
// 65,536 triangles, three of each: 10.9 ms with whole walks, 1.97 with these.
struct ExactHit {
  int32_t prim;
  float t;
};
template <bool ANY>
__device__ __forceinline__ ExactHit retrace4(const Exact4 &X, const RaySoA &RS, int64_t ray, float near,
                                             uint32_t *err) {
  // Entries: (tnear rounded down | BVH2 ref, or ~(first << 3 | count - 1)).
  uint64_t stk[kRetryStack];
  float3 o, d, inv;
  float tmin, tmax;
  load_ray(RS, ray, o, d, inv, tmin, tmax);
  const int32_t root = scene_root(X.roots, X.ray_off, X.n_scenes, ray);
  ExactHit h{-1, tmax};
  if (root == INT32_MIN) return h;
  bool again;
  do {
    float best = near >= 0.0f ? fminf(near * (1.0f + kAround), tmax) : tmax;
    // a hit may lie that far from its triangle
    const float slack = fabsf(near) * max3f(fabsf(d.x), fabsf(d.y), fabsf(d.z)) * 3.814697265625e-06f;  // 2^-18
    bool have = false;
    int sp = 0;
    int32_t cur = root < 0 ? ~((~root) << 3) : root;
    int64_t left = X.most;
    while (true) {
      bool next = false;
      if (--left < 0) {  // a broken tree
        atomicOr(err, kErrQueue);
        break;
      }
      if (cur >= 0) {
        Cand c[4];
        int nc;
        open_wide<4>(X.nodes2, X.R, X.leaf_size, cur, c, nc);
        uint32_t key[4];
        int32_t ref[4];
        int nh = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          key[k] = ~0u;
          ref[k] = 0;
          if (k < nc) {
            float reach;
            const float t0 = slab_exact(c[k].lo, c[k].hi, o, inv, best, slack, reach);
            if (t0 == t0 && !(reach < near * (1.0f - kAround))) {
              key[k] = (__float_as_uint(t0) & 0x7FFFFFFCu) | (uint32_t)k;
              ++nh;
            }
            ref[k] = c[k].ref < 0 || c[k].count <= X.leaf_size ? ~((c[k].first << 3) | (c[k].count - 1)) : c[k].ref;
          }
        }
        sort_keys<4>(key);
        if (sp + nh > kRetryStack) {
          atomicOr(err, kErrStack);
          break;
        }
#pragma unroll
        for (int k = 3; k >= 1; --k)
          if (k < nh) stk[sp++] = key_entry<4>(key[k], ref);
        if (nh > 0) {
          cur = key_ref<4>(key[0], ref);
          next = true;
        }
      } else {
        const int32_t enc = ~cur;
        const int64_t first = (int64_t)((uint32_t)enc >> 3);
        const int count = (enc & 7) + 1;
        for (int j = 0; j < count; ++j) {
          if (ANY) {
            if (test_tri_any(X.tris, first + j, o, d, tmin, tmax)) return ExactHit{(int32_t)(first + j), tmax};
          } else {
            test_tri(X.tris, first + j, o, d, tmin, best, have, h.prim);
          }
        }
      }
      while (!next && sp > 0) {
        const uint64_t e = stk[--sp];
        if (__uint_as_float((uint32_t)(e >> 32)) > best) continue;
        cur = (int32_t)(uint32_t)e;
        next = true;
      }
      if (!next) break;
    }
    if (have) h.t = best;
    again = near >= 0.0f && !have;
    near = -1.0f;
  } while (again);
  return h;
}

// Which of two sorted positions of a scene the exact traversal of a ray tests
// first: at the wide node where their paths part, the child that is entered
// first; within a leaf range, the lower one.
__device__ __noinline__ int32_t first_of_two(const Exact4 &X, const RaySoA &RS, int64_t ray, int32_t p, int32_t q) {
  int32_t cur = scene_root(X.roots, X.ray_off, X.n_scenes, ray);
  for (int level = 0; cur >= 0 && level < 4096; ++level) {
    WalkCand c[4];
    int nc;
    walk_open(X.nodes2, X.R, X.leaf_size, cur, c, nc);
    int32_t next = INT32_MIN, bp = -1, bq = -1, sp = 0, sq = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k < nc) {
        if ((uint32_t)(p - c[k].first) < (uint32_t)c[k].count) {
          bp = c[k].box;
          sp = k;
          if (c[k].ref >= 0 && c[k].count > X.leaf_size) next = c[k].ref;
        }
        if ((uint32_t)(q - c[k].first) < (uint32_t)c[k].count) {
          bq = c[k].box;
          sq = k;
        }
      }
    }
    if (bp < 0 || bq < 0) break;  // a broken tree
    if (bp != bq) {
      float3 o, d, inv;
      float tmin, tmax;
      load_ray(RS, ray, o, d, inv, tmin, tmax);
      auto key = [&](int32_t box, int slot) {
        float lo[3], hi[3];
        walk_box(X.nodes2, box, lo, hi);
        return (__float_as_uint(slab_exact(lo, hi, o, inv, 3.402823466e+38f)) & 0x7FFFFFFCu) | (uint32_t)slot;
      };
      return key(bp, sp) < key(bq, sq) ? p : q;
    }
    cur = next;
  }
  return min(p, q);
}

// Final values of a closest hit: sorted position g, fp32 t.
__device__ __forceinline__ void finish_hit(const RaySoA &R, const Out &O, const TriRec *__restrict__ tris, int64_t i,
                                           int32_t g, float best) {
  const float3 o = make_float3(__ldg(R.ox + i), __ldg(R.oy + i), __ldg(R.oz + i));
  const float3 d = make_float3(__ldg(R.dx + i), __ldg(R.dy + i), __ldg(R.dz + i));
  const float4 *p = (const float4 *)(tris + g);
  const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  const float3 pa = make_float3(a.x, a.y, a.z), pb = make_float3(b.x, b.y, b.z), pc = make_float3(c.x, c.y, c.z);
  float u = 0.0f, v = 0.0f;
  if (!refine_tuv(pa, pb, pc, o, d, best, u, v)) {
    // N.D == 0: the fp32 barycentrics of the test stand (t stays the test's)
    float tf;
    pluecker(pa, pb, pc, o, d, tf, u, v);
  }
  O.prim[i] = __float_as_int(a.w);
  O.t[i] = best;
  O.u[i] = u;
  O.v[i] = v;
}

// Those of the closest hits that k_trace4 is sure of, one ray per thread; the rays
// that other threads settle are left alone: neither kListed nor a finished id
// has kPending.
__device__ __forceinline__ void finish_pending(const RaySoA &R, int64_t n, const Out &O,
                                               const TriRec *__restrict__ tris) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t g = O.prim[i];
    if (g < 0 || !(g & kPending)) continue;
    finish_hit(R, O, tris, i, g & ~kPending, O.t[i]);
  }
}

// Final values of a listed ray.
__device__ __noinline__ void settle(const RaySoA &R, const Out &O, const Exact4 &X, int64_t i, uint32_t *err) {
  const int32_t q = __float_as_int(O.v[i]);
  ExactHit h{__float_as_int(O.u[i]), O.t[i]};
  if (q >= 0) h.prim = first_of_two(X, R, i, h.prim, q);
  else h = retrace4<false>(X, R, i, q == kByWalk ? h.t : -1.0f, err);
  if (h.prim >= 0) {
    finish_hit(R, O, X.tris, i, h.prim, h.t);
  } else {
    O.prim[i] = -1;
    O.t[i] = h.t;
    O.u[i] = 0.0f;
    O.v[i] = 0.0f;
  }
}

// Clears the trace's counters for the next one, in the last block to get here
// (the word above the list's length counts them, and wraps to 0).
__device__ __forceinline__ void clear_counters(const Scratch &S) {
  __syncthreads();  // every thread has read the list's length
  if (threadIdx.x == 0 && atomicInc(S.ovf_count + 1, gridDim.x - 1) == gridDim.x - 1) {
    *S.work = 0ull;
    *S.ovf_count = 0u;
  }
}

// Settles the rays that k_trace4 left open and writes the final values of all.
// The list comes first: the walks of its rays take longer than the others'
// values, which hide them.  Up to kSettleWide rays with registers for the walks
// (five blocks of 128 threads per SM), above with as few as the values need: 921,600
// camera rays 222 -> 218 us against 64 registers, 1 M rays on layers of quads 258 ->
// 248; 31.6 M rays 20.15 -> 20.05 ms against five blocks of 128.
constexpr int64_t kSettleWide = 1 << 21;
template <int THREADS, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS)
    k_settle4(const __grid_constant__ RaySoA R, RayCount N, Out O, const __grid_constant__ Exact4 X, Scratch S) {
  after_wait();
  const uint32_t cnt = *S.ovf_count;
  const int64_t n = N.get();
  const int64_t t = (int64_t)blockIdx.x * THREADS + threadIdx.x, threads = (int64_t)gridDim.x * THREADS;
  const bool listed = cnt <= S.ovf_cap;  // else look for the marks
  const int64_t end = listed ? (int64_t)cnt : n;
  // a short list: a ray to a warp
  const int64_t first = end <= threads / 32 ? (t & 31) * (threads / 32) + (t >> 5) : t;
  for (int64_t j = first; j < end; j += threads) {
    const int64_t i = listed ? S.ovf[j] : j;
    if (O.prim[i] == kListed) settle(R, O, X, i, S.err);
  }
  finish_pending(R, n, O, X.tris);
  clear_counters(S);
}

// Any-hit rays that k_trace4 left open.
__global__ void __launch_bounds__(128)
    k_trace_retry4(const __grid_constant__ RaySoA R, RayCount N, Out O, const __grid_constant__ Exact4 X, Scratch S) {
  after_wait();
  const uint32_t cnt = *S.ovf_count;
  const bool listed = cnt <= S.ovf_cap;  // else look for the marks
  const int64_t end = listed ? (int64_t)cnt : N.get();
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < end; j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = listed ? S.ovf[j] : j;
    if (O.occ[i] == kOccListed) O.occ[i] = retrace4<true>(X, R, i, -1.0f, S.err).prim >= 0 ? 1 : 0;
  }
  clear_counters(S);
}

// The traversal: while-while with speculative leaf postponing (Aila & Laine,
// "Understanding the efficiency of ray traversal on GPUs", HPG 2009).  Each
// lane walks inner nodes; a lane that reaches a leaf parks it (up to two) and
// keeps walking until at most kLeafWait lanes of the warp still look for
// their first leaf; then the warp tests the parked leaves together, so node
// and leaf code run with most lanes active.  One wave of resident blocks at
// most; warps refill idle lanes from the ray counter once `refill` of them
// are idle.
//
// Stack: entries (key | ref) in shared memory, [slot][thread], over a sentinel
// that no culling removes and that names the end of the ray.  When it is full
// its lower half moves to the per-thread local array, and back when the
// sentinel is reached; a ray that overflows both is traced again with a deep
// stack (closest: k_settle4, any: k_trace_retry4).
//
// A ray is a chain of dependent steps, and a few rays visit ten times as many
// nodes as the average, so without more the last of them set the time of a
// launch (of half of it on camera rays of a surface), and the longest that of
// a small batch.  Once the counter is exhausted, idle lanes of a warp
// therefore help the others: each takes one of their stack entries, the lowest
// (farthest, and mostly largest) subtrees first, with a copy of the ray, and
// walks it as a ray of its own.  The lane that took the ray from the counter
// leads: at every turn of the outer loop it collects the group's closest hit,
// under the rules for a second candidate of the same ray, and all take its t
// for their limit; it retires once its helpers are done.
//
// leaf_wait: kLeafWait; for any hit (one scene) kLeafWaitAny in a tree of more than
// kLargeTree triangles.  The deeper the tree, the more the turns differ at which
// the lanes of a warp find their first leaf.  2 M shadow rays, 12 lanes against 8:
// displaced spheres of 1,280 triangles 281 / 271 us, 5,120 325 / 317, 20,480 374 /
// 370, 81,920 428 / 425, 327,680 490 / 492, 1.3 M 561 / 573 (200,000 rays: 5,120
// 87 / 82, 20,480 108 / 104, 81,920 136 / 136, 1.3 M 220 / 225); soups of 65,536 to 8 M
// triangles within 1 % of each other, 12 lanes ahead by 0.2 to 0.9 % at 2 M rays.
constexpr int kLeafWait = 8, kLeafWaitAny = 12;
constexpr int64_t kLargeTree = 1 << 18;
// Slots, the sentinel's included.  With the ray indices 32 KB per 256-thread
// block: four blocks leave 124 KB of an SM for L1, a byte more only 92.
constexpr int kStackSlots = 15;
constexpr int kStackMove = 8;    // entries moved at a time
constexpr int kStackLocal = 64;
// Turns of the node loop after the counter's end before lanes help, and
// between two rounds of helping: 4 / 4; us at 32 / 8, 16 / 4, 8 / 4, 4 / 4:
// 1 M camera rays on 327,680 triangles 199, 186, 183, 182 (240 without help),
// 2 M shadow rays 511, 490, 479, 475, a 640x360 x 4 image 1319, 1206, 1145,
// 1115, 4,096 rays on 20,001 triangles 60, 45, 42, 36 (96 at the time that every
// ray walked alone).
constexpr int kHelpAfter = 4;
constexpr int kHelpTurns = 4;

__device__ __forceinline__ void stack_store(uint32_t at, uint32_t key, int32_t ref) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at), "r"(key), "r"(ref) : "memory");
}
__device__ __forceinline__ void stack_load(uint32_t at, uint32_t &key, int32_t &ref) {
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(key), "=r"(ref) : "r"(at) : "memory");
}

// COUNTED: the number of rays stands in device memory (as a runtime choice it
// made long launches 0.5 % slower).
template <bool ANY, bool COUNTED>
__global__ void __launch_bounds__(256, 4)
    k_trace4(const NodeQ *__restrict__ nodes, const TriRec *__restrict__ tris, const int32_t *__restrict__ roots,
             const int64_t *__restrict__ ray_off, int n_scenes, RaySoA R, RayCount N, Out O, Scratch S, int refill,
             int lanes, int leaf_wait, float one) {
  // What a lane does next: a node (0 .. kPop - 1), a leaf (< 0), a pop, nothing
  // more for its ray, or nothing.  No parked leaf: 0.
  constexpr int32_t kPop = 0x7FFFFFFD, kDone = 0x7FFFFFFE, kIdle = 0x7FFFFFFF;
  constexpr uint32_t kSlot = 256 * sizeof(uint64_t);  // bytes between a thread's slots
  constexpr unsigned kAll = 0xFFFFFFFFu;
  // The upper word: bits 32 .. 47 of the ray's index; trace it again over the
  // exact boxes (its stack overflowed, an any-hit candidate's own box kept
  // it out, or its inverse direction is too small or too large); and, as
  // multiples of kHelper, its helpers at work.
  constexpr uint32_t kRayHigh = 0xFFFFu, kAgain = 1u << 16, kHelper = 1u << 17;
  // A second candidate near the closest hit: none, one within kNear but not
  // equal, two or more equal, or (>= 0) the one that is equal.
  constexpr int32_t kNone = -1, kSome = -2, kMany = -3;
  __shared__ uint64_t s_stk[kStackSlots][256];
  __shared__ uint32_t s_ray[2][256];  // the ray's index; in the upper word also its flags and helpers
  const uint32_t s_base = (uint32_t)__cvta_generic_to_shared(&s_stk[0][0]);
  const uint32_t bottom = s_base + threadIdx.x * (uint32_t)sizeof(uint64_t);
  uint32_t *crew = s_ray[1] + (threadIdx.x & ~31u);  // the upper words of the warp's lanes
  stack_store(bottom, 0xFF800000u, kDone);  // the sentinel: -inf
  after_wait();
  uint64_t stk[kStackLocal];
  float3 o = make_float3(0.f, 0.f, 0.f), d = o, inv = o;
  float tmin = 0.f;
  float best = 0.f;  // the ray's limit: tmax, and the closest t so far
  int32_t prim = -1, tie = kNone, cur = kIdle, leaf = 0, leaf2 = 0;
  uint32_t low = bottom;          // the lane's sentinel: entries given away lie below it
  uint32_t top = bottom + kSlot;  // the next free slot
  int moved = 0;                  // entries in the local array
  int scene = -1;
  int lead = 0;                   // the lane that leads this ray
  int phase = 0;                  // 0 at the start; 1 the counter has rays; then 2 + turns since it has none
  // The first `lanes` rays of every warp by its index, the others from the
  // counter, which starts behind them.
  const int64_t taken = (int64_t)gridDim.x * (blockDim.x >> 5) * lanes;

  while (true) {
    const int lane = threadIdx.x & 31;
    // Lanes that help hand their hits to the lane that leads, share its limit,
    // and are idle again once they are done.
    const bool helps = cur != kIdle && lead != lane;
    if (phase > kHelpAfter && __any_sync(kAll, helps)) {
      for (unsigned m = __ballot_sync(kAll, helps && (prim >= 0 || tie != kNone)); m != 0u; m &= m - 1u) {
        const int h = __ffs(m) - 1;
        const int to = __shfl_sync(kAll, lead, h);
        const float h_best = __shfl_sync(kAll, best, h);
        const int32_t h_prim = __shfl_sync(kAll, prim, h), h_tie = __shfl_sync(kAll, tie, h);
        if (lane == to) {
          if (ANY) {
            prim = h_prim;
            cur = kDone;
            leaf = leaf2 = 0;
          } else if (h_prim < 0) {
            if (tie == kNone) tie = kSome;
          } else if (h_best < best || (prim < 0 && h_best == best)) {
            tie = h_tie != kNone ? h_tie : best <= h_best * (1.0f + kNear) ? kSome : kNone;
            best = h_best;
            prim = h_prim;
          } else if (h_best == best) {
            tie = (tie == kNone || tie == kSome) && (h_tie == kNone || h_tie == kSome) ? h_prim : kMany;
          } else if (h_best <= best * (1.0f + kNear) && tie == kNone) {
            tie = kSome;
          }
        }
      }
      const float l_best = __shfl_sync(kAll, best, lead);
      const int32_t l_prim = __shfl_sync(kAll, prim, lead);
      if (helps) {
        prim = -1;
        tie = kNone;
        if (!ANY) best = l_best;
        if (ANY && l_prim >= 0) {
          cur = kDone;
          leaf = leaf2 = 0;
        }
        if (cur == kDone && leaf == 0) {
          cur = kIdle;
          atomicSub(crew + lead, kHelper);
        }
      }
      __syncwarp();
    }
    // Retire finished rays.
    if (cur == kDone && leaf == 0 && lead == lane && *(volatile uint32_t *)(crew + lane) < kHelper) {
      const uint32_t flags = crew[lane];
      const int64_t at = (int64_t)(flags & kRayHigh) << 32 | s_ray[0][threadIdx.x];
      const bool redo = (flags & kAgain) != 0u;
      if (ANY) {
        O.occ[at] = prim >= 0 ? 1 : redo ? kOccListed : 0;
        if (redo && prim < 0) {
          const uint32_t k = atomicAdd(S.ovf_count, 1u);
          if (k < S.ovf_cap) S.ovf[k] = at;  // past the end the mark is looked for
        }
      } else {
        bool listed = redo;
        int32_t other = -1;
        if (prim >= 0 && !listed) {
          // the winner's box, and that of a second triangle at the same t
          const float3 ie = make_float3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
          float lo[3], hi[3];
          tri_rec_box(tris, prim, lo, hi);
          float t0 = slab_exact(lo, hi, o, ie, 3.402823466e+38f);
          listed = tie == kNone ? !(t0 <= best * (1.0f + kNear)) : tie == kSome ? !(t0 <= best) : true;
          if (t0 <= best * (1.0f + 0.5f * kAround)) other = kByWalk;
          if (tie >= 0 && t0 <= best) {
            tri_rec_box(tris, tie, lo, hi);
            t0 = slab_exact(lo, hi, o, ie, 3.402823466e+38f);
            if (t0 <= best) other = tie;
          }
        }
        O.t[at] = best;  // of a miss, tmax
        O.prim[at] = listed ? kListed : prim >= 0 ? prim | kPending : -1;
        if (listed) {
          O.u[at] = __int_as_float(prim);
          O.v[at] = __int_as_float(other);
          const uint32_t k = atomicAdd(S.ovf_count, 1u);
          if (k < S.ovf_cap) S.ovf[k] = at;  // past the end the mark is looked for
        } else if (prim < 0) {
          O.u[at] = 0.0f;
          O.v[at] = 0.0f;
        }
      }
      cur = kIdle;
    }
    // Take new rays.
    const unsigned idle = __ballot_sync(kAll, cur == kIdle);
    const int nidle = __popc(idle);
    if (phase < 2 && nidle >= refill) {
      const int64_t n = COUNTED ? (int64_t)*N.at : N.most;
      int64_t my;
      if (phase == 0) {
        my = lane < lanes ? ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * lanes + lane : n;
        phase = taken >= n ? 2 : 1;
      } else {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(S.work, (unsigned long long)nidle);
        base = __shfl_sync(kAll, base, 0) + (unsigned long long)taken;
        my = (int64_t)base + __popc(idle & ((1u << lane) - 1u));
        if ((int64_t)base + nidle >= n) phase = 2;
      }
      if (cur == kIdle && my < n) {
        s_ray[0][threadIdx.x] = (uint32_t)my;
        crew[lane] = (uint32_t)(my >> 32);
        load_ray(R, my, o, d, inv, tmin, best);
        tie = kNone;
        prim = -1;
        cur = scene_root_walk(roots, ray_off, n_scenes, my, scene);
        if (cur == kEmptyChild) cur = kDone;
        if (odd_inv(inv) && cur != kDone && !inv_q(nodes + cur, o, d, best, inv)) {
          crew[lane] |= kAgain;
          cur = kDone;
        }
        low = bottom;
        top = bottom + kSlot;
        moved = 0;
        lead = lane;
      }
    } else if (phase >= 2 && idle != 0u) {
      if (idle == kAll) break;
      // Help: of the entries in the lanes' stacks, in lane order and each lane's
      // lowest first, the r-th idle lane takes the r-th.
      int left = phase > kHelpAfter && cur < kDone && moved == 0 ? (int)((top - low) / kSlot) - 1 : 0;
      int upto = left;  // entries in the lanes up to this one
#pragma unroll
      for (int w = 1; w < 32; w <<= 1) {
        const int v = __shfl_up_sync(kAll, upto, w);
        if (lane >= w) upto += v;
      }
      const int k = min(nidle, __shfl_sync(kAll, upto, 31));
      if (k > 0) {
        const int r = __popc(idle & ((1u << lane) - 1u));
        const bool take = cur == kIdle && r < k;
        int from = 0;  // the first lane whose entries reach past r
#pragma unroll
        for (int w = 16; w >= 1; w >>= 1)
          if (__shfl_sync(kAll, upto, (from + w - 1) & 31) <= r) from += w;
        if (!take) from = lane;
        const int before = upto - left, give = max(0, min(left, k - before));
        o.x = __shfl_sync(kAll, o.x, from);
        o.y = __shfl_sync(kAll, o.y, from);
        o.z = __shfl_sync(kAll, o.z, from);
        d.x = __shfl_sync(kAll, d.x, from);
        d.y = __shfl_sync(kAll, d.y, from);
        d.z = __shfl_sync(kAll, d.z, from);
        inv.x = __shfl_sync(kAll, inv.x, from);
        inv.y = __shfl_sync(kAll, inv.y, from);
        inv.z = __shfl_sync(kAll, inv.z, from);
        tmin = __shfl_sync(kAll, tmin, from);
        best = __shfl_sync(kAll, best, from);
        lead = __shfl_sync(kAll, lead, from);
        const uint32_t at = __shfl_sync(kAll, low, from) + (uint32_t)(1 + r - __shfl_sync(kAll, before, from)) * kSlot;
        if (take) {
          uint32_t key;
          stack_load(at, key, cur);
          tie = kNone;
          prim = -1;
          low = bottom;
          top = bottom + kSlot;
          moved = 0;
          atomicAdd(crew + lead, kHelper);
        }
        __syncwarp();  // the entries are read before a slot becomes a sentinel
        if (give > 0) {
          low += (uint32_t)give * kSlot;  // the last slot given away becomes the sentinel
          stack_store(low, 0xFF800000u, kDone);
        }
      }
    }

    // Inner nodes, parking the first two leaves found.  Ends once at most
    // kLeafWait lanes are still looking for their first leaf (waiting for the
    // last few cost more idle node iterations than the leaf tests they would
    // have joined), unless there is neither a leaf to test nor a ray to take;
    // with idle lanes that can only help, after kHelpTurns at the latest.
    unsigned seeking;
    int turns = 0;
    do {
      if (cur == kPop) {
        uint32_t key;
        do {
          top -= kSlot;
          stack_load(top, key, cur);
        } while (__uint_as_float(key & ~0xFFu) > best);
        if (cur == kDone && moved > 0) {
          moved -= kStackMove;
          for (int k = 0; k < kStackMove; ++k) {
            top += kSlot;
            stack_store(top, (uint32_t)(stk[moved + k] >> 32), (int32_t)(uint32_t)stk[moved + k]);
          }
          top += kSlot;
          cur = kPop;
        }
      }
      if ((uint32_t)cur < (uint32_t)kPop) {
        uint32_t key[4];
        int32_t base;
        visit_q(nodes + cur, o, inv, best, key, base);
        sort_keys<4>(key);
        const int32_t from = cur;
        cur = (int32_t)key[0] >= 0 ? child_ref(key[0], from, base) : kPop;
        if ((int32_t)key[1] >= 0) {
          // the other children, the farthest first
          if ((int32_t)key[2] >= 0) {
            if ((int32_t)key[3] >= 0) {
              stack_store(top, key[3], child_ref(key[3], from, base));
              top += kSlot;
            }
            stack_store(top, key[2], child_ref(key[2], from, base));
            top += kSlot;
          }
          stack_store(top, key[1], child_ref(key[1], from, base));
          top += kSlot;
          if (top >= s_base + (kStackSlots - 2) * kSlot) {
            // Fewer than three slots are left: reclaim those given away, and if
            // that was not enough move the lower entries to the local array.
            uint32_t at, key_m;
            int32_t ref_m;
            if (low != bottom) {
              const uint32_t shift = low - bottom;
              for (at = low; at < top; at += kSlot) {
                stack_load(at, key_m, ref_m);
                stack_store(at - shift, key_m, ref_m);
              }
              top -= shift;
              low = bottom;
            }
            if (top >= s_base + (kStackSlots - 2) * kSlot) {
              if (moved + kStackMove > kStackLocal) {
                atomicOr(crew + lead, kAgain);
                cur = kDone;
                leaf = leaf2 = 0;
              } else {
                at = bottom + kSlot;
                for (int k = 0; k < kStackMove; ++k, at += kSlot) {
                  stack_load(at, key_m, ref_m);
                  stk[moved + k] = (uint64_t)key_m << 32 | (uint32_t)ref_m;
                }
                for (; at < top; at += kSlot) {
                  stack_load(at, key_m, ref_m);
                  stack_store(at - kStackMove * kSlot, key_m, ref_m);
                }
                top -= kStackMove * kSlot;
                moved += kStackMove;
              }
            }
          }
        }
      }
      if (cur < 0 && leaf2 == 0) {
        leaf2 = leaf;
        leaf = cur;
        cur = kPop;
      }
      ++turns;
      seeking = __ballot_sync(kAll, leaf == 0 && cur < kDone);
    } while (__popc(seeking) > (ANY ? leaf_wait : kLeafWait)
                 ? !(phase >= 2 && idle != 0u && turns >= kHelpTurns)
                 : seeking != 0u && phase >= 2 && turns < kHelpTurns && !__any_sync(kAll, leaf != 0));
    if (phase >= 2 && phase <= kHelpAfter) phase += turns;

    // Test the (up to two) parked leaves together.
    if (leaf != 0) {
      const uint32_t s1 = (uint32_t)leaf & 0x7FFFFFFFu, s2 = (uint32_t)leaf2 & 0x7FFFFFFFu;
      const int32_t e1 = ~__ldg(nodes[s1 >> 2].leaf + (s1 & 3u));
      const int32_t e2 = leaf2 == 0 ? -1 : ~__ldg(nodes[s2 >> 2].leaf + (s2 & 3u));
      // an unused slot holds no range
      const int n1 = e1 < 0 ? 0 : (e1 & 7) + 1;
      const int total = e2 < 0 ? n1 : n1 + (e2 & 7) + 1;
      const int32_t f1 = (int32_t)((uint32_t)e1 >> 3), f2 = (int32_t)((uint32_t)e2 >> 3) - n1;
      for (int j = 0; j < total; ++j) {
        const int32_t g = (j < n1 ? f1 : f2) + j;
        const float4 *p = (const float4 *)(tris + g);
        const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
        float t;
        if (!pluecker_t2(make_float3(a.x, a.y, a.z), make_float3(b.x, b.y, b.z), make_float3(c.x, c.y, c.z), o, d,
                         pack2(one, one), t))
          continue;
        if (ANY) {
          if (t >= tmin && !(t > best)) {
            const float3 ie = make_float3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
            float lo[3], hi[3];
            tri_rec_box(tris, g, lo, hi);
            const float t0 = slab_exact(lo, hi, o, ie, best);
            if (t0 == t0) {
              prim = g;
              cur = kDone;
              break;
            }
            atomicOr(crew + lead, kAgain);
          }
        } else if (t >= tmin && t <= best * (1.0f + kNear)) {
          if (t < best || (prim < 0 && t == best)) {
            tie = best <= t * (1.0f + kNear) ? kSome : kNone;
            best = t;
            prim = g;
          } else if (t == best) {
            tie = tie == kNone || tie == kSome ? g : kMany;
          } else if (tie == kNone) {
            tie = kSome;
          }
        }
      }
      leaf = 0;
      leaf2 = 0;
    }
  }
}

template <int W, bool ANY, bool MT = false>
__global__ void __launch_bounds__(128)
    k_trace_retry(const NodeW<8> *__restrict__ wide, const Node2 *__restrict__ nodes2,
                  const TriRec *__restrict__ tris, const int32_t *__restrict__ roots,
                  const int64_t *__restrict__ ray_off, int n_scenes, RaySoA R, Out O, Scratch S) {
  const uint32_t cnt = min((int64_t)*S.ovf_count, S.ovf_cap);
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt; j += gridDim.x * blockDim.x) {
    const int64_t i = S.ovf[j];
    float3 o, d, inv;
    float tmin, tmax;
    load_ray(R, i, o, d, inv, tmin, tmax);
    const int32_t root = scene_root(roots, ray_off, n_scenes, i);
    bool have;
    int32_t prim;
    float best;
    bool done;
    if constexpr (W == 2) {
      done = trace_bvh2<ANY, kRetryStack, MT>(nodes2, tris, root, o, d, inv, tmin, tmax, have, prim, best);
    } else {
      Tracer<W, ANY, kRetryStack> tr;
      tr.o = o; tr.d = d; tr.inv = inv; tr.tmin = tmin; tr.tmax = tmax;
      tr.start(root);
      while (!tr.step(wide, tris)) {
      }
      done = !tr.overflow;
      have = tr.have;
      prim = tr.prim;
      best = tr.best;
    }
    if (!done) atomicOr(S.err, kErrStack);
    else write_result(O, i, ANY, have, prim, best, tmax);
  }
}

// ----------------------------------------------------------------------------
// Host side.
// ----------------------------------------------------------------------------

// ----------------------------------------------------------------------------
// Ray sort (flg_trace_opts.ray_sort = 1): rays of a single-scene trace are
// reordered by a 30-bit key — direction octant (3 bits) above a 27-bit Morton
// code of the origin in the scene box enlarged by its extent on every side —
// traced in that order, and their hits written back in the caller's order.
// Neighbouring lanes then start in the same region heading the same way.
// ----------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    k_ray_keys(RaySoA R, int64_t n, const float *__restrict__ box, uint32_t *__restrict__ keys,
               uint32_t *__restrict__ hist) {
  __shared__ uint32_t s_hist[4][256];
  for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) (&s_hist[0][0])[i] = 0u;
  __syncthreads();
  float lo[3], sc[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float e = box[3 + k] - box[k];
    lo[k] = box[k] - e;
    sc[k] = e > 0.0f ? 1.0f / (3.0f * e) : 0.0f;
  }
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float o[3] = {__ldg(R.ox + i), __ldg(R.oy + i), __ldg(R.oz + i)};
    const float d[3] = {__ldg(R.dx + i), __ldg(R.dy + i), __ldg(R.dz + i)};
    uint32_t q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float u = fminf(fmaxf((o[k] - lo[k]) * sc[k], 0.0f), 1.0f);
      q[k] = min((uint32_t)(u * 512.0f), 511u);  // NaN origins land in cell 0
    }
    const uint32_t oct = (d[0] < 0.0f ? 1u : 0u) | (d[1] < 0.0f ? 2u : 0u) | (d[2] < 0.0f ? 4u : 0u);
    const uint32_t key = (oct << 27) | (left_shift3(q[2]) << 2) | (left_shift3(q[1]) << 1) | left_shift3(q[0]);
    keys[i] = key;
#pragma unroll
    for (int p = 0; p < 4; ++p) atomicAdd(&s_hist[p][(key >> (8 * p)) & 0xFFu], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) {
    const uint32_t c = (&s_hist[0][0])[i];
    if (c) atomicAdd(&hist[i], c);
  }
}

// Sorted position j takes ray perm[j].
__global__ void k_ray_gather(RaySoA R, int64_t n, const uint32_t *__restrict__ perm, float *__restrict__ out) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = perm[j];
    if (i < 0 || i >= n) continue;  // only a timed-out sort leaves such slots (error word set)
    out[j] = __ldg(R.ox + i);
    out[n + j] = __ldg(R.oy + i);
    out[2 * n + j] = __ldg(R.oz + i);
    out[3 * n + j] = __ldg(R.dx + i);
    out[4 * n + j] = __ldg(R.dy + i);
    out[5 * n + j] = __ldg(R.dz + i);
    out[6 * n + j] = R.tmin ? __ldg(R.tmin + i) : R.tmin_c;
    out[7 * n + j] = R.tmax ? __ldg(R.tmax + i) : R.tmax_c;
  }
}

// Hits of sorted position j go back to ray perm[j].
__global__ void k_ray_scatter(int64_t n, const uint32_t *__restrict__ perm, const int32_t *__restrict__ prim,
                              const float *__restrict__ t, const float *__restrict__ u, const float *__restrict__ v,
                              const uint8_t *__restrict__ occ, Out O) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = perm[j];
    if (i < 0 || i >= n) continue;
    if (occ) {
      O.occ[i] = occ[j];
    } else {
      O.prim[i] = prim[j];
      O.t[i] = t[j];
      O.u[i] = u[j];
      O.v[i] = v[j];
    }
  }
}

static int ensure_trace_scratch(flg_ctx ctx) {
  if (ctx->d_ovf) return FLG_OK;
  if (ctx->capturing) return set_error(ctx, FLG_ERR_STATE, "first trace allocates; not allowed during capture");
  ctx->ovf_cap = 1 << 20;
  // Two sets (index 0: default stream, 1: staging second stream).
  FLG_CUDA(ctx, cudaMalloc((void **)&ctx->d_ovf, sizeof(int64_t) * ctx->ovf_cap * 2));
  FLG_CUDA(ctx, cudaMalloc((void **)&ctx->d_trace_ctr, sizeof(unsigned long long) * 8));
  FLG_CUDA(ctx, cudaMemsetAsync(ctx->d_trace_ctr, 0, sizeof(unsigned long long) * 8, ctx->stream));
  return FLG_OK;
}

static Scratch scratch_for(flg_ctx ctx, int set) {
  unsigned long long *c = ctx->d_trace_ctr + 2 * set;  // [0] rays taken, [1] entries of the list
  return Scratch{ctx->d_ovf + (set & 1) * ctx->ovf_cap, (uint32_t *)(c + 1), ctx->ovf_cap, c, ctx->d_err};
}

static int check_rays(flg_ctx ctx, const flg_rays *r, int64_t n) {
  if (!r) return set_error(ctx, FLG_ERR_ARG, "rays is NULL");
  if (n < 0) return set_error(ctx, FLG_ERR_ARG, "n < 0");
  if (n > 0 && (!r->ox || !r->oy || !r->oz || !r->dx || !r->dy || !r->dz))
    return set_error(ctx, FLG_ERR_ARG, "ray origin/direction pointer is NULL");
  return FLG_OK;
}

// ----------------------------------------------------------------------------
// Persistent while-while traversal with speculative leaf postponing (Aila &
// Laine, "Understanding the efficiency of ray traversal on GPUs", HPG 2009),
// on wide nodes.  Each lane walks inner nodes; a lane that reaches a leaf
// parks it (up to two) and keeps walking inner nodes until all but
// kLeafWait lanes of the warp hold a parked leaf (or have no inner node
// left); then the warp tests the parked leaves together.  Node and leaf code
// thus run with most lanes active, instead of the two branches diverging at
// every step.  Measured on config 3 (32 scenes): waiting for every lane kept
// only 37 % of the lanes at a node per node iteration; two parked leaves and
// kLeafWait = 4 give 21 % more rays/s.  Finished lanes are refilled from the
// global ray counter once `refill` of them are idle.
// ----------------------------------------------------------------------------
constexpr int kLeafWaitWW = 4;
// Shared-memory stack entries per lane (a power of two; 32 KB per 256-thread
// CTA).  16 measured 3.7 % faster than a local-memory stack, 8 gave 2 %.
constexpr int kStackTop = 16;

template <int W, bool ANY, int STACK>
__global__ void __launch_bounds__(256, 4)
    k_trace_ww(const NodeW<W> *__restrict__ nodes, const TriRec *__restrict__ tris, const int32_t *__restrict__ roots,
               const int64_t *__restrict__ ray_off, int n_scenes, RaySoA R, int64_t n, Out O, Scratch S, int refill) {
  constexpr int32_t kNone = kEmptyChild;  // "no node" / "no parked leaf"
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt = (1u << lane) - 1u;
  float3 o = make_float3(0.f, 0.f, 0.f), d = o, inv = o;
  float tmin = 0.f, tmax = 0.f, best = 0.f;
  int32_t prim = -1, cur = kNone, leaf = kNone, leaf2 = kNone;
  int sp = 0, scene = -1;
  bool have = false, active = false, overflow = false, exhausted = false;
  int64_t ray = -1;
  // Two-level stack: the top kStackTop entries of every lane live in shared
  // memory (a ring indexed by sp, laid out [slot][thread] so that a warp's
  // accesses fall in distinct banks); deeper entries spill to the per-thread
  // local array.  Most rays never go below the shared part, so pops no longer
  // wait on local-memory misses (57 % of the local-stack loads missed L1).
  uint64_t stk[STACK];
  constexpr int KS = kStackTop;
  __shared__ uint64_t s_stk[KS][256];
  const int tid = threadIdx.x;
  auto push = [&](uint64_t e) {
    if (sp >= KS) stk[sp - KS] = s_stk[sp & (KS - 1)][tid];
    s_stk[sp & (KS - 1)][tid] = e;
    ++sp;
  };

  auto pop = [&]() -> int32_t {
    const float lim = ANY ? tmax : best;
    while (sp > 0) {
      --sp;
      const uint64_t e = s_stk[sp & (KS - 1)][tid];
      if (sp >= KS) s_stk[sp & (KS - 1)][tid] = stk[sp - KS];
      if (__uint_as_float((uint32_t)(e >> 32)) > lim) continue;
      return (int32_t)(uint32_t)e;
    }
    return kNone;
  };

  while (true) {
    // Retire finished rays.
    if (active && cur == kNone && leaf == kNone && leaf2 == kNone) {
      if (overflow) record_overflow(S, ray);
      else write_result(O, ray, ANY, have, prim, best, tmax);
      active = false;
    }
    // Refill idle lanes.
    const unsigned idle = __ballot_sync(0xFFFFFFFFu, !active);
    const int nidle = __popc(idle);
    if (!exhausted && nidle >= refill) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(S.work, (unsigned long long)nidle);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (!active) {
        const int64_t my = (int64_t)base + __popc(idle & lt);
        if (my < n) {
          ray = my;
          load_ray(R, ray, o, d, inv, tmin, tmax);
          best = tmax;
          have = false;
          overflow = false;
          prim = -1;
          sp = 0;
          leaf = kNone;
          leaf2 = kNone;
          cur = scene_root_walk(roots, ray_off, n_scenes, ray, scene);
          if (cur == INT32_MIN) cur = kNone;
          active = true;
        }
      }
      if ((int64_t)base + nidle >= n) exhausted = true;
    }
    if (__ballot_sync(0xFFFFFFFFu, active) == 0u) {
      if (exhausted) break;
      continue;
    }

    // Inner nodes, parking the first two leaves found.
    while (true) {
      if (active && cur < 0) {
        if (leaf == kNone) {
          leaf = cur;
          cur = pop();
        } else if (leaf2 == kNone) {
          leaf2 = cur;
          cur = pop();
        }
      }
      const bool at_node = active && cur >= 0 && cur != kNone;
      if (!__any_sync(0xFFFFFFFFu, at_node)) break;
      if (at_node) {
        uint32_t key[W];
        int32_t ref[W];
        const int nh = visit_node<W>(nodes + cur, o, inv, ANY ? tmax : best, key, ref);
        if (nh == 0) {
          cur = pop();
        } else {
          sort_keys<W>(key);
          if (sp + nh - 1 > STACK + KS) {
            overflow = true;
            cur = kNone;
            leaf = kNone;
            leaf2 = kNone;
          } else {
#pragma unroll
            for (int k = W - 1; k >= 1; --k)
              if (k < nh) push(key_entry<W>(key[k], ref));
            cur = key_ref<W>(key[0], ref);
          }
        }
      }
      // Leave once at most kLeafWait active lanes are still looking for
      // their first leaf: waiting for the last few cost more idle node
      // iterations than the leaf tests they would have joined.
      const bool ready = !active || leaf != kNone || cur == kNone || (cur < 0 && leaf != kNone);
      if (__popc(__ballot_sync(0xFFFFFFFFu, !ready)) <= kLeafWaitWW) break;
    }

    // Test the (up to two) parked leaves together.
    for (int q = 0; q < 2; ++q) {
      const int32_t lf = q == 0 ? leaf : leaf2;
      if (active && lf != kNone && !(ANY && have)) {
        const int32_t enc = ~lf;
        const int64_t first = (int64_t)((uint32_t)enc >> 3);
        const int count = (enc & 7) + 1;
        for (int j = 0; j < count; ++j) {
          if (ANY) {
            if (test_tri_any(tris, first + j, o, d, tmin, tmax)) {
              have = true;
              cur = kNone;
              break;
            }
          } else {
            test_tri(tris, first + j, o, d, tmin, best, have, prim);
          }
        }
      }
    }
    leaf = kNone;
    leaf2 = kNone;
  }
}

constexpr int kRefill4 = 8;

// One trace over the 4-wide layout: the traversal, then the hit values (any
// hit: the overflow list).
//
// A warp runs through the paths of its rays in turn, so the fewer it has the
// sooner they end; but past a few warps per scheduler thinner warps only add
// instructions.  A batch too small to give sixteen full warps to every SM is
// spread over that many (before lanes helped: 4,096 rays on 20,001 triangles 72
// us, 92 in full warps, 96 in one-ray warps), and its blocks are made smaller
// until they cover the SMs.  Refills at kRefill4 idle lanes at most: with the
// quantised nodes 8 beat 16 and 24 (24.0 against 25.6 and 29.6 ms on 31.6 M
// scattered rays).
template <bool ANY>
static int launch4(flg_ctx ctx, cudaStream_t st, flg_bvh b, const RaySoA &R, int64_t n, const int32_t *n_dev,
                   const Out &O, const Scratch &S, const int64_t *ray_off, int n_scenes, const flg_trace_opts &op, bool &open) {
  const int lanes = (int)std::min<int64_t>(32, ceil_div(n, (int64_t)ctx->num_sms * 16));
  int threads = op.block_threads;
  while (threads > 32 && ceil_div(n, (int64_t)lanes * (threads / 32)) < ctx->num_sms) threads >>= 1;
  int64_t g = ceil_div(n, (int64_t)lanes * (threads / 32));
  if (g > ctx->num_sms) {  // no more than can be resident
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace4<ANY, false>, threads, 0);
    g = std::min<int64_t>(g, (int64_t)std::max(per_sm, 1) * ctx->num_sms);
  }
  const int refill = std::max(1, std::min(kRefill4, op.refill_lanes));
  const RayCount N{n, n_dev};
  const Exact4 X{b->d_nodes2, b->d_tris, Ranges{b->d_rfirst, b->d_rcount}, b->leaf_size, b->d_root, ray_off, n_scenes,
                 2 * b->n_tri};
  open = true;  // until the kernel that clears the counters is launched
  FLG_CUDA(ctx, launch_after(n_dev ? k_trace4<ANY, true> : k_trace4<ANY, false>, (unsigned)g, threads, st,
                             (const NodeQ *)b->d_wide, b->d_tris, b->d_wide_root, ray_off, n_scenes, R, N, O, S, refill,
                             lanes, b->n_tri > kLargeTree ? kLeafWaitAny : kLeafWait, 1.0f));
  FLG_LAUNCH_CHECK(ctx, "k_trace4");
  stage_mark(ctx, st, "trace");
  if (ANY) {
    FLG_CUDA(ctx, launch_after(k_trace_retry4, grid_for(n, 128, (int64_t)ctx->num_sms * 4), 128, st, R, N, O, X, S));
    FLG_LAUNCH_CHECK(ctx, "k_trace_retry4");
  } else {
    FLG_CUDA(ctx, n > kSettleWide
                      ? launch_after(k_settle4<256, 4>, grid_for(n, 256, (int64_t)ctx->num_sms * 16), 256, st, R, N, O, X, S)
                      : launch_after(k_settle4<128, 5>, grid_for(n, 128, (int64_t)ctx->num_sms * 32), 128, st, R, N, O, X, S));
    FLG_LAUNCH_CHECK(ctx, "k_settle4");
  }
  open = false;
  stage_mark(ctx, st, ANY ? "trace_retry" : "trace_finish");
  return FLG_OK;
}

template <int W, bool ANY>
static void launch_wide(flg_ctx ctx, cudaStream_t st, flg_bvh b, const RaySoA &R, int64_t n, const Out &O,
                        const Scratch &S, const int64_t *ray_off, int n_scenes, const flg_trace_opts &op) {
  const NodeW<W> *nodes = (const NodeW<W> *)b->d_wide;
  const int threads = op.block_threads;
  if (op.persistent == 2) {
    int per_sm = 0;
    if (op.stack_depth <= 32)
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace_ww<W, ANY, 32>, threads, 0);
    else
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace_ww<W, ANY, 64>, threads, 0);
    if (per_sm < 1) per_sm = 1;
    int64_t g = std::min<int64_t>((int64_t)per_sm * ctx->num_sms, ceil_div(n, threads));
    if (g < 1) g = 1;
    const int refill = std::max(1, std::min(32, op.refill_lanes));
    if (op.stack_depth <= 32)
      k_trace_ww<W, ANY, 32><<<(unsigned)g, threads, 0, st>>>(nodes, b->d_tris, b->d_wide_root, ray_off, n_scenes, R,
                                                              n, O, S, refill);
    else
      k_trace_ww<W, ANY, 64><<<(unsigned)g, threads, 0, st>>>(nodes, b->d_tris, b->d_wide_root, ray_off, n_scenes, R,
                                                              n, O, S, refill);
  } else if (op.persistent) {
    int per_sm = 0;
    if (op.stack_depth <= 32)
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace_persistent<W, ANY, 32>, threads, 0);
    else
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace_persistent<W, ANY, 64>, threads, 0);
    if (per_sm < 1) per_sm = 1;
    int64_t want = ceil_div(n, threads);
    int64_t g = std::min<int64_t>((int64_t)per_sm * ctx->num_sms, want);
    if (g < 1) g = 1;
    const int refill = std::max(1, std::min(32, op.refill_lanes));
    if (op.stack_depth <= 32)
      k_trace_persistent<W, ANY, 32><<<(unsigned)g, threads, 0, st>>>(nodes, b->d_tris, b->d_wide_root, ray_off,
                                                                      n_scenes, R, n, O, S, refill);
    else
      k_trace_persistent<W, ANY, 64><<<(unsigned)g, threads, 0, st>>>(nodes, b->d_tris, b->d_wide_root, ray_off,
                                                                      n_scenes, R, n, O, S, refill);
  } else {
    const unsigned g = (unsigned)ceil_div(n, threads);
    if (op.stack_depth <= 32)
      k_trace_wide<W, ANY, 32><<<g, threads, 0, st>>>(nodes, b->d_tris, b->d_wide_root, ray_off, n_scenes, R, n, O,
                                                      S);
    else
      k_trace_wide<W, ANY, 64><<<g, threads, 0, st>>>(nodes, b->d_tris, b->d_wide_root, ray_off, n_scenes, R, n, O,
                                                      S);
  }
}

// Enqueues one traversal of n rays on stream st with scratch set `set`.
// Closest hits: the hit-value pass after every traversal kernel of a call.
static int finish_enqueue(flg_ctx ctx, cudaStream_t st, const RaySoA &R, int64_t n, const Out &O, flg_bvh b,
                          bool any) {
  if (any || n <= 0) return FLG_OK;
  k_trace_finish<<<grid_for(n, 256, (int64_t)ctx->num_sms * 16), 256, 0, st>>>(R, n, O, b->d_tris);
  FLG_LAUNCH_CHECK(ctx, "k_trace_finish");
  stage_mark(ctx, st, "trace_finish");
  return FLG_OK;
}

bool trace_takes_device_count(flg_bvh b, const flg_trace_opts *opts) {
  return b->width == 4 && (!opts || (opts->tri_test == 0 && opts->ray_sort == 0));
}

int trace_enqueue(flg_ctx ctx, cudaStream_t st, int set, flg_bvh b, const flg_rays *rays, int64_t n,
                  const flg_trace_opts *opts, const int64_t *ray_off_dev, int n_scenes, flg_hits *hits,
                  uint8_t *occ, const int32_t *n_dev) {
  flg_trace_opts op{};
  if (opts) op = *opts;
  if (op.stack_depth == 0) op.stack_depth = 64;
  if (op.block_threads == 0) op.block_threads = 256;
  if (op.refill_lanes == 0) op.refill_lanes = 16;
  if (op.stack_depth != 32 && op.stack_depth != 64) return set_error(ctx, FLG_ERR_ARG, "stack_depth must be 32 or 64");
  if (op.block_threads != 64 && op.block_threads != 128 && op.block_threads != 256)
    return set_error(ctx, FLG_ERR_ARG, "block_threads must be 64, 128 or 256");
  if (op.ray_sort != 0 && op.ray_sort != 1) return set_error(ctx, FLG_ERR_ARG, "ray_sort must be 0 or 1");
  if (op.ray_sort && (ray_off_dev || n_scenes != 1))
    return set_error(ctx, FLG_ERR_UNSUPPORTED, "ray_sort applies to single-scene traces");
  if (op.ray_sort && n > ((int64_t)1 << 28)) return set_error(ctx, FLG_ERR_UNSUPPORTED, "ray_sort: at most 2^28 rays");
  if (op.tri_test != 0 && op.tri_test != 1) return set_error(ctx, FLG_ERR_ARG, "tri_test must be 0 or 1");
  int rc = ensure_trace_scratch(ctx);
  if (rc) return rc;
  if (n == 0) return FLG_OK;
  RaySoA R{rays->ox, rays->oy, rays->oz, rays->dx, rays->dy, rays->dz, rays->tmin, rays->tmax,
           rays->tmin_const, rays->tmax_const};
  if (n_dev && !trace_takes_device_count(b, &op))
    return set_error(ctx, FLG_ERR_STATE, "this trace needs its number of rays on the host");
  if (op.ray_sort) {
    // Scratch: keys and indices (2 x 2), digit counts and offsets, look-back,
    // tile counters, the sorted rays (8 arrays) and their hits (4 arrays).
    const int64_t tiles = sort_tiles(n, kSortItemsLarge);
    const size_t w = (size_t)n * 4;
    const size_t need = 4 * w + 2 * 4 * 256 * 4 + (size_t)4 * tiles * 256 * 4 + 64 + 8 * w + 4 * w + 16 * 256;
    if (ctx->rs_bytes < need) {
      if (ctx->capturing) return set_error(ctx, FLG_ERR_STATE, "ray-sort scratch grows; not allowed during capture");
      cudaFree(ctx->rs_buf);
      ctx->rs_buf = nullptr;
      ctx->rs_bytes = 0;
      FLG_CUDA(ctx, cudaMalloc(&ctx->rs_buf, need));
      ctx->rs_bytes = need;
    }
    char *bp = (char *)ctx->rs_buf;
    auto take = [&](size_t bytes) {
      char *p = bp;
      bp += (bytes + 255) & ~(size_t)255;
      return (void *)p;
    };
    uint32_t *keys[2] = {(uint32_t *)take(w), (uint32_t *)take(w)};
    uint32_t *vals[2] = {(uint32_t *)take(w), (uint32_t *)take(w)};
    uint32_t *hist = (uint32_t *)take(2 * 4 * 256 * 4);
    uint32_t *lookback = (uint32_t *)take((size_t)4 * tiles * 256 * 4);
    uint32_t *tile_ctr = (uint32_t *)take(64);
    float *sr = (float *)take(8 * w);
    float *sh = (float *)take(4 * w);
    if (bp > (char *)ctx->rs_buf + need) return set_error(ctx, FLG_ERR_STATE, "ray-sort buffer layout");
    FLG_CUDA(ctx, cudaMemsetAsync(hist, 0, sizeof(uint32_t) * 4 * 256, st));
    const unsigned g = grid_for(n, 256, (int64_t)ctx->num_sms * 8);
    k_ray_keys<<<g, 256, 0, st>>>(R, n, b->d_scene_box, keys[0], hist);
    FLG_LAUNCH_CHECK(ctx, "k_ray_keys");
    rc = sort_pairs_enqueue(ctx, st, n, 4, keys, vals, hist, lookback, tile_ctr);
    if (rc) return rc;
    const uint32_t *perm = vals[0];  // 4 passes: the result is back in buffer 0
    k_ray_gather<<<g, 256, 0, st>>>(R, n, perm, sr);
    FLG_LAUNCH_CHECK(ctx, "k_ray_gather");
    flg_rays sorted{sr, sr + n, sr + 2 * n, sr + 3 * n, sr + 4 * n, sr + 5 * n, sr + 6 * n, sr + 7 * n, 0.0f, 0.0f};
    flg_trace_opts op2 = op;
    op2.ray_sort = 0;
    uint8_t *socc = occ ? (uint8_t *)sh : nullptr;
    flg_hits shits{(int32_t *)sh, sh + n, sh + 2 * n, sh + 3 * n};
    rc = trace_enqueue(ctx, st, set, b, &sorted, n, &op2, nullptr, 1, occ ? nullptr : &shits, socc);
    if (rc) return rc;
    Out O{hits ? hits->prim : nullptr, hits ? hits->t : nullptr, hits ? hits->u : nullptr,
          hits ? hits->v : nullptr, occ};
    k_ray_scatter<<<g, 256, 0, st>>>(n, perm, (const int32_t *)sh, sh + n, sh + 2 * n, sh + 3 * n, socc, O);
    FLG_LAUNCH_CHECK(ctx, "k_ray_scatter");
    return FLG_OK;
  }
  Out O{hits ? hits->prim : nullptr, hits ? hits->t : nullptr, hits ? hits->u : nullptr,
        hits ? hits->v : nullptr, occ};
  const bool any = occ != nullptr;
  // Traces over the 4-wide layout end with their counters cleared, so they
  // keep a pair of their own (sets 2 and 3).
  const bool clears = b->width == 4 && op.tri_test == 0;
  Scratch S = scratch_for(ctx, clears ? set + 2 : set);
  stage_mark(ctx, st, "start");
  if (!clears || ctx->trace4_open[set])
    FLG_CUDA(ctx, cudaMemsetAsync(S.work, 0, 2 * sizeof(unsigned long long), st));  // both counters
  if (op.tri_test == 1) {
    // The live renderer's Moller-Trumbore test: one ray per thread over the
    // BVH2 layout (kept by every handle), overflow retried with a deep stack.
    const unsigned g = (unsigned)ceil_div(n, 256);
    if (any)
      k_trace_bvh2<true, true><<<g, 256, 0, st>>>(b->d_nodes2, b->d_tris, b->d_root, ray_off_dev, n_scenes, R, n, O,
                                                  S);
    else
      k_trace_bvh2<false, true><<<g, 256, 0, st>>>(b->d_nodes2, b->d_tris, b->d_root, ray_off_dev, n_scenes, R, n, O,
                                                   S);
    FLG_LAUNCH_CHECK(ctx, "trace kernel");
    stage_mark(ctx, st, "trace");
    const unsigned rg = (unsigned)ctx->num_sms;
    if (any)
      k_trace_retry<2, true, true><<<rg, 128, 0, st>>>(nullptr, b->d_nodes2, b->d_tris, b->d_root, ray_off_dev,
                                                       n_scenes, R, O, S);
    else
      k_trace_retry<2, false, true><<<rg, 128, 0, st>>>(nullptr, b->d_nodes2, b->d_tris, b->d_root, ray_off_dev,
                                                        n_scenes, R, O, S);
    FLG_LAUNCH_CHECK(ctx, "trace retry kernel");
    stage_mark(ctx, st, "trace_retry");
    return finish_enqueue(ctx, st, R, n, O, b, any);
  }
  if (b->width == 2) {
    const unsigned g = (unsigned)ceil_div(n, 256);
    if (any)
      k_trace_bvh2<true><<<g, 256, 0, st>>>(b->d_nodes2, b->d_tris, b->d_root, ray_off_dev, n_scenes, R, n, O, S);
    else
      k_trace_bvh2<false><<<g, 256, 0, st>>>(b->d_nodes2, b->d_tris, b->d_root, ray_off_dev, n_scenes, R, n, O, S);
  } else if (b->width == 4) {
    return any ? launch4<true>(ctx, st, b, R, n, n_dev, O, S, ray_off_dev, n_scenes, op, ctx->trace4_open[set])
               : launch4<false>(ctx, st, b, R, n, n_dev, O, S, ray_off_dev, n_scenes, op, ctx->trace4_open[set]);
  } else {
    if (any) launch_wide<8, true>(ctx, st, b, R, n, O, S, ray_off_dev, n_scenes, op);
    else launch_wide<8, false>(ctx, st, b, R, n, O, S, ray_off_dev, n_scenes, op);
  }
  FLG_LAUNCH_CHECK(ctx, "trace kernel");
  stage_mark(ctx, st, "trace");
  const unsigned rg = (unsigned)ctx->num_sms;
  const NodeW<8> *wide = (const NodeW<8> *)b->d_wide;
  const int32_t *roots = b->width == 2 ? b->d_root : b->d_wide_root;
  if (b->width == 2 && any)
    k_trace_retry<2, true><<<rg, 128, 0, st>>>(wide, b->d_nodes2, b->d_tris, roots, ray_off_dev, n_scenes, R, O, S);
  else if (b->width == 2)
    k_trace_retry<2, false><<<rg, 128, 0, st>>>(wide, b->d_nodes2, b->d_tris, roots, ray_off_dev, n_scenes, R, O, S);
  else if (any)
    k_trace_retry<8, true><<<rg, 128, 0, st>>>(wide, b->d_nodes2, b->d_tris, roots, ray_off_dev, n_scenes, R, O, S);
  else
    k_trace_retry<8, false><<<rg, 128, 0, st>>>(wide, b->d_nodes2, b->d_tris, roots, ray_off_dev, n_scenes, R, O, S);
  FLG_LAUNCH_CHECK(ctx, "trace retry kernel");
  stage_mark(ctx, st, "trace_retry");
  return finish_enqueue(ctx, st, R, n, O, b, any);
}

}  // namespace flg

using namespace flg;

FLG_API int flg_trace_closest(flg_ctx ctx, flg_bvh bvh, const flg_rays *rays, int64_t n,
                              const flg_trace_opts *opts, flg_hits *out) {
  if (!ctx || !bvh || !out) return ctx ? set_error(ctx, FLG_ERR_ARG, "NULL argument") : FLG_ERR_ARG;
  int rc = check_rays(ctx, rays, n);
  if (rc) return rc;
  if (n > 0 && (!out->prim || !out->t || !out->u || !out->v))
    return set_error(ctx, FLG_ERR_ARG, "hit output pointer is NULL");
  if (bvh->n_scenes != 1) return set_error(ctx, FLG_ERR_ARG, "batched handle: use flg_trace_closest_batched");
  return trace_enqueue(ctx, ctx->stream, 0, bvh, rays, n, opts, nullptr, 1, out, nullptr);
}

FLG_API int flg_trace_any(flg_ctx ctx, flg_bvh bvh, const flg_rays *rays, int64_t n, const flg_trace_opts *opts,
                          uint8_t *occluded) {
  if (!ctx || !bvh) return ctx ? set_error(ctx, FLG_ERR_ARG, "NULL argument") : FLG_ERR_ARG;
  int rc = check_rays(ctx, rays, n);
  if (rc) return rc;
  if (n > 0 && !occluded) return set_error(ctx, FLG_ERR_ARG, "occluded is NULL");
  if (bvh->n_scenes != 1) return set_error(ctx, FLG_ERR_ARG, "batched handle: use flg_trace_closest_batched");
  return trace_enqueue(ctx, ctx->stream, 0, bvh, rays, n, opts, nullptr, 1, nullptr, occluded);
}

FLG_API int flg_trace_closest_batched(flg_ctx ctx, flg_bvh bvh, const flg_rays *rays,
                                      const int64_t *ray_offsets_host, const flg_trace_opts *opts,
                                      flg_hits *out) {
  if (!ctx || !bvh || !out || !ray_offsets_host)
    return ctx ? set_error(ctx, FLG_ERR_ARG, "NULL argument") : FLG_ERR_ARG;
  const int ns = bvh->n_scenes;
  if (ray_offsets_host[0] != 0) return set_error(ctx, FLG_ERR_ARG, "ray_offsets[0] must be 0");
  for (int s = 0; s < ns; ++s)
    if (ray_offsets_host[s + 1] < ray_offsets_host[s])
      return set_error(ctx, FLG_ERR_ARG, "ray_offsets must be non-decreasing");
  const int64_t n = ray_offsets_host[ns];
  int rc = check_rays(ctx, rays, n);
  if (rc) return rc;
  if (n > 0 && (!out->prim || !out->t || !out->u || !out->v))
    return set_error(ctx, FLG_ERR_ARG, "hit output pointer is NULL");
  // Device copy of the offsets, refreshed only when they change (so a
  // captured graph replays without a host copy).
  std::vector<int64_t> &cached = ctx->ray_off_h;
  bool same = ctx->d_ray_off && ctx->ray_off_cap >= ns + 1 && cached.size() == (size_t)(ns + 1) &&
              std::equal(cached.begin(), cached.end(), ray_offsets_host);
  if (!same) {
    if (ctx->capturing) return set_error(ctx, FLG_ERR_STATE, "new ray offsets inside a capture; call once before");
    if (ctx->ray_off_cap < ns + 1) {
      cudaFree(ctx->d_ray_off);
      FLG_CUDA(ctx, cudaMalloc((void **)&ctx->d_ray_off, sizeof(int64_t) * (ns + 1)));
      ctx->ray_off_cap = ns + 1;
    }
    // Stream-ordered: earlier traces on this stream read the old offsets
    // first.  From pageable memory the source is staged before the call
    // returns, and the host does not wait for the stream's earlier work.
    FLG_CUDA(ctx, cudaMemcpyAsync(ctx->d_ray_off, ray_offsets_host, sizeof(int64_t) * (ns + 1),
                                  cudaMemcpyHostToDevice, ctx->stream));
    cached.assign(ray_offsets_host, ray_offsets_host + ns + 1);
  }
  return trace_enqueue(ctx, ctx->stream, 0, bvh, rays, n, opts, ctx->d_ray_off, ns, out, nullptr);
}

// Host-buffer entry point: chunks of rays are staged through two device
// buffers.  Every copy runs on the copy stream, in the order H0 H1 D0 H2 D1
// H3 ... (Hi: chunk i's rays in, Di: its hits out, once its trace on the
// context's stream is done), so copies overlap the traces but never each
// other: a host-to-device and a device-to-host copy that run at once each
// drop to about a third of their bandwidth alone.
FLG_API int flg_trace_closest_host(flg_ctx ctx, flg_bvh bvh, const flg_rays *rh, int64_t n,
                                   const flg_trace_opts *opts, flg_hits *oh) {
  if (!ctx || !bvh || !oh) return ctx ? set_error(ctx, FLG_ERR_ARG, "NULL argument") : FLG_ERR_ARG;
  int rc = check_rays(ctx, rh, n);
  if (rc) return rc;
  if (ctx->capturing) return set_error(ctx, FLG_ERR_STATE, "host staging cannot be captured");
  if (bvh->n_scenes != 1) return set_error(ctx, FLG_ERR_ARG, "batched handle");
  if (n > 0 && (!oh->prim || !oh->t || !oh->u || !oh->v))
    return set_error(ctx, FLG_ERR_ARG, "hit output pointer is NULL");
  if ((rc = ensure_trace_scratch(ctx))) return rc;
  const int64_t chunk = std::min<int64_t>(n, (int64_t)1 << 22);
  if (chunk == 0) return FLG_OK;
  // Per buffer: 8 ray arrays + 4 hit arrays, 4 bytes each.
  const size_t per_buf = (size_t)chunk * 12 * sizeof(float);
  if (ctx->stage_bytes < 2 * per_buf) {
    cudaFree(ctx->stage);
    ctx->stage = nullptr;
    ctx->stage_bytes = 0;
    FLG_CUDA(ctx, cudaMalloc(&ctx->stage, 2 * per_buf));
    ctx->stage_bytes = 2 * per_buf;
  }
  cudaStream_t cs = ctx->stream, cp = ctx->copy_stream;
  cudaEvent_t *in_done = ctx->ev, *traced = ctx->ev + 2;  // per buffer
  // The copy stream must not start before earlier work on the context's stream.
  FLG_CUDA(ctx, cudaEventRecord(traced[0], cs));
  FLG_CUDA(ctx, cudaStreamWaitEvent(cp, traced[0], 0));
  const int64_t n_chunks = (n + chunk - 1) / chunk;
  auto buffers = [&](int k, float *(&arr)[12]) {
    float *base = (float *)((char *)ctx->stage + k * per_buf);
    for (int a = 0; a < 12; ++a) arr[a] = base + (size_t)a * chunk;
  };
  auto copy_in = [&](int64_t ci) -> int {
    const int k = (int)(ci & 1);
    const int64_t c0 = ci * chunk, m = std::min(chunk, n - c0);
    float *arr[12];
    buffers(k, arr);
    const float *src[8] = {rh->ox, rh->oy, rh->oz, rh->dx, rh->dy, rh->dz, rh->tmin, rh->tmax};
    for (int a = 0; a < 8; ++a)
      if (src[a]) FLG_CUDA(ctx, cudaMemcpyAsync(arr[a], src[a] + c0, sizeof(float) * m, cudaMemcpyHostToDevice, cp));
    FLG_CUDA(ctx, cudaEventRecord(in_done[k], cp));
    return FLG_OK;
  };
  if ((rc = copy_in(0))) return rc;
  if (n_chunks > 1 && (rc = copy_in(1))) return rc;
  for (int64_t ci = 0; ci < n_chunks; ++ci) {
    const int k = (int)(ci & 1);
    const int64_t c0 = ci * chunk, m = std::min(chunk, n - c0);
    float *arr[12];
    buffers(k, arr);
    flg_rays dr{arr[0], arr[1], arr[2], arr[3], arr[4], arr[5], rh->tmin ? arr[6] : nullptr,
                rh->tmax ? arr[7] : nullptr, rh->tmin_const, rh->tmax_const};
    flg_hits dh{(int32_t *)arr[8], arr[9], arr[10], arr[11]};
    flg_trace_opts op{};
    if (opts) op = *opts;
    op.persistent = 0;
    FLG_CUDA(ctx, cudaStreamWaitEvent(cs, in_done[k], 0));
    rc = trace_enqueue(ctx, cs, k, bvh, &dr, m, &op, nullptr, 1, &dh, nullptr);
    if (rc) return rc;
    FLG_CUDA(ctx, cudaEventRecord(traced[k], cs));
    FLG_CUDA(ctx, cudaStreamWaitEvent(cp, traced[k], 0));
    FLG_CUDA(ctx, cudaMemcpyAsync(oh->prim + c0, dh.prim, sizeof(int32_t) * m, cudaMemcpyDeviceToHost, cp));
    FLG_CUDA(ctx, cudaMemcpyAsync(oh->t + c0, dh.t, sizeof(float) * m, cudaMemcpyDeviceToHost, cp));
    FLG_CUDA(ctx, cudaMemcpyAsync(oh->u + c0, dh.u, sizeof(float) * m, cudaMemcpyDeviceToHost, cp));
    FLG_CUDA(ctx, cudaMemcpyAsync(oh->v + c0, dh.v, sizeof(float) * m, cudaMemcpyDeviceToHost, cp));
    // this buffer's next rays: after its hits are out (same stream)
    if (ci + 2 < n_chunks && (rc = copy_in(ci + 2))) return rc;
  }
  FLG_CUDA(ctx, cudaStreamSynchronize(ctx->copy_stream));
  FLG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return flg_ctx_sync(ctx);
}

namespace flg {

// Staged search of the traversal configuration on a given workload (node
// width and leaf size, then the kernel, then the block size; single-scene
// handles also try the ray-sort key).  Options that a layout's kernel does not
// read are not varied: the 4-wide one has one kernel, which refills at kRefill4
// idle lanes at most.  Every trial is one untimed launch and `reps` launches timed
// one by one with events; the trial's time is their median.  Leaves the handle at
// the fastest layout.
struct Tuner {
  flg_ctx ctx;
  flg_bvh bvh;
  const flg_rays *rays;
  int64_t n;
  const int64_t *ray_off;
  int n_scenes, reps;
  flg_hits h;
  std::vector<cudaEvent_t> ev;
  std::string rec = "{\"trials\": [";
  bool first = true;
  float best_ms = 1e30f;
  flg_trace_opts best{};
  int best_w = 4, best_leaf = 1;

  int trial(int w, int leaf, const flg_trace_opts &op, const char *stage) {
    int rc = trace_enqueue(ctx, ctx->stream, 0, bvh, rays, n, &op, ray_off, n_scenes, &h, nullptr);
    if (rc) return rc;
    for (int r = 0; r < reps; ++r) {
      FLG_CUDA(ctx, cudaEventRecord(ev[2 * r], ctx->stream));
      rc = trace_enqueue(ctx, ctx->stream, 0, bvh, rays, n, &op, ray_off, n_scenes, &h, nullptr);
      if (rc) return rc;
      FLG_CUDA(ctx, cudaEventRecord(ev[2 * r + 1], ctx->stream));
    }
    FLG_CUDA(ctx, cudaEventSynchronize(ev[2 * reps - 1]));
    std::vector<float> ms(reps);
    for (int r = 0; r < reps; ++r) FLG_CUDA(ctx, cudaEventElapsedTime(&ms[r], ev[2 * r], ev[2 * r + 1]));
    std::sort(ms.begin(), ms.end());
    const float med = reps % 2 ? ms[reps / 2] : 0.5f * (ms[reps / 2 - 1] + ms[reps / 2]);
    char line[384];
    snprintf(line, sizeof(line),
             "%s{\"stage\": \"%s\", \"node_width\": %d, \"leaf_size\": %d, \"stack_depth\": %d, \"persistent\": %d, "
             "\"refill_lanes\": %d, \"block_threads\": %d, \"ray_sort\": %d, \"ms\": %.5f, \"ms_min\": %.5f, "
             "\"ms_max\": %.5f, \"mrays_s\": %.2f}",
             first ? "" : ", ", stage, w, leaf, op.stack_depth, op.persistent, op.refill_lanes, op.block_threads,
             op.ray_sort, med, ms.front(), ms.back(), n / (med * 1e3));
    first = false;
    rec += line;
    if (med < best_ms) {
      best_ms = med;
      best = op;
      best_w = w;
      best_leaf = leaf;
    }
    return FLG_OK;
  }

  static flg_trace_opts kernel_opts(int w, int pers, int refill, int stack, int threads) {
    flg_trace_opts op{};
    op.stack_depth = stack;
    op.persistent = w == 2 ? 0 : pers;
    op.refill_lanes = refill;
    op.block_threads = threads;
    return op;
  }

  int run() {
    int rc;
    // 1. layout, with the default kernel of each width
    for (int w : {2, 4, 8}) {
      for (int leaf : {1, 2, 3, 4}) {
        if (w == 2 && leaf > 1) continue;
        rc = flg_bvh_set_width(ctx, bvh, w, leaf);
        if (rc) return rc;
        rc = trial(w, leaf, kernel_opts(w, 2, 8, 64, 256), "layout");
        if (rc) return rc;
      }
    }
    const int w = best_w, leaf = best_leaf;
    rc = flg_bvh_set_width(ctx, bvh, w, leaf);
    if (rc) return rc;
    // 2. kernel on that layout
    if (w == 4) {
      for (int refill : {2, 4, 6}) {
        rc = trial(w, leaf, kernel_opts(w, 2, refill, 64, 256), "kernel");
        if (rc) return rc;
      }
    } else if (w > 2) {
      for (int pers : {0, 1, 2})
        for (int refill : {4, 8, 16})
          for (int stack : {32, 64}) {
            if (pers == 0 && refill != 8) continue;
            if (pers == 2 && refill == 8 && stack == 64) continue;  // tried in stage 1
            rc = trial(w, leaf, kernel_opts(w, pers, refill, stack, 256), "kernel");
            if (rc) return rc;
          }
    } else {
      rc = trial(w, leaf, kernel_opts(w, 0, 8, 32, 256), "kernel");
      if (rc) return rc;
    }
    // 3. block size
    const flg_trace_opts kernel = best;
    for (int threads : {64, 128}) {
      if (threads == 64 && w != 4) continue;
      flg_trace_opts op = kernel;
      op.block_threads = threads;
      rc = trial(w, leaf, op, "block");
      if (rc) return rc;
    }
    // 4. ray-sort key (single-scene traces): pays when neighbouring rays are
    // scattered, costs a sort and two gathers when they are not
    if (!ray_off && n_scenes == 1 && n <= ((int64_t)1 << 28)) {
      flg_trace_opts op = best;
      op.ray_sort = 1;
      rc = trial(w, leaf, op, "ray_sort");
      if (rc) return rc;
    }
    char tail[384];
    snprintf(tail, sizeof(tail),
             "], \"reps\": %d, \"rays\": %lld, \"scenes\": %d, \"best\": {\"node_width\": %d, \"leaf_size\": %d, "
             "\"stack_depth\": %d, \"persistent\": %d, \"refill_lanes\": %d, \"block_threads\": %d, \"ray_sort\": %d, "
             "\"ms\": %.5f, \"mrays_s\": %.2f}}",
             reps, (long long)n, n_scenes, best_w, best_leaf, best.stack_depth, best.persistent, best.refill_lanes,
             best.block_threads, best.ray_sort, best_ms, n / (best_ms * 1e3));
    rec += tail;
    return FLG_OK;
  }
};

static int autotune(flg_ctx ctx, flg_bvh bvh, const flg_rays *rays, int64_t n, const int64_t *ray_off,
                    int n_scenes, int reps, flg_trace_opts *best, int32_t *best_width, int32_t *best_leaf,
                    char *json, size_t json_len) {
  if (ctx->capturing) return set_error(ctx, FLG_ERR_STATE, "autotuning cannot be captured");
  if (reps < 1 || reps > 64) return set_error(ctx, FLG_ERR_ARG, "reps must be in [1, 64]");
  if (n <= 0) return set_error(ctx, FLG_ERR_ARG, "autotuning needs rays");
  void *buf = nullptr;
  FLG_CUDA(ctx, cudaMalloc(&buf, sizeof(float) * 4 * (size_t)n));
  Tuner T{ctx, bvh, rays, n, ray_off, n_scenes, reps,
          flg_hits{(int32_t *)buf, (float *)buf + n, (float *)buf + 2 * n, (float *)buf + 3 * n}};
  T.ev.assign(2 * reps, nullptr);
  int rc = FLG_OK;
  for (auto &e : T.ev)
    if (cudaEventCreate(&e) != cudaSuccess) {
      cudaGetLastError();
      rc = set_error(ctx, FLG_ERR_CUDA, "cudaEventCreate failed");
      break;
    }
  if (!rc) rc = T.run();
  for (auto &e : T.ev)
    if (e) cudaEventDestroy(e);
  cudaFree(buf);
  if (rc) return rc;
  *best = T.best;
  if (best_width) *best_width = T.best_w;
  if (best_leaf) *best_leaf = T.best_leaf;
  if (json && json_len) {
    if (T.rec.size() + 1 > json_len)
      return set_error(ctx, FLG_ERR_ARG, "json buffer too small (%zu bytes needed)", T.rec.size() + 1);
    std::memcpy(json, T.rec.c_str(), T.rec.size() + 1);
  }
  return flg_ctx_sync(ctx);
}

}  // namespace flg

FLG_API int flg_autotune_trace(flg_ctx ctx, flg_bvh bvh, const flg_rays *rays, int64_t n, flg_trace_opts *best,
                               int32_t *best_width, char *json, size_t json_len) {
  if (!ctx || !bvh || !best) return ctx ? set_error(ctx, FLG_ERR_ARG, "NULL argument") : FLG_ERR_ARG;
  int rc = check_rays(ctx, rays, n);
  if (rc) return rc;
  if (bvh->n_scenes != 1) return set_error(ctx, FLG_ERR_ARG, "batched handle: use flg_autotune_trace_batched");
  return autotune(ctx, bvh, rays, n, nullptr, 1, 5, best, best_width, nullptr, json, json_len);
}

FLG_API int flg_autotune_trace_batched(flg_ctx ctx, flg_bvh bvh, const flg_rays *rays,
                                       const int64_t *ray_offsets_host, int32_t reps, flg_trace_opts *best,
                                       int32_t *best_width, int32_t *best_leaf, char *json, size_t json_len) {
  if (!ctx || !bvh || !best || !ray_offsets_host)
    return ctx ? set_error(ctx, FLG_ERR_ARG, "NULL argument") : FLG_ERR_ARG;
  const int ns = bvh->n_scenes;
  if (ray_offsets_host[0] != 0) return set_error(ctx, FLG_ERR_ARG, "ray_offsets[0] must be 0");
  for (int s = 0; s < ns; ++s)
    if (ray_offsets_host[s + 1] < ray_offsets_host[s])
      return set_error(ctx, FLG_ERR_ARG, "ray_offsets must be non-decreasing");
  const int64_t n = ray_offsets_host[ns];
  int rc = check_rays(ctx, rays, n);
  if (rc) return rc;
  if (ctx->capturing) return set_error(ctx, FLG_ERR_STATE, "autotuning cannot be captured");
  if (ctx->ray_off_cap < ns + 1) {
    cudaFree(ctx->d_ray_off);
    ctx->d_ray_off = nullptr;
    ctx->ray_off_cap = 0;
    FLG_CUDA(ctx, cudaMalloc((void **)&ctx->d_ray_off, sizeof(int64_t) * (ns + 1)));
    ctx->ray_off_cap = ns + 1;
  }
  FLG_CUDA(ctx, cudaMemcpy(ctx->d_ray_off, ray_offsets_host, sizeof(int64_t) * (ns + 1), cudaMemcpyHostToDevice));
  ctx->ray_off_h.assign(ray_offsets_host, ray_offsets_host + ns + 1);
  return autotune(ctx, bvh, rays, n, ctx->d_ray_off, ns, reps, best, best_width, best_leaf, json, json_len);
}

// ---------------------------------------------------------------------------
// Closest hit that allocates nothing.
//
// flg_trace_closest takes its traversal scratch (the list of rays whose short
// stack overflowed, plus two counters) from the context and allocates it with
// cudaMalloc on the context's first trace.  Some callers cannot allocate at
// that moment: a renderer recording its frame loop into a CUDA graph (an
// allocation inside a stream capture is refused), an application whose
// device memory is handed out once, up front, by its own arena (as the
// reference's Resource arena owns every allocation, src/resource.hpp:45-120),
// or a latency-critical loop in which a cudaMalloc would synchronise the
// device.  This entry point runs the same traversal kernels with the scratch
// in a fixed file-scope device array instead.
//
// The array holds the overflow list for at most kNoAllocMaxRays rays (8 MB
// plus 256 bytes of counters) and stays resident on every GPU that loads the
// library until the process exits.  All calls share it: calls that overlap
// on the GPU (concurrent streams or contexts) race on it and must not be
// issued.  Its counters are cleared at the start of every call.
// ---------------------------------------------------------------------------
constexpr int64_t kNoAllocMaxRays = int64_t(1) << 20;
// words: [0] overflow count (low 32 bits), [1] work counter, [2, 32) unused,
// [32, 32 + kNoAllocMaxRays) overflow list of ray indices
static __device__ __align__(256) unsigned long long g_noalloc_scratch[32 + kNoAllocMaxRays];

static std::mutex g_noalloc_mu;
static unsigned long long *g_noalloc_ptr[64] = {};

// Device address of the scratch array on ctx's device.  In host code the
// array's name is only a host-side stand-in, so the address is looked up
// once per device with that device current, and cached.  The lookup may load
// the library's device code, which a stream capture does not allow: a first
// call on a device inside a capture is refused, as allocating calls are.
static int noalloc_scratch(flg_ctx ctx, unsigned long long **out) {
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (ctx->device < 0 || ctx->device >= 64) return set_error(ctx, FLG_ERR_UNSUPPORTED, "device index >= 64");
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (!g_noalloc_ptr[ctx->device] &&
      (ctx->capturing || (cudaStreamIsCapturing(ctx->stream, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone)))
    return set_error(ctx, FLG_ERR_STATE,
                     "the first flg_trace_closest_noalloc on a device looks up its scratch; not allowed during capture");
  if (!g_noalloc_ptr[ctx->device]) {
    int prev = 0;
    FLG_CUDA(ctx, cudaGetDevice(&prev));
    FLG_CUDA(ctx, cudaSetDevice(ctx->device));
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    cudaError_t e2 = cudaSetDevice(prev);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaGetSymbolAddress(g_noalloc_scratch)");
    if (e2 != cudaSuccess) return cuda_fail(ctx, e2, "cudaSetDevice");
    g_noalloc_ptr[ctx->device] = (unsigned long long *)p;
  }
  *out = g_noalloc_ptr[ctx->device];
  return FLG_OK;
}

FLG_API int flg_trace_closest_noalloc(flg_ctx ctx, flg_bvh bvh, const flg_rays *rays, int64_t n, flg_hits *out) {
  if (!ctx || !bvh || !out) return ctx ? set_error(ctx, FLG_ERR_ARG, "NULL argument") : FLG_ERR_ARG;
  int rc = check_rays(ctx, rays, n);
  if (rc) return rc;
  if (n > kNoAllocMaxRays)
    return set_error(ctx, FLG_ERR_ARG, "flg_trace_closest_noalloc: n = %lld exceeds its maximum of %lld rays",
                     (long long)n, (long long)kNoAllocMaxRays);
  if (n > 0 && (!out->prim || !out->t || !out->u || !out->v))
    return set_error(ctx, FLG_ERR_ARG, "hit output pointer is NULL");
  if (bvh->n_scenes != 1) return set_error(ctx, FLG_ERR_ARG, "batched handle: use flg_trace_closest_batched");
  unsigned long long *s = nullptr;
  if ((rc = noalloc_scratch(ctx, &s))) return rc;
  if (n == 0) return FLG_OK;
  cudaStream_t st = ctx->stream;
  // Clear the shared counters left by the previous call.
  FLG_CUDA(ctx, cudaMemsetAsync(s, 0, 2 * sizeof(unsigned long long), st));
  Scratch S{(int64_t *)(s + 32), (uint32_t *)s, kNoAllocMaxRays, s + 1, ctx->d_err};
  RaySoA R{rays->ox, rays->oy, rays->oz, rays->dx, rays->dy, rays->dz, rays->tmin, rays->tmax,
           rays->tmin_const, rays->tmax_const};
  Out O{out->prim, out->t, out->u, out->v, nullptr};
  const unsigned g = (unsigned)ceil_div(n, 256);
  const unsigned rg = (unsigned)ctx->num_sms;
  if (bvh->width == 2) {
    k_trace_bvh2<false><<<g, 256, 0, st>>>(bvh->d_nodes2, bvh->d_tris, bvh->d_root, nullptr, 1, R, n, O, S);
    FLG_LAUNCH_CHECK(ctx, "k_trace_bvh2");
    k_trace_retry<2, false><<<rg, 128, 0, st>>>(nullptr, bvh->d_nodes2, bvh->d_tris, bvh->d_root, nullptr, 1, R, O, S);
  } else if (bvh->width == 4) {
    flg_trace_opts op{};
    op.block_threads = 256;
    op.refill_lanes = 16;
    bool open;  // the counters are cleared above, on every call
    return launch4<false>(ctx, st, bvh, R, n, nullptr, O, S, nullptr, 1, op, open);
  } else {
    k_trace_wide<8, false, 64><<<g, 256, 0, st>>>((const NodeW<8> *)bvh->d_wide, bvh->d_tris, bvh->d_wide_root,
                                                  nullptr, 1, R, n, O, S);
    FLG_LAUNCH_CHECK(ctx, "k_trace_wide");
    k_trace_retry<8, false><<<rg, 128, 0, st>>>((const NodeW<8> *)bvh->d_wide, bvh->d_nodes2, bvh->d_tris,
                                                bvh->d_wide_root, nullptr, 1, R, O, S);
  }
  FLG_LAUNCH_CHECK(ctx, "k_trace_retry");
  return finish_enqueue(ctx, st, R, n, O, bvh, false);
}
