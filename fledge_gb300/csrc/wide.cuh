// wide.cuh — the wide-node layouts' device code shared by the collapse
// (collapse.cu) and the traversal (trace.cu): which BVH2 nodes become the
// children of a wide node, and the quantised 4-wide record.
#pragma once

#include "common.cuh"
#include "internal.h"

namespace flg {

struct Cand {
  int32_t ref;     // BVH2 ref (>=0 internal, <0 ~leaf position)
  int32_t first;   // first sorted triangle of the subtree
  int32_t count;   // triangles in the subtree
  float lo[3], hi[3];
};

__device__ __forceinline__ float half_area(const Cand &c) {
  float dx = c.hi[0] - c.lo[0], dy = c.hi[1] - c.lo[1], dz = c.hi[2] - c.lo[2];
  return dx * dy + dy * dz + dz * dx;
}

// Leaf ranges of internal nodes.  LBVH records carry their own range
// (d.z, d.w: first and last sorted triangle) and split (the left child ref
// names it, node slots being numbered by sorted position), so both children's
// ranges come from the parent's record; PLOC trees keep explicit depth-first
// ranges (rfirst / rcount) per node.
struct Ranges {
  const int32_t *rfirst, *rcount;
};

__device__ __forceinline__ void child_cands(const Node2 &nd, const Ranges &R, Cand &c0, Cand &c1) {
  int32_t r[2] = {nd.d.x, nd.d.y};
  Cand *o[2] = {&c0, &c1};
  const float lo[2][3] = {{nd.a.x, nd.a.z, nd.c.x}, {nd.b.x, nd.b.z, nd.c.z}};
  const float hi[2][3] = {{nd.a.y, nd.a.w, nd.c.y}, {nd.b.y, nd.b.w, nd.c.w}};
  const int32_t split = r[0] >= 0 ? r[0] : ~r[0];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    Cand &c = *o[k];
    c.ref = r[k];
    for (int a = 0; a < 3; ++a) {
      c.lo[a] = lo[k][a];
      c.hi[a] = hi[k][a];
    }
    if (!R.rfirst) {
      c.first = k == 0 ? nd.d.z : split + 1;
      c.count = k == 0 ? split - nd.d.z + 1 : nd.d.w - split;
    } else if (r[k] < 0) {
      c.first = ~r[k];
      c.count = 1;
    } else {
      c.first = R.rfirst[r[k]];
      c.count = R.rcount[r[k]];
    }
  }
}

// Children of the wide node that stands for BVH2 node `node`: starting from
// its two children, the child of largest surface area (the first of equals)
// is opened until there are W or none holds more than leaf_size triangles.
// The records of both children that may be opened are fetched together: the
// first opening takes one of them and the second usually the other, so most
// wide nodes wait on two dependent loads instead of three.
template <int W>
__device__ __forceinline__ void open_wide(const Node2 *__restrict__ nodes2, const Ranges &R, int leaf_size,
                                          int32_t node, Cand (&c)[W], int &nc) {
  nc = 2;
  child_cands(nodes2[node], R, c[0], c[1]);
  Node2 pf0, pf1;
  const int32_t pf0_ref = c[0].ref >= 0 && c[0].count > leaf_size ? c[0].ref : -1;
  const int32_t pf1_ref = c[1].ref >= 0 && c[1].count > leaf_size ? c[1].ref : -1;
  if (pf0_ref >= 0) pf0 = nodes2[pf0_ref];
  if (pf1_ref >= 0) pf1 = nodes2[pf1_ref];
  while (nc < W) {
    int best = -1;
    float ba = -1.0f;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      if (k < nc && c[k].ref >= 0 && c[k].count > leaf_size) {
        float a = half_area(c[k]);
        if (a > ba) {
          ba = a;
          best = k;
        }
      }
    }
    if (best < 0) break;
    Cand a, b;
    int32_t r = 0;
#pragma unroll
    for (int k = 0; k < W; ++k)
      if (k == best) r = c[k].ref;
    if (r == pf0_ref) child_cands(pf0, R, a, b);
    else if (r == pf1_ref) child_cands(pf1, R, a, b);
    else child_cands(nodes2[r], R, a, b);
#pragma unroll
    for (int k = 0; k < W; ++k) {
      if (k == best) c[k] = a;
      if (k == nc) c[k] = b;
    }
    ++nc;
  }
}

// A child of a 4-wide node by what chooses it: as Cand, with its area and the
// place of its box (BVH2 node x 2 + side) instead of the box, which keeps the
// choice of four children in half the registers.
struct WalkCand {
  int32_t ref, first, count, box;
  float area;
};

__device__ __forceinline__ void walk_cands(const Node2 *__restrict__ nodes2, const Ranges &R, int32_t node,
                                           WalkCand &a, WalkCand &b) {
  const float4 *np = (const float4 *)(nodes2 + node);
  Node2 nd;
  nd.a = __ldg(np);
  nd.b = __ldg(np + 1);
  nd.c = __ldg(np + 2);
  nd.d = __ldg((const int4 *)(np + 3));
  Cand c, e;
  child_cands(nd, R, c, e);
  a = WalkCand{c.ref, c.first, c.count, 2 * node, half_area(c)};
  b = WalkCand{e.ref, e.first, e.count, 2 * node + 1, half_area(e)};
}

// Box of a WalkCand.
__device__ __forceinline__ void walk_box(const Node2 *__restrict__ nodes2, int32_t box, float *lo, float *hi) {
  const float4 *np = (const float4 *)(nodes2 + (box >> 1));
  const float4 ab = __ldg(np + (box & 1));
  const float2 z = __ldg((const float2 *)(np + 2) + (box & 1));
  lo[0] = ab.x;
  hi[0] = ab.y;
  lo[1] = ab.z;
  hi[1] = ab.w;
  lo[2] = z.x;
  hi[2] = z.y;
}

// The children of a 4-wide node, as open_wide<4> picks them.  The records of
// both children of `node` that may be opened are read at once: the first
// opening takes one of them and the second usually the other.
__device__ __forceinline__ void walk_open(const Node2 *__restrict__ nodes2, const Ranges &R, int leaf_size,
                                          int32_t node, WalkCand (&c)[4], int &nc) {
  nc = 2;
  walk_cands(nodes2, R, node, c[0], c[1]);
  const int32_t r0 = c[0].ref >= 0 && c[0].count > leaf_size ? c[0].ref : -1;
  const int32_t r1 = c[1].ref >= 0 && c[1].count > leaf_size ? c[1].ref : -1;
  WalkCand g0[2], g1[2];
  if (r0 >= 0) walk_cands(nodes2, R, r0, g0[0], g0[1]);
  if (r1 >= 0) walk_cands(nodes2, R, r1, g1[0], g1[1]);
  while (nc < 4) {
    int best = -1;
    float ba = -1.0f;
    int32_t r = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k < nc && c[k].ref >= 0 && c[k].count > leaf_size && c[k].area > ba) {
        ba = c[k].area;
        best = k;
        r = c[k].ref;
      }
    }
    if (best < 0) break;
    WalkCand a, b;
    if (r == r0) {
      a = g0[0];
      b = g0[1];
    } else if (r == r1) {
      a = g1[0];
      b = g1[1];
    } else {
      walk_cands(nodes2, R, r, a, b);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k == best) c[k] = a;
      if (k == nc) c[k] = b;
    }
    ++nc;
  }
}

// Quantises the children's boxes of a 4-wide node (NodeQ): per axis an origin
// and a power-of-two step, as in Ylitie, Karras and Laine's nodes; every child's lower plane rounds down and its
// upper plane up, both with at least 1/64 step to spare.  The slack covers
// the rounding of the traversal's plane distances, so that a box test on the
// record never rejects a box that the exact test accepts (visit_q).  The
// record holds the exponent of 2^16 steps, as visit_q takes it.  An axis
// whose planes are not finite, or more than 2^118 apart, gets an infinite
// step and zero bytes, which constrain nothing.
__device__ __forceinline__ void quantise(const Cand (&c)[4], int nc, NodeQ &out) {
  out.step = 0u;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float lo = c[0].lo[a], hi = c[0].hi[a];
#pragma unroll
    for (int k = 1; k < 4; ++k) {
      if (k < nc) {
        lo = fminf(lo, c[k].lo[a]);
        hi = fmaxf(hi, c[k].hi[a]);
      }
    }
    // 253 steps cover the extent and two ulps of the largest coordinate (the
    // origin is rounded down), never finer than 2^-40.
    const float m = fmaxf(fabsf(lo), fabsf(hi));
    const float ext = __fadd_ru(__fsub_ru(hi, lo), m * 2.384185791015625e-07f);
    const uint32_t b = __float_as_uint(__fmul_ru(ext, 0.0039525693f));  // just above 1 / 253
    uint32_t e = (b >> 23) + ((b & 0x7FFFFFu) ? 1u : 0u);
    e = max(e, 87u);
    uint32_t qlo = 0u, qhi = 0u;
    float org = 0.0f;
    // ext < inf and not NaN (lo <= hi, so ext >= 0); 2^16 steps stay finite
    if (ext < __int_as_float(0x7f800000) && e <= 238u) {
      const float s = __uint_as_float(e << 23), rs = __uint_as_float((254u - e) << 23);
      org = __fsub_rd(lo, s * 0.03125f);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        // an unused slot gets an inverted box (and an empty leaf range)
        const float l = k < nc ? floorf(__fsub_rd(c[k].lo[a], org) * rs - 0.015625f) : 255.0f;
        const float h = k < nc ? ceilf(__fsub_ru(c[k].hi[a], org) * rs + 0.015625f) : 0.0f;
        qlo |= (uint32_t)fminf(fmaxf(l, 0.0f), 255.0f) << (8 * k);
        qhi |= (uint32_t)fminf(fmaxf(h, 0.0f), 255.0f) << (8 * k);
      }
      e += 16u;
    } else {
      e = 255u;
    }
    out.step |= e << (a == 0 ? 7 : a == 1 ? 23 : 15);
    out.org[a] = org;
    out.qlo[a] = qlo;
    out.qhi[a] = qhi;
  }
}

}  // namespace flg
