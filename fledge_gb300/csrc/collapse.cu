// collapse.cu — re-lays out a built Karras BVH2 as 4- or 8-wide nodes for
// traversal.  Top-down, level by level (one cooperative launch with a grid
// barrier between levels): each queued BVH2 node becomes a wide node whose children are found by
// repeatedly opening the child with the largest surface area (Wald, Benthin,
// Boulos 2008 style collapsing).
// A BVH2 subtree covers a contiguous run of sorted triangles, so any subtree
// with at most leaf_size triangles becomes a leaf range [first, first+count).
// The Karras topology itself (the parity object) is unchanged.
#include <algorithm>
#include <climits>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "wide.cuh"

namespace flg {

constexpr int kMaxLevels = 64;
constexpr int kCollapseThreads = 128;
constexpr int kCollapseNodes = 4;
// 4-wide layouts hold leaf ranges of at most this many triangles, whatever
// the handle's leaf_size: with quantised nodes a visit costs about as much as
// a triangle test, and ranges of 1 / 2 / 3 / 4 traced 24 batched scenes in
// 20.7 / 20.5 / 22.0 / 23.8 ms (64 k soup 890 / 913 / 985 / 1061 us, camera
// rays 243 / 228 / 228 / 236).  The hits stay those of ranges of leaf_size:
// k_trace4's superset argument does not depend on the ranges, and retrace4 and
// first_of_two form the exact tree with leaf_size.
constexpr int kLeaf4 = 2;
// Collapse counters: [0] wide nodes allocated, [1] its initial value, [2 .. 4]
// the barrier; the initial values of these kCtrLive words follow as a static
// copy.
constexpr int kCtrLive = 5;

// One wide node per queued BVH2 node of a level (cnt items in q_in).  A warp
// claims the slots of its new wide nodes with one atomic on node_ctr (prefix
// sum of the lanes' internal children); the queue of the next level holds the
// new nodes in slot order, so a node's place in it is its slot less the level's
// first (q_base).  Claims by block cost more in barriers than they save (4 M
// triangles: 230 against 220 us).  Queue entries are read through L2 (__ldcg):
// this SM may still hold lines of the same buffer from two levels before.
template <int W>
__device__ __forceinline__ void collapse_level(const Node2 *__restrict__ nodes2, const Ranges &R, int leaf_size,
                                               const int2 *__restrict__ q_in, int cnt, int2 *__restrict__ q_out,
                                               int q_base, int32_t *node_ctr, int64_t cap,
                                               typename WideRec<W>::T *__restrict__ wide, uint32_t *err) {
  const int lane = threadIdx.x & 31;
  // Warp-uniform loop: all lanes of a warp share it0.
  for (int it0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) & ~31u); it0 < cnt; it0 += gridDim.x * blockDim.x) {
    const int it = it0 + lane;
    const bool valid = it < cnt;
    int2 item = make_int2(0, 0);
    Cand c[W];
    int nc = 0;
    if (valid) {
      item = __ldcg(q_in + it);
      // cap = BVH2 node count + 1: item.x names a BVH2 node, item.y a wide slot.
      if (item.x < 0 || item.y < 0 || item.x >= cap - 1 || item.y >= cap)
        atomicOr(err, kErrQueue);  // a hole left by an overflowing level
      else
        open_wide<W>(nodes2, R, leaf_size, item.x, c, nc);
    }
    // Children that become wide nodes of the next level.
    int need = 0;
#pragma unroll
    for (int k = 0; k < W; ++k)
      if (k < nc && c[k].ref >= 0 && c[k].count > leaf_size) ++need;
    int incl = need;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += v;
    }
    int slot0 = 0;
    if (lane == 31 && incl > 0) slot0 = atomicAdd(node_ctr, incl);
    slot0 = __shfl_sync(0xFFFFFFFFu, slot0, 31) + incl - need;
    if (!valid || nc == 0) continue;
    int32_t child[W];
#pragma unroll
    for (int k = 0; k < W; ++k) {
      child[k] = kEmptyChild;
      if (k < nc) {
        if (c[k].ref < 0 || c[k].count <= leaf_size) {
          child[k] = ~((c[k].first << 3) | (c[k].count - 1));
        } else {
          const int slot = slot0++, q = slot - q_base;
          if (slot >= cap) {
            atomicOr(err, kErrQueue);
            if (q < cap) q_out[q] = make_int2(-1, -1);  // the next level skips it
          } else {
            q_out[q] = make_int2(c[k].ref, slot);
            child[k] = slot;
          }
        }
      }
    }
    typename WideRec<W>::T out;
    if constexpr (W == 4) {
      quantise(c, nc, out);
      // This lane's inner children took consecutive slots.
      out.base = 0;
      out.kind = 0u;
      uint32_t rank = 0u;
#pragma unroll
      for (int k = 3; k >= 0; --k)
        if (child[k] >= 0 && child[k] != kEmptyChild) out.base = child[k];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool inner = child[k] >= 0 && child[k] != kEmptyChild;
        out.kind |= (inner ? rank : 0x80u | (uint32_t)k) << (8 * k);
        rank += inner ? 1u : 0u;
        out.leaf[k] = inner ? kEmptyChild : child[k];
      }
    } else {
#pragma unroll
      for (int k = 0; k < W; ++k) {
        const float inf = __int_as_float(0x7f800000);  // unused slots: +inf boxes, which no ray enters
        out.lox[k] = k < nc ? c[k].lo[0] : inf;
        out.loy[k] = k < nc ? c[k].lo[1] : inf;
        out.loz[k] = k < nc ? c[k].lo[2] : inf;
        out.hix[k] = k < nc ? c[k].hi[0] : inf;
        out.hiy[k] = k < nc ? c[k].hi[1] : inf;
        out.hiz[k] = k < nc ? c[k].hi[2] : inf;
        out.child[k] = child[k];
      }
    }
    wide[item.y] = out;
  }
}

// Barrier over all CTAs of a cooperative launch (all resident): bar[0]
// counts arrivals, bar[1] is the generation.  Fences make each CTA's writes
// of the level visible before it arrives and the others' after it leaves.
// The last CTA to arrive notes *ctr in bar[2]; every thread returns that
// value (the next barrier, which all have to reach first, replaces it).
// The wait is bounded: on a timeout the error word is set and the CTA goes
// on (the tree is then wrong, the device keeps answering).
__device__ __forceinline__ int grid_barrier(uint32_t *bar, const int32_t *ctr, uint32_t limit, uint32_t *err) {
  __shared__ int s_now;
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t gen = ld_volatile(bar + 1);
    __threadfence();
    if (atomicAdd(bar, 1u) == gridDim.x - 1) {
      __threadfence();
      *(volatile uint32_t *)(bar + 2) = ld_volatile((const uint32_t *)ctr);
      *(volatile uint32_t *)bar = 0u;
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      for (uint32_t spins = 0; ld_volatile(bar + 1) == gen; ++spins) {
        if (spins >= limit) {
          atomicOr(err, kErrTimeout);
          break;
        }
        if (spins > 64) __nanosleep(128);
      }
    }
    __threadfence();
    s_now = (int)ld_volatile(bar + 2);
  }
  __syncthreads();
  return s_now;
}

// The whole collapse in one cooperative launch: level after level with a
// grid barrier between them, until a level is empty.  Replaces up to 64
// launches (most of them empty) by one.
template <int W>
__global__ void __launch_bounds__(kCollapseThreads)
    k_collapse_all(const Node2 *__restrict__ nodes2, Ranges R, int leaf_size, int n_roots, int2 *q0, int2 *q1,
                   int32_t *ctr, uint32_t *bar, int64_t cap, typename WideRec<W>::T *__restrict__ wide,
                   uint32_t spin_limit, uint32_t *err) {
  int cnt = n_roots, end = ctr[1];  // the level's queue; where its new nodes begin (ctr[0] moves on)
  for (int L = 0; L < kMaxLevels && cnt > 0; ++L) {
    collapse_level<W>(nodes2, R, leaf_size, (L & 1) ? q1 : q0, cnt, (L & 1) ? q0 : q1, end, ctr, cap, wide, err);
    const int now = grid_barrier(bar, ctr, spin_limit, err);
    // Counts beyond the queue capacity only arise from a corrupted tree.
    cnt = (int)min((int64_t)(now - end), cap);
    end = now;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && cnt > 0) atomicOr(err, kErrQueue);  // deeper than kMaxLevels
}

int collapse_reserve(flg_ctx ctx, flg_bvh b) {
  // Every wide node corresponds to a distinct BVH2 internal node.
  const int64_t cap = b->n_nodes + 1;
  const size_t rec = b->width == 4 ? sizeof(NodeQ) : sizeof(NodeW<8>);
  int rc = FLG_OK;
  if (b->d_wide) {
    cudaFree(b->d_wide);
    b->allocs.erase(std::find(b->allocs.begin(), b->allocs.end(), b->d_wide));
    b->device_bytes -= (int64_t)(b->wide_cap * (b->wide_rec));
    b->d_wide = nullptr;
  }
  uint8_t *w = nullptr;
  rc = halloc(b, &w, rec * (size_t)cap);
  if (rc) return rc;
  b->d_wide = w;
  b->wide_cap = cap;
  b->wide_rec = (int64_t)rec;
  if (!b->d_wide_root) {
    if ((rc = halloc(b, &b->d_wide_root, b->n_scenes))) return rc;
    if ((rc = halloc(b, &b->d_wide_ctr, 2 * kCtrLive))) return rc;
    if ((rc = halloc(b, &b->d_queue[0], cap))) return rc;
    if ((rc = halloc(b, &b->d_queue[1], cap))) return rc;
    if ((rc = halloc(b, &b->d_queue_init, b->n_scenes))) return rc;
  }
  // Scenes of one triangle: their root is the leaf in the 8-wide layout; in
  // the 4-wide one a node, written here once, whose one box constrains
  // nothing.
  std::vector<int32_t> roots(b->n_scenes);
  std::vector<int2> q;
  std::vector<NodeQ> lone;  // records of slots [0, lone.size())
  int32_t slots = 0;
  for (int s = 0; s < b->n_scenes; ++s) {
    int64_t c = b->tri_off_h[s + 1] - b->tri_off_h[s];
    if (c >= 2) {
      roots[s] = slots;
      q.push_back(make_int2((int)b->node_off_h[s], slots++));
    } else if (c == 1 && b->width == 4) {
      NodeQ nd = {};
      nd.step = kLoneStep;
      nd.kind = 0x83828180u;
      nd.leaf[0] = ~(int32_t)(b->tri_off_h[s] << 3);
      nd.leaf[1] = nd.leaf[2] = nd.leaf[3] = kEmptyChild;
      roots[s] = slots++;
      lone.resize(slots);  // the ones between are written by every collapse
      lone.back() = nd;
    } else if (c == 1) {
      roots[s] = ~(int32_t)(b->tri_off_h[s] << 3);
    } else {
      roots[s] = kEmptyChild;
    }
  }
  b->n_wide_roots = (int32_t)q.size();
  std::vector<int32_t> ctr(2 * kCtrLive, 0);
  ctr[0] = ctr[1] = ctr[kCtrLive] = ctr[kCtrLive + 1] = slots;
  cudaStream_t st = ctx->stream;
  cudaError_t e = cudaMemcpyAsync(b->d_wide_root, roots.data(), sizeof(int32_t) * b->n_scenes,
                                  cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && !q.empty())
    e = cudaMemcpyAsync(b->d_queue_init, q.data(), sizeof(int2) * q.size(), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(b->d_wide_ctr, ctr.data(), sizeof(int32_t) * ctr.size(), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && !lone.empty())
    e = cudaMemcpyAsync(b->d_wide, lone.data(), sizeof(NodeQ) * lone.size(), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "collapse upload");
  return FLG_OK;
}

template <int W>
static int collapse_levels(flg_ctx ctx, flg_bvh b) {
  cudaStream_t st = ctx->stream;
  using Rec = typename WideRec<W>::T;
  Rec *wide = (Rec *)b->d_wide;
  const Ranges R{b->d_rfirst, b->d_rcount};
  const int leaf = W == 4 ? std::min<int>(b->leaf_size, kLeaf4) : b->leaf_size;
  // Level sizes are only known on the device: one cooperative launch walks the
  // levels with a grid barrier in between.  A barrier costs by its CTAs, so a
  // small tree takes fewer than a resident wave: one thread per kCollapseNodes
  // nodes covers its widest levels.
  static const int per_sm = [] {
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_collapse_all<W>, kCollapseThreads, 0) != cudaSuccess ||
        v < 1)
      v = 1;
    return v;
  }();
  int32_t *ctr = b->d_wide_ctr;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid_for(ceil_div(b->n_nodes, kCollapseNodes), kCollapseThreads, (int64_t)ctx->num_sms * per_sm));
  cfg.blockDim = dim3(kCollapseThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  FLG_CUDA(ctx, cudaLaunchKernelEx(&cfg, k_collapse_all<W>, (const Node2 *)b->d_nodes2, R, leaf, (int)b->n_wide_roots,
                                   b->d_queue[0], b->d_queue[1], ctr, (uint32_t *)(ctr + 2), (int64_t)b->wide_cap, wide,
                                   ctx->spin_limit, ctx->d_err));
  FLG_LAUNCH_CHECK(ctx, "k_collapse_all");
  return FLG_OK;
}

int collapse_ctr_words() { return kCtrLive; }

// Expects the counters and the first level's queue at their initial values
// (k_build_setup, or flg_bvh_set_width's copies).
int collapse_enqueue(flg_ctx ctx, flg_bvh b, int width) {
  if (b->n_wide_roots == 0) return FLG_OK;
  cudaStream_t st = ctx->stream;
  const int rc = width == 4 ? collapse_levels<4>(ctx, b) : collapse_levels<8>(ctx, b);
  if (rc == FLG_OK) stage_mark(ctx, st, "collapse");
  return rc;
}

}  // namespace flg

using namespace flg;

FLG_API int flg_bvh_set_width(flg_ctx ctx, flg_bvh bvh, int32_t node_width, int32_t leaf_size) {
  if (!ctx || !bvh) return FLG_ERR_ARG;
  if (node_width != 2 && node_width != 4 && node_width != 8)
    return set_error(ctx, FLG_ERR_ARG, "node_width must be 2, 4 or 8");
  if (leaf_size < 1 || leaf_size > 8) return set_error(ctx, FLG_ERR_ARG, "leaf_size must be in [1, 8]");
  if (node_width == bvh->width && leaf_size == bvh->leaf_size) return FLG_OK;
  const int old_w = bvh->width;
  bvh->width = node_width;
  bvh->leaf_size = leaf_size;
  if (node_width == 2) return FLG_OK;
  if (ctx->capturing && (old_w != node_width || !bvh->d_wide))
    return set_error(ctx, FLG_ERR_STATE, "re-layout allocates; not allowed during capture");
  if (!bvh->d_wide || old_w != node_width) {
    int rc = collapse_reserve(ctx, bvh);
    if (rc) return rc;
  }
  if (bvh->n_wide_roots > 0) {
    FLG_CUDA(ctx, cudaMemcpyAsync(bvh->d_wide_ctr, bvh->d_wide_ctr + kCtrLive, sizeof(int32_t) * kCtrLive,
                                  cudaMemcpyDeviceToDevice, ctx->stream));
    FLG_CUDA(ctx, cudaMemcpyAsync(bvh->d_queue[0], bvh->d_queue_init, sizeof(int2) * bvh->n_wide_roots,
                                  cudaMemcpyDeviceToDevice, ctx->stream));
  }
  return collapse_enqueue(ctx, bvh, node_width);
}
