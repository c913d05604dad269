// collapse.cu — re-lays out a built Karras BVH2 as 4- or 8-wide nodes for
// traversal, top-down: a BVH2 node becomes a wide node whose children are found
// by repeatedly opening the child with the largest surface area (Wald, Benthin,
// Boulos 2008 style collapsing).  Large scenes go level by level in one
// cooperative launch with a grid barrier between levels (k_collapse_all),
// smaller ones in subtrees (k_collapse_top, k_collapse_rest).
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
// Counters of a collapse; the initial values of these kCtrLive words follow as a
// static copy.
enum {
  kCtrNodes = 0,  // slots taken
  kCtrFirst = 1,  // slots that the roots have
  kCtrBar = 2,    // k_collapse_all's barrier: arrivals, generation, kCtrNodes when all had arrived
  kCtrReady = 5,  // k_collapse_top: subtrees listed
  kCtrClaim = 6,  // subtrees taken
  kCtrLive = 7
};

// Child k of an opened node becomes a wide node of its own.
template <int W>
__device__ __forceinline__ bool is_inner(const Cand (&c)[W], int nc, int k, int leaf_size) {
  return k < nc && c[k].ref >= 0 && c[k].count > leaf_size;
}

// Record of an opened node whose inner children take the slots from slot0 on
// (those from cap on: unused, the caller has set the error word).
template <int W>
__device__ __forceinline__ typename WideRec<W>::T wide_record(const Cand (&c)[W], int nc, int leaf_size, int slot0,
                                                              int64_t cap) {
  int32_t child[W];
  int slot = slot0;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    child[k] = kEmptyChild;
    if (is_inner<W>(c, nc, k, leaf_size)) {
      if (slot < cap) child[k] = slot;
      ++slot;
    } else if (k < nc) {
      child[k] = ~((c[k].first << 3) | (c[k].count - 1));
    }
  }
  typename WideRec<W>::T out;
  if constexpr (W == 4) {
    quantise(c, nc, out);
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
  return out;
}

// Opens item (BVH2 node, wide slot); nc stays 0 if it names neither: a hole left
// by an overflow, or a broken tree.
template <int W>
__device__ __forceinline__ void open_item(const Node2 *__restrict__ nodes2, const Ranges &R, int leaf_size,
                                          const int2 &item, int64_t cap, Cand (&c)[W], int &nc, uint32_t *err) {
  // cap = BVH2 node count + 1: item.x names a BVH2 node, item.y a wide slot.
  if (item.x < 0 || item.y < 0 || item.x >= cap - 1 || item.y >= cap) atomicOr(err, kErrQueue);
  else open_wide<W>(nodes2, R, leaf_size, item.x, c, nc);
}

// What a collapse works on.
struct Collapse {
  const Node2 *nodes2;
  Ranges R;
  int leaf_size;
  int64_t cap;        // slots
  const int2 *roots;  // (BVH2 node, slot)
  int n_roots;
  int2 *queue[2];     // k_collapse_all: the nodes of a level, (BVH2 node, slot)
  int small;          // k_collapse_top: most triangles of a subtree that it lists
  int32_t *ref;       // BVH2 node by slot
  int32_t *ready;     // slots of the listed subtrees
  int32_t *large[2];  // slots of the large nodes of a level
  int32_t *ctr;
  uint32_t spin_limit, *err;
};

__device__ __forceinline__ int warp_inclusive(int v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= o) v += x;
  }
  return v;
}

// k_collapse_all: one wide node per queued BVH2 node of a level (cnt items in
// q_in).  A warp claims the slots of its new wide nodes with one atomic (prefix
// sum of the lanes' inner children); the queue of the next level holds the new
// nodes in slot order, so a node's place in it is its slot less the level's
// first (q_base).  Claims by block cost more in barriers than they save (4 M
// triangles: 230 against 220 us), as do separate lists of slots (246).  Queue
// entries are read through L2 (__ldcg): this SM may still hold lines of the same
// buffer from two levels before.
template <int W>
__device__ __forceinline__ void collapse_level(const Collapse &X, const int2 *__restrict__ q_in, int cnt,
                                               int2 *__restrict__ q_out, int q_base,
                                               typename WideRec<W>::T *__restrict__ wide) {
  const int lane = threadIdx.x & 31;
  // Warp-uniform loop: all lanes of a warp share it0.
  for (int it0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) & ~31u); it0 < cnt; it0 += gridDim.x * blockDim.x) {
    const int it = it0 + lane;
    int2 item = make_int2(0, 0);
    Cand c[W];
    int nc = 0;
    if (it < cnt) {
      item = __ldcg(q_in + it);
      open_item<W>(X.nodes2, X.R, X.leaf_size, item, X.cap, c, nc, X.err);
    }
    int need = 0;
#pragma unroll
    for (int k = 0; k < W; ++k) need += is_inner<W>(c, nc, k, X.leaf_size) ? 1 : 0;
    const int incl = warp_inclusive(need, lane);
    int base = 0;
    if (lane == 31 && incl > 0) base = atomicAdd(X.ctr + kCtrNodes, incl);
    base = __shfl_sync(0xFFFFFFFFu, base, 31);
    if (nc == 0) continue;
    const int slot0 = base + incl - need;
    int slot = slot0;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      if (!is_inner<W>(c, nc, k, X.leaf_size)) continue;
      const int q = slot - q_base;
      if (slot >= X.cap) atomicOr(X.err, kErrQueue);
      if (q < X.cap) q_out[q] = slot < X.cap ? make_int2(c[k].ref, slot) : make_int2(-1, -1);  // the next level skips it
      ++slot;
    }
    wide[item.y] = wide_record<W>(c, nc, X.leaf_size, slot0, X.cap);
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
// grid barrier between them, until a level is empty.
template <int W>
__global__ void __launch_bounds__(kCollapseThreads)
    k_collapse_all(const __grid_constant__ Collapse X, typename WideRec<W>::T *__restrict__ wide) {
  int cnt = X.n_roots, end = X.ctr[kCtrFirst];  // the level's queue; where its new nodes begin
  for (int L = 0; L < kMaxLevels && cnt > 0; ++L) {
    collapse_level<W>(X, L == 0 ? X.roots : X.queue[L & 1], cnt, X.queue[(L + 1) & 1], end, wide);
    const int now = grid_barrier((uint32_t *)X.ctr + kCtrBar, X.ctr + kCtrNodes, X.spin_limit, X.err);
    // Counts beyond the queue capacity only arise from a corrupted tree.
    cnt = (int)min((int64_t)(now - end), X.cap);
    end = now;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && cnt > 0) atomicOr(X.err, kErrQueue);  // deeper than kMaxLevels
}

// Up to kTopMax triangles a collapse is two launches without a wait for another
// SM.  k_collapse_top, one CTA, opens level after level the nodes of more than
// `small` triangles and lists their other inner children; k_collapse_rest gives
// these subtrees to warps.  A level of k_collapse_all takes 4 us, half of it in
// the barrier, whatever its size, and the last ones, of a few nodes each, are
// half of them.  us per collapse, k_collapse_all -> this: 5,000 triangles 48 ->
// 29, 20,001 54 -> 31, 65,536 62 -> 37, 200,000 73 -> 46, 600,000 97 -> 80,
// 1,000,000 108 -> 105, 2,000,000 152 -> 196.  `small`: 1.4 n / 2^k for the k at which
// n / 2^k falls to 181, at most 10.
// The top CTA is bound by instructions, so smaller subtrees cost (20,001
// triangles in subtrees of 64: 51 us); and a warp takes long over larger ones
// (200,000 in n / 256: 79).  Large scenes keep the levels: a warp's steps run
// with half of the lanes.
constexpr int64_t kTopMax = 1 << 20;
constexpr int kTopThreads = 256;
constexpr int kTopRoots = 1024;
constexpr int kTopSplit = 1024;
constexpr int kSmallTree = 181;

// Entries that this kernel writes and reads go through L2.
__device__ __forceinline__ int2 item_at(const Collapse &X, int slot) {
  return make_int2(slot >= 0 && slot < X.cap ? __ldcg(X.ref + slot) : -1, slot);
}

// Lists the inner children of an opened node, which take the slots from slot0 on:
// the large ones from list[large] on, the others from X.ready[other] on.
template <int W>
__device__ __forceinline__ void list_children(const Collapse &X, const Cand (&c)[W], int nc, int slot0, int32_t *list,
                                              int large, int64_t most, int other) {
  int slot = slot0;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    if (!is_inner<W>(c, nc, k, X.leaf_size)) continue;
    const bool big = c[k].count > X.small;
    int &at = big ? large : other;
    if (slot < X.cap && at < (big ? most : X.cap)) {
      X.ref[slot] = c[k].ref;
      (big ? list : X.ready)[at] = slot;
    } else {
      atomicOr(X.err, kErrQueue);  // counts that do not add up: a broken tree
    }
    ++at;
    ++slot;
  }
}

// Inner children of an opened node, and in the upper half the large ones.
template <int W>
__device__ __forceinline__ int count_children(const Collapse &X, const Cand (&c)[W], int nc) {
  int need = 0;
#pragma unroll
  for (int k = 0; k < W; ++k)
    if (is_inner<W>(c, nc, k, X.leaf_size)) need += c[k].count > X.small ? 0x10001 : 1;
  return need;
}

// The listed subtrees.  A warp takes one, opens up to 32 of its nodes at a time,
// claims the slots of their inner children with one atomic and stacks them as
// one run of slots.  Last in, first out: a run on the stack lies deeper in the
// tree than the one below it, so kMaxLevels runs suffice.
template <int W>
__device__ __forceinline__ void collapse_rest(const Collapse &X, int n_ready,
                                              typename WideRec<W>::T *__restrict__ wide) {
  __shared__ int2 s_run[kCollapseThreads / 32][kMaxLevels];
  const int lane = threadIdx.x & 31;
  int2 *run = s_run[threadIdx.x >> 5];
  const int warps = gridDim.x * (kCollapseThreads / 32);
  const int take = min(max(n_ready / (2 * warps), 1), 32);  // at a time
  int mine = (blockIdx.x * (kCollapseThreads / 32) + (threadIdx.x >> 5)) * take;
  int depth = 0;
  while (true) {
    int slot = -1;
    if (depth == 0) {
      if (mine >= n_ready) break;
      if (lane < take && mine + lane < n_ready) slot = __ldcg(X.ready + mine + lane);
      if (lane == 0) mine = warps * take + atomicAdd(X.ctr + kCtrClaim, take);
      mine = __shfl_sync(0xFFFFFFFFu, mine, 0);
    } else {
      const int2 r = run[depth - 1];
      const int m = min(r.y, 32);
      if (lane < m) slot = r.x + r.y - m + lane;
      __syncwarp();
      if (r.y == m) --depth;
      else if (lane == 0) run[depth - 1].y = r.y - m;
    }
    Cand c[W];
    int nc = 0;
    if (slot >= 0) open_item<W>(X.nodes2, X.R, X.leaf_size, item_at(X, slot), X.cap, c, nc, X.err);
    int need = 0;
#pragma unroll
    for (int k = 0; k < W; ++k) need += is_inner<W>(c, nc, k, X.leaf_size) ? 1 : 0;
    const int incl = warp_inclusive(need, lane);
    const int all = __shfl_sync(0xFFFFFFFFu, incl, 31);
    int base = 0;
    if (lane == 0 && all > 0) base = atomicAdd(X.ctr + kCtrNodes, all);
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (nc > 0) {
      const int slot0 = base + incl - need;
      int to = slot0;
#pragma unroll
      for (int k = 0; k < W; ++k) {
        if (!is_inner<W>(c, nc, k, X.leaf_size)) continue;
        if (to < X.cap) X.ref[to] = c[k].ref;
        ++to;
      }
      wide[slot] = wide_record<W>(c, nc, X.leaf_size, slot0, X.cap);
    }
    if (all > 0) {
      // only a broken tree needs more slots, or more levels, than there are
      const int left = base < X.cap ? (int)min((int64_t)all, X.cap - base) : 0;
      if ((left < all || depth == kMaxLevels) && lane == 0) atomicOr(X.err, kErrQueue);
      if (left > 0 && depth < kMaxLevels) {
        if (lane == 0) run[depth] = make_int2(base, left);
        ++depth;
      }
    }
    __syncwarp();
  }
}

template <int W>
__global__ void __launch_bounds__(kTopThreads)
    k_collapse_top(const __grid_constant__ Collapse X, typename WideRec<W>::T *__restrict__ wide) {
  __shared__ int s_wsum[kTopThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  after_wait();
  int slots = X.ctr[kCtrFirst], n_ready = 0;
  int cnt = X.n_roots;
  for (int L = 0; L < kMaxLevels && cnt > 0; ++L) {
    const int32_t *in = X.large[L & 1];
    int next = 0;
    for (int it0 = 0; it0 < cnt; it0 += kTopThreads) {
      int2 item = make_int2(0, 0);
      Cand c[W];
      int nc = 0;
      if (it0 + tid < cnt) {
        item = L == 0 ? X.roots[it0 + tid] : item_at(X, __ldcg(in + it0 + tid));
        open_item<W>(X.nodes2, X.R, X.leaf_size, item, X.cap, c, nc, X.err);
      }
      const int need = count_children<W>(X, c, nc), incl = warp_inclusive(need, lane);
      if (lane == 31) s_wsum[warp] = incl;
      __syncthreads();
      int before = incl - need, all = 0;
#pragma unroll
      for (int w = 0; w < kTopThreads / 32; ++w) {
        const int x = s_wsum[w];
        if (w < warp) before += x;
        all += x;
      }
      if (nc > 0) {
        const int slot0 = slots + (before & 0xFFFF);
        list_children<W>(X, c, nc, slot0, X.large[(L + 1) & 1], next + (before >> 16), X.cap,
                         n_ready + (before & 0xFFFF) - (before >> 16));
        wide[item.y] = wide_record<W>(c, nc, X.leaf_size, slot0, X.cap);
      }
      slots += all & 0xFFFF;
      next += all >> 16;
      n_ready += (all & 0xFFFF) - (all >> 16);
      __syncthreads();
    }
    cnt = (int)min((int64_t)next, X.cap);
  }
  if (tid == 0) {
    X.ctr[kCtrNodes] = slots;
    X.ctr[kCtrReady] = (int32_t)min((int64_t)n_ready, X.cap);
    if (cnt > 0) atomicOr(X.err, kErrQueue);  // deeper than kMaxLevels
  }
}

template <int W>
__global__ void __launch_bounds__(kCollapseThreads)
    k_collapse_rest(const __grid_constant__ Collapse X, typename WideRec<W>::T *__restrict__ wide) {
  after_wait();
  collapse_rest<W>(X, X.ctr[kCtrReady], wide);
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
  for (int i : {(int)kCtrNodes, (int)kCtrFirst}) ctr[i] = ctr[kCtrLive + i] = slots;
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
  Collapse X;
  X.nodes2 = b->d_nodes2;
  X.R = Ranges{b->d_rfirst, b->d_rcount};
  X.leaf_size = b->leaf_size;
  X.roots = b->d_queue_init;
  X.n_roots = b->n_wide_roots;
  X.cap = b->wide_cap;
  X.queue[0] = b->d_queue[0];
  X.queue[1] = b->d_queue[1];
  X.small = 0;
  X.ref = (int32_t *)b->d_queue[0];
  X.ready = X.ref + X.cap;
  X.large[0] = (int32_t *)b->d_queue[1];
  X.large[1] = X.large[0] + X.cap;
  X.ctr = b->d_wide_ctr;
  X.spin_limit = ctx->spin_limit;
  X.err = ctx->d_err;
  static const int rest_per_sm = [] {
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_collapse_rest<W>, kCollapseThreads, 0) != cudaSuccess ||
        v < 1)
      v = 1;
    return v;
  }();
  if (b->n_tri <= kTopMax && b->n_wide_roots <= kTopRoots) {
    // n / 2^k triangles are what a node of depth k has on average: cut between two
    // depths, not through the middle of one (builds with small = max(128, n / 700)
    // against this, us: 8,192 triangles 77 -> 67, 32,768 93 -> 84, 45,000 100 -> 95).
    int64_t nodes = 1;
    while (nodes < kTopSplit && b->n_tri > kSmallTree * nodes) nodes *= 2;
    X.small = (int)(b->n_tri * 181 / (128 * nodes));
    FLG_CUDA(ctx, launch_after(k_collapse_top<W>, 1, kTopThreads, st, X, wide));
    FLG_LAUNCH_CHECK(ctx, "k_collapse_top");
    FLG_CUDA(ctx, launch_after(k_collapse_rest<W>,
                               grid_for(b->n_nodes, 2 * kCollapseThreads, (int64_t)ctx->num_sms * rest_per_sm),
                               kCollapseThreads, st, X, wide));
    FLG_LAUNCH_CHECK(ctx, "k_collapse_rest");
    return FLG_OK;
  }
  static const int per_sm = [] {
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_collapse_all<W>, kCollapseThreads, 0) != cudaSuccess ||
        v < 1)
      v = 1;
    return v;
  }();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid_for(ceil_div(b->n_nodes, kCollapseNodes), kCollapseThreads, (int64_t)ctx->num_sms * per_sm));
  cfg.blockDim = dim3(kCollapseThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  FLG_CUDA(ctx, cudaLaunchKernelEx(&cfg, k_collapse_all<W>, X, wide));
  FLG_LAUNCH_CHECK(ctx, "k_collapse_all");
  return FLG_OK;
}

int collapse_ctr_words() { return kCtrLive; }

// Expects the counters at their initial values (k_build_setup, or
// flg_bvh_set_width's copy).
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
  if (bvh->n_wide_roots > 0)
    FLG_CUDA(ctx, cudaMemcpyAsync(bvh->d_wide_ctr, bvh->d_wide_ctr + kCtrLive, sizeof(int32_t) * kCtrLive,
                                  cudaMemcpyDeviceToDevice, ctx->stream));
  return collapse_enqueue(ctx, bvh, node_width);
}
