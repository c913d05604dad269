// volume.cu — participating media on a dense density grid:
//   k_volume_tr        ratio-tracking transmittance (OpenVDBVolume::tr,
//                      volume.cpp:75-107), one ray per thread, optional
//                      checkpoint of the state after the last roulette
//   k_volume_tr_adj    its adjoint with respect to the grid, replaying the
//                      ray's Philox stream from the checkpoint (or from the
//                      start) and scattering fp32 atomics into dL/dgrid
//   k_volume_sample    delta tracking (OpenVDBVolume::sample, :109-148)
// The grid is a vertex-centred lattice (x fastest) over the box; trilinear
// interpolation with background 0, the dense restatement of OpenVDB's
// tools::Sampler<1> lookups (volume.cpp:94,133).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "internal.h"
#include "volume.cuh"

namespace flg {

struct VRays {
  const float *ox, *oy, *oz, *dx, *dy, *dz, *tmax;
  float tmax_c;
};

__device__ __forceinline__ void load_vray(const VRays &R, int64_t i, float3 &o, float3 &d, float &tmax) {
  o = make_float3(__ldg(R.ox + i), __ldg(R.oy + i), __ldg(R.oz + i));
  d = make_float3(__ldg(R.dx + i), __ldg(R.dy + i), __ldg(R.dz + i));
  tmax = R.tmax ? __ldg(R.tmax + i) : R.tmax_c;
}

// The tracking kernels are latency-bound on dependent grid taps: they run at
// 4 CTAs per SM (64 registers, no spills), 32 % faster than at the 3 that 74
// registers allowed; 5 CTAs spill and lose again.
//
// Rays take very different numbers of steps (geometric: the longest of 32 takes
// about four times the mean), so a warp does not run 32 rays to their end: it
// owns a contiguous chunk of the rays, and lanes whose ray has ended take the
// next ones together once kVolRefill of them are idle.  A lane's step (of delta
// tracking: two, a Philox block's draws) is one turn of the warp's loop.
// Together with one bounds test and one address per lattice cell (grid_cell), us
// before -> after: delta tracking of 2 M rays through a 192^3 sparse grid 927 ->
// 547, with two steps to a turn 460, with refills at 4 idle lanes 434 (8: 446), and
// with a pointer to each of the two layers of bricks 1.5 % less; of 1 M rays
// through a 256^3 dense one 83 -> 52 -> 47.  Ratio tracking of the latter became 5 %
// faster, its adjoint 3 %: it waits for one dependent lookup after the other
// (stalls on loads: 5.4 and 10.2 per issued instruction; L1 at 61 and 36 % of
// its rate, L2 at 50 and 41, DRAM at 28 and 56, 17.7 and 12.1 of 32 lanes active).
// It gains nothing from turns of four draws (75 -> 76 us, the adjoint 79 -> 85), nor
// from lookups of steps ahead; with refills at 4 idle lanes it takes 81 us, at 16 77.
constexpr int kVolRefill = 8, kSampleRefill = 4;

struct WarpChunk {
  int64_t next, end;
  int refill;  // idle lanes that make the warp take rays
  bool fresh;  // the rays just taken are those of all lanes
  __device__ __forceinline__ WarpChunk(int64_t n, int refill_) : refill(refill_), fresh(false) {
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int64_t per = (n + warps - 1) / warps;
    next = min(per * (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), n);
    end = min(next + per, n);
  }
  // The ray that this lane takes now, or -1; all lanes call it.  `left`: false
  // once every lane is idle and the chunk is empty.
  __device__ __forceinline__ int64_t take(bool busy, bool &left) {
    const unsigned idle = __ballot_sync(0xFFFFFFFFu, !busy);
    const int nidle = __popc(idle);
    left = next < end || nidle < 32;
    fresh = false;
    if (next >= end || nidle < refill) return -1;
    fresh = nidle == 32;
    const int64_t my = next + __popc(idle & ((1u << (threadIdx.x & 31u)) - 1u));
    next += nidle;
    return !busy && my < end ? my : -1;
  }
  // After 32 rays have been taken together (`mine`: one of them is this lane's):
  // a warp whose rays lie side by side takes all of the next ones together, too.
  __device__ __forceinline__ void adapt(const GridDev &G, bool mine, const float3 &o, const float3 &d) {
    const int src = __ffs(__ballot_sync(0xFFFFFFFFu, mine)) - 1;
    const float ox = (o.x - __shfl_sync(0xFFFFFFFFu, o.x, src)) * G.scale[0];
    const float oy = (o.y - __shfl_sync(0xFFFFFFFFu, o.y, src)) * G.scale[1];
    const float oz = (o.z - __shfl_sync(0xFFFFFFFFu, o.z, src)) * G.scale[2];
    const float ex = __shfl_sync(0xFFFFFFFFu, d.x, src), ey = __shfl_sync(0xFFFFFFFFu, d.y, src),
                ez = __shfl_sync(0xFFFFFFFFu, d.z, src);
    const float dot = d.x * ex + d.y * ey + d.z * ez;
    const bool near = ox * ox + oy * oy + oz * oz <= 256.0f && dot > 0.0f &&
                      dot * dot >= 0.999f * (d.x * d.x + d.y * d.y + d.z * d.z) * (ex * ex + ey * ey + ez * ez);
    refill = __all_sync(0xFFFFFFFFu, !mine || near) ? 32 : kVolRefill;
  }
};

template <bool SP>
__global__ void __launch_bounds__(256, 4)
    k_volume_tr(GridDev G, VRays R, int64_t n, uint64_t seed, float *__restrict__ T, float *__restrict__ ck_t,
                uint32_t *__restrict__ ck_k, float *__restrict__ ck_c, bool adapt) {
  after_wait();
  const float maj = __ldg(G.params), inv_maj = __ldg(G.params + 1);
  const float max_mu = G.sigma_t * maj;
  WarpChunk chunk(n, kVolRefill);
  RatioState s;
  int64_t ray = -1;
  int steps = 0;
  while (true) {
    bool left, go = ray >= 0;
    const int64_t my = chunk.take(go, left);
    if (!left) break;
    if (my >= 0) {
      ray = my;
      float tmax;
      load_vray(R, ray, s.o, s.d, tmax);
      go = ratio_start(G, s, tmax, seed, ray);
      steps = 0;
    }
    if (adapt && chunk.fresh) chunk.adapt(G, my >= 0, s.o, s.d);
    if (go) go = ratio_step<SP>(G, max_mu, inv_maj, s) && ++steps < kMaxTrackSteps;
    if (!go && ray >= 0) {
      T[ray] = s.tr;
      if (ck_t) {
        ck_t[ray] = s.ck_t;
        ck_k[ray] = s.ck_k;
        ck_c[ray] = s.ck_c;
      }
      ray = -1;
    }
  }
}

// Adds v0, v1 to grad[e], grad[e + 1] (nv values in all).  One reduction
// operation where the pair lies in an aligned group of two, or inside one of
// four whose ends take +0 (the L2 takes a vector reduction in the time of a
// scalar one); two otherwise.
__device__ __forceinline__ void add_pair(float *grad, int64_t e, int64_t nv, bool aligned, float v0, float v1) {
  if (aligned && (e & 1) == 0) {
    atomicAdd(reinterpret_cast<float2 *>(grad + e), make_float2(v0, v1));
  } else if (aligned && (e & 3) == 1 && e + 2 < nv) {
    atomicAdd(reinterpret_cast<float4 *>(grad + e - 1), make_float4(0.0f, v0, v1, 0.0f));
  } else {
    atomicAdd(grad + e, v0);
    atomicAdd(grad + e + 1, v1);
  }
}

// Adjoint: T = c * prod_{last segment} (1 - d_i/rho_max); with the majorant
// fixed, dT/drho_v = sum_i -T/(1 - d_i/rho_max) * w_iv / rho_max.  Bound by its
// reductions into L2: two of the eight values of a step share a row.
template <bool SP>
__global__ void __launch_bounds__(256, 4)
    k_volume_tr_adj(GridDev G, VRays R, int64_t n, uint64_t seed, const float *__restrict__ dLdT,
                    const float *__restrict__ T, const float *__restrict__ ck_t, const uint32_t *__restrict__ ck_k,
                    float *__restrict__ grad, int64_t nv) {
  after_wait();
  const float maj = __ldg(G.params), inv_maj = __ldg(G.params + 1);
  const float max_mu = G.sigma_t * maj;
  const bool aligned = (reinterpret_cast<uintptr_t>(grad) & 15u) == 0u;
  WarpChunk chunk(n, kVolRefill);
  float3 o = make_float3(0.0f, 0.0f, 0.0f), d = o;
  float t = 0.0f, t_max = 0.0f, base = 0.0f;
  RayStream rs;
  bool go = false;
  int steps = 0;
  while (true) {
    bool left;
    const int64_t i = chunk.take(go, left);
    if (!left) break;
    if (i >= 0) {
      const float g = __ldg(dLdT + i);
      const float Tf = __ldg(T + i);
      if (!(g == 0.0f || Tf == 0.0f)) {
        float tmax, t_min;
        load_vray(R, i, o, d, tmax);
        uint32_t k;
        if (ck_t) {
          t = __ldg(ck_t + i);
          k = __ldg(ck_k + i);
        } else {
          float cc;
          ratio_track<SP>(G, maj, inv_maj, o, d, tmax, seed, i, t, k, cc);
        }
        go = box_pbrt(G, o, d, tmax, t_min, t_max);
        t_max = fminf(t_max, tmax);
        base = -g * Tf * inv_maj;
        rs.init(seed, (uint64_t)i, k);
        steps = 0;
      }
    }
    if (go) {
      const float u = rs.next();
      t += -flg_logf(1.0f - u) / max_mu;
      go = !(t >= t_max);
    }
    if (go) {
      int x, y, z;
      float fx, fy, fz;
      const float dens = sample_grid<SP>(G, o.x + d.x * t, o.y + d.y * t, o.z + d.z * t, x, y, z, fx, fy, fz);
      const float xr = dens * inv_maj;
      if (xr > 0.0f) {
        const float coef = base / (1.0f - xr);
        const float wx[2] = {1.0f - fx, fx}, wy[2] = {1.0f - fy, fy}, wz[2] = {1.0f - fz, fz};
        const bool inside = (unsigned)x < (unsigned)(G.nx - 1) && (unsigned)y < (unsigned)(G.ny - 1) &&
                            (unsigned)z < (unsigned)(G.nz - 1);
        if (inside && (!SP || (unsigned)x % kBrick < kBrick - 1)) {
          // rows of two values, contiguous
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int cy = c & 1, cz = c >> 1;
            int64_t e = ((int64_t)(z + cz) * G.ny + (y + cy)) * G.nx + x;
            if (SP) {
              e = grid_voxel<true>(G, x, y + cy, z + cz);
              if (e < 0) continue;  // an empty brick of a sparse grid is not a parameter
            }
            add_pair(grad, e, nv, aligned, coef * (wx[0] * wy[cy] * wz[cz]), coef * (wx[1] * wy[cy] * wz[cz]));
          }
        } else {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const int cx = c & 1, cy = (c >> 1) & 1, cz = c >> 2;
            const int X = x + cx, Y = y + cy, Z = z + cz;
            if (X < 0 || Y < 0 || Z < 0 || X >= G.nx || Y >= G.ny || Z >= G.nz) continue;
            int64_t off = ((int64_t)Z * G.ny + Y) * G.nx + X;
            if (SP) {
              off = grid_voxel<true>(G, X, Y, Z);
              if (off < 0) continue;
            }
            atomicAdd(grad + off, coef * (wx[cx] * wy[cy] * wz[cz]));
          }
        }
      }
      go = ++steps < kMaxTrackSteps;
    }
  }
}

template <bool SP>
__global__ void __launch_bounds__(256, 4)
    k_volume_sample(GridDev G, VRays R, int64_t n, uint64_t seed, uint8_t *__restrict__ success,
                    float *__restrict__ p, float *__restrict__ weight) {
  after_wait();
  const float maj = __ldg(G.params);
  const float max_mu = G.sigma_t * maj;
  WarpChunk chunk(n, kSampleRefill);
  TrackState s;
  int64_t ray = -1;
  while (true) {
    bool left;
    const int64_t my = chunk.take(ray >= 0, left);
    if (!left) break;
    int r = ray >= 0 ? 0 : -1;
    if (my >= 0) {
      ray = my;
      float tmax;
      load_vray(R, ray, s.o, s.d, tmax);
      s.ray = ray;
      r = s.start(G, tmax) ? 0 : -1;
    }
    float3 q = make_float3(0.0f, 0.0f, 0.0f);
    if (r == 0) r = delta_turn<SP>(G, max_mu, seed, s, q);
    if (r != 0 && ray >= 0) {
      const bool ok = r == 1;
      success[ray] = ok ? 1 : 0;
      p[3 * ray] = q.x;
      p[3 * ray + 1] = q.y;
      p[3 * ray + 2] = q.z;
      weight[ray] = ok ? G.sigma_s / G.sigma_t : 1.0f;
      ray = -1;
    }
  }
}

__device__ __forceinline__ void atomic_max_nonneg(float *a, float v) {
  if (v >= 0.0f) atomicMax((int *)a, __float_as_int(v));
}

__global__ void k_grid_max(const float *__restrict__ rho, int64_t nv, float *params) {
  float m = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += (int64_t)gridDim.x * blockDim.x)
    m = fmaxf(m, rho[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  if ((threadIdx.x & 31) == 0) atomic_max_nonneg(params, m);
}

__global__ void k_grid_inv(float *params) {
  // volume.cpp:55: 1.0 / m_maxDensity in double, stored as Float.
  params[1] = (float)(1.0 / (double)params[0]);
}

// One wave of the tracking kernels' blocks (4 per SM by their launch bounds); where
// a warp would own more than kTrackMost rays, blocks of warps of kTrackRays, which
// come in order as others end: neighbouring chunks are under way at the same time,
// so that rays that lie side by side find the grid in L2, and rays that miss the box
// leave no SM idle.  Ratio tracking then also looks whether a warp's rays lie side by
// side (WarpChunk::adapt).  us, one wave -> this (one ray per thread before): 8.3 M
// camera rays through 512^3 ratio tracking 1370 -> 790 (745), adjoint 1222 -> 755
// (955), delta tracking 628 -> 458 (533), through a sparse grid 1721 -> 1574 (2622).
// Scattered rays: 4.2 M through 256^3 271 -> 275 (301), 8.4 M through 100^3 485 -> 470
// (547); warps of 128 rays are as fast there, of 64 lose 4 to 25 %.
constexpr int kTrackMost = 512, kTrackRays = 256;
static bool many_waves(flg_ctx ctx, int64_t n) { return n > (int64_t)ctx->num_sms * 4 * 8 * kTrackMost; }
static unsigned track_blocks(flg_ctx ctx, int64_t n) {
  return many_waves(ctx, n) ? (unsigned)ceil_div(n, 8 * kTrackRays) : grid_for(n, 256, (int64_t)ctx->num_sms * 4);
}

static int vrays(flg_ctx ctx, const flg_rays *r, int64_t n, VRays &V) {
  if (!r) return set_error(ctx, FLG_ERR_ARG, "rays is NULL");
  if (n < 0) return set_error(ctx, FLG_ERR_ARG, "n < 0");
  if (n > 0 && (!r->ox || !r->oy || !r->oz || !r->dx || !r->dy || !r->dz))
    return set_error(ctx, FLG_ERR_ARG, "ray pointer is NULL");
  V = VRays{r->ox, r->oy, r->oz, r->dx, r->dy, r->dz, r->tmax, r->tmax_const};
  return FLG_OK;
}

// Sparse grids.  One CTA of 128 threads per brick; a brick is kept when one
// of its voxels differs from +0 (background), and keeps its slot in brick
// order (k_brick_scan), so the layout is deterministic.
__global__ void k_brick_flags(const float *__restrict__ rho, int nx, int ny, int nz, int bnx, int bny,
                              int32_t *__restrict__ bidx) {
  const int64_t b = blockIdx.x;
  const int bx = (int)(b % bnx), by = (int)((b / bnx) % bny), bz = (int)(b / ((int64_t)bnx * bny));
  int any = 0;
  for (int v = threadIdx.x; v < kBrick * kBrick * kBrick; v += blockDim.x) {
    const int x = bx * kBrick + v % kBrick, y = by * kBrick + (v / kBrick) % kBrick, z = bz * kBrick + v / (kBrick * kBrick);
    if (x < nx && y < ny && z < nz && __float_as_uint(rho[((int64_t)z * ny + y) * nx + x]) != 0u) any = 1;
  }
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) bidx[b] = any;
}

// Exclusive scan of the 0/1 flags into slots (-1 for empty bricks), one CTA.
__global__ void k_brick_scan(int32_t *bidx, int64_t nb, int64_t *count) {
  __shared__ int64_t s_part[1024];
  const int t = threadIdx.x;
  const int64_t per = (nb + blockDim.x - 1) / blockDim.x;
  const int64_t a = t * per, e = min(a + per, nb);
  int64_t c = 0;
  for (int64_t i = a; i < e; ++i) c += bidx[i];
  s_part[t] = c;
  __syncthreads();
  if (t == 0) {
    int64_t run = 0;
    for (int i = 0; i < (int)blockDim.x; ++i) {
      const int64_t x = s_part[i];
      s_part[i] = run;
      run += x;
    }
    *count = run;
  }
  __syncthreads();
  int64_t run = s_part[t];
  for (int64_t i = a; i < e; ++i) {
    const int32_t f = bidx[i];
    bidx[i] = f ? (int32_t)run : -1;
    run += f;
  }
}

__global__ void k_brick_copy(const float *__restrict__ rho, int nx, int ny, int nz, int bnx, int bny,
                             const int32_t *__restrict__ bidx, float *__restrict__ bricks) {
  const int64_t b = blockIdx.x;
  const int32_t slot = bidx[b];
  if (slot < 0) return;
  const int bx = (int)(b % bnx), by = (int)((b / bnx) % bny), bz = (int)(b / ((int64_t)bnx * bny));
  for (int v = threadIdx.x; v < kBrick * kBrick * kBrick; v += blockDim.x) {
    const int x = bx * kBrick + v % kBrick, y = by * kBrick + (v / kBrick) % kBrick, z = bz * kBrick + v / (kBrick * kBrick);
    const float val = (x < nx && y < ny && z < nz) ? rho[((int64_t)z * ny + y) * nx + x] : 0.0f;
    bricks[(int64_t)slot * (kBrick * kBrick * kBrick) + v] = val;
  }
}

}  // namespace flg

using namespace flg;

// Shared by the dense and the sparse constructors: rho holds nv values (the
// dense lattice, or the bricks), over which the majorant is taken.
static int grid_new(flg_ctx ctx, const float *density, int64_t nv, const int32_t *bidx, int64_t n_bricks,
                    int32_t nx, int32_t ny, int32_t nz, const float *lo, const float *hi, const flg_medium *medium,
                    flg_grid *out) {
  if (!ctx || !out) return FLG_ERR_ARG;
  *out = nullptr;
  if (!density || !lo || !hi || !medium) return set_error(ctx, FLG_ERR_ARG, "NULL argument");
  if (nx < 2 || ny < 2 || nz < 2) return set_error(ctx, FLG_ERR_ARG, "grid needs at least 2 samples per axis");
  for (int k = 0; k < 3; ++k)
    if (!(hi[k] > lo[k])) return set_error(ctx, FLG_ERR_ARG, "empty box");
  if (!(medium->sigma_s >= 0.0f) || !(medium->sigma_a >= 0.0f) || !(medium->sigma_s + medium->sigma_a > 0.0f))
    return set_error(ctx, FLG_ERR_ARG, "sigma_s, sigma_a must be >= 0 with a positive sum");
  if (ctx->capturing) return set_error(ctx, FLG_ERR_STATE, "grid creation allocates");
  flg_grid g = new flg_grid_t();
  g->ctx = ctx;
  g->rho = density;
  g->bidx = bidx;
  g->n_bricks = n_bricks;
  g->bnx = (nx + kBrick - 1) / kBrick;
  g->bny = (ny + kBrick - 1) / kBrick;
  g->bnz = (nz + kBrick - 1) / kBrick;
  g->nx = nx;
  g->ny = ny;
  g->nz = nz;
  const int dims[3] = {nx, ny, nz};
  for (int k = 0; k < 3; ++k) {
    g->lo[k] = lo[k];
    g->hi[k] = hi[k];
    g->scale[k] = (float)(dims[k] - 1) / (hi[k] - lo[k]);
  }
  g->medium = *medium;
  g->sigma_t = medium->sigma_a + medium->sigma_s;  // volume.cpp:38
  cudaError_t e = cudaMalloc((void **)&g->d_params, 4 * sizeof(float));
  if (e != cudaSuccess) {
    delete g;
    cudaGetLastError();
    return set_error(ctx, FLG_ERR_OOM, "cudaMalloc failed");
  }
  cudaStream_t st = ctx->stream;
  if (medium->majorant > 0.0f) {
    float prm[4] = {medium->majorant, (float)(1.0 / (double)medium->majorant), 0.0f, 0.0f};
    e = cudaMemcpyAsync(g->d_params, prm, sizeof(prm), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  } else {
    e = cudaMemsetAsync(g->d_params, 0, 4 * sizeof(float), st);
    if (e == cudaSuccess && nv > 0) {
      k_grid_max<<<grid_for(nv, 256, (int64_t)ctx->num_sms * 8), 256, 0, st>>>(density, nv, g->d_params);
      k_grid_inv<<<1, 1, 0, st>>>(g->d_params);
      e = cudaGetLastError();
    }
  }
  if (e != cudaSuccess) {
    cudaFree(g->d_params);
    delete g;
    return cuda_fail(ctx, e, "grid create");
  }
  *out = g;
  return FLG_OK;
}

FLG_API int flg_grid_create(flg_ctx ctx, const float *density, int32_t nx, int32_t ny, int32_t nz,
                            const float *lo, const float *hi, const flg_medium *medium, flg_grid *out) {
  return grid_new(ctx, density, (int64_t)nx * ny * nz, nullptr, 0, nx, ny, nz, lo, hi, medium, out);
}

FLG_API int flg_grid_create_sparse(flg_ctx ctx, const int32_t *brick_index, const float *bricks, int64_t n_bricks,
                                   int32_t nx, int32_t ny, int32_t nz, const float *lo, const float *hi,
                                   const flg_medium *medium, flg_grid *out) {
  if (!ctx) return FLG_ERR_ARG;
  if (!brick_index) return set_error(ctx, FLG_ERR_ARG, "brick_index is NULL");
  if (n_bricks < 0 || (n_bricks > 0 && !bricks)) return set_error(ctx, FLG_ERR_ARG, "bad brick array");
  static const float kNoBricks[1] = {0.0f};  // never read: every slot is -1
  return grid_new(ctx, n_bricks > 0 ? bricks : kNoBricks, n_bricks * kBrick * kBrick * kBrick, brick_index,
                  n_bricks, nx, ny, nz, lo, hi, medium, out);
}

FLG_API int flg_grid_sparsify(flg_ctx ctx, const float *density, int32_t nx, int32_t ny, int32_t nz,
                              int32_t *brick_index, float *bricks, int64_t max_bricks, int64_t *n_bricks) {
  if (!ctx || !n_bricks) return FLG_ERR_ARG;
  if (!density || !brick_index) return set_error(ctx, FLG_ERR_ARG, "NULL argument");
  if (nx < 1 || ny < 1 || nz < 1) return set_error(ctx, FLG_ERR_ARG, "bad grid size");
  if (ctx->capturing) return set_error(ctx, FLG_ERR_STATE, "sparsify reads its count back to the host");
  const int bnx = (nx + kBrick - 1) / kBrick, bny = (ny + kBrick - 1) / kBrick, bnz = (nz + kBrick - 1) / kBrick;
  const int64_t nb = (int64_t)bnx * bny * bnz;
  if (nb > ((int64_t)1 << 31) - 1) return set_error(ctx, FLG_ERR_UNSUPPORTED, "too many bricks");
  cudaStream_t st = ctx->stream;
  int64_t *d_count = nullptr;
  FLG_CUDA(ctx, cudaMalloc((void **)&d_count, sizeof(int64_t)));
  k_brick_flags<<<(unsigned)nb, kBrick * kBrick * kBrick / 4, 0, st>>>(density, nx, ny, nz, bnx, bny, brick_index);
  cudaError_t e = cudaGetLastError();
  ++ctx->launches;
  if (e == cudaSuccess) {
    k_brick_scan<<<1, 1024, 0, st>>>(brick_index, nb, d_count);
    e = cudaGetLastError();
    ++ctx->launches;
  }
  int64_t count = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&count, d_count, sizeof(int64_t), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFree(d_count);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "sparsify");
  *n_bricks = count;
  if (!bricks) return FLG_OK;  // counting call
  if (count > max_bricks) return set_error(ctx, FLG_ERR_ARG, "brick array too small (%lld bricks)", (long long)count);
  k_brick_copy<<<(unsigned)nb, kBrick * kBrick * kBrick / 4, 0, st>>>(density, nx, ny, nz, bnx, bny, brick_index,
                                                                       bricks);
  FLG_LAUNCH_CHECK(ctx, "k_brick_copy");
  return FLG_OK;
}

FLG_API int flg_grid_destroy(flg_grid g) {
  if (!g) return FLG_OK;
  cudaFree(g->d_params);
  delete g;
  return FLG_OK;
}

FLG_API int flg_grid_majorant(flg_grid g, float *maj) {
  if (!g || !maj) return FLG_ERR_ARG;
  cudaError_t e = cudaMemcpyAsync(maj, g->d_params, sizeof(float), cudaMemcpyDeviceToHost, g->ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(g->ctx->stream);
  if (e != cudaSuccess) return cuda_fail(g->ctx, e, "majorant");
  return FLG_OK;
}

FLG_API int flg_volume_tr(flg_ctx ctx, flg_grid grid, const flg_rays *rays, int64_t n, uint64_t seed, float *T,
                          const flg_tr_ckpt *ckpt) {
  if (!ctx || !grid) return FLG_ERR_ARG;
  VRays V;
  int rc = vrays(ctx, rays, n, V);
  if (rc) return rc;
  if (n > 0 && !T) return set_error(ctx, FLG_ERR_ARG, "T is NULL");
  if (ckpt && (!ckpt->t || !ckpt->k || !ckpt->c)) return set_error(ctx, FLG_ERR_ARG, "checkpoint array is NULL");
  if (n == 0) return FLG_OK;
  auto *kern = grid->bidx ? k_volume_tr<true> : k_volume_tr<false>;
  FLG_CUDA(ctx, launch_after(kern, track_blocks(ctx, n), 256, ctx->stream, grid_dev(grid), V, n, seed, T,
                             ckpt ? ckpt->t : nullptr, ckpt ? ckpt->k : nullptr, ckpt ? ckpt->c : nullptr,
                             many_waves(ctx, n)));
  FLG_LAUNCH_CHECK(ctx, "k_volume_tr");
  return FLG_OK;
}

FLG_API int flg_volume_tr_adjoint(flg_ctx ctx, flg_grid grid, const flg_rays *rays, int64_t n, uint64_t seed,
                                  const float *dLdT, const float *T, const flg_tr_ckpt *ckpt, float *grad) {
  if (!ctx || !grid) return FLG_ERR_ARG;
  VRays V;
  int rc = vrays(ctx, rays, n, V);
  if (rc) return rc;
  if (n > 0 && (!dLdT || !T || !grad)) return set_error(ctx, FLG_ERR_ARG, "NULL argument");
  if (ckpt && (!ckpt->t || !ckpt->k)) return set_error(ctx, FLG_ERR_ARG, "checkpoint array is NULL");
  if (n == 0) return FLG_OK;
  auto *kern = grid->bidx ? k_volume_tr_adj<true> : k_volume_tr_adj<false>;
  const int64_t nv = grid->bidx ? grid->n_bricks * kBrick * kBrick * kBrick : (int64_t)grid->nx * grid->ny * grid->nz;
  FLG_CUDA(ctx, launch_after(kern, track_blocks(ctx, n), 256, ctx->stream, grid_dev(grid), V, n, seed, dLdT, T,
                             ckpt ? ckpt->t : nullptr, ckpt ? ckpt->k : nullptr, grad, nv));
  FLG_LAUNCH_CHECK(ctx, "k_volume_tr_adj");
  return FLG_OK;
}

FLG_API int flg_volume_sample(flg_ctx ctx, flg_grid grid, const flg_rays *rays, int64_t n, uint64_t seed,
                              uint8_t *success, float *p, float *weight) {
  if (!ctx || !grid) return FLG_ERR_ARG;
  VRays V;
  int rc = vrays(ctx, rays, n, V);
  if (rc) return rc;
  if (n > 0 && (!success || !p || !weight)) return set_error(ctx, FLG_ERR_ARG, "NULL output");
  if (n == 0) return FLG_OK;
  auto *kern = grid->bidx ? k_volume_sample<true> : k_volume_sample<false>;
  FLG_CUDA(ctx, launch_after(kern, track_blocks(ctx, n), 256, ctx->stream, grid_dev(grid), V, n, seed, success, p, weight));
  FLG_LAUNCH_CHECK(ctx, "k_volume_sample");
  return FLG_OK;
}
