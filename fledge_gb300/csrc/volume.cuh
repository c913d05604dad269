// volume.cuh — device functions of the dense-grid medium shared by the
// volume kernels (volume.cu) and the volumetric path tracer (pathtrace.cu):
// the grid lookup, the box clip, ratio tracking (OpenVDBVolume::tr,
// volume.cpp:75-107), delta tracking (OpenVDBVolume::sample, :109-148) and
// the Henyey-Greenstein phase function (math_utils.h:103-128).
#pragma once

#include "common.cuh"
#include "internal.h"

namespace flg {

// Edge of a sparse grid's bricks (voxels per axis).
constexpr int kBrick = 8;

// Kernel-side grid: dense ([nz][ny][nx], x fastest) or, with bidx, sparse:
// bidx[bz][by][bx] is the slot of an 8^3 brick in rho (z, y, x inside the
// brick, x fastest) or -1 for a brick of background (0) values.
struct GridDev {
  const float *rho;
  int nx, ny, nz;
  float lo[3], hi[3], scale[3];
  float sigma_s, sigma_a, sigma_t, rr;
  const float *params;  // [0] majorant, [1] 1/majorant (double quotient as float)
  const int32_t *bidx;  // sparse bricks, or NULL for a dense grid
  int bnx, bny;
  int64_t layer;  // bricks of a layer
};

// Offset of voxel (x, y, z) in rho, or -1 outside the grid or in an empty
// brick.  SP selects the sparse lookup at compile time, so the dense kernels
// keep their plain index arithmetic.
template <bool SP>
__device__ __forceinline__ int64_t grid_voxel(const GridDev &G, int x, int y, int z) {
  if (x < 0 || y < 0 || z < 0 || x >= G.nx || y >= G.ny || z >= G.nz) return -1;
  if (!SP) return ((int64_t)z * G.ny + y) * G.nx + x;
  const int32_t slot = __ldg(G.bidx + ((int64_t)(z / kBrick) * G.bny + y / kBrick) * G.bnx + x / kBrick);
  if (slot < 0) return -1;
  return (int64_t)slot * (kBrick * kBrick * kBrick) + ((z % kBrick) * kBrick + y % kBrick) * kBrick + x % kBrick;
}

// Density at lattice point (x, y, z), background 0 outside.  The dense path
// tests the bounds before forming the index (as a plain branch around the
// load): routing it through grid_voxel's -1 sentinel cost 25 % of the
// tracking throughput.
template <bool SP>
__device__ __forceinline__ float gat(const GridDev &G, int x, int y, int z) {
  if (x < 0 || y < 0 || z < 0 || x >= G.nx || y >= G.ny || z >= G.nz) return 0.0f;
  if (!SP) return __ldg(G.rho + ((int64_t)z * G.ny + y) * G.nx + x);
  const int64_t o = grid_voxel<true>(G, x, y, z);
  return o < 0 ? 0.0f : __ldg(G.rho + o);
}

__device__ __forceinline__ float lerpf(float a, float b, float w) { return a + (b - a) * w; }

// The eight lattice values around (x, y, z), x fastest.  Almost every lookup
// lies inside the lattice: one bounds test then stands for those of the eight
// points, whose addresses follow from one base (dense), or from the brick slots
// and the offsets of both planes per axis (sparse; seven of the slots are loaded
// only where the cell straddles bricks, which a third of the lookups do: nearly
// every warp has both kinds, and one path for them takes fewer instructions than
// two).
template <bool SP>
__device__ __forceinline__ void grid_cell(const GridDev &G, int x, int y, int z, float (&v)[8]) {
  if ((unsigned)x < (unsigned)(G.nx - 1) && (unsigned)y < (unsigned)(G.ny - 1) && (unsigned)z < (unsigned)(G.nz - 1)) {
    if (!SP) {
      const float *p = G.rho + ((int64_t)z * G.ny + y) * G.nx + x;
      const int64_t sz = (int64_t)G.ny * G.nx;
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = __ldg(p + (c >> 2) * sz + (c >> 1 & 1) * (int64_t)G.nx + (c & 1));
    } else {
      // 64 bits for a brick's index: a table of 2^32 bricks is 17 GB, and fits.  (All
      // indices from one 64-bit offset: 2 M rays 435 us; a pointer per layer 416.)
      const unsigned ox = (unsigned)x % kBrick, oy = (unsigned)y % kBrick, oz = (unsigned)z % kBrick;
      const int32_t *brick = G.bidx + ((unsigned)z / kBrick * G.layer +
                                       ((int64_t)((unsigned)y / kBrick) * G.bnx + (unsigned)x / kBrick));
      // brick step and offset in the brick of the upper plane of each axis
      const bool nx = ox == kBrick - 1, ny = oy == kBrick - 1, nz = oz == kBrick - 1;
      const uint32_t sx = nx, sy = ny ? G.bnx : 0;
      const int32_t *upper = nz ? brick + G.layer : brick;
      const uint32_t ux = nx ? 0 : ox + 1, uy = (ny ? 0 : oy + 1) * kBrick, uz = (nz ? 0 : oz + 1) * kBrick * kBrick;
      const uint32_t ly = oy * kBrick, lz = oz * kBrick * kBrick;
      int32_t slot[8];
      slot[0] = __ldg(brick);
#pragma unroll
      for (int c = 1; c < 8; ++c)
        slot[c] = ((c & 1) && nx) || ((c & 2) && ny) || ((c & 4) && nz)
                      ? __ldg((c & 4 ? upper : brick) + ((c & 2 ? sy : 0) + (c & 1 ? sx : 0)))
                      : slot[0];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float *p = G.rho + ((c & 4 ? uz : lz) + (c & 2 ? uy : ly) + (c & 1 ? ux : ox));
        v[c] = slot[c] < 0 ? 0.0f : __ldg(p + (int64_t)slot[c] * (kBrick * kBrick * kBrick));
      }
    }
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = gat<SP>(G, x + (c & 1), y + (c >> 1 & 1), z + (c >> 2));
  }
}

template <bool SP>
__device__ __forceinline__ float sample_grid(const GridDev &G, float px, float py, float pz, int &x, int &y, int &z,
                                             float &fx, float &fy, float &fz) {
  float gx = (px - G.lo[0]) * G.scale[0];
  float gy = (py - G.lo[1]) * G.scale[1];
  float gz = (pz - G.lo[2]) * G.scale[2];
  float x0 = floorf(gx), y0 = floorf(gy), z0 = floorf(gz);
  x = (int)x0;
  y = (int)y0;
  z = (int)z0;
  fx = gx - x0;
  fy = gy - y0;
  fz = gz - z0;
  float v[8];
  grid_cell<SP>(G, x, y, z, v);
  float c00 = lerpf(v[0], v[1], fx);
  float c10 = lerpf(v[2], v[3], fx);
  float c01 = lerpf(v[4], v[5], fx);
  float c11 = lerpf(v[6], v[7], fx);
  float c0 = lerpf(c00, c10, fy);
  float c1 = lerpf(c01, c11, fy);
  return lerpf(c0, c1, fz);
}

// AABB::intersect_pbrt (common/aabb.h:38-59) with t1 starting at tMax.
__device__ __forceinline__ bool box_pbrt(const GridDev &G, const float3 &o, const float3 &d, float tmax, float &t0o,
                                         float &t1o) {
  float t0 = 0.0f, t1 = tmax;
  const float oo[3] = {o.x, o.y, o.z}, dd[3] = {d.x, d.y, d.z};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    float inv = __frcp_rn(dd[i]);
    float tn = (G.lo[i] - oo[i]) * inv;
    float tf = (G.hi[i] - oo[i]) * inv;
    bool s = tn > tf;
    float a = s ? tf : tn, b = s ? tn : tf;
    t0 = a > t0 ? a : t0;
    t1 = b < t1 ? b : t1;
    if (t0 > t1) return false;
  }
  t0o = t0;
  t1o = t1;
  return true;
}

// What the trackers keep of a ray.  They work in turns of a Philox block's four
// draws, so that the lanes of a warp compute their blocks together: drawn one
// by one, some lane of every warp needs a new block at every step.
struct TrackState {
  float3 o, d;
  float t, t_max;
  uint32_t k;  // draws taken
  int steps;
  int64_t ray;

  // The block of draw k.
  __device__ __forceinline__ uint4 block(uint64_t seed) const {
    return philox4x32_10(make_uint4(k >> 2, (uint32_t)ray, (uint32_t)((uint64_t)ray >> 32), 0x7e5u), (uint32_t)seed,
                         (uint32_t)(seed >> 32));
  }
  // False if the ray misses the grid's box.
  __device__ __forceinline__ bool start(const GridDev &G, float tmax) {
    float t_min;
    k = 0u;
    steps = 0;
    if (!box_pbrt(G, o, d, tmax, t_min, t_max)) return false;
    t = fmaxf(t_min, 0.0f);
    t_max = fminf(t_max, tmax);
    return true;
  }
};

__device__ __forceinline__ float free_path(uint32_t x, float max_mu) { return -flg_logf(1.0f - u01(x)) / max_mu; }

// Ratio tracking of one ray, a step at a time: T so far in tr, and the state
// after the last roulette survival (the adjoint's checkpoint).
struct RatioState {
  float3 o, d;
  float t, t_max, tr;
  float ck_t, ck_c;
  uint32_t ck_k;
  RayStream rs;
};

// False if the ray misses the grid's box (T = 1).
__device__ __forceinline__ bool ratio_start(const GridDev &G, RatioState &s, float tmax, uint64_t seed, int64_t ray) {
  s.ck_t = 0.0f;
  s.ck_k = 0u;
  s.ck_c = 1.0f;
  s.tr = 1.0f;
  float t_min;
  if (!box_pbrt(G, s.o, s.d, tmax, t_min, s.t_max)) return false;
  s.t = fmaxf(t_min, 0.0f);
  s.t_max = fminf(s.t_max, tmax);
  s.rs.init(seed, (uint64_t)ray, 0u);
  s.ck_t = s.t;
  return true;
}

// One step; false once the ray has left the box or been absorbed.
template <bool SP>
__device__ __forceinline__ bool ratio_step(const GridDev &G, float max_mu, float inv_maj, RatioState &s) {
  const float u = s.rs.next();
  s.t += -flg_logf(1.0f - u) / max_mu;
  if (s.t >= s.t_max) return false;
  int x, y, z;
  float fx, fy, fz;
  const float dens =
      sample_grid<SP>(G, s.o.x + s.d.x * s.t, s.o.y + s.d.y * s.t, s.o.z + s.d.z * s.t, x, y, z, fx, fy, fz);
  s.tr *= 1.0f - fmaxf(0.0f, dens * inv_maj);
  if (s.tr < G.rr) {
    const float q = fmaxf(0.05f, 1.0f - s.tr);
    if (s.rs.next() < q) {
      s.tr = 0.0f;
      return false;
    }
    s.tr /= 1.0f - q;
    s.ck_t = s.t;
    s.ck_k = s.rs.k;
    s.ck_c = s.tr;
  }
  return true;
}

template <bool SP>
__device__ __forceinline__ float ratio_track(const GridDev &G, float maj, float inv_maj, const float3 &o,
                                             const float3 &d, float tmax, uint64_t seed, int64_t ray, float &ck_t,
                                             uint32_t &ck_k, float &ck_c) {
  RatioState s;
  s.o = o;
  s.d = d;
  if (ratio_start(G, s, tmax, seed, ray)) {
    const float max_mu = G.sigma_t * maj;
    for (int step_ = 0; step_ < kMaxTrackSteps; ++step_)
      if (!ratio_step<SP>(G, max_mu, inv_maj, s)) break;
  }
  ck_t = s.ck_t;
  ck_k = s.ck_k;
  ck_c = s.ck_c;
  return s.tr;
}

// Kernel-side view of a grid handle.
inline GridDev grid_dev(flg_grid g) {
  GridDev G;
  G.rho = g->rho;
  G.nx = g->nx;
  G.ny = g->ny;
  G.nz = g->nz;
  for (int k = 0; k < 3; ++k) {
    G.lo[k] = g->lo[k];
    G.hi[k] = g->hi[k];
    G.scale[k] = g->scale[k];
  }
  G.sigma_s = g->medium.sigma_s;
  G.sigma_a = g->medium.sigma_a;
  G.sigma_t = g->sigma_t;
  G.rr = g->medium.rr_threshold;
  G.params = g->d_params;
  G.bidx = g->bidx;
  G.bnx = g->bnx;
  G.bny = g->bny;
  G.layer = (int64_t)g->bnx * g->bny;
  return G;
}

// One turn of delta tracking (volume.cpp:109-148): two steps, each with one
// uniform for its free path and one for its collision test.  1: a real
// collision (its position in p), -1: out of the box, 0: go on.
template <bool SP>
__device__ __forceinline__ int delta_turn(const GridDev &G, float max_mu, uint64_t seed, TrackState &s, float3 &p) {
  const uint4 b = s.block(seed);  // k is a multiple of 4
  s.k += 4u;
#pragma unroll
  for (int w = 0; w < 4; w += 2) {
    s.t += free_path(w ? b.z : b.x, max_mu);
    if (s.t >= s.t_max) return -1;
    const float qx = s.o.x + s.d.x * s.t, qy = s.o.y + s.d.y * s.t, qz = s.o.z + s.d.z * s.t;
    int x, y, z;
    float fx, fy, fz;
    const float dens = sample_grid<SP>(G, qx, qy, qz, x, y, z, fx, fy, fz);
    const float p_s = G.sigma_s * dens / max_mu;
    const float p_a = G.sigma_a * dens / max_mu;
    const float p_n = 1.0f - p_s - p_a;
    if (u01(w ? b.w : b.y) > p_n) {
      p = make_float3(qx, qy, qz);
      return 1;
    }
    if (++s.steps >= kMaxTrackSteps) return -1;
  }
  return 0;
}

template <bool SP>
__device__ __forceinline__ bool delta_track(const GridDev &G, float maj, const float3 &o, const float3 &d,
                                            float tmax, uint64_t seed, int64_t ray, float3 &p) {
  TrackState s;
  s.o = o;
  s.d = d;
  s.ray = ray;
  int r = -1;
  if (s.start(G, tmax)) {
    const float max_mu = G.sigma_t * maj;
    do r = delta_turn<SP>(G, max_mu, seed, s, p);
    while (r == 0);
  }
  return r == 1;
}

// Henyey-Greenstein phase function HGP(wi, wo, g) (math_utils.h:103-107).
__device__ __forceinline__ float hg_p(const float3 &wi, const float3 &wo, float g) {
  const float cos_theta = wi.x * wo.x + wi.y * wo.y + wi.z * wo.z;
  const float denom = 1.0f + g * g + 2.0f * g * cos_theta;
  return (1.0f - g * g) / (denom * sqrtf(denom)) * 0.07957747154594766788f;
}

// HGSampleP (math_utils.h:111-128): direction wi around wo for uniforms u, v,
// in the frame of CoordinateSystem(wo) (math_utils.h:57-66).
__device__ __forceinline__ float3 hg_sample(const float3 &wo, float u, float v, float g) {
  float cos_theta;
  if (fabsf(g) < 1e-3f) {
    cos_theta = 1.0f - 2.0f * u;
  } else {
    const float tmp = (1.0f - g * g) / (1.0f + g - 2.0f * g * u);
    cos_theta = -(1.0f + g * g - tmp * tmp) / (2.0f * g);
  }
  const float phi = 2.0f * 3.14159265358979f * v;
  const float sin_theta = sqrtf(fmaxf(0.0f, 1.0f - cos_theta * cos_theta));
  float3 v1;
  if (fabsf(wo.x) > fabsf(wo.y)) {
    const float l = sqrtf(wo.x * wo.x + wo.z * wo.z);
    v1 = make_float3(-wo.z / l, 0.0f, wo.x / l);
  } else {
    const float l = sqrtf(wo.y * wo.y + wo.z * wo.z);
    v1 = make_float3(0.0f, wo.z / l, -wo.y / l);
  }
  const float3 v2 = make_float3(wo.y * v1.z - wo.z * v1.y, wo.z * v1.x - wo.x * v1.z, wo.x * v1.y - wo.y * v1.x);
  const float a = sin_theta * cosf(phi), b = sin_theta * sinf(phi);
  return make_float3(a * v1.x + b * v2.x + cos_theta * wo.x, a * v1.y + b * v2.y + cos_theta * wo.y,
                     a * v1.z + b * v2.z + cos_theta * wo.z);
}

// Philox stream of one tracking call of the volumetric path tracer: pixel,
// sample, bounce and purpose (0: free-flight sampling along the path,
// 1: transmittance of the shadow ray).
__device__ __host__ __forceinline__ uint64_t path_stream_id(int64_t pix, int s, int depth, int purpose) {
  return (uint64_t)pix | ((uint64_t)s << 26) | ((uint64_t)depth << 42) | ((uint64_t)purpose << 50);
}

}  // namespace flg
