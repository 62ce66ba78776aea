// Voxel-SDF path: bake a field into a grid, the .rsdf file format, and
// sphere tracing of the sampled grid at three quality levels.
//
// Replaces, in the reference (hadalhw17/RayEngine, "RE/" = RayEngine/src/):
//   generate_noise (bake)   RE/cuda-src/renderer.cu:106-126,813-836
//   .rsdf read / write      RE/World/Grid.cpp:23-64, renderer.cu:839-870
//                           (int dim[3], float spacing[3], then float2
//                           {distance, material} per voxel, x fastest)
//   get_distance            RE/cuda-src/sdf_functions.cuh:394-419 with
//     LOW    nearest voxel                       (tex3D point lookup)
//     MEDIUM trilinear between voxels            (interpolate, :231-262)
//     HIGH   tricubic B-spline, 64 voxels        (cubicTex3DSimple, :296-329)
//
// Grid coordinates: u = (p - origin) / spacing per axis; voxel (i, j, k)
// holds the field at origin + (i, j, k) * spacing.  Lookups outside the grid
// clamp to the edge voxels (the reference's texture uses a zero border,
// which reads as a surface along the grid boundary).  The reference's
// texture fetches filter in hardware (linear mode with 8-bit weights); here
// every lookup reads exact voxel values and blends in FP32 with the
// reference's formulas, so results are reproducible on the CPU.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "re_common.hpp"
#include "re_math.cuh"
#include "re_noise.cuh"

namespace re {
namespace voxel {

struct GridDev {
  const float2* __restrict__ v;
  int dim[3];
  float spacing[3], origin[3];
};

__device__ __forceinline__ int clampi(int v, int dim) { return min(max(v, 0), dim - 1); }

__device__ __forceinline__ const float2* voxel_row(const GridDev& g, int y, int z) {
  return g.v + (size_t)g.dim[0] * ((size_t)y + (size_t)g.dim[1] * z);
}

// x / 6 for x in [0, 1] (zero or at least 2^-69 here): the product with the
// rounded reciprocal, corrected once by its exact remainder, is the rounded
// quotient (Markstein 1990, division by a constant with fused multiply-add;
// compared with the division over every mantissa).
__device__ __forceinline__ float sixth(float x) {
  const float y = 1.0f / 6.0f, q = x * y;
  return __fmaf_rn(__fmaf_rn(-6.0f, q, x), y, q);
}

// The cubic B-spline at -1 - f, -f, 1 - f and 2 - f for a fraction f in
// [0, 1]: with t its argument's magnitude and a = 2 - t, 2/3 - t^2 a / 2
// below 1 and a^3 / 6 from 1 to 2.  The outer two are always in the second
// range, the inner two in the first or at t = 1.  A NaN fraction (a lookup
// at an infinite coordinate) has no weight anywhere.
__device__ __forceinline__ void bspline4(float f, float (&w)[4]) {
  const float t0 = fabsf(-1.0f - f), t1 = fabsf(f), t2 = fabsf(1.0f - f), t3 = fabsf(2.0f - f);
  const float a0 = 2.0f - t0, a1 = 2.0f - t1, a2 = 2.0f - t2, a3 = 2.0f - t3;
  const bool some = f >= 0.0f;
  w[0] = some ? sixth(a0 * a0 * a0) : 0.0f;
  w[1] = some ? (t1 < 1.0f ? 2.0f / 3.0f - 0.5f * t1 * t1 * a1 : 1.0f / 6.0f) : 0.0f;
  w[2] = some ? (t2 < 1.0f ? 2.0f / 3.0f - 0.5f * t2 * t2 * a2 : 1.0f / 6.0f) : 0.0f;
  w[3] = some ? sixth(a3 * a3 * a3) : 0.0f;
}

__device__ __forceinline__ float bilerp(float tx, float ty, float c00, float c10, float c01,
                                        float c11) {
  return (1.0f - tx) * (1.0f - ty) * c00 + tx * (1.0f - ty) * c10 + (1.0f - tx) * ty * c01 +
         tx * ty * c11;
}

// Lookup at p.  The clamped indices are found once per axis, and a cell
// whose N x N x N voxels (2 or 4 a side) all lie inside the grid is read
// through one pointer and the two strides, each row with constant offsets.
// The arithmetic is the plain form's: weights bx (by bz), products added in
// x, y, z order.
// Measured on B200 (one edit and the 1280x720 frame of a 192x96x192 grid at
// HIGH, with k_trace_high and k_brush below): 2.40 -> 0.81 ms; each of the 64
// lookups had taken its own three clamps, 64-bit index and three B-spline
// evaluations.
// WARP: all 32 lanes call it, and one whose cell reaches past the grid takes
// the others with it: of points in no order nearly every warp would run both
// paths.  2,000,000 points about and in a 32^3 grid at HIGH 195 -> 166 us (each
// lookup with its own 64 clamps, as it was, 170), MEDIUM 30.8 -> 28.8.
template <uint32_t Q, bool WARP = false>
__device__ __forceinline__ float sample(const GridDev& g, V3 p) {
  const float u[3] = {(p.x - g.origin[0]) / g.spacing[0], (p.y - g.origin[1]) / g.spacing[1],
                      (p.z - g.origin[2]) / g.spacing[2]};
  if (Q == RE_VOXEL_LOW) {
    const int x = clampi(__float2int_rd(u[0]), g.dim[0]),
              y = clampi(__float2int_rd(u[1]), g.dim[1]),
              z = clampi(__float2int_rd(u[2]), g.dim[2]);
    return __ldg(&voxel_row(g, y, z)[x].x);
  }
  constexpr int N = Q == RE_VOXEL_MEDIUM ? 2 : 4;
  constexpr int kFirst = Q == RE_VOXEL_MEDIUM ? 0 : -1;
  // HIGH: B-spline weights about the voxel below u - 0.5
  constexpr float kShift = Q == RE_VOXEL_MEDIUM ? 0.0f : 0.5f;
  float fr[3];
  int c[3];  // the lowest voxel of the cell
  bool inside = true;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float cg = Q == RE_VOXEL_MEDIUM ? u[k] : u[k] - kShift;
    fr[k] = cg - floorf(cg);
    // kept near the grid before any offset is added: a coordinate beyond the
    // integers converts to the largest one, and adding to that would wrap
    // past the clamps below
    c[k] = min(max(__float2int_rd(cg), -N), g.dim[k] + N) + kFirst;
    inside = inside && c[k] >= 0 && c[k] <= g.dim[k] - N;
  }
  if (WARP) inside = __all_sync(0xFFFFFFFFu, inside);
  // v(x, y, z) of the cell, x innermost; rows by pointer
  float w[3][4];
  if (Q == RE_VOXEL_HIGH) {
#pragma unroll
    for (int k = 0; k < 3; ++k) bspline4(fr[k], w[k]);
  }
  float result = 0.0f, ef[2] = {0.0f, 0.0f};
  auto layer = [&](int z, auto row) {  // row(y, x): voxel (x, y) of layer z
    if (Q == RE_VOXEL_MEDIUM) {
      ef[z] = bilerp(fr[0], fr[1], row(0, 0), row(0, 1), row(1, 0), row(1, 1));
    } else {
      // rows y and y + 1 in the halves of packed registers, added one after
      // the other
#pragma unroll
      for (int y = 0; y < N; y += 2) {
        const f32x2 byz = mul2(pack2(w[1][y], w[1][y + 1]), pack2(w[2][z], w[2][z]));
        float lo[N], hi[N];
#pragma unroll
        for (int x = 0; x < N; ++x)
          unpack2(mul2(mul2(pack2(w[0][x], w[0][x]), byz), pack2(row(y, x), row(y + 1, x))), lo[x],
                  hi[x]);
#pragma unroll
        for (int x = 0; x < N; ++x) result = __fadd_rn(result, lo[x]);
#pragma unroll
        for (int x = 0; x < N; ++x) result = __fadd_rn(result, hi[x]);
      }
    }
  };
  if (inside) {
    const float2* base = voxel_row(g, c[1], c[2]) + c[0];
    const size_t sy = (size_t)g.dim[0], sz = sy * (size_t)g.dim[1];
#pragma unroll
    for (int z = 0; z < N; ++z)
      layer(z, [&](int y, int x) { return __ldg(&(base + z * sz + y * sy)[x].x); });
  } else {
    int xs[N], ys[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      xs[i] = clampi(c[0] + i, g.dim[0]);
      ys[i] = clampi(c[1] + i, g.dim[1]);
    }
#pragma unroll
    for (int z = 0; z < N; ++z) {
      const int zc = clampi(c[2] + z, g.dim[2]);
      layer(z, [&](int y, int x) { return __ldg(&voxel_row(g, ys[y], zc)[xs[x]].x); });
    }
  }
  if (Q == RE_VOXEL_MEDIUM) return ef[0] * (1.0f - fr[2]) + ef[1] * fr[2];
  return result;
}

// Whether a grid of n voxels is baked on the rows: their 128 KB take 2 us more
// to fill than the copies, and a single octave past an even number costs a
// pair.  Measured on B200, copies | rows, us: 8 octaves 32^3 8.3 | 10.3, 48^3
// 12.4 | 12.4, 64^3 18.6 | 16.5; 4 octaves 48^3 8.4 | 10.4, 64^3 12.4 | 12.4; 5
// octaves 128^3 65.7 | 65.7; 3 octaves 128^3 47.2 | 49.3, 256^3 332 | 331; one
// octave 256^3 176 | 212.
inline bool bake_on_rows(uint32_t octaves, uint64_t n) {
  const bool odd = octaves < 7u && octaves % 2u != 0u;
  return octaves > 1u && n >= (odd ? 1u << 22 : 200000u);
}

template <class FORM>
__global__ void __launch_bounds__(FORM::kThreads) k_bake(PermTable perm, uint32_t octaves,
                                                         float scale, float amp, GridDev g,
                                                         float2* __restrict__ out) {
  extern __shared__ uint32_t rows_smem[];
  const auto P = FORM::load(perm, rows_smem);
  size_t n = (size_t)g.dim[0] * g.dim[1] * g.dim[2];
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    uint32_t x = (uint32_t)(i % g.dim[0]), y = (uint32_t)((i / g.dim[0]) % g.dim[1]),
             z = (uint32_t)(i / ((size_t)g.dim[0] * g.dim[1]));
    V3 p = v3(__fmaf_rn((float)x, g.spacing[0], g.origin[0]), __fmaf_rn((float)y, g.spacing[1], g.origin[1]),
              __fmaf_rn((float)z, g.spacing[2], g.origin[2]));
    out[i] = make_float2(terrain_density(P, p, octaves, scale, amp), 0.0f);
  }
}

template <uint32_t Q>
__global__ void __launch_bounds__(256) k_sample(GridDev g, const float* __restrict__ pts,
                                                uint32_t n, float* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const size_t at = 3 * (size_t)min(i, n - 1u);  // past the last point: its value, not stored
  const float v = sample<Q, true>(g, v3(pts[at], pts[at + 1], pts[at + 2]));
  if (i < n) out[i] = v;
}

struct MarchDev {
  float step_factor, eps, tmax;
  uint32_t max_steps;
};

// Sphere tracing of the sampled grid inside its box (the box holds the
// voxel centres, origin .. origin + (dim - 1) spacing): the exact tracer's
// rule t += step_factor * d, hit when d < eps; normal by central
// differences with delta = half the smallest spacing.  Output as re_sdf_hit.

// The ray of pixel (x, y) and its span [t0, t1) in the box.
__device__ __forceinline__ void grid_ray(const GridDev& g, const MarchDev& m, const CamDev& cam,
                                         uint32_t w, uint32_t h, uint32_t x, uint32_t y, V3& o,
                                         V3& d, float& t0, float& t1) {
  generate_ray(cam, w, h, x, y, o, d);
  const float o3[3] = {o.x, o.y, o.z}, d3[3] = {d.x, d.y, d.z};
  t0 = 0.0f;
  t1 = m.tmax;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float lo = g.origin[k], hi = __fmaf_rn((float)(g.dim[k] - 1), g.spacing[k], g.origin[k]);
    float inv = 1.0f / d3[k];
    float ta = (lo - o3[k]) * inv, tb = (hi - o3[k]) * inv;
    t0 = fmaxf(t0, fminf(ta, tb));
    t1 = fminf(t1, fmaxf(ta, tb));
  }
}

// n: the differences along the axes (hits only).
__device__ __forceinline__ void store_record(float4* out, uint32_t pix, V3 p, V3 n,
                                             uint32_t steps, uint32_t status) {
  float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0;
  if (status == 1) {
    n = normalize(n);
    r0 = make_float4(p.x, p.y, p.z, n.x);
    r1 = make_float4(n.y, n.z, 0.f, 0.f);
  }
  r1.z = __uint_as_float(steps);
  r1.w = __uint_as_float(status);
  out[2 * (size_t)pix] = r0;
  out[2 * (size_t)pix + 1] = r1;
}

// LOW and MEDIUM, a thread per pixel: the march, then the six lookups of the
// normal side by side (their loads overlap; one after another as below they
// took a 160x90 frame from 78 to 110 us).
template <uint32_t Q>
__global__ void __launch_bounds__(256) k_trace_pixel(GridDev g, MarchDev m, CamDev cam, uint32_t w,
                                                     uint32_t h, float4* __restrict__ out) {
  const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= w * h) return;
  V3 o, d, p = {0.f, 0.f, 0.f}, n = p;
  float t, t1;
  grid_ray(g, m, cam, w, h, pix % w, pix / w, o, d, t, t1);
  uint32_t steps = 0, status = 0;
  if (t < t1) {
    for (;;) {
      p = v3(__fmaf_rn(t, d.x, o.x), __fmaf_rn(t, d.y, o.y), __fmaf_rn(t, d.z, o.z));
      const float v = sample<Q>(g, p);
      ++steps;
      if (v < m.eps) {
        status = 1;
        break;
      }
      t = __fmaf_rn(m.step_factor, v, t);
      if (t > t1) break;
      if (steps >= m.max_steps) {
        status = 2;
        break;
      }
    }
  }
  if (status == 1) {
    const float e = 0.5f * fminf(g.spacing[0], fminf(g.spacing[1], g.spacing[2]));
    n.x = sample<Q>(g, v3(p.x + e, p.y, p.z)) - sample<Q>(g, v3(p.x - e, p.y, p.z));
    n.y = sample<Q>(g, v3(p.x, p.y + e, p.z)) - sample<Q>(g, v3(p.x, p.y - e, p.z));
    n.z = sample<Q>(g, v3(p.x, p.y, p.z + e)) - sample<Q>(g, v3(p.x, p.y, p.z - e));
  }
  store_record(out, pix, p, n, steps, status);
}

// HIGH, a per-lane state machine with one lookup per trip (phase 0 marches,
// phases 1..6 are the normal's taps), so rays that hit early take their taps
// while others march, and the long lookup is in the code once.  A warp takes
// its next 8x4 pixel tile when all its rays have ended: the loads bound it
// (64 a lookup, L1 74 % busy), and lanes of one tile read the same few
// voxels, which lanes refilled from another do not (measured, frame above:
// next pixels at 8 idle lanes 906 us, at 24 861, at 32 808; 2 blocks an SM
// 803, 4 972).  A block owns the tiles blockIdx, blockIdx + gridDim, ...; its
// warps claim them from a counter in shared memory.
__global__ void __launch_bounds__(256) k_trace_high(GridDev g, MarchDev m, CamDev cam, uint32_t w,
                                                    uint32_t h, float4* __restrict__ out) {
  __shared__ uint32_t cursor;
  if (threadIdx.x == 0) cursor = 0u;
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t tiles_x = (w + 7) / 8, tiles = tiles_x * ((h + 3) / 4);
  const uint32_t mine = (tiles - blockIdx.x + gridDim.x - 1u) / gridDim.x;  // grid <= tiles
  const float delta = 0.5f * fminf(g.spacing[0], fminf(g.spacing[1], g.spacing[2]));
  bool live = false;
  uint32_t pix = 0, steps = 0, phase = 0;
  V3 o = {0.f, 0.f, 0.f}, d = {0.f, 0.f, 1.f}, p = o, n = o;
  float t = 0.f, t1 = 0.f, plus = 0.f;
  for (;;) {
    if (__ballot_sync(0xFFFFFFFFu, live) == 0u) {
      uint32_t k = 0;
      if (lane == 0) k = atomicAdd(&cursor, 1u);
      k = __shfl_sync(0xFFFFFFFFu, k, 0);
      if (k >= mine) break;
      const uint32_t tile = blockIdx.x + k * gridDim.x;
      const uint32_t x = (tile % tiles_x) * 8 + (lane & 7u),
                     y = (tile / tiles_x) * 4 + (lane >> 3);
      if (x < w && y < h) {
        grid_ray(g, m, cam, w, h, x, y, o, d, t, t1);
        pix = y * w + x;
        steps = 0;
        phase = 0;
        live = t < t1;
        if (!live) store_record(out, pix, p, n, 0u, 0u);  // the ray passes the grid by
      }
    }
    if (!live) continue;
    V3 q;
    if (phase == 0) {
      q = v3(__fmaf_rn(t, d.x, o.x), __fmaf_rn(t, d.y, o.y), __fmaf_rn(t, d.z, o.z));
    } else {
      const float sd = (phase & 1u) ? delta : -delta;
      q = p;
      if (phase <= 2) q.x = p.x + sd;
      else if (phase <= 4) q.y = p.y + sd;
      else q.z = p.z + sd;
    }
    const float v = sample<RE_VOXEL_HIGH>(g, q);
    uint32_t status = 3;  // 3 = keep going
    if (phase == 0) {
      ++steps;
      if (v < m.eps) {
        p = q;
        phase = 1;
      } else {
        t = __fmaf_rn(m.step_factor, v, t);
        if (t > t1) status = 0;
        else if (steps >= m.max_steps) status = 2;
      }
    } else {
      if (phase & 1u) {
        plus = v;
      } else {
        const float diff = plus - v;
        if (phase == 2) n.x = diff;
        else if (phase == 4) n.y = diff;
        else n.z = diff;
      }
      if (phase == 6) status = 1;
      else ++phase;
    }
    if (status != 3) {
      store_record(out, pix, p, n, steps, status);
      live = false;
    }
  }
}

// Brush edit of every voxel (insert_sphere_to_texture, renderer.cu:31-92):
// q = voxel position - centre; SPHERE_ADD smooth union (sdf_smin, k),
// SPHERE_SUBTRACT max(v, -sphere), CUBE_ADD component-wise min of the
// {distance, material} pairs (as the reference's fminf on float2),
// CUBE_SUBTRACT max(v, -box); sphere = |q| - r, box as aabb_distance
// (sdf_functions.cuh:424-436).
__device__ __forceinline__ float len3(float x, float y, float z) { return sqrtf(x * x + y * y + z * z); }

__global__ void __launch_bounds__(256) k_brush(GridDev g, uint32_t type, float cx, float cy, float cz, float ex, float ey,
                        float ez, float mat, float k, float2* __restrict__ v) {
  // at most 2^31 voxels: 32-bit indices, two divisions a voxel
  const uint32_t nx = (uint32_t)g.dim[0], ny = (uint32_t)g.dim[1], n = nx * ny * (uint32_t)g.dim[2];
#pragma unroll 4
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t yz = i / nx, x = i - yz * nx, z = yz / ny, y = yz - z * ny;
    float qx = __fmaf_rn((float)x, g.spacing[0], g.origin[0]) - cx;
    float qy = __fmaf_rn((float)y, g.spacing[1], g.origin[1]) - cy;
    float qz = __fmaf_rn((float)z, g.spacing[2], g.origin[2]) - cz;
    float2 a = v[i], r = a;
    if (type == RE_BRUSH_SPHERE_ADD || type == RE_BRUSH_SPHERE_SUBTRACT) {
      float sd = len3(qx, qy, qz) - ex;
      if (type == RE_BRUSH_SPHERE_ADD) {
        float h = fmaxf(k - fabsf(a.x - sd), 0.0f) / k;
        float2 m = a.x < sd ? a : make_float2(sd, mat);
        float c = h * h * k * 0.25f;
        r = make_float2(m.x - c, m.y);
      } else {
        r = a.x > -sd ? a : make_float2(-sd, mat);
      }
    } else {
      float dx = fabsf(qx) - ex, dy = fabsf(qy) - ey, dz = fabsf(qz) - ez;
      float bd = len3(fmaxf(dx, 0.0f), fmaxf(dy, 0.0f), fmaxf(dz, 0.0f)) +
                 fminf(fmaxf(dx, fmaxf(dy, dz)), 0.0f);
      if (type == RE_BRUSH_CUBE_ADD) r = make_float2(fminf(a.x, bd), fminf(a.y, mat));
      else r = a.x > -bd ? a : make_float2(-bd, mat);
    }
    // an untouched voxel is not written: most of an edit's traffic is the read
    if (__float_as_uint(r.x) != __float_as_uint(a.x) || __float_as_uint(r.y) != __float_as_uint(a.y))
      v[i] = r;
  }
}

}  // namespace voxel
}  // namespace re

namespace re {
namespace {

re_status check_grid(const re_voxel_grid* g, const char* fn) {
  if (!g) return fail(RE_ERR_INVALID_ARG, "%s: null grid", fn);
  for (int k = 0; k < 3; ++k) {
    if (g->dim[k] < 2 || g->dim[k] > 4096) return fail(RE_ERR_INVALID_ARG, "%s: dim out of [2, 4096]", fn);
    if (!(g->spacing[k] > 0.f)) return fail(RE_ERR_INVALID_ARG, "%s: spacing must be > 0", fn);
  }
  if ((uint64_t)g->dim[0] * g->dim[1] * g->dim[2] > (1ull << 31))
    return fail(RE_ERR_LIMIT, "%s: more than 2^31 voxels", fn);
  return RE_OK;
}

voxel::GridDev grid_dev(const re_voxel_grid* g, const float* d_grid) {
  voxel::GridDev d;
  d.v = reinterpret_cast<const float2*>(d_grid);
  for (int k = 0; k < 3; ++k) {
    d.dim[k] = (int)g->dim[k];
    d.spacing[k] = g->spacing[k];
    d.origin[k] = g->origin[k];
  }
  return d;
}

CamDev cam_of_voxel(const re_camera& c) {
  CamBasis b;
  camera_basis(c, b);
  CamDev d;
  d.campos = {b.campos[0], b.campos[1], b.campos[2]};
  d.middle = {b.middle[0], b.middle[1], b.middle[2]};
  d.horizontal = {b.horizontal[0], b.horizontal[1], b.horizontal[2]};
  d.vertical = {b.vertical[0], b.vertical[1], b.vertical[2]};
  d.focal = b.focal;
  return d;
}

}  // namespace
}  // namespace re

extern "C" {

RE_API re_status re_voxel_bake(const re_sdf_params* field, const re_voxel_grid* g, float* d_grid,
                               void* stream) {
  re_status st = re::check_grid(g, "re_voxel_bake");
  if (st != RE_OK) return st;
  if (!field || !d_grid || field->octaves < 1 || field->octaves > 16)
    return re::fail(RE_ERR_INVALID_ARG, "re_voxel_bake: bad arguments");
  uint32_t full[512];
  re::perlin_permutation(field->seed, full);
  re::PermTable t;
  for (int i = 0; i < 512; ++i) t.p[i] = (uint8_t)full[i];
  const uint64_t n = (uint64_t)g->dim[0] * g->dim[1] * g->dim[2];
  const bool rows = re::voxel::bake_on_rows(field->octaves, n);
  auto k = rows ? re::voxel::k_bake<re::RowsForm> : re::voxel::k_bake<re::CopyForm>;
  const uint32_t threads = rows ? re::RowsForm::kThreads : re::CopyForm::kThreads;
  const uint32_t smem = rows ? re::RowsForm::kBytes : re::CopyForm::kBytes;
  RE_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k<<<(rows ? 1 : 2) * re::sm_count(), threads, smem, (cudaStream_t)stream>>>(
      t, field->octaves, field->scale, field->amplitude, re::grid_dev(g, d_grid),
      reinterpret_cast<float2*>(d_grid));
  RE_CHECK_LAUNCH("re_voxel_bake: launch");
  return RE_OK;
}

RE_API re_status re_voxel_sample(const float* d_grid, const re_voxel_grid* g, uint32_t quality,
                                 const float* d_pts, uint32_t n, float* d_out, void* stream) {
  re_status st = re::check_grid(g, "re_voxel_sample");
  if (st != RE_OK) return st;
  if (!d_grid || !d_pts || !d_out || quality > RE_VOXEL_HIGH)
    return re::fail(RE_ERR_INVALID_ARG, "re_voxel_sample: bad arguments");
  if (n == 0) return RE_OK;
  auto k = quality == RE_VOXEL_LOW      ? re::voxel::k_sample<RE_VOXEL_LOW>
           : quality == RE_VOXEL_MEDIUM ? re::voxel::k_sample<RE_VOXEL_MEDIUM>
                                        : re::voxel::k_sample<RE_VOXEL_HIGH>;
  k<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(re::grid_dev(g, d_grid), d_pts, n, d_out);
  RE_CHECK_LAUNCH("re_voxel_sample: launch");
  return RE_OK;
}

RE_API re_status re_voxel_trace(const float* d_grid, const re_voxel_grid* g, uint32_t quality,
                                const re_sdf_params* march, const re_camera* cam, uint32_t w,
                                uint32_t h, re_sdf_hit* d_out, void* stream) {
  re_status st = re::check_grid(g, "re_voxel_trace");
  if (st != RE_OK) return st;
  if (!d_grid || !march || !cam || !d_out || quality > RE_VOXEL_HIGH || w < 2 || h < 2 ||
      !(march->step_factor > 0.f) || march->max_steps == 0)
    return re::fail(RE_ERR_INVALID_ARG, "re_voxel_trace: bad arguments");
  if ((uint64_t)w * h > (1ull << 30)) return re::fail(RE_ERR_LIMIT, "re_voxel_trace: image too large");
  re::voxel::MarchDev m{march->step_factor, march->eps, march->tmax, march->max_steps};
  const re::voxel::GridDev gd = re::grid_dev(g, d_grid);
  const re::CamDev cd = re::cam_of_voxel(*cam);
  float4* out = reinterpret_cast<float4*>(d_out);
  cudaStream_t cs = (cudaStream_t)stream;
  if (quality == RE_VOXEL_HIGH) {
    auto k = re::voxel::k_trace_high;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, 0) != cudaSuccess ||
        per_sm < 1)
      per_sm = 1;
    const uint32_t tiles = ((w + 7) / 8) * ((h + 3) / 4);
    const uint32_t grid = std::min<uint32_t>((uint32_t)(per_sm * re::sm_count()), tiles);
    k<<<grid, 256, 0, cs>>>(gd, m, cd, w, h, out);
  } else {
    auto k = quality == RE_VOXEL_LOW ? re::voxel::k_trace_pixel<RE_VOXEL_LOW>
                                     : re::voxel::k_trace_pixel<RE_VOXEL_MEDIUM>;
    k<<<(w * h + 255) / 256, 256, 0, cs>>>(gd, m, cd, w, h, out);
  }
  RE_CHECK_LAUNCH("re_voxel_trace: launch");
  return RE_OK;
}

RE_API re_status re_voxel_brush(float* d_grid, const re_voxel_grid* g, const re_voxel_brush_params* b,
                                void* stream) {
  re_status st = re::check_grid(g, "re_voxel_brush");
  if (st != RE_OK) return st;
  if (!d_grid || !b || b->type > RE_BRUSH_CUBE_SUBTRACT ||
      (b->type == RE_BRUSH_SPHERE_ADD && !(b->smooth > 0.f)))
    return re::fail(RE_ERR_INVALID_ARG, "re_voxel_brush: bad arguments");
  re::voxel::k_brush<<<8 * re::sm_count(), 256, 0, (cudaStream_t)stream>>>(
      re::grid_dev(g, d_grid), b->type, b->center[0], b->center[1], b->center[2], b->extent[0],
      b->extent[1], b->extent[2], b->material, b->smooth, reinterpret_cast<float2*>(d_grid));
  RE_CHECK_LAUNCH("re_voxel_brush: launch");
  return RE_OK;
}

// .rsdf: int32 dim[3], float spacing[3], then {distance, material} float
// pairs with x fastest (Grid.cpp:23-64; the reference's save_map writes
// the same order).  The origin is not stored (0 on load).
RE_API re_status re_voxel_save(const char* path, const re_voxel_grid* g, const float* host_grid) {
  re_status st = re::check_grid(g, "re_voxel_save");
  if (st != RE_OK) return st;
  if (!path || !host_grid) return re::fail(RE_ERR_INVALID_ARG, "re_voxel_save: bad arguments");
  FILE* f = std::fopen(path, "wb");
  if (!f) return re::fail(RE_ERR_INVALID_ARG, "re_voxel_save: cannot open %s", path);
  int32_t dim[3] = {(int32_t)g->dim[0], (int32_t)g->dim[1], (int32_t)g->dim[2]};
  size_t n = (size_t)dim[0] * dim[1] * dim[2];
  bool ok = std::fwrite(dim, 4, 3, f) == 3 && std::fwrite(g->spacing, 4, 3, f) == 3 &&
            std::fwrite(host_grid, 8, n, f) == n;
  ok = (std::fclose(f) == 0) && ok;
  if (!ok) return re::fail(RE_ERR_INTERNAL, "re_voxel_save: write failed for %s", path);
  return RE_OK;
}

RE_API re_status re_voxel_load(const char* path, re_voxel_grid* g, float* host_grid,
                               uint64_t capacity_voxels) {
  if (!path || !g) return re::fail(RE_ERR_INVALID_ARG, "re_voxel_load: bad arguments");
  FILE* f = std::fopen(path, "rb");
  if (!f) return re::fail(RE_ERR_INVALID_ARG, "re_voxel_load: cannot open %s", path);
  int32_t dim[3];
  float sp[3];
  bool ok = std::fread(dim, 4, 3, f) == 3 && std::fread(sp, 4, 3, f) == 3;
  re_voxel_grid tmp;
  std::memset(&tmp, 0, sizeof(tmp));
  if (ok)
    for (int k = 0; k < 3; ++k) {
      tmp.dim[k] = dim[k] > 0 ? (uint32_t)dim[k] : 0u;
      tmp.spacing[k] = sp[k];
    }
  re_status st = ok ? re::check_grid(&tmp, "re_voxel_load")
                    : re::fail(RE_ERR_INVALID_ARG, "re_voxel_load: %s: short header", path);
  if (st != RE_OK) {
    std::fclose(f);
    return st;
  }
  *g = tmp;
  size_t n = (size_t)tmp.dim[0] * tmp.dim[1] * tmp.dim[2];
  if (host_grid) {
    if (capacity_voxels < n) {
      std::fclose(f);
      return re::fail(RE_ERR_LIMIT, "re_voxel_load: buffer holds %llu of %zu voxels",
                      (unsigned long long)capacity_voxels, n);
    }
    ok = std::fread(host_grid, 8, n, f) == n;
  }
  std::fclose(f);
  if (!ok) return re::fail(RE_ERR_INVALID_ARG, "re_voxel_load: %s: truncated", path);
  return RE_OK;
}

}  // extern "C"
