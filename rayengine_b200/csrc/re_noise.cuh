// Improved-Perlin noise and fBm on the device.
//
// Value part of eval() (RayEngine/src/cuda-src/sdf_functions.cuh:84-135):
// lattice cell from floor & 255, quintic fade (:57-60), 16-case gradient dot
// (:26-47) and the k0..k7 polynomial form of the trilinear blend.  The
// reference's hash (:77-81) reads a linearly filtered, normalised-float
// texture and cannot be reproduced; the lattice hash here is
// P[P[P[x] + y] + z] over RPerlinNoise's table (PerlinNoise.h:16-52), which
// the kernels keep in shared memory.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "re_common.hpp"
#include "re_math.cuh"

namespace re {

struct PermTable {
  uint8_t p[512];
};

// One octave at a time (the caller-point fBm and the heightfield; the terrain
// field reads FieldTable below): the table in 16 interleaved copies, entry j
// of lane c at word 16*j + (c & 15), so that of a warp's 32 divergent lookups
// only lanes c and c + 16 can meet in a bank (when their entries have the
// same parity).  512 entries x 16 copies x 4 B = 32 KB, four blocks to an SM;
// 32 conflict-free copies (64 KB) allow one block fewer.  Each
// word holds P[j] in bits 0-7 and the gradient case h = P[j] & 15 decoded
// for grad_dot in bits 28-31: bit 28 set when its first operand is y (else
// x), bit 29 when its second operand is y (else z), bit 30 when the second
// operand is negated and bit 31 when the first one is (so that negation is
// an XOR of the operand's sign bit with the word).  Bits 28-31 fall out of
// the interleaved table's 32-bit index arithmetic (Perm::word), so chained
// lookups use the word unmasked.
constexpr uint32_t kPermSmemBytes = 512 * 16 * 4;

__host__ __device__ __forceinline__ uint32_t perm_word(uint32_t p) {
  const uint32_t h = p & 15u;
  return p | (((0xCF00u >> h) & 1u) << 28) | (((0x300Fu >> h) & 1u) << 29) |
         (((0x8CCCu >> h) & 1u) << 30) | (((0xEAAAu >> h) & 1u) << 31);
}

__device__ __forceinline__ void load_perm(const PermTable& t, uint32_t* s) {
  for (uint32_t i = threadIdx.x; i < 512 * 16; i += blockDim.x) s[i] = perm_word(t.p[i >> 4]);
  __syncthreads();
}

// Permutation-table views: idx(j) = P[j] (a lattice index), grad(j) = the
// perm_word() of P[j] (its gradient case decoded).
struct Perm {
  const uint32_t* __restrict__ s;
  uint32_t lane;
  // j may carry a word's bits 28-31: the 32-bit shift drops them, and the
  // rest (an index below 512) stays inside the 8192-word table
  __device__ __forceinline__ uint32_t word(uint32_t j) const { return s[(j << 4) + lane]; }
  // the raw word: as the next lookup's index its bits 28-31 do not count
  __device__ __forceinline__ uint32_t idx(uint32_t j) const { return word(j); }
  __device__ __forceinline__ uint32_t grad(uint32_t j) const { return word(j); }
};

__device__ __forceinline__ Perm perm_view(const uint32_t* s) { return Perm{s, threadIdx.x & 15u}; }

// Single shared tables for several seeds side by side (the batched
// renderer; no per-lane copies, lookups may share banks): perm_word()
// entries, 2 KB per seed (measured 4 % faster on the batch), or plain bytes,
// 512 B per seed, for batches with many seeds.
struct PermWords {
  const uint32_t* __restrict__ s;
  __device__ __forceinline__ uint32_t idx(uint32_t j) const { return s[j] & 255u; }
  __device__ __forceinline__ uint32_t grad(uint32_t j) const { return s[j]; }
};

struct PermBytes {
  const uint8_t* __restrict__ s;
  __device__ __forceinline__ uint32_t idx(uint32_t j) const { return s[j]; }
  __device__ __forceinline__ uint32_t grad(uint32_t j) const { return perm_word(s[j]); }
};

// gradientDotV (sdf_functions.cuh:26-47) without branches: each case is a
// sum of two signed coordinates, picked here from the decoded case bits of
// perm_word().  The operands and their signs are exactly the reference's,
// so the single rounded addition is unchanged:
//   first operand is y for cases 8-11, 14, 15 (x otherwise), negated for
//   1, 3, 5, 7, 9, 11, 13, 14, 15; second operand is y for 0-3, 12 and 13
//   (z otherwise), negated for 2, 3, 6, 7, 10, 11, 15.
// Case 12 is the reference's y + x, taken here as x + y: IEEE addition is
// commutative, so the sum is the same, and the second operand needs one
// select instead of two.  Negating the first operand flips its sign bit
// with the word's bit 31.  (Measured on B200: the field evaluation is bound
// by the ALU pipe, where these selects run.)
// g: a grad() lookup.
__device__ __forceinline__ float grad_dot(uint32_t g, float x, float y, float z) {
  float u = (g & 0x10000000u) ? y : x;
  u = __uint_as_float(__float_as_uint(u) ^ (g & 0x80000000u));
  float v = (g & 0x20000000u) ? y : z;
  v = (g & 0x40000000u) ? -v : v;
  return u + v;
}

__device__ __forceinline__ float quintic(float t) {
  float in = __fmaf_rn(t, 6.0f, -15.0f);
  in = __fmaf_rn(t, in, 10.0f);
  return ((t * t) * t) * in;
}

// PT: a permutation-table view with idx() and grad() (Perm: interleaved
// shared copies; PermWords: one word table).  The table's second half repeats the
// first (P[256 + i] = P[i], RPerlinNoise), so the upper lattice corners
// index it with xi0 + 1 etc. unmasked, which reads the same entries as the
// reference's (xi0 + 1) & 255.
template <class PT>
__device__ __forceinline__ float perlin(const PT& P, float x, float y, float z) {
  float fx = floorf(x), fy = floorf(y), fz = floorf(z);
  uint32_t xi0 = ((int)fx) & 255, yi0 = ((int)fy) & 255, zi0 = ((int)fz) & 255;
  uint32_t xi1 = xi0 + 1, yi1 = yi0 + 1, zi1 = zi0 + 1;
  float tx = x - fx, ty = y - fy, tz = z - fz;
  float u = quintic(tx), v = quintic(ty), w = quintic(tz);
  float x1 = tx - 1.0f, y1 = ty - 1.0f, z1 = tz - 1.0f;
  uint32_t px0 = P.idx(xi0), px1 = P.idx(xi1);
  uint32_t p00 = P.idx(px0 + yi0), p10 = P.idx(px1 + yi0);
  uint32_t p01 = P.idx(px0 + yi1), p11 = P.idx(px1 + yi1);
  float a = grad_dot(P.grad(p00 + zi0), tx, ty, tz);
  float b = grad_dot(P.grad(p10 + zi0), x1, ty, tz);
  float c = grad_dot(P.grad(p01 + zi0), tx, y1, tz);
  float d = grad_dot(P.grad(p11 + zi0), x1, y1, tz);
  float e = grad_dot(P.grad(p00 + zi1), tx, ty, z1);
  float f = grad_dot(P.grad(p10 + zi1), x1, ty, z1);
  float g = grad_dot(P.grad(p01 + zi1), tx, y1, z1);
  float h = grad_dot(P.grad(p11 + zi1), x1, y1, z1);
  float k1 = b - a;
  float k2 = c - a;
  float k3 = e - a;
  float k4 = ((a + d) - b) - c;
  float k5 = ((a + f) - b) - e;
  float k6 = ((a + g) - c) - e;
  float k7 = ((((((b + c) + e) + h) - a) - d) - f) - g;
  float r = __fmaf_rn(k1, u, a);
  r = __fmaf_rn(k2, v, r);
  r = __fmaf_rn(k3, w, r);
  r = __fmaf_rn(k4, u * v, r);
  r = __fmaf_rn(k5, u * w, r);
  r = __fmaf_rn(k6, v * w, r);
  r = __fmaf_rn(k7, (u * v) * w, r);
  return r;
}

template <class PT>
__device__ __forceinline__ float fbm(const PT& P, float x, float y, float z,
                                     uint32_t octaves, float lacunarity, float gain) {
  float sum = 0.0f, amp = 1.0f;
#pragma unroll 4
  for (uint32_t i = 0; i < octaves; ++i) {
    sum = __fmaf_rn(amp, perlin(P, x, y, z), sum);
    x *= lacunarity;
    y *= lacunarity;
    z *= lacunarity;
    amp *= gain;
  }
  return sum;
}

// d(p) = p.y - amp * fbm(scale * p), lacunarity 2, gain 0.5
template <class PT>
__device__ __forceinline__ float terrain_density(const PT& P, V3 p,
                                                 uint32_t octaves, float scale, float amp) {
  float f = fbm(P, scale * p.x, scale * p.y, scale * p.z, octaves, 2.0f, 0.5f);
  return __fmaf_rn(-amp, f, p.y);
}

// ------------------------------------------------- two octaves at a time
// The same field for the kernels that spend their time in it: octaves i and
// i + 1 are evaluated together in the two halves of packed FP32 registers
// (add/mul/fma.f32x2, each half rounded as the scalar instruction rounds),
// in perlin()'s operations and order, so every result is the scalar form's.
//
// What changes is how the lattice is read.  The table is 512 rows of 256
// bytes: row j holds, for each of the 32 lanes, an A word with the rows of
// P[j] and P[j + 1] as byte offsets in its halves (P << 8), then, for each
// lane, a G word with the gradient of case P[j] & 15 as three bytes (x in
// bits 24-31, y in 16-23, z in 0-7), each the top byte of the float +2, -2
// or 0.  One A word answers both lattice neighbours, so a cell takes 3 A and
// 8 G lookups instead of 14, and with a copy per lane no two lanes meet in a
// bank (16 copies cost two shared-memory passes per divergent lookup).  A
// corner's value is then a three-term dot product: the two non-zero terms
// are exact, so its one rounding is grad_dot's addition at twice the scale,
// and the doubled noise times half the amplitude is the same product.  (A
// corner that is zero may differ in its sign, which the sum over the octaves,
// starting at +0, does not keep; a noise value below 2^-126 keeps more bits.)
// The lattice cell comes from one addition rounded down to a multiple of 1:
// 1.5 * 2^23 + floor(x), its low byte the masked index, where floor and a
// conversion run on the quarter-rate unit.  That holds for |x| < 2^22;
// beyond, field_far() finds the cells as perlin() does.
//
// Measured on B200 (a march of 8-octave evaluations, no other work): 33.3 G
// evaluations/s against 26.3 of perlin() on 16 copies.  Per octave 99
// instructions against 147; the multiply-add pipes, 73 % busy, are what is
// left (the scalar form of this layout: 29.9 G/s).  Frames, one octave at a
// time on 16 copies against this form alone: the 1080p terrain 3.18 -> 2.56
// ms, the shaded terrain at 1366x768 2.65 -> 2.10 ms (1.95 with several lanes
// to a ray, terrain_density_shared), the 1080p neural tracer 2.27 -> 1.85 ms
// (1.77 with the normals' gradient in this form too, perlin_grad2).
// FieldTable<STRIDE, G>: rows STRIDE bytes apart, G words G bytes past A words.
constexpr uint32_t kRowBytes = 256;
constexpr uint32_t kRowsSmemBytes = 512 * kRowBytes;
// One block per SM, whose warps share the table.  640 threads: 5 warps per
// sub-partition with 96 registers to keep both cells' lookups in flight
// (1080p terrain frame 2.62 ms; 512 threads 2.75, 768 2.69, 1024 2.74).  One,
// two and four pairs of octaves unrolled: 2.62, 2.58, 2.56; kernels that hold
// the forms with several lanes to a ray as well unroll two (warp_density).
constexpr uint32_t kRowsThreads = 640;

// How a frame of n rays spreads over `blocks` blocks of kRowsThreads: the rays
// a warp takes at once (32, or 16 or 8 with several lanes to a ray,
// terrain_density_shared) and the warps of a block that take any.  A warp
// claims that many rays when it starts, so the first blocks would claim all of
// a small frame.
struct RowsSpread {
  uint32_t rays, warps;
};
inline RowsSpread rows_spread(uint64_t n, uint32_t blocks) {
  const uint64_t warps = (uint64_t)blocks * (kRowsThreads / 32u);
  const uint32_t rays = n <= 8u * warps ? 8u : n <= 16u * warps ? 16u : 32u;
  const uint64_t per = ((n + rays - 1u) / rays + blocks - 1u) / blocks;
  return {rays, (uint32_t)(per < kRowsThreads / 32u ? (per ? per : 1u) : kRowsThreads / 32u)};
}

template <uint32_t STRIDE, uint32_t G>
struct FieldTable {
  uint32_t base;  // shared-memory address of this lane's column
};
using FieldRows = FieldTable<kRowBytes, 128>;

// One copy of the table per seed, 512 A words then 512 G words (the batched
// renderer, which holds several seeds; lanes may meet in a bank).
constexpr uint32_t kFieldWordsBytes = 2 * 512 * 4;
using FieldWords = FieldTable<4, 2048>;

template <uint32_t STRIDE>
__host__ __device__ __forceinline__ uint32_t field_a_word(uint32_t p, uint32_t next) {
  return p * STRIDE | (next * STRIDE) << 16;
}

__host__ __device__ __forceinline__ uint32_t grad_bytes(uint32_t p) {
  const uint32_t h = perm_word(p) >> 28;  // bit 0: first is y, 1: second is y, 2, 3: negated
  const uint32_t f = (h & 8u) ? 0xC0u : 0x40u, s = (h & 4u) ? 0xC0u : 0x40u;
  const uint32_t gx = (h & 1u) ? 0u : f, gz = (h & 2u) ? 0u : s;
  const uint32_t gy = (h & 1u) ? f : (h & 2u) ? s : 0u;
  return (gx << 24) | (gy << 16) | gz;
}

// A table's base address, for row_word(), whose loads the compiler takes for
// functions of the address alone: they depend on this value, and it comes
// from behind the barrier that publishes the table.
__device__ __forceinline__ uint32_t after_barrier(uint32_t base) {
  asm volatile("" : "+r"(base) : : "memory");
  return base;
}

// smem: kRowsSmemBytes; every thread of the block calls it.
__device__ __forceinline__ FieldRows load_rows(const PermTable& t, uint32_t* smem) {
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t j = threadIdx.x >> 5; j < 512u; j += blockDim.x >> 5) {
    const uint32_t p = t.p[j], q = t.p[(j + 1u) & 511u];
    smem[64u * j + lane] = field_a_word<kRowBytes>(p, q);
    smem[64u * j + 32u + lane] = grad_bytes(p);
  }
  __syncthreads();
  return FieldRows{after_barrier((uint32_t)__cvta_generic_to_shared(smem) + 4u * lane)};
}

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2_down(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
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

// A word of a table whose base went through after_barrier().
template <uint32_t OFF>
__device__ __forceinline__ uint32_t row_word(uint32_t addr) {
  uint32_t r;
  asm("ld.shared.u32 %0, [%1+%2];" : "=r"(r) : "r"(addr), "n"(OFF));
  return r;
}

// The 8 corner G words of the cell whose masked indices are the low bytes of
// x, y and z (corner order a..h: x fastest, then y, z).  Every row index is
// a sum of two bytes, at most 510, and a corner at z + 1 is the next row.
template <uint32_t STRIDE, uint32_t G>
__device__ __forceinline__ void cell_words(const FieldTable<STRIDE, G>& R, uint32_t x, uint32_t y,
                                           uint32_t z, uint32_t (&g)[8]) {
  const uint32_t wx = row_word<0>((x & 255u) * STRIDE + R.base);
  const uint32_t ry = (y & 255u) * STRIDE + R.base, rz = (z & 255u) * STRIDE + R.base;
  const uint32_t w0 = row_word<0>(__dp2a_lo(wx, 1u, ry)), w1 = row_word<0>((wx >> 16) + ry);
  const uint32_t r00 = __dp2a_lo(w0, 1u, rz), r01 = (w0 >> 16) + rz;
  const uint32_t r10 = __dp2a_lo(w1, 1u, rz), r11 = (w1 >> 16) + rz;
  g[0] = row_word<G>(r00);
  g[1] = row_word<G>(r10);
  g[2] = row_word<G>(r01);
  g[3] = row_word<G>(r11);
  g[4] = row_word<G + STRIDE>(r00);
  g[5] = row_word<G + STRIDE>(r10);
  g[6] = row_word<G + STRIDE>(r01);
  g[7] = row_word<G + STRIDE>(r11);
}

// Twice the corner values of both octaves.
__device__ __forceinline__ f32x2 corner2(uint32_t lo, uint32_t hi, f32x2 x, f32x2 y, f32x2 z) {
  const f32x2 gx =
      pack2(__uint_as_float(lo & 0xFF000000u), __uint_as_float(hi & 0xFF000000u));
  const f32x2 gy = pack2(__uint_as_float(__byte_perm(lo, 0u, 0x2444)),
                         __uint_as_float(__byte_perm(hi, 0u, 0x2444)));
  const f32x2 gz = pack2(__uint_as_float(lo << 24), __uint_as_float(hi << 24));
  return fma2(gz, z, fma2(gy, y, mul2(gx, x)));
}

__device__ __forceinline__ f32x2 quintic2(f32x2 t) {
  f32x2 in = fma2(t, pack2(6.0f, 6.0f), pack2(-15.0f, -15.0f));
  in = fma2(t, in, pack2(10.0f, 10.0f));
  return mul2(mul2(mul2(t, t), t), in);
}

// The cells (lattice indices, of which the low bytes count) and the fractions
// of two coordinates.  FAR: as perlin() takes them, at any magnitude; otherwise
// below 2^22, from one addition rounded down.
template <bool FAR>
__device__ __forceinline__ f32x2 lattice2(f32x2 x, uint32_t& lo, uint32_t& hi) {
  if (FAR) {
    float x0, x1;
    unpack2(x, x0, x1);
    const float f0 = floorf(x0), f1 = floorf(x1);
    lo = (uint32_t)(int)f0;
    hi = (uint32_t)(int)f1;
    return sub2(x, pack2(f0, f1));
  }
  const f32x2 kInt = pack2(12582912.0f, 12582912.0f), i = add2_down(x, kInt);
  lo = (uint32_t)i;
  hi = (uint32_t)(i >> 32);
  return sub2(x, sub2(i, kInt));
}

// Twice the noise of two octaves; unless FAR every coordinate below 2^22.
template <bool FAR = false, class FT>
__device__ __forceinline__ f32x2 perlin2(const FT& R, f32x2 x, f32x2 y, f32x2 z) {
  const f32x2 kOne = pack2(1.0f, 1.0f);
  uint32_t xl, xh, yl, yh, zl, zh;
  const f32x2 tx = lattice2<FAR>(x, xl, xh), ty = lattice2<FAR>(y, yl, yh),
              tz = lattice2<FAR>(z, zl, zh);
  uint32_t lo[8], hi[8];
  cell_words(R, xl, yl, zl, lo);
  cell_words(R, xh, yh, zh, hi);
  const f32x2 x1 = sub2(tx, kOne), y1 = sub2(ty, kOne), z1 = sub2(tz, kOne);
  const f32x2 u = quintic2(tx), v = quintic2(ty), w = quintic2(tz);
  const f32x2 a = corner2(lo[0], hi[0], tx, ty, tz), b = corner2(lo[1], hi[1], x1, ty, tz);
  const f32x2 c = corner2(lo[2], hi[2], tx, y1, tz), d = corner2(lo[3], hi[3], x1, y1, tz);
  const f32x2 e = corner2(lo[4], hi[4], tx, ty, z1), f = corner2(lo[5], hi[5], x1, ty, z1);
  const f32x2 g = corner2(lo[6], hi[6], tx, y1, z1), h = corner2(lo[7], hi[7], x1, y1, z1);
  const f32x2 k1 = sub2(b, a), k2 = sub2(c, a), k3 = sub2(e, a);
  const f32x2 k4 = sub2(sub2(add2(a, d), b), c);
  const f32x2 k5 = sub2(sub2(add2(a, f), b), e);
  const f32x2 k6 = sub2(sub2(add2(a, g), c), e);
  const f32x2 k7 = sub2(sub2(sub2(sub2(add2(add2(add2(b, c), e), h), a), d), f), g);
  f32x2 r = fma2(k1, u, a);
  r = fma2(k2, v, r);
  r = fma2(k3, w, r);
  r = fma2(k4, mul2(u, v), r);
  r = fma2(k5, mul2(u, w), r);
  r = fma2(k6, mul2(v, w), r);
  return fma2(k7, mul2(mul2(u, v), w), r);
}

// perlin()'s view of the table.
template <uint32_t STRIDE>
struct PermRows {
  uint32_t base;
  __device__ __forceinline__ uint32_t idx(uint32_t j) const {
    return (row_word<0>(base + j * STRIDE) & 0xFFFFu) / STRIDE;
  }
  __device__ __forceinline__ uint32_t grad(uint32_t j) const { return perm_word(idx(j)); }
};

// The octaves' sum at any coordinates (infinities and NaN among them); out of
// line, so that the callers' registers are those of the near form.  In pairs
// on the rows; an octave at a time on FieldWords, for the registers of the
// batched renderer (which takes other tables for such fields).  Measured on
// B200, 480x270 frames whose rays are all or mostly past the near form's
// range, an octave at a time | in pairs: 8 octaves at scale 1000 674 | 408 us
// (one octave at a time on 16 copies, four times the warps: 366), 20 octaves
// 1892 | 1116 (1157); 1920x1080 at scale 1000: 2176 (2644).
template <uint32_t STRIDE, uint32_t G>
static __device__ __noinline__ float field_far(uint32_t base, float x, float y, float z,
                                               uint32_t octaves) {
  float sum = 0.0f, a = 1.0f;
  if (STRIDE != kRowBytes) {
    PermRows<STRIDE> P{base};
#pragma unroll 1
    for (uint32_t i = 0; i < octaves; ++i) {
      sum = __fmaf_rn(a, perlin(P, x, y, z), sum);
      x *= 2.0f;
      y *= 2.0f;
      z *= 2.0f;
      a *= 0.5f;
    }
    return sum;
  }
  const FieldTable<STRIDE, G> R{base};
  const f32x2 kFour = pack2(4.0f, 4.0f);
  f32x2 X = pack2(x, 2.0f * x), Y = pack2(y, 2.0f * y), Z = pack2(z, 2.0f * z);
#pragma unroll 1
  for (uint32_t i = 0; i < octaves; i += 2) {
    float r0, r1;
    unpack2(perlin2<true>(R, X, Y, Z), r0, r1);
    sum = __fmaf_rn(0.5f * a, r0, sum);
    // the octave past an odd last one may be infinite or NaN
    if (i + 1u < octaves) sum = __fmaf_rn(0.25f * a, r1, sum);
    a *= 0.25f;
    X = mul2(X, kFour);
    Y = mul2(Y, kFour);
    Z = mul2(Z, kFour);
  }
  return sum;
}

// The octaves' sum on a field table.  The near form evaluates octaves in pairs,
// an odd last one with an octave past it at amplitude zero, so the largest
// coordinate it meets is below 2^octaves times the first one's.
// UNROLL: pairs in the code at once.
template <int UNROLL, uint32_t STRIDE, uint32_t G>
__device__ __forceinline__ float field_near(const FieldTable<STRIDE, G>& R, float x, float y,
                                            float z, uint32_t octaves) {
  const f32x2 kFour = pack2(4.0f, 4.0f);
  f32x2 X = pack2(x, 2.0f * x), Y = pack2(y, 2.0f * y), Z = pack2(z, 2.0f * z);
  float sum = 0.0f, a = 0.5f;
#pragma unroll UNROLL
  for (uint32_t i = 0; i < octaves; i += 2) {
    float r0, r1;
    unpack2(perlin2(R, X, Y, Z), r0, r1);
    sum = __fmaf_rn(a, r0, sum);
    sum = __fmaf_rn(i + 1u < octaves ? 0.5f * a : 0.0f, r1, sum);
    a *= 0.25f;
    X = mul2(X, kFour);
    Y = mul2(Y, kFour);
    Z = mul2(Z, kFour);
  }
  return sum;
}

// Whether the near form holds: coordinates below 2^(22 - octaves), octaves <= 32.
__device__ __forceinline__ bool is_near(float x, float y, float z, uint32_t octaves) {
  const float lim = __uint_as_float((127u + 22u - octaves) << 23);
  return fabsf(x) < lim && fabsf(y) < lim && fabsf(z) < lim;
}

// terrain_density() on a field table.
template <int UNROLL = 4, uint32_t STRIDE, uint32_t G>
__device__ __forceinline__ float terrain_density(const FieldTable<STRIDE, G>& R, V3 p,
                                                 uint32_t octaves, float scale, float amp) {
  const float x = scale * p.x, y = scale * p.y, z = scale * p.z;
  const float sum = is_near(x, y, z, octaves) ? field_near<UNROLL>(R, x, y, z, octaves)
                                              : field_far<STRIDE, G>(R.base, x, y, z, octaves);
  return __fmaf_rn(-amp, sum, p.y);
}

// The position of the n-th (from 0) set bit of m.
__device__ __forceinline__ uint32_t nth_set(uint32_t m, uint32_t n) {
  uint32_t pos = 0;
#pragma unroll
  for (uint32_t s = 16; s > 0; s >>= 1)
    if ((uint32_t)__popc(m & ((1u << (pos + s)) - 1u)) <= n) pos += s;
  return pos;
}

// terrain_density() at the points of a warp's few live lanes (at most 32 / L
// of them, `live` their mask), L = 2 or 4 lanes to a point: the pairs of
// octaves are dealt to them in turn, and the point's lane adds their noise up
// in the octaves' order, so the sum is the same.  All 32 lanes call it; the
// live lanes get their value.  For frames with fewer rays than lanes and for
// the end of any frame, when what is left is the chain of the longest rays:
// an evaluation takes a warp alone 1.2 us, with 4 lanes to the point 0.8.
// The field may differ between the lanes (FieldWords: and its table with it;
// FieldRows: one table, every lane its own copy).
template <uint32_t L, uint32_t STRIDE, uint32_t G>
__device__ __forceinline__ float terrain_density_shared(const FieldTable<STRIDE, G>& R, V3 p,
                                                        uint32_t live, uint32_t octaves,
                                                        float scale, float amp) {
  const uint32_t lane = threadIdx.x & 31u;
  const float x = scale * p.x, y = scale * p.y, z = scale * p.z;
  const bool mine = (live >> lane) & 1u;
  float sum = 0.0f;
  if (__any_sync(0xFFFFFFFFu, mine && !is_near(x, y, z, octaves))) {
    if (mine) sum = field_far<STRIDE, G>(R.base, x, y, z, octaves);
    return __fmaf_rn(-amp, sum, p.y);
  }
  const uint32_t src = nth_set(live, lane / L);  // past the last point: lane 31's, unused
  const float sx = __shfl_sync(0xFFFFFFFFu, x, src), sy = __shfl_sync(0xFFFFFFFFu, y, src),
              sz = __shfl_sync(0xFFFFFFFFu, z, src);
  FieldTable<STRIDE, G> T = R;
  uint32_t oct = octaves, most = octaves;  // of the point this lane helps with; of any
  if (STRIDE != kRowBytes) {
    T.base = __shfl_sync(0xFFFFFFFFu, R.base, src);
    oct = __shfl_sync(0xFFFFFFFFu, octaves, src);
    most = __reduce_max_sync(0xFFFFFFFFu, mine ? octaves : 0u);
  }
  const bool helps = lane / L < (uint32_t)__popc(live);
  const uint32_t from = L * (uint32_t)__popc(live & ((1u << lane) - 1u));  // this point's helpers
  float a = 1.0f;
#pragma unroll 1
  for (uint32_t c = 0; c < most; c += 2u * L) {
    const uint32_t k = c + 2u * (lane & (L - 1u));
    float r0 = 0.0f, r1 = 0.0f;
    if (helps && k < oct) {
      const float f = __uint_as_float((127u + k) << 23);  // 2^k
      unpack2(perlin2(T, pack2(f * sx, 2.0f * (f * sx)), pack2(f * sy, 2.0f * (f * sy)),
                      pack2(f * sz, 2.0f * (f * sz))),
              r0, r1);
    }
#pragma unroll
    for (uint32_t j = 0; j < L; ++j) {
      const float v0 = __shfl_sync(0xFFFFFFFFu, r0, (from + j) & 31u);
      const float v1 = __shfl_sync(0xFFFFFFFFu, r1, (from + j) & 31u);
      const uint32_t o = c + 2u * j;
      if (o < octaves) sum = __fmaf_rn(0.5f * a, v0, sum);
      if (o + 1u < octaves) sum = __fmaf_rn(0.25f * a, v1, sum);
      a *= 0.25f;
    }
  }
  return __fmaf_rn(-amp, sum, p.y);
}

// terrain_density() at the points of the live lanes, with more lanes to a
// point where they are few.  All 32 lanes call it.
// SHARED2: two lanes to a point as well as four (a third copy of the code).
template <int UNROLL = 2, bool SHARED2 = true, uint32_t STRIDE, uint32_t G>
__device__ __forceinline__ float warp_density(const FieldTable<STRIDE, G>& R, V3 p, bool live,
                                              uint32_t octaves, float scale, float amp) {
  const uint32_t mask = __ballot_sync(0xFFFFFFFFu, live);
  const uint32_t n = __popc(mask);
  if (n <= 8u) return terrain_density_shared<4>(R, p, mask, octaves, scale, amp);
  if (SHARED2 && n <= 16u) return terrain_density_shared<2>(R, p, mask, octaves, scale, amp);
  if (STRIDE != kRowBytes) return live ? terrain_density<UNROLL>(R, p, octaves, scale, amp) : 0.0f;
  // one far lane takes the others with it: the far form's result is the near
  // one's, and the warp then runs one of the two
  const float x = scale * p.x, y = scale * p.y, z = scale * p.z;
  if (!__all_sync(0xFFFFFFFFu, !live || is_near(x, y, z, octaves)))
    return live ? __fmaf_rn(-amp, field_far<STRIDE, G>(R.base, x, y, z, octaves), p.y) : 0.0f;
  return live ? __fmaf_rn(-amp, field_near<UNROLL>(R, x, y, z, octaves), p.y) : 0.0f;
}

template <class PT>
__device__ __forceinline__ float warp_density(const PT& P, V3 p, bool live, uint32_t octaves,
                                              float scale, float amp) {
  return live ? terrain_density(P, p, octaves, scale, amp) : 0.0f;
}

// How a kernel holds the field: pairs of octaves on the rows, or an octave at a
// time on 16 copies of the permutation, with up to twice the warps.
struct RowsForm {
  static constexpr uint32_t kThreads = kRowsThreads, kBytes = kRowsSmemBytes;
  static __device__ __forceinline__ FieldRows load(const PermTable& t, uint32_t* smem) {
    return load_rows(t, smem);
  }
};
struct CopyForm {
  static constexpr uint32_t kThreads = 256, kBytes = kPermSmemBytes;
  static __device__ __forceinline__ Perm load(const PermTable& t, uint32_t* smem) {
    load_perm(t, smem);
    return perm_view(smem);
  }
};

// Whether the marches' kernels take the rows: a single octave is half a pair,
// and two are too little work to need few warps until the frame is large.
// Measured on B200, exact terrain, copies | rows: one octave 480x270 340 | 513
// us, 1920x1080 1245 | 1682; two octaves 428 | 475, 960x540 762 | 683; three 565
// | 512.  STENCIL: the neural tracer's exact phase with a stencil for the
// normal, which mixes a warp's rays: two octaves 492 | 578, 1920x1080 1589 |
// 1686; three 64x36 184 | 169, 160x90 472 | 491, 1920x1080 1915 | 2011.
template <bool STENCIL = false>
inline bool field_on_rows(uint32_t octaves, uint64_t rays) {
  if (STENCIL) return octaves > 3u || (octaves == 3u && rays < (1u << 13));
  return octaves > 2u || (octaves == 2u && rays >= (1u << 18));
}

// Launches the kernel's form for a frame of `rays` rays: call(kernel, grid,
// threads, shared bytes, spread).  extra(warps): shared bytes past the table.
template <class K, class E, class F>
re_status launch_field(bool rows, K rows_kernel, K copy_kernel, uint64_t rays, E extra, F call) {
  const uint32_t threads = rows ? RowsForm::kThreads : CopyForm::kThreads;
  const uint32_t smem = (rows ? RowsForm::kBytes : CopyForm::kBytes) + extra(threads / 32u);
  const K kernel = rows ? rows_kernel : copy_kernel;
  RE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 1;
  if (!rows && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int)threads,
                                                              smem) != cudaSuccess ||
                per_sm < 1))
    per_sm = 1;
  call(kernel, per_sm * sm_count(), threads, smem,
       rows ? rows_spread(rays, (uint32_t)sm_count()) : RowsSpread{32u, CopyForm::kThreads / 32u});
  return RE_OK;
}

// Gradient of perlin() at (x, y, z), from the same lattice, fade and blend
// differentiated in closed form.  With corner values a..h (corner gradient
// vector ga..gh dotted with the offset to the corner) the blend is
//   n = a + k1 u + k2 v + k3 w + k4 uv + k5 uw + k6 vw + k7 uvw,
// u = fade(tx) etc., so
//   dn/dx = [sum over corners of (its trilinear weight in u, v, w) g].x
//           + fade'(tx) (k1 + k4 v + k5 w + k7 vw),
// likewise for y and z, with fade'(t) = 30 t^2 (t - 1)^2.  A corner's
// gradient vector is s1 e_op1 + s2 e_op2 (grad_dot's operands and signs), so
// the weighted sum adds the signed weight to the operands' components
// instead of multiplying.
template <class PT>
__device__ __forceinline__ V3 perlin_grad(const PT& P, float x, float y, float z) {
  float fx = floorf(x), fy = floorf(y), fz = floorf(z);
  uint32_t xi0 = ((int)fx) & 255, yi0 = ((int)fy) & 255, zi0 = ((int)fz) & 255;
  uint32_t xi1 = xi0 + 1, yi1 = yi0 + 1, zi1 = zi0 + 1;
  float tx = x - fx, ty = y - fy, tz = z - fz;
  float u = quintic(tx), v = quintic(ty), w = quintic(tz);
  float x1 = tx - 1.0f, y1 = ty - 1.0f, z1 = tz - 1.0f;
  float du = 30.0f * (tx * tx) * (x1 * x1);
  float dv = 30.0f * (ty * ty) * (y1 * y1);
  float dw = 30.0f * (tz * tz) * (z1 * z1);
  uint32_t px0 = P.idx(xi0), px1 = P.idx(xi1);
  uint32_t p00 = P.idx(px0 + yi0), p10 = P.idx(px1 + yi0);
  uint32_t p01 = P.idx(px0 + yi1), p11 = P.idx(px1 + yi1);
  const uint32_t G[8] = {P.grad(p00 + zi0), P.grad(p10 + zi0), P.grad(p01 + zi0),
                         P.grad(p11 + zi0), P.grad(p00 + zi1), P.grad(p10 + zi1),
                         P.grad(p01 + zi1), P.grad(p11 + zi1)};
  const float a = grad_dot(G[0], tx, ty, tz), b = grad_dot(G[1], x1, ty, tz);
  const float c = grad_dot(G[2], tx, y1, tz), d = grad_dot(G[3], x1, y1, tz);
  const float e = grad_dot(G[4], tx, ty, z1), f = grad_dot(G[5], x1, ty, z1);
  const float g = grad_dot(G[6], tx, y1, z1), h = grad_dot(G[7], x1, y1, z1);
  float k1 = b - a, k2 = c - a, k3 = e - a;
  float k4 = ((a + d) - b) - c;
  float k5 = ((a + f) - b) - e;
  float k6 = ((a + g) - c) - e;
  float k7 = ((((((b + c) + e) + h) - a) - d) - f) - g;
  float uv = u * v, uw = u * w, vw = v * w, uvw = uv * w;
  // trilinear weights of the corners (order a..h: x fastest, then y, z)
  const float cw[8] = {1.0f - u - v - w + uv + uw + vw - uvw, u - uv - uw + uvw,
                       v - uv - vw + uvw, uv - uvw, w - uw - vw + uvw, uw - uvw, vw - uvw, uvw};
  float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t gk = G[k];
    const float c1 = __uint_as_float(__float_as_uint(cw[k]) ^ (gk & 0x80000000u));  // s1 w
    const float c2 = (gk & 0x40000000u) ? -cw[k] : cw[k];                          // s2 w
    // first operand x or y, second y or z
    sx += (gk & 0x10000000u) ? 0.0f : c1;
    sy += ((gk & 0x10000000u) ? c1 : 0.0f) + ((gk & 0x20000000u) ? c2 : 0.0f);
    sz += (gk & 0x20000000u) ? 0.0f : c2;
  }
  V3 r;
  r.x = sx + du * (k1 + k4 * v + k5 * w + k7 * vw);
  r.y = sy + dv * (k2 + k4 * u + k6 * w + k7 * uw);
  r.z = sz + dw * (k3 + k5 * u + k6 * v + k7 * uv);
  return r;
}

// The octaves' gradients at any coordinates, summed (out of line, as
// field_far is).
template <uint32_t STRIDE>
static __device__ __noinline__ V3 gradient_far(uint32_t base, float x, float y, float z,
                                               uint32_t octaves) {
  PermRows<STRIDE> P{base};
  V3 s = v3(0.f, 0.f, 0.f);
#pragma unroll 1
  for (uint32_t i = 0; i < octaves; ++i) {
    V3 gi = perlin_grad(P, x, y, z);
    s = v3(s.x + gi.x, s.y + gi.y, s.z + gi.z);
    x *= 2.0f;
    y *= 2.0f;
    z *= 2.0f;
  }
  return s;
}

// a + b and a - b where one of them may be a product: as a product with one,
// so that the two roundings stay two.  (A packed product feeding a packed
// addition is contracted, a product with a one known to the compiler too;
// `one` comes from the caller's arguments.)
__device__ __forceinline__ f32x2 plus2(f32x2 a, f32x2 b, float one) {
  return fma2(b, pack2(one, one), a);
}
__device__ __forceinline__ f32x2 minus2(f32x2 a, f32x2 b, float one) {
  return fma2(b, pack2(-one, -one), a);
}

// Twice perlin_grad() of two octaves; every coordinate below 2^22.  The
// corners' gradient bytes are +2, -2 and 0, so perlin_grad's selections by
// gradient case are products here, exact ones, and every value is twice
// perlin_grad's.
template <class FT>
__device__ __forceinline__ void perlin_grad2(const FT& R, f32x2 x, f32x2 y, f32x2 z, float one,
                                             f32x2& rx, f32x2& ry, f32x2& rz) {
  const f32x2 kOne = pack2(1.0f, 1.0f), k30 = pack2(30.0f, 30.0f);
  uint32_t xl, xh, yl, yh, zl, zh;
  const f32x2 tx = lattice2<false>(x, xl, xh), ty = lattice2<false>(y, yl, yh),
              tz = lattice2<false>(z, zl, zh);
  uint32_t lo[8], hi[8];
  cell_words(R, xl, yl, zl, lo);
  cell_words(R, xh, yh, zh, hi);
  const f32x2 x1 = sub2(tx, kOne), y1 = sub2(ty, kOne), z1 = sub2(tz, kOne);
  const f32x2 u = quintic2(tx), v = quintic2(ty), w = quintic2(tz);
  const f32x2 uv = mul2(u, v), uw = mul2(u, w), vw = mul2(v, w), uvw = mul2(uv, w);
  const auto plus = [one](f32x2 a, f32x2 b) { return plus2(a, b, one); };
  const auto minus = [one](f32x2 a, f32x2 b) { return minus2(a, b, one); };
  // trilinear weights of the corners (order a..h: x fastest, then y, z)
  const f32x2 cw[8] = {
      minus(plus(plus(plus(minus(minus(minus(kOne, u), v), w), uv), uw), vw), uvw),
      plus(minus(minus(u, uv), uw), uvw),
      plus(minus(minus(v, uv), vw), uvw),
      minus(uv, uvw),
      plus(minus(minus(w, uw), vw), uvw),
      minus(uw, uvw),
      minus(vw, uvw),
      uvw};
  f32x2 c[8], sx = 0ull, sy = 0ull, sz = 0ull;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const f32x2 gx =
        pack2(__uint_as_float(lo[k] & 0xFF000000u), __uint_as_float(hi[k] & 0xFF000000u));
    const f32x2 gy = pack2(__uint_as_float(__byte_perm(lo[k], 0u, 0x2444)),
                           __uint_as_float(__byte_perm(hi[k], 0u, 0x2444)));
    const f32x2 gz = pack2(__uint_as_float(lo[k] << 24), __uint_as_float(hi[k] << 24));
    c[k] = fma2(gz, k & 4 ? z1 : tz, fma2(gy, k & 2 ? y1 : ty, mul2(gx, k & 1 ? x1 : tx)));
    sx = fma2(cw[k], gx, sx);
    sy = fma2(cw[k], gy, sy);
    sz = fma2(cw[k], gz, sz);
  }
  const f32x2 k1 = sub2(c[1], c[0]), k2 = sub2(c[2], c[0]), k3 = sub2(c[4], c[0]);
  const f32x2 k4 = sub2(sub2(add2(c[0], c[3]), c[1]), c[2]);
  const f32x2 k5 = sub2(sub2(add2(c[0], c[5]), c[1]), c[4]);
  const f32x2 k6 = sub2(sub2(add2(c[0], c[6]), c[2]), c[4]);
  const f32x2 k7 =
      sub2(sub2(sub2(sub2(add2(add2(add2(c[1], c[2]), c[4]), c[7]), c[0]), c[3]), c[5]), c[6]);
  const f32x2 du = mul2(mul2(k30, mul2(tx, tx)), mul2(x1, x1));
  const f32x2 dv = mul2(mul2(k30, mul2(ty, ty)), mul2(y1, y1));
  const f32x2 dw = mul2(mul2(k30, mul2(tz, tz)), mul2(z1, z1));
  rx = plus(sx, mul2(du, plus(plus(plus(k1, mul2(k4, v)), mul2(k5, w)), mul2(k7, vw))));
  ry = plus(sy, mul2(dv, plus(plus(plus(k2, mul2(k4, u)), mul2(k6, w)), mul2(k7, uw))));
  rz = plus(sz, mul2(dw, plus(plus(plus(k3, mul2(k5, u)), mul2(k6, v)), mul2(k7, uv))));
}

// Gradient of terrain_density: (0, 1, 0) - amp * scale * sum_i gain^i
// lacunarity^i grad perlin(lacunarity^i scale p), lacunarity 2, gain 0.5
// (each octave's amplitude x frequency is 1).  Octaves in pairs, as
// terrain_density() evaluates them.  one: 1.0f (plus2).
template <uint32_t STRIDE, uint32_t G>
__device__ __forceinline__ V3 terrain_gradient(const FieldTable<STRIDE, G>& R, V3 p,
                                               uint32_t octaves, float scale, float amp,
                                               float one) {
  const float x = scale * p.x, y = scale * p.y, z = scale * p.z;
  const float lim = __uint_as_float((127u + 22u - octaves) << 23);
  V3 s = v3(0.f, 0.f, 0.f);
  if (fabsf(x) < lim && fabsf(y) < lim && fabsf(z) < lim) {
    const f32x2 kFour = pack2(4.0f, 4.0f);
    f32x2 X = pack2(x, 2.0f * x), Y = pack2(y, 2.0f * y), Z = pack2(z, 2.0f * z);
#pragma unroll 1
    for (uint32_t i = 0; i < octaves; i += 2) {
      f32x2 gx, gy, gz;
      perlin_grad2(R, X, Y, Z, one, gx, gy, gz);
      float x0, x1, y0, y1, z0, z1;
      unpack2(gx, x0, x1);
      unpack2(gy, y0, y1);
      unpack2(gz, z0, z1);
      s = v3(s.x + 0.5f * x0, s.y + 0.5f * y0, s.z + 0.5f * z0);
      if (i + 1u < octaves) s = v3(s.x + 0.5f * x1, s.y + 0.5f * y1, s.z + 0.5f * z1);
      X = mul2(X, kFour);
      Y = mul2(Y, kFour);
      Z = mul2(Z, kFour);
    }
  } else {
    s = gradient_far<STRIDE>(R.base, x, y, z, octaves);
  }
  const float k = -amp * scale;
  return v3(k * s.x, __fmaf_rn(k, s.y, 1.0f), k * s.z);
}

}  // namespace re
