// Neural SDF surrogate of the volumetric terrain (config 3 of the path).
//
// The reference has no learned component.  The network stands in for the
// fBm terrain density (sdf_functions.cuh:147-206, d(p) = p.y - 3 fBm(p/4) in
// the configs) during sphere tracing; the exact field stays the arbiter and
// finishes every hit (sphere_tracing.cuh:183-216 restated in re_noise.cu).
//
//   data      k_nsdf_data: 50% points uniform in the view box, 50% near the
//             surface (exact-traced camera hits + N(0, 0.02) offsets),
//             labelled by the exact field's first-order distance d / |grad d|
//   training  tcgen05 as well: k_tc_train runs a tile's features, 4 MMA layers
//             with FP32 bias + softplus epilogues, head, L1 loss and the whole
//             backward pass (dA_prev = dZ W and dW^T = A^T dZ) without leaving
//             the SM, pre-activations and weight gradients in tensor memory,
//             BF16 operands and FP32 accumulation; then k_train_reduce sums
//             the CTAs' gradients and applies hand-written Adam; one step is
//             captured once in a CUDA graph and replayed
//   inference tcgen05 (sm_100a): 128-point tiles, BF16 operands in shared
//             memory (K-major canonical layout, no swizzle), FP32
//             accumulators in tensor memory, one elected thread issues the
//             MMAs and commits to an mbarrier; softplus epilogue from TMEM
//   tracing   k_nsdf_march (persistent, lane refill) steps by the network's
//             distance scaled by its measured Lipschitz bound until it is
//             within `switch_dist` of the surface, then k_sdf_refine finishes
//             the ray with exact-field steps and the exact normal.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <random>
#include <vector>

#include "re_common.hpp"
#include "re_noise.cuh"
#include "re_nsdf.cuh"

namespace re {
namespace nsdf {

// ------------------------------------------------------------ shared
struct FieldDev {
  uint32_t octaves, max_steps;
  float scale, amp, step_factor, eps, tmax;
};

__device__ __forceinline__ uint32_t mix32(uint32_t a, uint32_t b, uint32_t c) {
  return hash_u32(a, b, c);
}
__device__ __forceinline__ float u01(uint32_t h) { return (float)(h >> 8) * 5.9604644775390625e-08f; }

// ------------------------------------------------------ data generation
// 768 threads: with 640 a second round of rays begins at 94,720 points (130,000
// points 750 -> 647 us, one octave at a time on 16 copies 693); 1,000 points
// 256 -> 131 us with a warp to each SM.
constexpr uint32_t kDataThreads = 768;

__global__ void __launch_bounds__(kDataThreads) k_nsdf_data(PermTable perm, FieldDev f, CamDev cam,
                                                            uint32_t w, uint32_t h, float3 bmin,
                                                            float3 bmax, uint32_t n, uint32_t seed,
                                                            float4* __restrict__ out) {
  extern __shared__ uint32_t rows_smem[];
  const FieldRows P = load_rows(perm, rows_smem);
  // the warps of all blocks in turn, so that few points spread over the SMs
  const uint32_t first = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32u + (threadIdx.x & 31u);
  for (uint32_t i = first; i < n; i += gridDim.x * blockDim.x) {
    float px = 0.f, py = 0.f, pz = 0.f;
    bool placed = false;
    if (i & 1u) {
      // near-surface sample: an exact-traced camera hit plus N(0, 0.02) per axis
      uint32_t pix = mix32(seed, i, 11u) % (w * h);
      V3 o, d;
      generate_ray(cam, w, h, pix % w, pix / w, o, d);
      float t = 0.f;
      for (uint32_t s = 0; s < f.max_steps; ++s) {
        V3 p = v3(__fmaf_rn(t, d.x, o.x), __fmaf_rn(t, d.y, o.y), __fmaf_rn(t, d.z, o.z));
        float dist = terrain_density(P, p, f.octaves, f.scale, f.amp);
        if (dist < f.eps) {
          float u1 = fmaxf(u01(mix32(seed, i, 12u)), 1e-7f), u2 = u01(mix32(seed, i, 13u));
          float u3 = fmaxf(u01(mix32(seed, i, 14u)), 1e-7f), u4 = u01(mix32(seed, i, 15u));
          float r1 = sqrtf(-2.f * __logf(u1)), r2 = sqrtf(-2.f * __logf(u3));
          float s1, c1, s2, c2;
          __sincosf(6.28318531f * u2, &s1, &c1);
          __sincosf(6.28318531f * u4, &s2, &c2);
          px = p.x + 0.02f * r1 * c1;
          py = p.y + 0.02f * r1 * s1;
          pz = p.z + 0.02f * r2 * c2;
          placed = px >= bmin.x && px <= bmax.x && py >= bmin.y && py <= bmax.y &&
                   pz >= bmin.z && pz <= bmax.z;
          break;
        }
        t = __fmaf_rn(f.step_factor, dist, t);
        if (t > f.tmax) break;
      }
    }
    if (!placed) {
      px = bmin.x + (bmax.x - bmin.x) * u01(mix32(seed, i, 1u));
      py = bmin.y + (bmax.y - bmin.y) * u01(mix32(seed, i, 2u));
      pz = bmin.z + (bmax.z - bmin.z) * u01(mix32(seed, i, 3u));
    }
    // label: first-order distance d / |grad d| of the exact field, clipped
    const float e = 1e-3f;
    float d0 = terrain_density(P, v3(px, py, pz), f.octaves, f.scale, f.amp);
    float gx = terrain_density(P, v3(px + e, py, pz), f.octaves, f.scale, f.amp) -
               terrain_density(P, v3(px - e, py, pz), f.octaves, f.scale, f.amp);
    float gy = terrain_density(P, v3(px, py + e, pz), f.octaves, f.scale, f.amp) -
               terrain_density(P, v3(px, py - e, pz), f.octaves, f.scale, f.amp);
    float gz = terrain_density(P, v3(px, py, pz + e), f.octaves, f.scale, f.amp) -
               terrain_density(P, v3(px, py, pz - e), f.octaves, f.scale, f.amp);
    float g = sqrtf(gx * gx + gy * gy + gz * gz) / (2.f * e);
    float label = d0 / fmaxf(g, 0.25f);
    label = fminf(fmaxf(label, -4.f), 4.f);
    out[i] = make_float4(px, py, pz, label);
  }
}

// ------------------------------------------------------------- training
// One step on a batch of B rows (a multiple of 512): k_tc_train (below) leaves
// one partial gradient and loss per CTA, k_train_reduce sums them and, when
// training, applies Adam.
constexpr int kRowsBwd = 512;   // batch granularity of the training API
constexpr int kTrRows = 128;    // rows per tensor-core tile
// one CTA's partial sums: the gradient in the parameters' order, then the loss
constexpr uint32_t kPartStride = (uint32_t)kNumParams + 1u;

// Sum of the partial gradients, in a fixed order: 8 warps of a block each sum
// every 8th CTA's partials of the block's 32 parameters, then one warp adds
// the 8 sums.  adam_m null: grad gets the sums.  Otherwise the parameters
// get one Adam step, the step's loss is appended to loss_hist, and the last
// block to finish advances the step counter (ctr[0]; ctr[1] counts blocks).
// A thread per parameter that walked every partial by itself took as long as
// its chain of loads (82 blocks, 444 + 512 dependent additions); here 651
// blocks walk at most 19.
constexpr uint32_t kReduceWarps = 8;
__global__ void __launch_bounds__(32 * kReduceWarps) k_train_reduce(
    const float* __restrict__ part, uint32_t nparts, float* __restrict__ grad,
    float* __restrict__ params, float* __restrict__ adam_m, float* __restrict__ adam_v,
    float* __restrict__ loss_hist, uint32_t* __restrict__ ctr, float lr, uint32_t batch) {
  __shared__ float sums[kReduceWarps][32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t p = blockIdx.x * 32u + lane;
  float s = 0.f;
  if (p < kPartStride) {
#pragma unroll 4
    for (uint32_t b = warp; b < nparts; b += kReduceWarps) s += part[(size_t)b * kPartStride + p];
  }
  sums[warp][lane] = s;
  __syncthreads();
  if (warp != 0) return;
#pragma unroll
  for (uint32_t k = 1; k < kReduceWarps; ++k) s += sums[k][lane];
  if (!adam_m) {
    if (p < (uint32_t)kNumParams) grad[p] = s;
    return;
  }
  const uint32_t step = *(volatile const uint32_t*)ctr;
  if (p < (uint32_t)kNumParams) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    float mm = b1 * adam_m[p] + (1.f - b1) * s;
    float vv = b2 * adam_v[p] + (1.f - b2) * s * s;
    adam_m[p] = mm;
    adam_v[p] = vv;
    float mh = mm / (1.f - powf(b1, (float)(step + 1u)));
    float vh = vv / (1.f - powf(b2, (float)(step + 1u)));
    params[p] -= lr * mh / (sqrtf(vh) + eps);
  } else if (p == (uint32_t)kNumParams) {
    loss_hist[step] = s / (float)batch;
  }
  __syncwarp();
  if (lane == 0) {
    __threadfence();  // this block has read the step before it counts as done
    if (atomicAdd(&ctr[1], 1u) == gridDim.x - 1u) {
      ctr[1] = 0u;
      ctr[0] = step + 1u;
    }
  }
}

// ------------------------------------------------ tensor-core inference
// Canonical K-major BF16 layout without swizzle: 8 rows x 8 k-elements
// (16 B per row) form a 128-byte core matrix; core matrices follow each
// other along K every 128 B (LBO) and along rows every K*16 B (SBO).
__host__ __device__ __forceinline__ uint32_t canon_off(uint32_t row, uint32_t k, uint32_t K) {
  return (row >> 3) * (K * 16u) + (k >> 3) * 128u + (row & 7u) * 16u + (k & 7u) * 2u;
}

// Packed inference weights: W1 (64x128), W2..W4 (64x64) in the canonical
// layout, then FP32 b1..b4, w5 (BF16-rounded) and b5.
constexpr uint32_t kPackW1 = kHidden * kIn * 2;            // 16384
constexpr uint32_t kPackWh = kHidden * kHidden * 2;        // 8192
constexpr uint32_t kPackWBytes = kPackW1 + 3 * kPackWh;    // 40960
constexpr uint32_t kPackFloats = 4 * kHidden + kHidden + 1;
constexpr uint32_t kPackBytes = kPackWBytes + kPackFloats * 4;
constexpr uint32_t kBiasCol = 99;    // feature = 1.0; W1 column = BF16(b1)
constexpr uint32_t kBiasColLo = 100; // feature = 1.0; W1 column = b1 - BF16(b1)

// The inference kernels feed 1.0 at W1 columns 99 and 100 (unused by the
// features), so those columns carry b1 as a BF16 high part and a BF16
// remainder and the first layer's bias comes out of the MMA.
__global__ void k_pack(const float* __restrict__ params, unsigned char* __restrict__ pack) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < (uint32_t)(kHidden * kIn)) {
    uint32_t n = i / kIn, k = i % kIn;
    float v = params[OFF_W1 + i];
    if (k == kBiasCol) v = bf16_round(params[OFF_B1 + n]);
    if (k == kBiasColLo) v = params[OFF_B1 + n] - bf16_round(params[OFF_B1 + n]);
    *reinterpret_cast<__nv_bfloat16*>(pack + canon_off(n, k, kIn)) = __float2bfloat16_rn(v);
  }
  if (i < (uint32_t)(3 * kHidden * kHidden)) {
    uint32_t l = i / (kHidden * kHidden), e = i % (kHidden * kHidden);
    uint32_t n = e / kHidden, k = e % kHidden;
    *reinterpret_cast<__nv_bfloat16*>(pack + kPackW1 + l * kPackWh + canon_off(n, k, kHidden)) =
        __float2bfloat16_rn(params[w_off(1 + l) + e]);
  }
  if (i < kPackFloats) {
    float* f = reinterpret_cast<float*>(pack + kPackWBytes);
    float v;
    if (i < 4u * kHidden)
      v = params[b_off(i / kHidden) + i % kHidden];
    else if (i < 5u * kHidden)
      v = bf16_round(params[OFF_W5 + i - 4 * kHidden]);
    else
      v = params[OFF_B5];
    f[i] = v;
  }
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Operand descriptor.  sbo: stride between groups of 8 along M or N; lbo:
// between groups of 8 along K (128 bytes when K is the contiguous dimension).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t sbo_bytes,
                                              uint32_t lbo_bytes = 128u) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: D FP32, A/B BF16, both K-major, N = 64, M = 128
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((64u >> 3) << 17) |
                            ((128u >> 4) << 24);

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t acc,
                                         uint32_t idesc = kIdesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_addr(bar))
      : "memory");
}

// Bounded wait on an mbarrier phase; false if the bound was reached.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  uint32_t a = smem_addr(bar);
  for (uint32_t i = 0; i < (1u << 24); ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Sets an error word in host memory (re_nsdf::sync_err).
__device__ __forceinline__ void report(int* word) {
  *reinterpret_cast<volatile int*>(word) = 1;
  __threadfence_system();
}

// The end of a kernel whose threads each kept whether their own waits came
// through: all of them call it, and one that ran out, whichever thread's it
// was, is reported.
__device__ __forceinline__ void report_block(bool ok, int* word) {
  ok = __syncthreads_and(ok);
  if (!ok && threadIdx.x == 0) report(word);
}

__device__ __forceinline__ void fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// ---- packed BF16x2 arithmetic (two activations per instruction)
__device__ __forceinline__ uint32_t bf2_fma(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t bf2_mul(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t bf2_max(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t bf2_ex2(uint32_t a) {
  uint32_t d;
  asm("ex2.approx.ftz.bf16x2 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}

// BF16 pairs {lo, hi} of constants
constexpr uint32_t bf2_const(uint32_t bits) { return bits | (bits << 16); }
constexpr uint32_t kBf2Log2e = bf2_const(0x3FB9u);   // 1.4453125 ~ log2(e)
constexpr uint32_t kBf2C1 = bf2_const(0x3F7Cu);      // 0.984375
constexpr uint32_t kBf2C2 = bf2_const(0xBECFu);      // -0.404296875
constexpr uint32_t kBf2C3 = bf2_const(0x3DE6u);      // 0.1123046875

// softplus of two BF16 pre-activations in BF16 arithmetic:
// max(z, 0) + u (c1 + u (c2 + u c3)) with u = 2^(-|z| log2 e), the cubic a
// least-squares fit of log1p(u) / u on [0, 1] (coefficients rounded to
// BF16).  Against softplus in FP32 rounded once to BF16 (the training
// arithmetic) the pre-activation is rounded twice; the difference is at
// most one BF16 unit in the last place of the activation.
__device__ __forceinline__ uint32_t softplus_bf16x2(uint32_t z) {
  uint32_t u = bf2_ex2(bf2_mul(z | 0x80008000u, kBf2Log2e));
  uint32_t q = bf2_fma(kBf2C3, u, kBf2C2);
  q = bf2_fma(q, u, kBf2C1);
  return bf2_fma(q, u, bf2_max(z, 0u));
}

// Tensor-core inference: each CTA runs kGroups independent pipelines of 128
// rows (one thread per row, 4 warps per group, one warp of every group on
// each SM sub-partition).  A group computes its rows' features, then for
// each layer: one elected thread issues the MMAs into the group's 64 TMEM
// columns and commits to the group's mbarrier; the group reads its
// accumulators back, applies bias and softplus, and writes the next
// layer's BF16 input.  While one group waits on its MMAs the others run
// their epilogues, which hides the tensor-core latency.
constexpr int kGroups = 4;
constexpr int kGroupRows = 128;
constexpr int kTcThreads = kGroups * kGroupRows;  // 512
constexpr uint32_t kTmemCols = 64 * kGroups;      // 256

struct __align__(1024) TcSmem {
  unsigned char w[kPackWBytes];               // W1..W4, canonical
  unsigned char x[kGroups][kGroupRows * kIn * 2];  // per-group layer input (K = 128 or 64)
  float bias[3][kHidden];                     // b2..b4 (b1 rides in W1)
  float w5[kHidden];
  float b5;
  uint64_t bar[kGroups];
  uint32_t tmem;
};

__device__ __forceinline__ void group_sync(int g) {
  asm volatile("bar.sync %0, 128;" ::"r"(g + 1) : "memory");
}
__device__ __forceinline__ bool group_and(int g, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "r"(g + 1)
      : "memory");
  return r != 0u;
}
__device__ __forceinline__ bool group_or(int g, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "bar.red.or.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "r"(g + 1)
      : "memory");
  return r != 0u;
}

__device__ __forceinline__ void store_chunk(unsigned char* x, int row, int k, uint32_t K, uint32_t a,
                                            uint32_t b, uint32_t c, uint32_t d) {
  *reinterpret_cast<uint4*>(x + canon_off(row, k, K)) = make_uint4(a, b, c, d);
}

// Network value of this thread's row (q = normalised point).  Called by the
// 128 threads of group g together; `ok` turns false if an MMA did not
// complete within the wait bound (the caller makes it group-uniform).
__device__ __forceinline__ float mlp_row(TcSmem& s, const InputMap& m, int g, int row,
                                         const float q[3], uint32_t& phase, bool& ok) {
  unsigned char* x = s.x[g];
  {
    float v[48];
#pragma unroll
    for (int chain = 0; chain < 2; ++chain) {
      chain_features(m, q, chain, v);
#pragma unroll
      for (int c = 0; c < 6; ++c)
        store_chunk(x, row, (chain * 6 + c) * 8, kIn, pack_bf16x2(v[c * 8 + 0], v[c * 8 + 1]),
                    pack_bf16x2(v[c * 8 + 2], v[c * 8 + 3]), pack_bf16x2(v[c * 8 + 4], v[c * 8 + 5]),
                    pack_bf16x2(v[c * 8 + 6], v[c * 8 + 7]));
    }
    // k = 96..103: q.xyz, the two bias inputs (1.0), zeros; 104..127 zero
    store_chunk(x, row, 96, kIn, pack_bf16x2(q[0], q[1]), pack_bf16x2(q[2], 1.0f),
                pack_bf16x2(1.0f, 0.f), 0u);
#pragma unroll
    for (int c = 13; c < 16; ++c) store_chunk(x, row, c * 8, kIn, 0u, 0u, 0u, 0u);
  }
  const uint32_t wq = (uint32_t)(row >> 5);  // warp within the group = TMEM lane quarter
  const uint32_t tcol = s.tmem + ((32u * wq) << 16) + 64u * (uint32_t)g;
  float d = 0.f;
#pragma unroll 1
  for (int layer = 0; layer < 4; ++layer) {
    const uint32_t K = layer == 0 ? kIn : kHidden;
    fence_async_smem();
    fence_before();
    group_sync(g);
    fence_after();
    if (row == 0) {
      uint32_t xa = smem_addr(x);
      uint32_t wa = smem_addr(s.w + (layer == 0 ? 0u : kPackW1 + (layer - 1) * kPackWh));
#pragma unroll 1
      for (uint32_t kk = 0; kk < K / 16; ++kk)
        mma_bf16(s.tmem + 64u * (uint32_t)g, umma_desc(xa + kk * 256u, K * 16u),
                 umma_desc(wa + kk * 256u, K * 16u), kk > 0 ? 1u : 0u);
      mma_commit(&s.bar[g]);
    }
    ok = mbar_wait(&s.bar[g], phase) && ok;
    phase ^= 1u;
    __syncwarp();
    fence_after();
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float acc[32];
      tmem_ld32(tcol + 32u * (uint32_t)half, acc);
      if (layer > 0) {
        const float4* b4 = reinterpret_cast<const float4*>(s.bias[layer - 1]) + 8 * half;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float4 bb = b4[j];
          acc[4 * j] += bb.x;
          acc[4 * j + 1] += bb.y;
          acc[4 * j + 2] += bb.z;
          acc[4 * j + 3] += bb.w;
        }
      }
      uint32_t a[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) a[j] = softplus_bf16x2(pack_bf16x2(acc[2 * j], acc[2 * j + 1]));
      if (layer < 3) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          store_chunk(x, row, 32 * half + 8 * c, kHidden, a[4 * c], a[4 * c + 1], a[4 * c + 2],
                      a[4 * c + 3]);
      } else {
        const float4* w4 = reinterpret_cast<const float4*>(s.w5) + 8 * half;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float4 ww = w4[j];
          d = __fmaf_rn(__uint_as_float(a[2 * j] << 16), ww.x, d);
          d = __fmaf_rn(__uint_as_float(a[2 * j] & 0xFFFF0000u), ww.y, d);
          d = __fmaf_rn(__uint_as_float(a[2 * j + 1] << 16), ww.z, d);
          d = __fmaf_rn(__uint_as_float(a[2 * j + 1] & 0xFFFF0000u), ww.w, d);
        }
      }
    }
    // every thread has read its accumulators before the next MMA overwrites them
    fence_before();
  }
  return d + s.b5;
}

__device__ __forceinline__ void tc_setup(TcSmem& s, const unsigned char* __restrict__ pack) {
  int tid = threadIdx.x;
  for (uint32_t i = tid; i < kPackWBytes / 16; i += blockDim.x)
    reinterpret_cast<uint4*>(s.w)[i] = __ldg(reinterpret_cast<const uint4*>(pack) + i);
  const float* f = reinterpret_cast<const float*>(pack + kPackWBytes);
  for (uint32_t i = tid; i < 3 * kHidden; i += blockDim.x)
    s.bias[i / kHidden][i % kHidden] = f[kHidden + i];
  for (uint32_t i = tid; i < kHidden; i += blockDim.x) s.w5[i] = f[4 * kHidden + i];
  if (tid == 0) {
    s.b5 = f[5 * kHidden];
    for (int g = 0; g < kGroups; ++g)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s.bar[g])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if ((tid >> 5) == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(&s.tmem)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
}

__device__ __forceinline__ void tc_teardown(TcSmem& s) {
  fence_before();
  __syncthreads();
  fence_after();
  if ((threadIdx.x >> 5) == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s.tmem),
                 "r"(kTmemCols));
}

__device__ __forceinline__ TcSmem& tc_smem(unsigned char* raw) {
  return *reinterpret_cast<TcSmem*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
}

// Reference evaluation with the training arithmetic (SIMT FP32, BF16-rounded
// weights and activations), one thread per point.
__global__ void __launch_bounds__(128) k_ref_eval(InputMap m, const float* __restrict__ params,
                                                  const float* __restrict__ pts, uint32_t n,
                                                  float* __restrict__ out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float x[kIn];
  float q[3];
  normalise(m, pts[3 * (size_t)i], pts[3 * (size_t)i + 1], pts[3 * (size_t)i + 2], q);
  float v[48];
  chain_features(m, q, 0, v);
  for (int k = 0; k < 48; ++k) x[k] = bf16_round(v[k]);
  chain_features(m, q, 1, v);
  for (int k = 0; k < 48; ++k) x[48 + k] = bf16_round(v[k]);
  x[96] = bf16_round(q[0]);
  x[97] = bf16_round(q[1]);
  x[98] = bf16_round(q[2]);
  for (int k = 99; k < kIn; ++k) x[k] = 0.f;
  float h[kHidden], h2[kHidden];
  for (int c = 0; c < kHidden; ++c) {
    float z = 0.f;
    for (int k = 0; k < kIn; ++k) z = __fmaf_rn(x[k], bf16_round(params[OFF_W1 + c * kIn + k]), z);
    h[c] = bf16_round(softplus_approx(z + params[OFF_B1 + c]));
  }
  for (int l = 1; l < 4; ++l) {
    for (int c = 0; c < kHidden; ++c) {
      float z = 0.f;
      for (int k = 0; k < kHidden; ++k)
        z = __fmaf_rn(h[k], bf16_round(params[w_off(l) + c * kHidden + k]), z);
      h2[c] = bf16_round(softplus_approx(z + params[b_off(l) + c]));
    }
    for (int c = 0; c < kHidden; ++c) h[c] = h2[c];
  }
  float d = 0.f;
  for (int c = 0; c < kHidden; ++c) d = __fmaf_rn(h[c], bf16_round(params[OFF_W5 + c]), d);
  out[i] = d + params[OFF_B5];
}

// ------------------------------------------------ tensor-core training
// k_tc_train: one CTA takes 128-row tiles of the batch and carries each
// through the forward pass, the loss and the backward pass.
//
// Four threads share a row (warp w: rows 32 (w & 3) .. + 31, the lanes of
// tensor memory it may read; columns 16 (w >> 2) .. + 15 of a layer), so an
// epilogue holds 16 values a thread and 16 warps are there to hide the
// latency of the chain MMA -> load -> softplus -> store -> MMA, 8 links a
// tile.
//
// Nothing of a tile goes to memory.  The pre-activations Z1..Z4 stay in
// tensor memory as FP32 accumulators (columns 0..255) until the backward
// pass has read them; dA of the layer below then takes the same columns.
// The weight gradients dW1^T..dW4^T stay in columns 256..511 over all of the
// CTA's tiles.  Activations (BF16, the MMA operands) stay in shared memory.
//
// Every operand is stored once: a core matrix of 8 rows x 16 bytes reads as
// K-major when the contiguous 8 elements run along K, and as MN-major when
// they run along M or N, with the two strides exchanged.  So A_prev (rows x
// inputs) is the A operand of the layer (K = inputs) and, transposed by the
// descriptor, of dW^T = A_prev^T dZ (M = inputs, K = rows); dZ is the A
// operand of dA = dZ W and the B operand of dW^T; W (outputs x inputs) is
// the B operand of the layer and of dA.
//
// The bias gradient rides in dW^T: an input column of ones (99 of the
// features, whose weights are packed as zero, and 64 of the activations)
// makes that accumulator row sum_b dZ.  With 64 inputs, M = 128 reads past
// the ones column into the next row group; those accumulator rows are never
// read.
//
// Measured on B200, 65,536 rows: one forward launch that stored 257 MB of
// activations and four backward launches that read them back and transposed
// the operands with 2-byte stores, the reduction and the copies took 308 us
// a re_nsdf_loss_grad call; this kernel 60 us, the reduction 7 us, the call
// 80 us.  What is left is the chain of links (issue slots 41 % busy on the 128
// SMs in use, 4 rounds of tiles at 15 us).
constexpr int kTrainThreads = 512;
constexpr uint32_t kActCols = 72;       // 64 activations, the ones column, 7 zeros
constexpr uint32_t kOnesX = 99;         // column of ones in the features
constexpr uint32_t kFeatK = 112;        // features in use (99) and the ones, in steps of 16
constexpr uint32_t kTrainCols = 512;    // tensor-memory columns
constexpr uint32_t kIdescTransA = 1u << 15, kIdescTransB = 1u << 16;  // MN-major A, B

struct __align__(1024) TrainSmem {
  unsigned char w[kPackWBytes];                   // W1..W4, canonical
  unsigned char x[kTrRows * kIn * 2];             // features
  unsigned char a[3][kTrRows * kActCols * 2];     // activations of layers 1..3
  unsigned char dz[2][kTrRows * kHidden * 2];     // dZ, two layers in turn
  float bias[4][kHidden];
  float w5[kHidden];
  float head[4][kTrRows];                         // the row's output by column quarter
  float red[4][kHidden + 2];                      // w5, b5 and loss sums by row quarter
  float b5;
  uint64_t bar;
  uint32_t tmem;
};
constexpr size_t kTrainSmemBytes = sizeof(TrainSmem) + 1024;

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Octaves 4 half .. 4 half + 3 of a chain's features (chain_features, 24 of
// its 48 values), the doublings below them carried through.
__device__ __forceinline__ void half_chain(const InputMap& m, const float q[3], int chain,
                                           int half, float out[24]) {
  float f = chain ? m.f0 * 1.41421356f : m.f0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    float arg = f * q[j];
    float r = arg - rintf(arg);
    float s, c;
    __sincosf(6.28318531f * r, &s, &c);
    for (int o = 0; o < 4 * half; ++o) {
      float s2 = 2.0f * s * c;
      c = __fmaf_rn(-2.0f * s, s, 1.0f);
      s = s2;
    }
#pragma unroll
    for (int o = 0; o < kOctaves / 2; ++o) {
      out[o * 6 + 2 * j] = s;
      out[o * 6 + 2 * j + 1] = c;
      float s2 = 2.0f * s * c;
      c = __fmaf_rn(-2.0f * s, s, 1.0f);
      s = s2;
    }
  }
}

// softplus_approx of two values, rounded to BF16, and its derivative (u times
// the derivative of the polynomial; one minus that for x > 0), the
// polynomials in packed FP32 (each half rounded as the scalar form rounds).
__device__ __forceinline__ f32x2 splat2(float c) { return pack2(c, c); }
__device__ __forceinline__ f32x2 exp_neg_abs2(float x0, float x1) {
  return pack2(__expf(-fabsf(x0)), __expf(-fabsf(x1)));
}
__device__ __forceinline__ uint32_t softplus_pair(float x0, float x1) {
  const f32x2 u = exp_neg_abs2(x0, x1);
  f32x2 p = fma2(u, splat2(-0.017806457f), splat2(0.083866805f));
  p = fma2(u, p, splat2(-0.19167475f));
  p = fma2(u, p, splat2(0.31643057f));
  p = fma2(u, p, splat2(-0.49753284f));
  p = fma2(u, p, splat2(0.9998613f));
  float a, b;
  unpack2(mul2(u, p), a, b);
  return pack_bf16x2(__fadd_rn(fmaxf(x0, 0.0f), a), __fadd_rn(fmaxf(x1, 0.0f), b));
}
__device__ __forceinline__ f32x2 softplus_deriv2(float x0, float x1) {
  const f32x2 u = exp_neg_abs2(x0, x1);
  f32x2 p = fma2(u, splat2(6.0f * -0.017806457f), splat2(5.0f * 0.083866805f));
  p = fma2(u, p, splat2(4.0f * -0.19167475f));
  p = fma2(u, p, splat2(3.0f * 0.31643057f));
  p = fma2(u, p, splat2(2.0f * -0.49753284f));
  p = fma2(u, p, splat2(0.9998613f));
  float g0, g1;
  unpack2(mul2(u, p), g0, g1);
  return pack2(x0 > 0.0f ? __fsub_rn(1.0f, g0) : g0, x1 > 0.0f ? __fsub_rn(1.0f, g1) : g1);
}

// z += this thread's 16 biases.
__device__ __forceinline__ void add_bias16(float (&z)[16], const float* bias) {
  const float4* b4 = reinterpret_cast<const float4*>(bias);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 b = b4[j];
    unpack2(add2(pack2(z[4 * j], z[4 * j + 1]), pack2(b.x, b.y)), z[4 * j], z[4 * j + 1]);
    unpack2(add2(pack2(z[4 * j + 2], z[4 * j + 3]), pack2(b.z, b.w)), z[4 * j + 2], z[4 * j + 3]);
  }
}

// Stores are visible to the MMAs and every thread's tensor-memory reads are
// done before the next ones are issued.
__device__ __forceinline__ void train_sync() {
  fence_async_smem();
  fence_before();
  __syncthreads();
  fence_after();
}

__global__ void __launch_bounds__(kTrainThreads, 1) k_tc_train(
    InputMap m, const float4* __restrict__ data, uint32_t npts,
    const uint32_t* __restrict__ step_ctr, uint32_t seed, int direct,
    const float* __restrict__ params, float* __restrict__ part, uint32_t batch,
    float* __restrict__ pred_out, int* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  TrainSmem& s = *reinterpret_cast<TrainSmem*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x;
  const int row = tid & 127, quarter = tid >> 7;  // quarter: columns 16 quarter .. + 15
  const int col = 16 * quarter;
  // BF16 weights, 8 inputs of an output at a time
  for (int i = tid; i < kHidden * (kIn + 3 * kHidden) / 8; i += kTrainThreads) {
    const bool first = i < kHidden * kIn / 8;
    const int l = first ? 0 : 1 + (i - kHidden * kIn / 8) / (kHidden * kHidden / 8);
    const int e = first ? i : (i - kHidden * kIn / 8) % (kHidden * kHidden / 8);
    const uint32_t K = first ? kIn : kHidden;
    const uint32_t n = (uint32_t)e / (K / 8), k = ((uint32_t)e % (K / 8)) * 8u;
    const float4* src = reinterpret_cast<const float4*>(params + w_off(l) + n * K + k);
    float4 u = src[0], v = src[1];
    if (first && k >= 96u) {  // the features end at column 98
      if (k > 96u) u = make_float4(0.f, 0.f, 0.f, 0.f);
      u.w = 0.f;
      v = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    store_chunk(s.w + (first ? 0u : kPackW1 + (uint32_t)(l - 1) * kPackWh), (int)n, (int)k, K,
                pack_bf16x2(u.x, u.y), pack_bf16x2(u.z, u.w), pack_bf16x2(v.x, v.y),
                pack_bf16x2(v.z, v.w));
  }
  if (tid < 4 * kHidden)
    s.bias[tid / kHidden][tid % kHidden] = params[b_off(tid / kHidden) + tid % kHidden];
  else if (tid < 5 * kHidden)
    s.w5[tid - 4 * kHidden] = bf16_round(params[OFF_W5 + tid - 4 * kHidden]);
  // the constant columns: zeros past the features, the activations' ones
  if (quarter == 0) {
#pragma unroll
    for (int c = 13; c < 16; ++c) store_chunk(s.x, row, 8 * c, kIn, 0u, 0u, 0u, 0u);
  } else {
    store_chunk(s.a[quarter - 1], row, kHidden, kActCols, 0x3F80u, 0u, 0u, 0u);
  }
  if (tid == 0) {
    s.b5 = params[OFF_B5];
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s.bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // every column of the SM: shared memory admits no second CTA of this
  // kernel, and the inference kernels' CTAs give theirs back when they end
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(&s.tmem)),
                 "r"(kTrainCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  train_sync();
  // this thread's lanes and columns of a 64-column accumulator
  const uint32_t tme = s.tmem + ((32u * (uint32_t)(row >> 5)) << 16) + (uint32_t)col;
  const uint32_t xa = smem_addr(s.x), aa = smem_addr(s.a), da = smem_addr(s.dz),
                 wa = smem_addr(s.w);
  constexpr uint32_t kActBytes = kTrRows * kActCols * 2, kDzBytes = kTrRows * kHidden * 2;
  const uint32_t step = *step_ctr;
  uint32_t phase = 0;
  bool ok = true, started = false;
  float gw5[16], gb5 = 0.f, loss = 0.f;
#pragma unroll
  for (int j = 0; j < 16; ++j) gw5[j] = 0.f;
  const uint32_t tiles = batch / kTrRows;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint32_t b = tile * kTrRows + (uint32_t)row;
    const uint32_t idx = direct ? b : mix32(seed, step, b) % npts;
    const float4 pt = __ldg(&data[idx]);
    float q[3];
    normalise(m, pt.x, pt.y, pt.z, q);
    {
      float v[24];
      const int chain = quarter >> 1, half = quarter & 1;
      half_chain(m, q, chain, half, v);
      // the previous tile's last MMAs read the features
      if (started && ok) ok = mbar_wait(&s.bar, phase);
      if (started) phase ^= 1u;
#pragma unroll
      for (int c = 0; c < 3; ++c)
        store_chunk(s.x, row, (chain * 6 + half * 3 + c) * 8, kIn,
                    pack_bf16x2(v[c * 8 + 0], v[c * 8 + 1]), pack_bf16x2(v[c * 8 + 2], v[c * 8 + 3]),
                    pack_bf16x2(v[c * 8 + 4], v[c * 8 + 5]), pack_bf16x2(v[c * 8 + 6], v[c * 8 + 7]));
      if (quarter == 0)
        store_chunk(s.x, row, 96, kIn, pack_bf16x2(q[0], q[1]), pack_bf16x2(q[2], 1.0f), 0u, 0u);
    }
    float z[16], d = 0.f;
    uint32_t a4[8];
#pragma unroll 1
    for (int l = 0; l < 4; ++l) {
      train_sync();
      if (tid == 0) {
        const uint32_t A = l == 0 ? xa : aa + (uint32_t)(l - 1) * kActBytes;
        const uint32_t B = l == 0 ? wa : wa + kPackW1 + (uint32_t)(l - 1) * kPackWh;
        const uint32_t sa = (l == 0 ? kIn : kActCols) * 16u, sb = (l == 0 ? kIn : kHidden) * 16u;
        const uint32_t steps = (l == 0 ? kFeatK : (uint32_t)kHidden) / 16u;
        for (uint32_t k = 0; k < steps; ++k)
          mma_bf16(s.tmem + 64u * (uint32_t)l, umma_desc(A + k * 256u, sa),
                   umma_desc(B + k * 256u, sb), k > 0u ? 1u : 0u);
        mma_commit(&s.bar);
      }
      if (ok) ok = mbar_wait(&s.bar, phase);
      phase ^= 1u;
      __syncwarp();
      fence_after();
      tmem_ld16(tme + 64u * (uint32_t)l, z);
      add_bias16(z, &s.bias[l][col]);
#pragma unroll
      for (int j = 0; j < 8; ++j) a4[j] = softplus_pair(z[2 * j], z[2 * j + 1]);
      if (l < 3) {
        store_chunk(s.a[l], row, col, kActCols, a4[0], a4[1], a4[2], a4[3]);
        store_chunk(s.a[l], row, col + 8, kActCols, a4[4], a4[5], a4[6], a4[7]);
      }
    }
    // head and L1 loss
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      d = __fmaf_rn(__uint_as_float(a4[j] << 16), s.w5[col + 2 * j], d);
      d = __fmaf_rn(__uint_as_float(a4[j] & 0xFFFF0000u), s.w5[col + 2 * j + 1], d);
    }
    s.head[quarter][row] = d;
    __syncthreads();
    const float pred =
        ((s.head[0][row] + s.head[1][row]) + (s.head[2][row] + s.head[3][row])) + s.b5;
    const float diff = pred - pt.w;
    const float g = (diff > 0.f ? 1.f : (diff < 0.f ? -1.f : 0.f)) / (float)batch;
    if (quarter == 0) {
      if (pred_out) pred_out[b] = pred;
      gb5 += g;
      loss += fabsf(diff);
    }
    float dv[16];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      gw5[2 * j] = __fmaf_rn(g, __uint_as_float(a4[j] << 16), gw5[2 * j]);
      gw5[2 * j + 1] = __fmaf_rn(g, __uint_as_float(a4[j] & 0xFFFF0000u), gw5[2 * j + 1]);
      dv[2 * j] = g * s.w5[col + 2 * j];
      dv[2 * j + 1] = g * s.w5[col + 2 * j + 1];
    }
    // backward: dv = dA and z = Z of layer l
#pragma unroll 1
    for (int l = 3; l >= 0; --l) {
      const uint32_t buf = (uint32_t)(3 - l) & 1u;
      uint32_t pk[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float d0, d1;
        unpack2(mul2(pack2(dv[2 * j], dv[2 * j + 1]), softplus_deriv2(z[2 * j], z[2 * j + 1])), d0,
                d1);
        pk[j] = pack_bf16x2(d0, d1);
      }
      store_chunk(s.dz[buf], row, col, kHidden, pk[0], pk[1], pk[2], pk[3]);
      store_chunk(s.dz[buf], row, col + 8, kHidden, pk[4], pk[5], pk[6], pk[7]);
      train_sync();
      if (tid == 0) {
        const uint32_t D = da + buf * kDzBytes;
        if (l > 0) {
          // dA of the layer below, in Z_l's columns (every thread has read them)
          const uint32_t W = wa + kPackW1 + (uint32_t)(l - 1) * kPackWh;
#pragma unroll 1
          for (uint32_t k = 0; k < kHidden / 16u; ++k)
            mma_bf16(s.tmem + 64u * (uint32_t)l, umma_desc(D + k * 256u, kHidden * 16u),
                     umma_desc(W + k * 2u * kHidden * 16u, 128u, kHidden * 16u), k > 0u ? 1u : 0u,
                     kIdesc | kIdescTransB);
          mma_commit(&s.bar);
        }
        // dW^T over the tile's rows; it runs while the next layer's dZ is
        // made, and the next commit covers it, so this dZ buffer is free
        // again two layers on
        const uint32_t A = l == 0 ? xa : aa + (uint32_t)(l - 1) * kActBytes;
        const uint32_t ga = (l == 0 ? kIn : kActCols) * 16u;
#pragma unroll 1
        for (uint32_t k = 0; k < kTrRows / 16u; ++k)
          mma_bf16(s.tmem + 256u + 64u * (uint32_t)l, umma_desc(A + k * 2u * ga, 128u, ga),
                   umma_desc(D + k * 2u * kHidden * 16u, 128u, kHidden * 16u),
                   started || k > 0u ? 1u : 0u, kIdesc | kIdescTransA | kIdescTransB);
        if (l == 0) mma_commit(&s.bar);
      }
      if (l > 0) {
        if (ok) ok = mbar_wait(&s.bar, phase);
        phase ^= 1u;
        __syncwarp();
        fence_after();
        tmem_ld16(tme + 64u * (uint32_t)l, dv);
        tmem_ld16(tme + 64u * (uint32_t)(l - 1), z);
        add_bias16(z, &s.bias[l - 1][col]);
      }
    }
    started = true;
  }
  // the grid has no CTA without a tile, so `started` holds here
  if (ok) ok = mbar_wait(&s.bar, phase);
  __syncwarp();
  fence_after();
  // this CTA's sums; tensor-memory lane = input k, column = output n
  float* pp = part + (size_t)blockIdx.x * kPartStride;
#pragma unroll 1
  for (int l = 0; l < 4; ++l) {
    const int Kin = l == 0 ? kIn : kHidden, ones = l == 0 ? (int)kOnesX : kHidden;
    float acc[16];
    tmem_ld16(tme + 256u + 64u * (uint32_t)l, acc);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (row < Kin) pp[w_off(l) + (col + j) * Kin + row] = row == ones ? 0.f : acc[j];
      if (row == ones) pp[b_off(l) + col + j] = acc[j];
    }
  }
  // w5, b5 and the loss over the CTA's rows
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int j = 0; j < 16; ++j) gw5[j] += __shfl_xor_sync(0xFFFFFFFFu, gw5[j], off);
    gb5 += __shfl_xor_sync(0xFFFFFFFFu, gb5, off);
    loss += __shfl_xor_sync(0xFFFFFFFFu, loss, off);
  }
  if ((tid & 31) == 0) {
#pragma unroll
    for (int j = 0; j < 16; ++j) s.red[row >> 5][col + j] = gw5[j];
    if (quarter == 0) {
      s.red[row >> 5][kHidden] = gb5;
      s.red[row >> 5][kHidden + 1] = loss;
    }
  }
  report_block(ok, err);
  if (tid < kHidden + 2)
    pp[OFF_W5 + tid] = (s.red[0][tid] + s.red[1][tid]) + (s.red[2][tid] + s.red[3][tid]);
  fence_before();
  __syncthreads();
  fence_after();
  if (tid < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s.tmem),
                 "r"(kTrainCols));
}

// Batch evaluation: out[i] = network(pts[i]), with mlp_row's arithmetic.
//
// What bounds it is the chain of a group's links (store, barrier, MMA, wait,
// load, softplus): 4 groups of 128 rows left the issue slots half idle.
// Here 8 groups share the SM, as many as tensor memory holds, one thread a
// row.  Their operand buffers fit because a row keeps 64 columns: the first
// layer runs as two MMAs over the features of one chain each (48 columns,
// then 48 with the position and bias inputs), which add in the order of one.
//
// Measured on B200, 1,000,003 points: a call 155 -> 128 us (issue slots 53 ->
// 65 % busy; 4 groups with two threads a row: 141 us).
constexpr int kEvalGroups = 8;
constexpr int kEvalThreads = kEvalGroups * kGroupRows;  // 1024
constexpr uint32_t kEvalCols = 64 * kEvalGroups;        // tensor-memory columns

struct __align__(1024) EvalSmem {
  unsigned char w[kPackWBytes];                             // W1..W4, canonical
  unsigned char x[kEvalGroups][kGroupRows * kHidden * 2];   // per-group MMA operand
  float bias[3][kHidden];                                   // b2..b4 (b1 rides in W1)
  float w5[kHidden];
  float b5;
  uint64_t bar[kEvalGroups];
  uint32_t tmem;
};
constexpr size_t kEvalSmemBytes = sizeof(EvalSmem) + 1024;

// One chain's 48 features (chain_features, packed as they are made).
__device__ __forceinline__ void eval_chain(unsigned char* x, const InputMap& m, int row,
                                           const float q[3], int chain) {
  const float f = chain ? m.f0 * 1.41421356f : m.f0;
  float s[3], c[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const float arg = f * q[j];
    const float r = arg - rintf(arg);
    __sincosf(6.28318531f * r, &s[j], &c[j]);
  }
  uint32_t w[4];
#pragma unroll
  for (int o = 0; o < kOctaves; ++o) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int k = 3 * o + j;
      w[k & 3] = pack_bf16x2(s[j], c[j]);
      if ((k & 3) == 3) store_chunk(x, row, 2 * (k - 3), kHidden, w[0], w[1], w[2], w[3]);
      const float s2 = 2.0f * s[j] * c[j];
      c[j] = __fmaf_rn(-2.0f * s[j], s[j], 1.0f);
      s[j] = s2;
    }
  }
}

__global__ void __launch_bounds__(kEvalThreads, 1) k_tc_eval(InputMap m,
                                                             const unsigned char* __restrict__ pack,
                                                             const float* __restrict__ pts,
                                                             uint32_t n, float* __restrict__ out,
                                                             int* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  EvalSmem& s = *reinterpret_cast<EvalSmem*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, g = tid >> 7, row = tid & 127;
  for (uint32_t i = tid; i < kPackWBytes / 16; i += kEvalThreads)
    reinterpret_cast<uint4*>(s.w)[i] = __ldg(reinterpret_cast<const uint4*>(pack) + i);
  const float* f = reinterpret_cast<const float*>(pack + kPackWBytes);
  if (tid < 3 * kHidden) s.bias[tid / kHidden][tid % kHidden] = f[kHidden + tid];
  else if (tid < 4 * kHidden) s.w5[tid - 3 * kHidden] = f[4 * kHidden + tid - 3 * kHidden];
  if (tid == 0) {
    s.b5 = f[5 * kHidden];
    for (int k = 0; k < kEvalGroups; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s.bar[k])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // every column: shared memory admits no second CTA of the kernels that use
  // tensor memory
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(&s.tmem)),
                 "r"(kEvalCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  unsigned char* x = s.x[g];
  const uint32_t dcol = s.tmem + 64u * (uint32_t)g;  // the group's accumulator
  const uint32_t tme = dcol + ((32u * (uint32_t)(row >> 5)) << 16);
  const uint32_t tiles = (n + kGroupRows - 1) / kGroupRows;
  uint32_t phase = 0;
  bool ok = true;
  // group 0 of every CTA first, so that a small call spreads over the SMs
  for (uint32_t tile = g * gridDim.x + blockIdx.x; tile < tiles;
       tile += gridDim.x * kEvalGroups) {
    const uint32_t i = tile * kGroupRows + row;
    const bool live = i < n;
    float q[3];
    normalise(m, live ? __ldg(&pts[3 * (size_t)i]) : 0.f,
              live ? __ldg(&pts[3 * (size_t)i + 1]) : 0.f,
              live ? __ldg(&pts[3 * (size_t)i + 2]) : 0.f, q);
    eval_chain(x, m, row, q, 0);
    float d = 0.f;
    // stage 0, 1: the first layer's two halves; 2, 3, 4: the hidden layers
#pragma unroll 1
    for (int stage = 0; stage < 5; ++stage) {
      fence_async_smem();
      fence_before();
      group_sync(g);
      fence_after();
      if (row == 0) {
        const uint32_t xa = smem_addr(x);
        const uint32_t wa =
            smem_addr(s.w) + (stage < 2 ? 768u * (uint32_t)stage  // inputs from column 48
                                        : kPackW1 + (uint32_t)(stage - 2) * kPackWh);
        const uint32_t sw = (stage < 2 ? (uint32_t)kIn : (uint32_t)kHidden) * 16u;
        const uint32_t steps = stage == 0 ? 3u : 4u;
#pragma unroll 1
        for (uint32_t k = 0; k < steps; ++k)
          mma_bf16(dcol, umma_desc(xa + k * 256u, kHidden * 16u), umma_desc(wa + k * 256u, sw),
                   stage == 1 || k > 0 ? 1u : 0u);
        mma_commit(&s.bar[g]);
      }
      if (ok) ok = mbar_wait(&s.bar[g], phase);
      phase ^= 1u;
      __syncwarp();
      fence_after();
      if (stage == 0) {
        eval_chain(x, m, row, q, 1);
        store_chunk(x, row, 48, kHidden, pack_bf16x2(q[0], q[1]), pack_bf16x2(q[2], 1.0f),
                    pack_bf16x2(1.0f, 0.f), 0u);
        store_chunk(x, row, 56, kHidden, 0u, 0u, 0u, 0u);
        continue;
      }
#pragma unroll
      for (int part = 0; part < 4; ++part) {
        float acc[16];
        uint32_t a[8];
        tmem_ld16(tme + 16u * (uint32_t)part, acc);
        if (stage > 1) add_bias16(acc, &s.bias[stage - 2][16 * part]);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = softplus_bf16x2(pack_bf16x2(acc[2 * j], acc[2 * j + 1]));
        if (stage < 4) {
          store_chunk(x, row, 16 * part, kHidden, a[0], a[1], a[2], a[3]);
          store_chunk(x, row, 16 * part + 8, kHidden, a[4], a[5], a[6], a[7]);
        } else {
          const float4* w4 = reinterpret_cast<const float4*>(s.w5) + 4 * part;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float4 ww = w4[j];
            d = __fmaf_rn(__uint_as_float(a[2 * j] << 16), ww.x, d);
            d = __fmaf_rn(__uint_as_float(a[2 * j] & 0xFFFF0000u), ww.y, d);
            d = __fmaf_rn(__uint_as_float(a[2 * j + 1] << 16), ww.z, d);
            d = __fmaf_rn(__uint_as_float(a[2 * j + 1] & 0xFFFF0000u), ww.w, d);
          }
        }
      }
    }
    if (live) out[i] = d + s.b5;
  }
  fence_before();
  report_block(ok, err);
  fence_after();
  if (tid < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s.tmem),
                 "r"(kEvalCols));
}

// report_block() with one thread whose wait ran out, for checking it.
__global__ void __launch_bounds__(kEvalThreads) k_check_report(uint32_t thread, int* err) {
  report_block(threadIdx.x != thread, err);
}

// ------------------------------------------------------------- tracing
struct MarchDev {
  float alpha;        // network step = alpha * network distance (safety / Lipschitz bound)
  float switch_dist;  // hand over to the exact field below this network distance
  float min_step;     // floor of a network step
  float tmax;
  uint32_t max_steps;  // network steps before handing over regardless
  float bmin[3], bmax[3];  // the network's box; the march stays inside it
};

// Exact phase parameters.
struct RefineDev {
  uint32_t max_steps;   // exact evaluations per ray (march + bracket + root)
  uint32_t root_steps;  // regula-falsi steps on a bracketed crossing
  float relax;          // an exact step may grow to relax x (step_factor * d) along a secant
  float root_tol;       // the root search ends when the secant point moves less than this
  float ceiling;        // no surface above this height (bound of the field)
  uint32_t normal_taps;  // 6: central differences; 4: tetrahedral; 1: none here (k_sdf_grad_normal)
  // cone starts (direct mode): pixel (x, y) starts at tile_t[(y / cone_tile)
  // * cone_tiles_x + x / cone_tile]; null: every pixel starts at t = 0
  const float* tile_t;
  uint32_t cone_tile, cone_tiles_x;
};

// Tap k of the tetrahedral normal (compute_sdf_normal_tet,
// sdf_functions.cuh:518-532): 0.5773 (2 b - 1) with b = (((k + 3) >> 1) & 1,
// (k >> 1) & 1, k & 1), i.e. the corners (+,-,-), (-,-,+), (-,+,-), (+,+,+)
// of a cube scaled to length ~1.
__device__ __forceinline__ V3 tet_dir(uint32_t k) {
  const float c = 0.5773f;
  return v3((((k + 3u) >> 1) & 1u) ? c : -c, ((k >> 1) & 1u) ? c : -c, (k & 1u) ? c : -c);
}

// Slab test of the ray against the box: [t0, t1] with t0 >= 0 (empty if t0 >= t1).
__device__ __forceinline__ void box_span(const MarchDev& md, const V3& o, const V3& d, float& t0,
                                         float& t1) {
  float o3[3] = {o.x, o.y, o.z}, d3[3] = {d.x, d.y, d.z};
  t0 = 0.f;
  t1 = md.tmax;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float inv = 1.0f / d3[k];
    float ta = (md.bmin[k] - o3[k]) * inv, tb = (md.bmax[k] - o3[k]) * inv;
    t0 = fmaxf(t0, fminf(ta, tb));
    t1 = fminf(t1, fmaxf(ta, tb));
  }
}

// Appends this lane's entry to the exact-phase queue (warp-aggregated).
__device__ __forceinline__ void queue_push(bool push, uint4 e, uint32_t* counters,
                                           uint4* __restrict__ queue) {
  uint32_t lane = threadIdx.x & 31u;
  uint32_t pm = __ballot_sync(0xFFFFFFFFu, push);
  if (pm == 0u) return;
  uint32_t leader = __ffs(pm) - 1u, base = 0;
  if (lane == leader) base = atomicAdd(&counters[1], (uint32_t)__popc(pm));
  base = __shfl_sync(0xFFFFFFFFu, base, leader);
  if (push) queue[base + __popc(pm & ((1u << lane) - 1u))] = e;
}

// Neural phase.  Each group of 128 threads marches 128 rays (one per
// thread) through the network; a warp refills its idle rows from the pixel
// cursor (claim order = 8x4 pixel tiles) once 8 of them are idle.  A ray
// starts where it enters the network's box and steps by
// max(alpha * d_net, min_step).  It is queued for the exact phase as
// {pixel, t, t_lo, steps} when d_net < switch_dist (t_lo = the previous
// network point, a bracket candidate), when it leaves the box before tmax
// (t = t_lo = exit), or after max_steps network steps; rays that reach tmax
// inside the box are written as misses.
__global__ void __launch_bounds__(kTcThreads, 1) k_nsdf_march(InputMap m,
                                                              const unsigned char* __restrict__ pack,
                                                              MarchDev md, CamDev cam, uint32_t w,
                                                              uint32_t h, uint32_t* __restrict__ counters,
                                                              unsigned long long* __restrict__ totals,
                                                              uint4* __restrict__ queue,
                                                              float4* __restrict__ out,
                                                              int* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  TcSmem& s = tc_smem(smem_raw);
  tc_setup(s, pack);
  const int tid = threadIdx.x, g = tid >> 7, row = tid & 127;
  const uint32_t lane = tid & 31u;
  uint32_t phase = 0;
  const uint32_t tiles_x = (w + 7) / 8;
  const uint32_t total = tiles_x * ((h + 3) / 4) * 32u;
  bool live = false, exhausted = false, ok = true;
  uint32_t pix = 0, steps = 0;
  V3 o = {0.f, 0.f, 0.f}, d = {0.f, 0.f, 1.f};
  float t = 0.f, t_lo = 0.f, t_end = 0.f;
  uint32_t n_live = 0, n_rows = 0;  // network evaluations of rays / rows computed
  for (uint32_t guard = 0; guard < (1u << 24); ++guard) {
    bool outside = false;  // a new ray that misses the box goes straight to the exact phase
    uint32_t idle = __ballot_sync(0xFFFFFFFFu, !live);
    uint32_t nidle = __popc(idle);
    if (!exhausted && nidle >= 8u) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(&counters[0], nidle);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (base + nidle >= total) exhausted = true;
      if (!live) {
        uint32_t i = base + __popc(idle & ((1u << lane) - 1u));
        uint32_t tile = i >> 5, l = i & 31u;
        uint32_t x = (tile % tiles_x) * 8 + (l & 7u), y = (tile / tiles_x) * 4 + (l >> 3);
        if (i < total && x < w && y < h) {
          generate_ray(cam, w, h, x, y, o, d);
          pix = y * w + x;
          steps = 0;
          float t0, t1;
          box_span(md, o, d, t0, t1);
          if (t0 < t1) {
            t = t0;
            t_lo = t0;
            t_end = t1;
            live = true;
          } else {
            outside = true;
          }
        }
      }
    }
    queue_push(outside, make_uint4(pix, 0u, 0u, 0u), counters, queue);
    if (!group_or(g, live || !exhausted)) break;
    float q[3];
    normalise(m, __fmaf_rn(t, d.x, o.x), __fmaf_rn(t, d.y, o.y), __fmaf_rn(t, d.z, o.z), q);
    float dn = mlp_row(s, m, g, row, q, phase, ok);
    if (!group_and(g, ok)) break;
    ++n_rows;
    n_live += live ? 1u : 0u;
    bool push = false;
    uint4 e = make_uint4(0u, 0u, 0u, 0u);
    if (live) {
      ++steps;
      if (dn < md.switch_dist) {
        push = true;
        e = make_uint4(pix, __float_as_uint(t), __float_as_uint(t_lo), steps);
      } else {
        t_lo = t;
        t += fmaxf(md.alpha * dn, md.min_step);
        if (t >= t_end) {
          if (t_end >= md.tmax) {
            out[2 * (size_t)pix] = make_float4(0.f, 0.f, 0.f, 0.f);
            out[2 * (size_t)pix + 1] =
                make_float4(0.f, 0.f, __uint_as_float(steps), __uint_as_float(0u));
            live = false;
          } else {
            push = true;
            e = make_uint4(pix, __float_as_uint(t_end), __float_as_uint(t_end), steps);
          }
        } else if (steps >= md.max_steps) {
          push = true;
          e = make_uint4(pix, __float_as_uint(t), __float_as_uint(t), steps);
        }
      }
      if (push) live = false;
    }
    queue_push(push, e, counters, queue);
  }
  n_live = __reduce_add_sync(0xFFFFFFFFu, n_live);
  n_rows = __reduce_add_sync(0xFFFFFFFFu, n_rows);
  if (lane == 0) {
    atomicAdd(&totals[0], (unsigned long long)n_live);
    atomicAdd(&totals[3], (unsigned long long)n_rows);
  }
  if (!ok && row == 0) atomicExch(err, 1);
  tc_teardown(s);
}

// Cone tiles of the network phase: tile x tile pixels, tiles_x x tiles_y of
// them; parent (may be null): start parameters of coarser tiles of
// parent_tile pixels (a multiple of tile), parent_tiles_x per row.
struct ConeDev {
  uint32_t tile, tiles_x, tiles_y;
  const float* parent;
  uint32_t parent_tile, parent_tiles_x;
};

// Cone phase.  Each tile's cone is marched by K consecutive lanes of a
// warp.  The axis is the normalised sum of the tile's four corner rays, and
// `s` the largest chord from the axis direction to a corner ray's.  The
// angle to the axis is quasi-convex over the image plane, so the corners
// bound it: every ray of the tile lies within t s of the axis point at the
// same parameter t, and a point of a tile ray within a further dt lies
// within dt + t s of the axis point.  The clearance c = d_net - t s (the
// network distance shrunk by the cone's radius) therefore bounds a step of
// alpha c for every ray of the tile, the per-ray rule's step.
//
// Speculation: in one pass lane j of a tile evaluates the axis at t + dt
// (r + r^2 + ... + r^j), dt the last accepted step and r = 0.9 x the ratio
// of the last two (the steps of a cone closing in on a surface shrink
// geometrically, in open space they grow).  The lanes' spheres are chained
// in order: a point that lies inside the part already cleared extends it to
// t_j + alpha c_j, a point beyond it ends the chain, and the first chained
// point whose clearance is below switch_dist stops the tile there.  Lane 0
// is at t, so a pass advances at least one sequential step, and up to K
// when the guesses land; K = 1 is plain cone marching.
//
// The axis starts at its entry into the network's box (or the parent tile's
// start, if later); a tile whose axis leaves the box stops at the exit, and
// one that makes max_steps passes stops where it is.  Every pixel of the
// tile then starts its exact phase at the tile's parameter (k_sdf_refine).
template <uint32_t K>
__global__ void __launch_bounds__(kTcThreads, 1) k_nsdf_cone(InputMap m,
                                                             const unsigned char* __restrict__ pack,
                                                             MarchDev md, ConeDev cd, CamDev cam,
                                                             uint32_t w, uint32_t h,
                                                             uint32_t* __restrict__ cursor,
                                                             unsigned long long* __restrict__ totals,
                                                             float* __restrict__ tile_t,
                                                             int* __restrict__ err) {
  static_assert(K == 1 || K == 2 || K == 4 || K == 8 || K == 16,
                "lanes per cone: 1, 2, 4, 8 or 16");
  extern __shared__ unsigned char smem_raw[];
  TcSmem& s = tc_smem(smem_raw);
  tc_setup(s, pack);
  const int tid = threadIdx.x, g = tid >> 7, row = tid & 127;
  const uint32_t lane = tid & 31u;
  const uint32_t j = lane & (K - 1u), lead = lane & ~(K - 1u);
  const uint32_t kmask = (K == 1 ? 1u : ((1u << K) - 1u)) << lead;
  uint32_t phase = 0;
  const uint32_t total = cd.tiles_x * cd.tiles_y;
  bool live = false, exhausted = false, ok = true;
  uint32_t tile = 0, passes = 0;
  V3 o = {0.f, 0.f, 0.f}, ax = {0.f, 0.f, 1.f};
  float t = 0.f, dt = 0.f, ratio = 1.f, t_end = 0.f, chord = 0.f;
  uint32_t n_live = 0, n_rows = 0;
  for (uint32_t guard = 0; guard < (1u << 24); ++guard) {
    // the K lanes of a tile share `live`, so a tile's first lane speaks for it
    const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !live && j == 0u);
    const uint32_t nidle = __popc(idle);
    if (!exhausted && nidle * K >= 8u) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(cursor, nidle);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (base + nidle >= total) exhausted = true;
      const uint32_t i =
          __shfl_sync(0xFFFFFFFFu, base + __popc(idle & ((1u << lane) - 1u)), lead);
      if (!live && i < total) {
        // every lane of the tile computes the same set-up
        tile = i;
        const uint32_t x0 = (i % cd.tiles_x) * cd.tile, y0 = (i / cd.tiles_x) * cd.tile;
        const uint32_t x1 = min(x0 + cd.tile - 1u, w - 1u), y1 = min(y0 + cd.tile - 1u, h - 1u);
        V3 c[4];
        generate_ray(cam, w, h, x0, y0, o, c[0]);
        generate_ray(cam, w, h, x1, y0, o, c[1]);
        generate_ray(cam, w, h, x0, y1, o, c[2]);
        generate_ray(cam, w, h, x1, y1, o, c[3]);
        ax = normalize(v3(c[0].x + c[1].x + c[2].x + c[3].x, c[0].y + c[1].y + c[2].y + c[3].y,
                          c[0].z + c[1].z + c[2].z + c[3].z));
        chord = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          V3 e = sub(c[k], ax);
          chord = fmaxf(chord, sqrtf(dot(e, e)));
        }
        // rounding of the corner rays and of the axis
        chord = chord * 1.001f + 1e-6f;
        float t0, t1;
        box_span(md, o, ax, t0, t1);
        float start =
            cd.parent ? cd.parent[(y0 / cd.parent_tile) * cd.parent_tiles_x + x0 / cd.parent_tile]
                      : 0.f;
        t = fmaxf(t0, start);
        t_end = t1;
        dt = 0.f;
        ratio = 1.f;
        passes = 0;
        if (t < t_end) live = true;
        else if (j == 0u) tile_t[tile] = start;
      }
    }
    if (!group_or(g, live || !exhausted)) break;
    float off = 0.f;
    {
      const float r = 0.9f * ratio;
      float rp = 1.f;
      for (uint32_t i = 0; i < j; ++i) {
        rp *= r;
        off += rp;
      }
    }
    const float tj = __fmaf_rn(off, dt, t);
    float q[3];
    normalise(m, __fmaf_rn(tj, ax.x, o.x), __fmaf_rn(tj, ax.y, o.y), __fmaf_rn(tj, ax.z, o.z), q);
    float dn = mlp_row(s, m, g, row, q, phase, ok);
    if (!group_and(g, ok)) break;
    ++n_rows;
    n_live += live ? 1u : 0u;
    if (live) {
      // all K lanes of the tile are here together and reach the same verdict
      const float cj = dn - tj * chord;
      float cov = t, t_stop = 0.f, s_last = dt, s_prev = dt;
      bool chained = true, stop = false;
#pragma unroll
      for (uint32_t k = 0; k < K; ++k) {
        const float tk = K == 1 ? tj : __shfl_sync(kmask, tj, lead + k);
        const float ck = K == 1 ? cj : __shfl_sync(kmask, cj, lead + k);
        if (chained && !stop) {
          if (tk > cov) {
            chained = false;
          } else if (ck < md.switch_dist) {
            stop = true;
            t_stop = tk;
          } else {
            cov = fmaxf(cov, tk + md.alpha * ck);
            s_prev = s_last;
            s_last = md.alpha * ck;
          }
        }
      }
      ++passes;
      if (stop) {
        if (j == 0u) tile_t[tile] = t_stop;
        live = false;
      } else {
        t = cov;
        ratio = s_prev > 0.f ? fminf(fmaxf(s_last / s_prev, 0.25f), 4.f) : 1.f;
        dt = s_last;
        if (t >= t_end) {
          if (j == 0u) tile_t[tile] = t_end;
          live = false;
        } else if (passes >= md.max_steps) {
          if (j == 0u) tile_t[tile] = t;
          live = false;
        }
      }
    }
  }
  n_live = __reduce_add_sync(0xFFFFFFFFu, n_live);
  n_rows = __reduce_add_sync(0xFFFFFFFFu, n_rows);
  if (lane == 0) {
    atomicAdd(&totals[0], (unsigned long long)n_live);
    atomicAdd(&totals[3], (unsigned long long)n_rows);
  }
  if (!ok && row == 0) atomicExch(err, 1);
  tc_teardown(s);
}

// Exact phase, one lane per ray with lane refill (from the queue, or from
// the pixel cursor when `direct`: every pixel from t = 0, the same method
// without the network).  One field evaluation per trip of a state machine:
//   march  t += step_factor * d (the exact tracer's rule); the step may
//          grow along the secant through the last two samples up to relax x
//          that (relax <= 1: plain rule).  d < eps: hit at t.  d < 0 (the
//          sample is inside): the crossing is bracketed by the last outside
//          sample and refined.  Going up above `ceiling`: miss.
//   probe  the ray arrived inside from the network: check the bracket
//          candidate t_lo; if it is outside the crossing lies in
//          [t_lo, t], else march again from t = 0 (the network skipped
//          over the surface).
//   root   Illinois regula falsi on the bracket, root_steps evaluations or
//          until |d| < 1e-6, or until the next secant point moves less than
//          root_tol (that point is the hit, unevaluated; a bracket already
//          narrower than root_tol gives its secant root at once).
//   normal the exact tracer's central differences (delta = 0.002 t), or,
//          with normal_taps 4, the reference's tetrahedral normal
//          (compute_sdf_normal_tet) at the same radius: sum of e_k d(p +
//          delta e_k) over the four tetrahedron directions e_k.  With
//          normal_taps 1 the hit is written without a normal and
//          k_sdf_grad_normal adds the field's analytic gradient afterwards.
// With cone starts a ray begins its march where its tile's cone stopped; a
// start that is already inside the terrain (the network overestimated the
// distance) marches again from the camera.
// The step count written is network steps + exact march/probe/root
// evaluations (normals excluded, as in the exact tracer).
enum : uint32_t { kMarch = 0, kProbe = 1, kRoot = 2, kNormal = 3 };

// the field's table, then the warps' rings (64 entries of 32 bytes each)
constexpr uint32_t kRefineRing = 64 * 32;

// NT: the normal (RefineDev::normal_taps), fixed at compile time so that
// the analytic-gradient form (1) carries no stencil state.
template <uint32_t NT, class FORM>
__global__ void __launch_bounds__(FORM::kThreads) k_sdf_refine(
    PermTable perm, FieldDev f, RefineDev rd, CamDev cam, uint32_t w, uint32_t h, RowsSpread spread,
    int direct, const uint4* __restrict__ queue, uint32_t* __restrict__ counters,
    unsigned long long* __restrict__ totals, float4* __restrict__ out) {
  extern __shared__ uint32_t rows_smem[];
  // Per-warp ring of set-up rays (64 entries): the warp claims 32 work
  // indices at a time and all its lanes set those rays up together (pixel,
  // two divisions and three normalisations for the direction, the cone
  // tile's start), so the set-up runs with every lane active instead of on
  // the few lanes that happen to be idle; idle lanes then take entries.
  // Entry: {d.xyz, t} and {pixel (0xFFFFFFFF: no ray), t_lo bits, base
  // steps, 0}.
  float4(*ring_a)[64] = reinterpret_cast<float4(*)[64]>(rows_smem + FORM::kBytes / 4);
  uint4(*ring_b)[64] = reinterpret_cast<uint4(*)[64]>(ring_a + FORM::kThreads / 32);
  const auto P = FORM::load(perm, rows_smem);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (warp >= spread.warps) return;
  // direct mode claims pixels in 8x4 tiles (claim i = lane i & 31 of tile
  // i >> 5), so a warp's rays start close together
  const uint32_t dtiles_x = (w + 7) / 8;
  const uint32_t total = direct ? dtiles_x * ((h + 3) / 4) * 32u : counters[1];
  const bool holds = lane < spread.rays;  // may hold a ray
  bool live = false, claimed_all = false, have_lo = false, restarted = false;
  uint32_t head = 0, tail = 0;  // ring positions (warp-uniform)
  uint32_t pix = 0, steps = 0, base_steps = 0, mode = kMarch, tap = 0, iters = 0;
  int side = 0;
  V3 o = cam.campos, d = {0, 0, 1}, p = {0, 0, 0};
  float t = 0.f, t_lo = 0.f, a = 0.f, va = 0.f, b = 0.f, vb = 0.f, delta = 0.f;
  float nx = 0.f, ny = 0.f, nz = 0.f, plus = 0.f;
  uint32_t n_exact = 0, n_normal = 0;  // evaluations: march/probe/root, normal taps
  for (;;) {
    uint32_t idle = __ballot_sync(0xFFFFFFFFu, holds && !live);
    uint32_t nidle = __popc(idle);
    if (nidle >= 4u && (!claimed_all || head != tail)) {
      if (tail - head < nidle && !claimed_all) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&counters[2], spread.rays);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base + spread.rays >= total) claimed_all = true;
        const uint32_t i = lane < spread.rays ? base + lane : total;
        uint32_t dx = 0, dy = 0;
        if (direct) {
          dx = ((i >> 5) % dtiles_x) * 8 + (i & 7u);
          dy = ((i >> 5) / dtiles_x) * 4 + ((i >> 3) & 3u);
        }
        float4 ea = make_float4(0.f, 0.f, 1.f, 0.f);
        uint4 eb = make_uint4(0xFFFFFFFFu, 0u, 0u, 0u);
        if (i < total && (!direct || (dx < w && dy < h))) {
          uint4 e = direct ? make_uint4(dy * w + dx, 0u, 0u, 0u) : queue[i];
          V3 ro, rd3;
          generate_ray(cam, w, h, e.x % w, e.x / w, ro, rd3);
          float t0 = __uint_as_float(e.y), tl = __uint_as_float(e.z);
          if (direct && rd.tile_t) {
            t0 = rd.tile_t[((e.x / w) / rd.cone_tile) * rd.cone_tiles_x + (e.x % w) / rd.cone_tile];
            tl = t0;
          }
          ea = make_float4(rd3.x, rd3.y, rd3.z, t0);
          eb = make_uint4(e.x, __float_as_uint(tl), e.w, 0u);
        }
        ring_a[warp][(tail + lane) & 63u] = ea;
        ring_b[warp][(tail + lane) & 63u] = eb;
        __syncwarp();
        tail += spread.rays;
      }
      const uint32_t avail = tail - head;
      if ((idle >> lane) & 1u) {
        const uint32_t r = __popc(idle & ((1u << lane) - 1u));
        if (r < avail) {
          const float4 ea = ring_a[warp][(head + r) & 63u];
          const uint4 eb = ring_b[warp][(head + r) & 63u];
          if (eb.x != 0xFFFFFFFFu) {
            pix = eb.x;
            d = v3(ea.x, ea.y, ea.z);
            t = ea.w;
            t_lo = __uint_as_float(eb.y);
            base_steps = eb.z;
            steps = 0;
            mode = kMarch;
            have_lo = false;
            restarted = false;
            live = true;
          }
        }
      }
      head += min(nidle, avail);
      __syncwarp();
    }
    if (__ballot_sync(0xFFFFFFFFu, live) == 0u) {
      if (claimed_all && head == tail) break;
      continue;
    }
    V3 qp;
    if (mode == kMarch) {
      qp = v3(__fmaf_rn(t, d.x, o.x), __fmaf_rn(t, d.y, o.y), __fmaf_rn(t, d.z, o.z));
    } else if (mode == kProbe) {
      qp = v3(__fmaf_rn(a, d.x, o.x), __fmaf_rn(a, d.y, o.y), __fmaf_rn(a, d.z, o.z));
    } else if (NT == 1u || mode == kRoot) {
      qp = v3(__fmaf_rn(t, d.x, o.x), __fmaf_rn(t, d.y, o.y), __fmaf_rn(t, d.z, o.z));
    } else if (NT == 4u) {
      V3 e = tet_dir(tap);
      qp = v3(__fmaf_rn(e.x, delta, p.x), __fmaf_rn(e.y, delta, p.y), __fmaf_rn(e.z, delta, p.z));
    } else {
      float sd = (tap & 1u) ? -delta : delta;
      qp = p;
      if (tap < 2) qp.x = p.x + sd;
      else if (tap < 4) qp.y = p.y + sd;
      else qp.z = p.z + sd;
    }
    float v = warp_density(P, qp, live, f.octaves, f.scale, f.amp);
    if (!live) continue;
    if (NT != 1u && mode == kNormal) ++n_normal;
    else ++n_exact;
    uint32_t status = 3;  // 3 = still running
    bool begin_root = false, hit_here = false;
    if (mode == kMarch) {
      ++steps;
      if (v < 0.f) {
        if (have_lo) {
          b = t;
          vb = v;
          begin_root = true;
        } else if (t_lo < t && !restarted) {
          b = t;
          vb = v;
          a = t_lo;
          mode = kProbe;
        } else if (rd.tile_t && !restarted) {
          // the cone start lies inside: march again from the camera
          t = 0.f;
          t_lo = 0.f;
          restarted = true;
          if (steps >= rd.max_steps) status = 2;
        } else {
          hit_here = true;
        }
      } else if (v < f.eps) {
        hit_here = true;
      } else if (d.y >= 0.f && qp.y > rd.ceiling) {
        status = 0;
      } else {
        float step = f.step_factor * v;
        if (have_lo && va > v && rd.relax > 1.f) {
          float sec = v * (t - a) / (va - v);  // distance to the secant's root
          step = fminf(fmaxf(step, sec), rd.relax * step);
        }
        a = t;
        va = v;
        have_lo = true;
        t += step;
        if (t > f.tmax) status = 0;
        else if (steps >= rd.max_steps) status = 2;
      }
    } else if (mode == kProbe) {
      ++steps;
      if (v > 0.f) {
        va = v;
        begin_root = true;
      } else {
        // the network passed the crossing: march again from the camera
        t = 0.f;
        t_lo = 0.f;
        have_lo = false;
        restarted = true;
        mode = kMarch;
        if (steps >= rd.max_steps) status = 2;
      }
    } else if (NT == 1u || mode == kRoot) {
      ++steps;
      if (fabsf(v) < 1e-6f || ++iters >= rd.root_steps) {
        hit_here = true;
      } else {
        if (v < 0.f) {
          b = t;
          vb = v;
          if (side < 0) va *= 0.5f;
          side = -1;
        } else {
          a = t;
          va = v;
          if (side > 0) vb *= 0.5f;
          side = 1;
        }
        const float tn = b - vb * (b - a) / (vb - va);
        // the next secant point moves less than root_tol: take it unevaluated
        if (fabsf(tn - t) < rd.root_tol) hit_here = true;
        t = tn;
      }
    } else if (NT == 4u) {
      V3 e = tet_dir(tap);
      nx = __fmaf_rn(e.x, v, nx);
      ny = __fmaf_rn(e.y, v, ny);
      nz = __fmaf_rn(e.z, v, nz);
      if (tap == 3) status = 1;
      else ++tap;
    } else {
      if ((tap & 1u) == 0u) {
        plus = v;
      } else {
        float diff = plus - v;
        if (tap == 1) nx = diff;
        else if (tap == 3) ny = diff;
        else nz = diff;
      }
      if (tap == 5) status = 1;
      else ++tap;
    }
    if (begin_root) {
      mode = kRoot;
      side = 0;
      iters = 0;
      t = b - vb * (b - a) / (vb - va);
      // a bracket narrower than root_tol: its secant root is the hit
      if (b - a < rd.root_tol) hit_here = true;
    }
    if (hit_here) {
      p = v3(__fmaf_rn(t, d.x, o.x), __fmaf_rn(t, d.y, o.y), __fmaf_rn(t, d.z, o.z));
      if (NT == 1u) {
        // the hit is final here; k_sdf_grad_normal adds the normal
        status = 1;
      } else {
        delta = 0.002f * t;
        mode = kNormal;
        tap = 0;
        nx = ny = nz = 0.f;
      }
    }
    if (status != 3) {
      float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1;
      uint32_t total_steps = base_steps + steps;
      if (status == 1) {
        V3 n = NT == 1u ? v3(0.f, 0.f, 0.f) : normalize(v3(nx, ny, nz));
        r0 = make_float4(p.x, p.y, p.z, n.x);
        r1 = make_float4(n.y, n.z, __uint_as_float(total_steps), __uint_as_float(status));
      } else {
        r1 = make_float4(0.f, 0.f, __uint_as_float(total_steps), __uint_as_float(status));
      }
      out[2 * (size_t)pix] = r0;
      out[2 * (size_t)pix + 1] = r1;
      live = false;
    }
  }
  n_exact = __reduce_add_sync(0xFFFFFFFFu, n_exact);
  n_normal = __reduce_add_sync(0xFFFFFFFFu, n_normal);
  if (lane == 0) {
    atomicAdd(&totals[1], (unsigned long long)n_exact);
    atomicAdd(&totals[2], (unsigned long long)n_normal);
  }
}

// normal_taps 1: the normal of every hit in `out` (status 1) is the exact
// field's analytic gradient at the hit position, normalised
// (terrain_gradient: one lattice walk per octave, about 1.5 field
// evaluations of work, against 4 or 6 for the finite-difference stencils,
// which at radius 0.002 t are coarse estimates of this gradient).  A
// separate pass, so that the exact phase's state machine keeps a single
// field call site and the gradient's lanes do not diverge from the march.
// Bound by instructions: octaves in pairs on the rows' table take 116 us of a
// 1080p frame, one octave at a time on 16 copies of the permutation took 169.
__global__ void __launch_bounds__(kRowsThreads, 1)
k_sdf_grad_normal(PermTable perm, FieldDev f, uint32_t n, float one, float4* __restrict__ out,
                  unsigned long long* __restrict__ totals) {
  extern __shared__ uint32_t rows_smem[];
  const FieldRows R = load_rows(perm, rows_smem);
  uint32_t count = 0;
  // the warps of all blocks in turn, so that a small frame spreads over the SMs
  const uint32_t first = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32u + (threadIdx.x & 31u);
  for (uint32_t i = first; i < n; i += gridDim.x * blockDim.x) {
    float4 r1 = out[2 * (size_t)i + 1];
    if (__float_as_uint(r1.w) != 1u) continue;
    float4 r0 = out[2 * (size_t)i];
    V3 nn = normalize(terrain_gradient(R, v3(r0.x, r0.y, r0.z), f.octaves, f.scale, f.amp, one));
    r0.w = nn.x;
    r1.x = nn.y;
    r1.y = nn.z;
    out[2 * (size_t)i] = r0;
    out[2 * (size_t)i + 1] = r1;
    ++count;
  }
  count = __reduce_add_sync(0xFFFFFFFFu, count);
  if ((threadIdx.x & 31u) == 0u && count) atomicAdd(&totals[2], (unsigned long long)count);
}

// Finite-difference gradient norm of the network at n sample points (vals
// holds 4 evaluations per point: p, p+hx, p+hy, p+hz).
__global__ void k_grad_norm(const float* __restrict__ vals, uint32_t n, float h,
                            float* __restrict__ norms) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float v0 = vals[4 * (size_t)i];
  float gx = (vals[4 * (size_t)i + 1] - v0) / h, gy = (vals[4 * (size_t)i + 2] - v0) / h,
        gz = (vals[4 * (size_t)i + 3] - v0) / h;
  norms[i] = sqrtf(gx * gx + gy * gy + gz * gz);
}

}  // namespace nsdf
}  // namespace re

// ----------------------------------------------------------------- host
struct re_nsdf {
  int device = 0;
  re::nsdf::InputMap map;
  uint32_t seed = 1;
  float* params = nullptr;  // [kNumParams]
  float* adam_m = nullptr;
  float* adam_v = nullptr;
  unsigned char* pack = nullptr;
  bool pack_valid = false;
  uint32_t* step_ctr = nullptr;  // [0] steps done [1] reduction blocks done
  float4* data = nullptr;
  uint32_t npts = 0;
  // partial gradients of the training CTAs, for `batch` rows
  uint32_t batch = 0;
  float* part = nullptr;
  int train_grid = 0;
  float* loss_hist = nullptr;
  uint32_t loss_cap = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graph_exec = nullptr;
  float graph_lr = -1.f;
  // tracing scratch
  // [0] pixel cursor [1] queue size [2] refine cursor; from byte 16, u64
  // totals of the last trace: network evaluations of rays, exact
  // evaluations (march/probe/root), exact normal taps, network rows computed
  uint32_t* counters = nullptr;
  uint4* queue = nullptr;
  size_t queue_cap = 0;
  int* err = nullptr;  // trace errors: word 12 of `counters`
  // error word of the calls that wait for their kernels (train, loss_grad,
  // eval): pinned host memory that a kernel writes only when a wait ran out,
  // so such a call neither clears nor copies anything on the device (a
  // 65,536-row loss_grad call 92.8 -> 78.9 us, a 1M-point eval 166 -> 155)
  volatile int* sync_err = nullptr;
  int* sync_err_dev = nullptr;
  // cone phase: start parameters of the fine tiles, then of the coarse ones;
  // the image and fine tile size of the last network phase that wrote them
  float* cone_t = nullptr;
  size_t cone_cap = 0;
  uint32_t cone_w = 0, cone_h = 0, cone_tile = 0, cone_tiles_x = 0;
  float lipschitz = 0.f;
  uint32_t total_steps_done = 0;
};

namespace re {
namespace {

using namespace nsdf;

// Forgets the captured training step.  It holds the model's input map, the
// training points' address and number, the loss history's address, the batch
// and the learning rate: whatever changes one of them calls this.
void drop_graph(re_nsdf* s) {
  if (s->graph_exec) cudaGraphExecDestroy(s->graph_exec);
  if (s->graph) cudaGraphDestroy(s->graph);
  s->graph_exec = nullptr;
  s->graph = nullptr;
}

void free_train(re_nsdf* s) {
  drop_graph(s);
  cudaFree(s->part);
  s->part = nullptr;
  s->batch = 0;
}

// One CTA per SM (512 tensor-memory columns), every CTA with the same number
// of tiles as far as they go round.
re_status alloc_train(re_nsdf* s, uint32_t batch) {
  if (s->batch == batch) return RE_OK;
  free_train(s);
  RE_CUDA(cudaFuncSetAttribute(k_tc_train, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kTrainSmemBytes));
  const uint32_t tiles = batch / kTrRows;
  const uint32_t rounds = (tiles + (uint32_t)sm_count() - 1u) / (uint32_t)sm_count();
  s->train_grid = (int)((tiles + rounds - 1u) / rounds);
  RE_CUDA(cudaMalloc(&s->part, (size_t)s->train_grid * kPartStride * 4));
  s->batch = batch;
  return RE_OK;
}

re_status check(const re_nsdf* s, const char* fn) {
  if (!s) return fail(RE_ERR_INVALID_ARG, "%s: null model", fn);
  int dev = -1;
  RE_CUDA(cudaGetDevice(&dev));
  if (dev != s->device)
    return fail(RE_ERR_INVALID_ARG, "%s: model lives on device %d, current device is %d", fn,
                s->device, dev);
  return RE_OK;
}

// One pass over a batch (sampled from s->data, or given points when direct):
// forward, L1 loss, backward and the reduction, whose sums go to `grad`, or
// into an Adam step when grad is null.
re_status enqueue_step(re_nsdf* s, const float4* data, uint32_t npts, int direct, float lr,
                       float* grad, float* pred, cudaStream_t st) {
  const uint32_t B = s->batch;
  k_tc_train<<<s->train_grid, kTrainThreads, kTrainSmemBytes, st>>>(
      s->map, data, npts, s->step_ctr, s->seed, direct, s->params, s->part, B, pred, s->sync_err_dev);
  k_train_reduce<<<(kPartStride + 31) / 32, 32 * kReduceWarps, 0, st>>>(
      s->part, (uint32_t)s->train_grid, grad, s->params, grad ? nullptr : s->adam_m, s->adam_v,
      s->loss_hist, s->step_ctr, lr, B);
  RE_CHECK_LAUNCH("nsdf training step launch");
  return RE_OK;
}

re_status ensure_pack(re_nsdf* s, cudaStream_t st) {
  if (s->pack_valid) return RE_OK;
  // one thread per element of the largest section (W2..W4: 3 x 64 x 64)
  constexpr int kPackThreads = 3 * kHidden * kHidden > kHidden * kIn ? 3 * kHidden * kHidden
                                                                      : kHidden * kIn;
  k_pack<<<(kPackThreads + 255) / 256, 256, 0, st>>>(s->params, s->pack);
  RE_CHECK_LAUNCH("nsdf pack launch");
  s->pack_valid = true;
  return RE_OK;
}

constexpr size_t kTcSmemBytes = sizeof(TcSmem) + 1024;

template <typename K>
int tc_grid(K kernel) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTcThreads, kTcSmemBytes) !=
          cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  per_sm = std::min(per_sm, 2);  // 2 x 256 TMEM columns of 512
  return per_sm * sm_count();
}

CamDev cam_dev(const re_camera& c) {
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

PermTable perm_of(uint32_t seed) {
  uint32_t full[512];
  perlin_permutation(seed, full);
  PermTable t;
  for (int i = 0; i < 512; ++i) t.p[i] = (uint8_t)full[i];
  return t;
}

FieldDev field_of(const re_sdf_params& p) {
  FieldDev f;
  f.octaves = p.octaves;
  f.max_steps = p.max_steps;
  f.scale = p.scale;
  f.amp = p.amplitude;
  f.step_factor = p.step_factor;
  f.eps = p.eps;
  f.tmax = p.tmax;
  return f;
}

re_status check_field(const re_sdf_params* p, const char* fn) {
  if (!p) return fail(RE_ERR_INVALID_ARG, "%s: null field", fn);
  if (p->octaves > 32) return fail(RE_ERR_LIMIT, "%s: octaves > 32", fn);
  if (p->max_steps == 0 || p->max_steps > (1u << 20))
    return fail(RE_ERR_LIMIT, "%s: max_steps must be in [1, 2^20]", fn);
  return RE_OK;
}

}  // namespace
}  // namespace re

extern "C" {

RE_API uint32_t re_nsdf_num_params(void) { return (uint32_t)re::nsdf::kNumParams; }

RE_API re_status re_nsdf_box_for_camera(const re_camera* cam, uint32_t w, uint32_t h, float tmax,
                                        float y_lo, float y_hi, float* box_min, float* box_max) {
  if (!cam || !box_min || !box_max || w < 2 || h < 2 || !(tmax > 0.f) || !(y_hi > y_lo))
    return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_box_for_camera: bad arguments");
  re::CamBasis b;
  re::camera_basis(*cam, b);
  double lo[3], hi[3];
  for (int k = 0; k < 3; ++k) lo[k] = hi[k] = b.campos[k];
  for (int cx = -1; cx <= 1; cx += 2)
    for (int cy = -1; cy <= 1; cy += 2) {
      double dir[3], n = 0;
      for (int k = 0; k < 3; ++k) {
        dir[k] = (b.middle[k] + cx * b.horizontal[k] + cy * b.vertical[k] - b.campos[k]) * b.focal;
        n += dir[k] * dir[k];
      }
      n = std::sqrt(n);
      for (int k = 0; k < 3; ++k) {
        double e = b.campos[k] + dir[k] / n * tmax;
        lo[k] = std::min(lo[k], e);
        hi[k] = std::max(hi[k], e);
      }
    }
  lo[1] = std::max(lo[1], (double)y_lo);
  hi[1] = std::min(hi[1], (double)y_hi);
  if (!(hi[1] > lo[1])) {
    lo[1] = y_lo;
    hi[1] = y_hi;
  }
  for (int k = 0; k < 3; ++k) {
    box_min[k] = (float)lo[k];
    box_max[k] = (float)hi[k];
  }
  return RE_OK;
}

RE_API re_status re_nsdf_create(const re_nsdf_config* cfg, re_nsdf** out) {
  using namespace re::nsdf;
  if (!cfg || !out) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_create: null argument");
  for (int k = 0; k < 3; ++k)
    if (!(cfg->box_max[k] > cfg->box_min[k]))
      return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_create: empty box");
  if (!(cfg->f0 > 0.f)) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_create: f0 must be > 0");
  re_nsdf* s = new (std::nothrow) re_nsdf();
  if (!s) return re::fail(RE_ERR_OUT_OF_MEMORY, "re_nsdf_create: host allocation");
  cudaError_t e = cudaGetDevice(&s->device);
  for (int k = 0; k < 3; ++k) {
    s->map.center[k] = 0.5f * (cfg->box_min[k] + cfg->box_max[k]);
    s->map.inv_half[k] = 2.0f / (cfg->box_max[k] - cfg->box_min[k]);
  }
  s->map.f0 = cfg->f0;
  s->seed = cfg->seed;
  if (e == cudaSuccess) e = cudaMalloc(&s->params, kNumParams * 4);
  if (e == cudaSuccess) e = cudaMalloc(&s->adam_m, kNumParams * 4);
  if (e == cudaSuccess) e = cudaMalloc(&s->adam_v, kNumParams * 4);
  if (e == cudaSuccess) e = cudaMalloc(&s->pack, re::nsdf::kPackBytes);
  if (e == cudaSuccess) e = cudaMalloc(&s->step_ctr, 16);
  if (e == cudaSuccess) e = cudaMalloc(&s->counters, 64);
  if (e == cudaSuccess) {
    s->err = reinterpret_cast<int*>(s->counters) + 12;
    int* word = nullptr;
    e = cudaHostAlloc(&word, sizeof(int), cudaHostAllocMapped);
    s->sync_err = word;
  }
  if (e == cudaSuccess)
    e = cudaHostGetDevicePointer(&s->sync_err_dev, const_cast<int*>(s->sync_err), 0);
  if (e == cudaSuccess) e = cudaMemset(s->adam_m, 0, kNumParams * 4);
  if (e == cudaSuccess) e = cudaMemset(s->adam_v, 0, kNumParams * 4);
  if (e == cudaSuccess) e = cudaMemset(s->step_ctr, 0, 16);
  if (e == cudaSuccess) e = cudaMemset(s->counters, 0, 64);
  if (e == cudaSuccess) {
    // Glorot-uniform weights, zero biases (std::mt19937 seeded by cfg->seed)
    std::vector<float> h(kNumParams, 0.f);
    std::mt19937 gen(cfg->seed);
    auto fill = [&](int off, int fan_out, int fan_in) {
      float a = std::sqrt(6.0f / (float)(fan_in + fan_out));
      std::uniform_real_distribution<float> U(-a, a);
      for (int i = 0; i < fan_out * fan_in; ++i) h[off + i] = U(gen);
    };
    fill(OFF_W1, kHidden, kIn);
    fill(OFF_W2, kHidden, kHidden);
    fill(OFF_W3, kHidden, kHidden);
    fill(OFF_W4, kHidden, kHidden);
    fill(OFF_W5, 1, kHidden);
    e = cudaMemcpy(s->params, h.data(), kNumParams * 4, cudaMemcpyHostToDevice);
  }
  if (e != cudaSuccess) {
    re_status st = re::cuda_fail(e, "re_nsdf_create");
    re_nsdf_destroy(s);
    return st;
  }
  *out = s;
  return RE_OK;
}

RE_API re_status re_nsdf_destroy(re_nsdf* s) {
  if (!s) return RE_OK;
  re::free_train(s);
  cudaFree(s->params);
  cudaFree(s->adam_m);
  cudaFree(s->adam_v);
  cudaFree(s->pack);
  cudaFree(s->step_ctr);
  cudaFree(s->data);
  cudaFree(s->loss_hist);
  cudaFree(s->counters);
  cudaFree(s->queue);
  cudaFree(s->cone_t);
  if (s->sync_err) cudaFreeHost(const_cast<int*>(s->sync_err));
  delete s;
  return RE_OK;
}

RE_API re_status re_nsdf_get_params(const re_nsdf* s, float* host) {
  re_status st = re::check(s, "re_nsdf_get_params");
  if (st != RE_OK) return st;
  if (!host) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_get_params: null output");
  RE_CUDA(cudaMemcpy(host, s->params, re::nsdf::kNumParams * 4, cudaMemcpyDeviceToHost));
  return RE_OK;
}

RE_API re_status re_nsdf_set_params(re_nsdf* s, const float* host) {
  re_status st = re::check(s, "re_nsdf_set_params");
  if (st != RE_OK) return st;
  if (!host) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_set_params: null input");
  RE_CUDA(cudaMemcpy(s->params, host, re::nsdf::kNumParams * 4, cudaMemcpyHostToDevice));
  s->pack_valid = false;
  s->lipschitz = 0.f;
  return RE_OK;
}

RE_API re_status re_nsdf_generate(re_nsdf* s, const re_sdf_params* field, const re_camera* cam,
                                  uint32_t w, uint32_t h, uint32_t num_points, uint32_t seed,
                                  void* stream) {
  re_status st = re::check(s, "re_nsdf_generate");
  if (st != RE_OK) return st;
  st = re::check_field(field, "re_nsdf_generate");
  if (st != RE_OK) return st;
  if (!cam || w < 2 || h < 2 || num_points < 2)
    return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_generate: bad arguments");
  if (num_points > (1u << 28)) return re::fail(RE_ERR_LIMIT, "re_nsdf_generate: > 2^28 points");
  cudaStream_t cs = (cudaStream_t)stream;
  if (s->npts != num_points) {
    RE_CUDA(cudaStreamSynchronize(cs));
    re::drop_graph(s);
    cudaFree(s->data);
    s->data = nullptr;
    s->npts = 0;
    RE_CUDA(cudaMalloc(&s->data, (size_t)num_points * sizeof(float4)));
    s->npts = num_points;
  }
  float3 bmin, bmax;
  bmin.x = s->map.center[0] - 1.f / s->map.inv_half[0];
  bmin.y = s->map.center[1] - 1.f / s->map.inv_half[1];
  bmin.z = s->map.center[2] - 1.f / s->map.inv_half[2];
  bmax.x = s->map.center[0] + 1.f / s->map.inv_half[0];
  bmax.y = s->map.center[1] + 1.f / s->map.inv_half[1];
  bmax.z = s->map.center[2] + 1.f / s->map.inv_half[2];
  RE_CUDA(cudaFuncSetAttribute(re::nsdf::k_nsdf_data, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)re::kRowsSmemBytes));
  re::nsdf::k_nsdf_data<<<re::sm_count(), re::nsdf::kDataThreads, re::kRowsSmemBytes, cs>>>(
      re::perm_of(field->seed), re::field_of(*field), re::cam_dev(*cam), w, h, bmin, bmax,
      num_points, seed, s->data);
  RE_CHECK_LAUNCH("re_nsdf_generate: launch");
  return RE_OK;
}

RE_API re_status re_nsdf_get_data(const re_nsdf* s, float* host_xyzl, uint32_t max_points) {
  re_status st = re::check(s, "re_nsdf_get_data");
  if (st != RE_OK) return st;
  if (!host_xyzl) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_get_data: null output");
  uint32_t n = std::min(max_points, s->npts);
  RE_CUDA(cudaMemcpy(host_xyzl, s->data, (size_t)n * 16, cudaMemcpyDeviceToHost));
  return RE_OK;
}

RE_API re_status re_nsdf_train(re_nsdf* s, uint32_t steps, uint32_t batch, float lr,
                               float* loss_out, void* stream) {
  re_status st = re::check(s, "re_nsdf_train");
  if (st != RE_OK) return st;
  if (!s->data || s->npts == 0) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_train: no data (call re_nsdf_generate)");
  if (batch == 0 || batch % re::nsdf::kRowsBwd != 0 || batch > (1u << 22))
    return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_train: batch must be a positive multiple of %d up to 2^22",
                    re::nsdf::kRowsBwd);
  if (steps == 0) return RE_OK;
  cudaStream_t cs = (cudaStream_t)stream;
  st = re::alloc_train(s, batch);
  if (st != RE_OK) return st;
  uint32_t done = s->total_steps_done;
  if (s->loss_cap < done + steps) {
    RE_CUDA(cudaStreamSynchronize(cs));
    float* nh = nullptr;
    uint32_t cap = std::max(done + steps, 2 * s->loss_cap);
    RE_CUDA(cudaMalloc(&nh, (size_t)cap * 4));
    if (s->loss_hist) {
      RE_CUDA(cudaMemcpy(nh, s->loss_hist, (size_t)s->loss_cap * 4, cudaMemcpyDeviceToDevice));
      cudaFree(s->loss_hist);
    }
    s->loss_hist = nh;
    s->loss_cap = cap;
    re::drop_graph(s);
  }
  if (!s->graph_exec || s->graph_lr != lr) {
    re::drop_graph(s);
    cudaStream_t cap_stream;
    RE_CUDA(cudaStreamCreateWithFlags(&cap_stream, cudaStreamNonBlocking));
    cudaError_t e = cudaStreamBeginCapture(cap_stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      st = re::enqueue_step(s, s->data, s->npts, 0, lr, nullptr, nullptr, cap_stream);
      e = cudaStreamEndCapture(cap_stream, &s->graph);
    }
    if (e == cudaSuccess && st == RE_OK) e = cudaGraphInstantiate(&s->graph_exec, s->graph, 0);
    cudaStreamDestroy(cap_stream);
    if (st != RE_OK) return st;
    if (e != cudaSuccess) return re::cuda_fail(e, "re_nsdf_train: graph capture");
    s->graph_lr = lr;
  }
  *s->sync_err = 0;
  for (uint32_t i = 0; i < steps; ++i) RE_CUDA(cudaGraphLaunch(s->graph_exec, cs));
  s->pack_valid = false;
  s->lipschitz = 0.f;
  if (loss_out)
    RE_CUDA(cudaMemcpyAsync(loss_out, s->loss_hist + done, (size_t)steps * 4,
                            cudaMemcpyDeviceToHost, cs));
  RE_CUDA(cudaStreamSynchronize(cs));
  s->total_steps_done = done + steps;
  if (*s->sync_err) return re::fail(RE_ERR_INTERNAL, "re_nsdf_train: tensor-core wait bound reached");
  return RE_OK;
}

// Loss gradient of a given batch (points + labels as float4), no update.
RE_API re_status re_nsdf_loss_grad(re_nsdf* s, const float* d_xyzl, uint32_t n, float* d_grad,
                                   float* d_pred, void* stream) {
  re_status st = re::check(s, "re_nsdf_loss_grad");
  if (st != RE_OK) return st;
  if (!d_xyzl || !d_grad || n == 0 || n % re::nsdf::kRowsBwd != 0)
    return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_loss_grad: n must be a positive multiple of %d",
                    re::nsdf::kRowsBwd);
  // a kernel writes the gradient: an address the device cannot reach is
  // refused here, as a copy to it would be
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, d_grad) != cudaSuccess || !at.devicePointer) {
    cudaGetLastError();
    return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_loss_grad: d_grad is not device memory");
  }
  cudaStream_t cs = (cudaStream_t)stream;
  st = re::alloc_train(s, n);
  if (st != RE_OK) return st;
  *s->sync_err = 0;
  st = re::enqueue_step(s, reinterpret_cast<const float4*>(d_xyzl), n, 1, 0.f, d_grad, d_pred, cs);
  if (st != RE_OK) return st;
  RE_CUDA(cudaStreamSynchronize(cs));
  if (*s->sync_err) return re::fail(RE_ERR_INTERNAL, "re_nsdf_loss_grad: tensor-core wait bound reached");
  return RE_OK;
}

RE_API re_status re_nsdf_eval(re_nsdf* s, const float* d_pts, uint32_t n, float* d_out,
                              void* stream) {
  re_status st = re::check(s, "re_nsdf_eval");
  if (st != RE_OK) return st;
  if (!d_pts || !d_out) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_eval: null buffer");
  if (n == 0) return RE_OK;
  cudaStream_t cs = (cudaStream_t)stream;
  st = re::ensure_pack(s, cs);
  if (st != RE_OK) return st;
  auto k = re::nsdf::k_tc_eval;
  RE_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)re::nsdf::kEvalSmemBytes));
  // one CTA per SM; no more CTAs than 128-row tiles, so that a small call's
  // tiles spread over the SMs
  const uint32_t tiles = (n + re::nsdf::kGroupRows - 1) / re::nsdf::kGroupRows;
  const int grid = (int)std::min<uint32_t>((uint32_t)re::sm_count(), tiles);
  *s->sync_err = 0;
  k<<<grid, re::nsdf::kEvalThreads, re::nsdf::kEvalSmemBytes, cs>>>(s->map, s->pack, d_pts, n,
                                                                    d_out, s->sync_err_dev);
  RE_CHECK_LAUNCH("re_nsdf_eval: launch");
  RE_CUDA(cudaStreamSynchronize(cs));
  if (*s->sync_err) return re::fail(RE_ERR_INTERNAL, "re_nsdf_eval: tensor-core wait bound reached");
  return RE_OK;
}

RE_API re_status re_nsdf_check_report(re_nsdf* s, uint32_t thread, int* reported) {
  re_status st = re::check(s, "re_nsdf_check_report");
  if (st != RE_OK) return st;
  if (!reported) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_check_report: null output");
  *s->sync_err = 0;
  re::nsdf::k_check_report<<<1, re::nsdf::kEvalThreads>>>(thread, s->sync_err_dev);
  RE_CHECK_LAUNCH("re_nsdf_check_report: launch");
  RE_CUDA(cudaStreamSynchronize(nullptr));
  *reported = *s->sync_err;
  return RE_OK;
}

RE_API re_status re_nsdf_eval_reference(re_nsdf* s, const float* d_pts, uint32_t n, float* d_out,
                                        void* stream) {
  re_status st = re::check(s, "re_nsdf_eval_reference");
  if (st != RE_OK) return st;
  if (!d_pts || !d_out) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_eval_reference: null buffer");
  if (n == 0) return RE_OK;
  re::nsdf::k_ref_eval<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>(s->map, s->params, d_pts,
                                                                            n, d_out);
  RE_CHECK_LAUNCH("re_nsdf_eval_reference: launch");
  return RE_OK;
}

// Lipschitz estimate of the network over `samples` training points: the
// `quantile` (1 = the maximum) of the forward-difference gradient norms
// with step h.
RE_API re_status re_nsdf_lipschitz(re_nsdf* s, uint32_t samples, float h, float quantile,
                                   float* out, void* stream) {
  re_status st = re::check(s, "re_nsdf_lipschitz");
  if (st != RE_OK) return st;
  if (!out || samples == 0 || !(h > 0.f) || !(quantile > 0.f && quantile <= 1.f) || !s->data)
    return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_lipschitz: bad arguments or no data");
  cudaStream_t cs = (cudaStream_t)stream;
  uint32_t n = std::min(samples, s->npts);
  std::vector<float4> pts(n);
  RE_CUDA(cudaMemcpy(pts.data(), s->data, (size_t)n * 16, cudaMemcpyDeviceToHost));
  std::vector<float> q(12 * (size_t)n);
  for (uint32_t i = 0; i < n; ++i) {
    float p[3] = {pts[i].x, pts[i].y, pts[i].z};
    for (int k = 0; k < 4; ++k)
      for (int a = 0; a < 3; ++a) q[12 * (size_t)i + 3 * k + a] = p[a] + ((k == a + 1) ? h : 0.f);
  }
  float *dq = nullptr, *dv = nullptr, *dn = nullptr;
  std::vector<float> norms(n);
  RE_CUDA(cudaMalloc(&dq, q.size() * 4));
  cudaError_t e = cudaMalloc(&dv, (size_t)n * 4 * 4);
  if (e == cudaSuccess) e = cudaMalloc(&dn, (size_t)n * 4);
  if (e == cudaSuccess) e = cudaMemcpy(dq, q.data(), q.size() * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    st = re_nsdf_eval(s, dq, 4 * n, dv, stream);
    if (st == RE_OK) {
      re::nsdf::k_grad_norm<<<(n + 255) / 256, 256, 0, cs>>>(dv, n, h, dn);
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaMemcpyAsync(norms.data(), dn, (size_t)n * 4, cudaMemcpyDeviceToHost, cs);
      if (e == cudaSuccess) e = cudaStreamSynchronize(cs);
    }
  }
  cudaFree(dq);
  cudaFree(dv);
  cudaFree(dn);
  if (st != RE_OK) return st;
  if (e != cudaSuccess) return re::cuda_fail(e, "re_nsdf_lipschitz");
  size_t k = std::min<size_t>(n - 1, (size_t)std::ceil((double)quantile * n) - 1);
  std::nth_element(norms.begin(), norms.begin() + k, norms.end());
  *out = norms[k];
  s->lipschitz = norms[k];
  return RE_OK;
}

namespace re {
namespace {
re_status trace_check(re_nsdf* s, const re_sdf_params* field, const re_nsdf_trace_params* tp,
                      const re_camera* cam, uint32_t w, uint32_t h, re_sdf_hit* d_out,
                      const char* fn) {
  re_status st = check(s, fn);
  if (st != RE_OK) return st;
  st = check_field(field, fn);
  if (st != RE_OK) return st;
  if (!tp || !cam || !d_out || w < 2 || h < 2) return fail(RE_ERR_INVALID_ARG, "%s: bad arguments", fn);
  if ((uint64_t)w * h > (1ull << 28)) return fail(RE_ERR_LIMIT, "%s: image > 2^28 pixels", fn);
  if (!(tp->flags & RE_NSDF_EXACT_ONLY) && !(tp->lipschitz > 0.f && tp->safety > 0.f))
    return fail(RE_ERR_INVALID_ARG, "%s: lipschitz and safety must be > 0", fn);
  if (tp->cone_tile > 256 ||
      (tp->cone_coarse && (tp->cone_tile == 0 || tp->cone_coarse > 1024 ||
                           tp->cone_coarse <= tp->cone_tile || tp->cone_coarse % tp->cone_tile)))
    return fail(RE_ERR_INVALID_ARG,
                "%s: cone_tile <= 256; cone_coarse 0 or a multiple of cone_tile above it, <= 1024",
                fn);
  if (tp->normal_taps != 0 && tp->normal_taps != 1 && tp->normal_taps != 4 &&
      tp->normal_taps != 6)
    return fail(RE_ERR_INVALID_ARG, "%s: normal_taps 0, 1, 4 or 6", fn);
  if (tp->cone_lanes > 16 || (tp->cone_lanes & (tp->cone_lanes - 1u)))
    return fail(RE_ERR_INVALID_ARG, "%s: cone_lanes 0, 1, 2, 4, 8 or 16", fn);
  return RE_OK;
}
}  // namespace
}  // namespace re

RE_API re_status re_nsdf_trace_network(re_nsdf* s, const re_sdf_params* field,
                                       const re_nsdf_trace_params* tp, const re_camera* cam,
                                       uint32_t w, uint32_t h, re_sdf_hit* d_out, void* stream) {
  re_status st = re::trace_check(s, field, tp, cam, w, h, d_out, "re_nsdf_trace_network");
  if (st != RE_OK) return st;
  cudaStream_t cs = (cudaStream_t)stream;
  const bool exact_only = (tp->flags & RE_NSDF_EXACT_ONLY) != 0u;
  const bool cone = !exact_only && tp->cone_tile > 0;
  size_t need = (size_t)w * h;
  const uint32_t T = tp->cone_tile, C = tp->cone_coarse;
  const uint32_t ctx = cone ? (w + T - 1) / T : 0, cty = cone ? (h + T - 1) / T : 0;
  const uint32_t pcx = cone && C ? (w + C - 1) / C : 0, pcy = cone && C ? (h + C - 1) / C : 0;
  const size_t cone_need = (size_t)ctx * cty + (size_t)pcx * pcy;
  if (cone && s->cone_cap < cone_need) {
    RE_CUDA(cudaStreamSynchronize(cs));
    cudaFree(s->cone_t);
    s->cone_t = nullptr;
    s->cone_cap = 0;
    RE_CUDA(cudaMalloc(&s->cone_t, cone_need * sizeof(float)));
    s->cone_cap = cone_need;
  }
  s->cone_w = s->cone_h = s->cone_tile = s->cone_tiles_x = 0;
  if (!exact_only && !cone && s->queue_cap < need) {
    RE_CUDA(cudaStreamSynchronize(cs));
    cudaFree(s->queue);
    s->queue = nullptr;
    s->queue_cap = 0;
    RE_CUDA(cudaMalloc(&s->queue, need * sizeof(uint4)));
    s->queue_cap = need;
  }
  RE_CUDA(cudaMemsetAsync(s->counters, 0, 64, cs));  // the error word among them
  if (exact_only) return RE_OK;
  st = re::ensure_pack(s, cs);
  if (st != RE_OK) return st;
  unsigned long long* totals = reinterpret_cast<unsigned long long*>(s->counters + 4);
  re::nsdf::MarchDev md;
  md.alpha = tp->safety / tp->lipschitz;
  md.switch_dist = tp->switch_dist;
  md.min_step = tp->min_step;
  md.tmax = field->tmax;
  md.max_steps = tp->max_network_steps ? tp->max_network_steps : 256;
  for (int k = 0; k < 3; ++k) {
    float half = 1.0f / s->map.inv_half[k];
    md.bmin[k] = s->map.center[k] - half;
    md.bmax[k] = s->map.center[k] + half;
  }
  if (cone) {
    const uint32_t K = tp->cone_lanes ? tp->cone_lanes : 1u;
    auto kc = K == 16u  ? re::nsdf::k_nsdf_cone<16>
              : K == 8u ? re::nsdf::k_nsdf_cone<8>
              : K == 4u ? re::nsdf::k_nsdf_cone<4>
              : K == 2u ? re::nsdf::k_nsdf_cone<2>
                        : re::nsdf::k_nsdf_cone<1>;
    RE_CUDA(cudaFuncSetAttribute(kc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)re::kTcSmemBytes));
    float* fine = s->cone_t;
    float* coarse = s->cone_t + (size_t)ctx * cty;
    re::nsdf::ConeDev cd{};
    if (C) {
      // coarse level from the box entry (cursor counters[0])
      cd.tile = C;
      cd.tiles_x = pcx;
      cd.tiles_y = pcy;
      cd.parent = nullptr;
      const int grid = std::min<int>(re::tc_grid(kc),
                                     (int)((pcx * pcy * K + re::nsdf::kTcThreads - 1) /
                                           re::nsdf::kTcThreads));
      kc<<<grid, re::nsdf::kTcThreads, re::kTcSmemBytes, cs>>>(
          s->map, s->pack, md, cd, re::cam_dev(*cam), w, h, s->counters, totals, coarse, s->err);
      RE_CHECK_LAUNCH("re_nsdf_trace_network: coarse cone launch");
    }
    // fine level, from the coarse tiles' starts (cursor counters[3])
    cd.tile = T;
    cd.tiles_x = ctx;
    cd.tiles_y = cty;
    cd.parent = C ? coarse : nullptr;
    cd.parent_tile = C;
    cd.parent_tiles_x = pcx;
    const int grid = std::min<int>(
        re::tc_grid(kc), (int)((ctx * cty * K + re::nsdf::kTcThreads - 1) / re::nsdf::kTcThreads));
    kc<<<grid, re::nsdf::kTcThreads, re::kTcSmemBytes, cs>>>(
        s->map, s->pack, md, cd, re::cam_dev(*cam), w, h, s->counters + 3, totals, fine, s->err);
    RE_CHECK_LAUNCH("re_nsdf_trace_network: cone launch");
    s->cone_w = w;
    s->cone_h = h;
    s->cone_tile = T;
    s->cone_tiles_x = ctx;
    return RE_OK;
  }
  auto k = re::nsdf::k_nsdf_march;
  RE_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)re::kTcSmemBytes));
  k<<<re::tc_grid(k), re::nsdf::kTcThreads, re::kTcSmemBytes, cs>>>(
      s->map, s->pack, md, re::cam_dev(*cam), w, h, s->counters, totals, s->queue,
      reinterpret_cast<float4*>(d_out), s->err);
  RE_CHECK_LAUNCH("re_nsdf_trace_network: march launch");
  return RE_OK;
}

RE_API re_status re_nsdf_trace_exact(re_nsdf* s, const re_sdf_params* field,
                                     const re_nsdf_trace_params* tp, const re_camera* cam,
                                     uint32_t w, uint32_t h, re_sdf_hit* d_out, void* stream) {
  re_status st = re::trace_check(s, field, tp, cam, w, h, d_out, "re_nsdf_trace_exact");
  if (st != RE_OK) return st;
  const bool exact_only = (tp->flags & RE_NSDF_EXACT_ONLY) != 0u;
  const bool cone = !exact_only && tp->cone_tile > 0;
  if (cone && !(s->cone_w == w && s->cone_h == h && s->cone_tile == tp->cone_tile))
    return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_trace_exact: no cone phase for this image");
  if (!exact_only && !cone && s->queue_cap < (size_t)w * h)
    return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_trace_exact: no network phase for this image");
  cudaStream_t cs = (cudaStream_t)stream;
  unsigned long long* totals = reinterpret_cast<unsigned long long*>(s->counters + 4);
  re::nsdf::RefineDev rd;
  rd.max_steps = tp->max_exact_steps ? tp->max_exact_steps : field->max_steps;
  rd.root_steps = tp->root_steps ? tp->root_steps : 4;
  rd.relax = tp->relax;
  rd.root_tol = tp->root_tol > 0.f ? tp->root_tol : 0.f;
  // |Perlin| <= 2 (each corner term |g . r| <= |r_x| + |r_y| <= 2 and the
  // interpolation is convex), so fBm <= 2 (2 - 2^(1 - octaves)) and the
  // density is positive above this height
  rd.ceiling =
      2.0f * std::fabs(field->amplitude) * (2.0f - std::ldexp(1.0f, 1 - (int)field->octaves)) + 1e-3f;
  rd.normal_taps = tp->normal_taps == 4u || tp->normal_taps == 1u ? tp->normal_taps : 6u;
  rd.tile_t = cone ? s->cone_t : nullptr;
  rd.cone_tile = cone ? s->cone_tile : 1u;
  rd.cone_tiles_x = cone ? s->cone_tiles_x : 0u;
  auto refine = [&](auto rows_kernel, auto copy_kernel) {
    return re::launch_field(
        rd.normal_taps == 1u ? re::field_on_rows(field->octaves, (uint64_t)w * h)
                             : re::field_on_rows<true>(field->octaves, (uint64_t)w * h),
        rows_kernel, copy_kernel, (uint64_t)w * h, [](uint32_t warps) { return warps * re::nsdf::kRefineRing; },
        [&](auto k, int grid, uint32_t threads, uint32_t smem, re::RowsSpread spread) {
          k<<<grid, threads, smem, cs>>>(re::perm_of(field->seed), re::field_of(*field), rd,
                                         re::cam_dev(*cam), w, h, spread,
                                         exact_only || cone ? 1 : 0, s->queue, s->counters, totals,
                                         reinterpret_cast<float4*>(d_out));
        });
  };
  using re::CopyForm;
  using re::RowsForm;
  st = rd.normal_taps == 1u ? refine(re::nsdf::k_sdf_refine<1u, RowsForm>,
                                     re::nsdf::k_sdf_refine<1u, CopyForm>)
       : rd.normal_taps == 4u ? refine(re::nsdf::k_sdf_refine<4u, RowsForm>,
                                       re::nsdf::k_sdf_refine<4u, CopyForm>)
                              : refine(re::nsdf::k_sdf_refine<6u, RowsForm>,
                                       re::nsdf::k_sdf_refine<6u, CopyForm>);
  if (st != RE_OK) return st;
  RE_CHECK_LAUNCH("re_nsdf_trace_exact: refine launch");
  if (rd.normal_taps == 1u) {
    RE_CUDA(cudaFuncSetAttribute(re::nsdf::k_sdf_grad_normal,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)re::kRowsSmemBytes));
    re::nsdf::k_sdf_grad_normal<<<re::sm_count(), re::kRowsThreads, re::kRowsSmemBytes, cs>>>(
        re::perm_of(field->seed), re::field_of(*field), w * h, 1.0f,
        reinterpret_cast<float4*>(d_out), totals);
    RE_CHECK_LAUNCH("re_nsdf_trace_exact: normal launch");
  }
  return RE_OK;
}

RE_API re_status re_nsdf_trace(re_nsdf* s, const re_sdf_params* field,
                               const re_nsdf_trace_params* tp, const re_camera* cam, uint32_t w,
                               uint32_t h, re_sdf_hit* d_out, void* stream) {
  re_status st = re_nsdf_trace_network(s, field, tp, cam, w, h, d_out, stream);
  if (st != RE_OK) return st;
  return re_nsdf_trace_exact(s, field, tp, cam, w, h, d_out, stream);
}

RE_API re_status re_nsdf_trace_status(re_nsdf* s, uint32_t* num_refined, int* error,
                                      uint64_t* evals) {
  re_status st = re::check(s, "re_nsdf_trace_status");
  if (st != RE_OK) return st;
  uint32_t c[16] = {};
  RE_CUDA(cudaMemcpy(c, s->counters, 64, cudaMemcpyDeviceToHost));
  if (num_refined) *num_refined = c[1];
  if (error) *error = (int)c[12];
  if (evals) std::memcpy(evals, c + 4, 4 * sizeof(uint64_t));
  return RE_OK;
}

// Checkpoint: 16-byte header ("RENSDF01", parameter count, steps done),
// the input map, then parameters and both Adam moments as FP32.
RE_API re_status re_nsdf_save(const re_nsdf* s, const char* path) {
  using namespace re::nsdf;
  re_status st = re::check(s, "re_nsdf_save");
  if (st != RE_OK) return st;
  if (!path) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_save: null path");
  std::vector<float> buf(3 * (size_t)kNumParams);
  RE_CUDA(cudaMemcpy(buf.data(), s->params, kNumParams * 4, cudaMemcpyDeviceToHost));
  RE_CUDA(cudaMemcpy(buf.data() + kNumParams, s->adam_m, kNumParams * 4, cudaMemcpyDeviceToHost));
  RE_CUDA(cudaMemcpy(buf.data() + 2 * kNumParams, s->adam_v, kNumParams * 4, cudaMemcpyDeviceToHost));
  uint32_t steps = 0;
  RE_CUDA(cudaMemcpy(&steps, s->step_ctr, 4, cudaMemcpyDeviceToHost));
  FILE* f = std::fopen(path, "wb");
  if (!f) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_save: cannot open %s", path);
  uint32_t hdr[4] = {0x534E4552u, 0x31304653u, (uint32_t)kNumParams, steps};
  bool ok = std::fwrite(hdr, 4, 4, f) == 4 && std::fwrite(&s->map, sizeof(s->map), 1, f) == 1 &&
            std::fwrite(buf.data(), 4, buf.size(), f) == buf.size();
  std::fclose(f);
  if (!ok) return re::fail(RE_ERR_INTERNAL, "re_nsdf_save: write failed");
  return RE_OK;
}

RE_API re_status re_nsdf_load(re_nsdf* s, const char* path) {
  using namespace re::nsdf;
  re_status st = re::check(s, "re_nsdf_load");
  if (st != RE_OK) return st;
  if (!path) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_load: null path");
  FILE* f = std::fopen(path, "rb");
  if (!f) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_load: cannot open %s", path);
  uint32_t hdr[4];
  InputMap m;
  std::vector<float> buf(3 * (size_t)kNumParams);
  bool ok = std::fread(hdr, 4, 4, f) == 4 && hdr[0] == 0x534E4552u && hdr[1] == 0x31304653u &&
            hdr[2] == (uint32_t)kNumParams && std::fread(&m, sizeof(m), 1, f) == 1 &&
            std::fread(buf.data(), 4, buf.size(), f) == buf.size();
  std::fclose(f);
  if (!ok) return re::fail(RE_ERR_INVALID_ARG, "re_nsdf_load: %s is not a checkpoint of this network", path);
  RE_CUDA(cudaMemcpy(s->params, buf.data(), kNumParams * 4, cudaMemcpyHostToDevice));
  RE_CUDA(cudaMemcpy(s->adam_m, buf.data() + kNumParams, kNumParams * 4, cudaMemcpyHostToDevice));
  RE_CUDA(cudaMemcpy(s->adam_v, buf.data() + 2 * kNumParams, kNumParams * 4, cudaMemcpyHostToDevice));
  RE_CUDA(cudaMemcpy(s->step_ctr, &hdr[3], 4, cudaMemcpyHostToDevice));
  re::drop_graph(s);
  s->map = m;
  s->total_steps_done = hdr[3];
  s->pack_valid = false;
  s->lipschitz = 0.f;
  return RE_OK;
}

}  // extern "C"
