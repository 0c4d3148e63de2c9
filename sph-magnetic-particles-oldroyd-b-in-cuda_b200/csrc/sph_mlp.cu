// sph_mlp.cu -- the surrogate network's kernels and C ABI (include/sph_mlp.h): an ensemble
// of independent MLPs ("heads") 6 -> 256 -> 256 -> 256 -> 4 with GELU, BF16 weights and
// activations, FP32 accumulation, trained with Adam on FP32 master weights.
//
// The 256 x 256 layers (forward, input gradient and weight gradient) run on the tensor
// cores through sph_tc_gemm.cuh (tcgen05, accumulators in TMEM); the 6-wide input layer
// and the 4-wide output layer are a few hundred multiply-adds per sample and run on the
// CUDA cores.  One kernel takes 128 samples of a head through all four layers, one takes
// them back through them (k_forward, k_backward); the weight gradients of both 256 x 256
// layers are one GEMM launch, and one kernel sums their slices, updates the parameters and
// rounds the new weights (k_update).  Every reduction has a fixed order: training is
// bit-reproducible.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <algorithm>
#include <string>
#include <utility>
#include <vector>

#include "sph_mlp.h"
#include "sph_tc_gemm.cuh"

using sph::tc::GemmArgs;
namespace tc = sph::tc;

namespace {

constexpr int IN = SPH_MLP_IN, HID = SPH_MLP_HIDDEN, OUT = SPH_MLP_OUT;
// parameter layout of one head (FP32 master copy, gradients and Adam moments alike)
constexpr int OFF_W1 = 0;
constexpr int OFF_B1 = OFF_W1 + HID * IN;
constexpr int OFF_W2 = OFF_B1 + HID;
constexpr int OFF_B2 = OFF_W2 + HID * HID;
constexpr int OFF_W3 = OFF_B2 + HID;
constexpr int OFF_B3 = OFF_W3 + HID * HID;
constexpr int OFF_W4 = OFF_B3 + HID;
constexpr int OFF_B4 = OFF_W4 + OUT * HID;
constexpr int NPARAM = OFF_B4 + OUT;
static_assert(NPARAM == SPH_MLP_NPARAMS, "parameter count");

// ---- the network's passes: one CTA carries 128 samples of one head through its layers ----
//
// The 128 x 256 activations live in shared memory as the next layer's A operand (four K
// chunks of 64 in the canonical layout); the 256 x 256 weights stream through a second
// region, four chunks of 32 KB, each layer's copied while the CUDA cores work on the layer
// before.  16 warps: warp w takes TMEM lanes (samples) 32 (w % 4) .. + 31 and columns
// 64 (w / 4) .. + 63, so a thread holds 64 neurons of one sample, the K chunk w / 4.
//
// R > 1: a CTA takes 128 / R samples, each in R rows of the operand (the tensor cores are nearly
// idle), and a thread 64 / R neurons of its row's sample, so that a batch of few tiles (8 per
// head at 1024 samples) spreads its GELUs over R times as many SMs.  R is chosen so that the
// tiles fit one wave (net_rep).
// What bounds it is the GELU arithmetic (erff) of 3 x 256 neurons per sample on the CUDA
// cores, 36 instructions each (77 M of them for 20,011 points and 5 heads: issue half of the
// cycles), and the weights each tile reads from L2 (256 KB).  Measured there, prediction by
// all heads: 2.29 ms with a kernel per layer, the activations in memory between them and 1024
// samples per pass, 0.18 ms so.  A training step (5 heads, batch 1024): 373 us in 15 launches,
// 107 us in 5.
constexpr int kNetThreads = 512;
constexpr int kNetA = tc::kTileM * HID * 2;       // bytes of the activations
constexpr int kNetChunkA = tc::kTileM * tc::kChunkK * 2;
constexpr int kNetChunkW = HID * tc::kChunkK * 2;
constexpr int kNetW = HID * HID * 2;              // bytes of one layer's weights
constexpr int kNetChunks = HID / tc::kChunkK;
static_assert(kNetChunks == 4 && kNetThreads == 128 * kNetChunks, "a K chunk per four warps");
struct NetSmall {
  float w1[HID][8];   // W1 row and its bias: w[0..5], b, 0
  float w4[HID][4];   // W4 by column
  float b2[HID], b3[HID], b4[4];
  float4 red[kNetChunks][tc::kTileM];  // output sums of the four column groups
  uint64_t bar;
  uint32_t tmem;
};
constexpr int kNetSmem = kNetA + kNetW + (int)sizeof(NetSmall);
static_assert(kNetSmem <= 227 * 1024, "shared memory of one CTA");

// Copies a 256 x 256 bf16 matrix (rows of 256) into the four chunks at dst, asynchronously:
// eight lanes fill the eight 16-byte rows of a core matrix (no bank conflicts), four such
// groups take 64 consecutive bytes of each row.
__device__ __forceinline__ void net_load_weights(uint8_t* dst, const __nv_bfloat16* w) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q = warp; q < (HID / 8) * (HID / 32); q += kNetThreads / 32) {
    const int row = (q >> 3) * 8 + (lane & 7), k8 = (q & 7) * 4 + (lane >> 3);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                     tc::smem_u32(dst + (k8 >> 3) * kNetChunkW + tc::core_offset(row, k8 & 7))),
                 "l"(w + (size_t)row * HID + k8 * 8)
                 : "memory");
  }
}

// Starts the layer's product: accumulator (128 x 256, FP32, TMEM) = A . W^T, once every thread's
// shared-memory writes and copies have landed.  Returns false if its completion was not
// observed in time (after a second bounded wait, which lets the MMAs that write TMEM finish).
__device__ __forceinline__ bool net_product(uint8_t* smem, NetSmall* s, uint32_t parity) {
  tc::cp_async_wait_all();
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (threadIdx.x == 0) {
    const uint32_t idesc = tc::idesc_bf16_f32(tc::kTileM, HID);
    const uint32_t sa = tc::smem_u32(smem), sw = sa + kNetA;
#pragma unroll
    for (int c = 0; c < kNetChunks; ++c)
#pragma unroll
      for (int q = 0; q < tc::kChunkK / 16; ++q)
        tc::mma_bf16(s->tmem, tc::smem_desc(sa + c * kNetChunkA + q * 256),
                     tc::smem_desc(sw + c * kNetChunkW + q * 256), idesc, c > 0 || q > 0 ? 1 : 0);
    tc::mma_commit(&s->bar);
  }
  const bool ok = __syncthreads_and(tc::mbar_wait(&s->bar, parity) ? 1 : 0) != 0;
  if (!ok) tc::mbar_wait(&s->bar, parity);
  tc::fence_after_sync();
  return ok;
}

__device__ __forceinline__ void net_open(NetSmall* s) {
  if (threadIdx.x < 32) tc::tmem_alloc(&s->tmem, tc::kTmemCols);
  if (threadIdx.x == 0) tc::mbar_init(&s->bar, 1);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
}
__device__ __forceinline__ void net_close(NetSmall* s, bool ok, int* err) {
  tc::cp_async_wait_all();
  if (!ok && threadIdx.x == 0) atomicExch(err, 1);
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc::fence_after_sync();
    tc::tmem_free(s->tmem, tc::kTmemCols);
  }
}

// 8 activations of a sample, moved 16 bytes at a time.
struct __align__(16) Act8 {
  __nv_bfloat16 v[8];
  __device__ __forceinline__ __nv_bfloat16& operator[](int q) { return v[q]; }
};
static_assert(sizeof(Act8) == sizeof(uint4) && alignof(Act8) == alignof(uint4), "one 16-byte move");

// Stores them, columns 8 k8 .. + 7 of chunk c, into the sample's rows of the A operand.
template <int R>
__device__ __forceinline__ void net_store8(uint8_t* smem, int c, int sample, int k8, const Act8& h) {
#pragma unroll
  for (int d = 0; d < R; ++d)
    *reinterpret_cast<uint4*>(smem + c * kNetChunkA +
                              tc::core_offset(sample + d * (tc::kTileM / R), k8)) =
        *reinterpret_cast<const uint4*>(&h);
}

// Reads this thread's 64 / R accumulator columns 16 at a time, the next 16 in flight while
// `use(k8, v)` works on the ones before (v: 8 columns from 8 k8 on).
template <int R, typename F>
__device__ __forceinline__ void net_columns(uint32_t tm, F use) {
  constexpr int kN = 4 / R;  // groups of 16 columns
  uint32_t r[2][16];
  tc::tmem_ld16_start(tm, r[0]);
  tc::tmem_ld16_finish(r[0]);
#pragma unroll
  for (int k = 0; k < kN; ++k) {
    if (k + 1 < kN) tc::tmem_ld16_start(tm + 16 * (k + 1), r[(k + 1) & 1]);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = __uint_as_float(r[k & 1][8 * p + q]);
      use(2 * k + p, v);
    }
    if (k + 1 < kN) tc::tmem_ld16_finish(r[(k + 1) & 1]);
  }
}

__device__ __forceinline__ float4 add4(const float4& a, const float4& b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

struct NetArgs {
  const float* x;       // n x IN
  const float* y;       // targets (training)
  const float* params;  // every head's FP32 parameters
  const __nv_bfloat16 *w1b, *wa, *wb, *w4b;  // forward: W2, W3; backward: W3^T, W2^T
  int n, heads;         // samples (a multiple of 128), heads
  float* out;           // heads x n x OUT
  // training: slopes GELU'(z) of the three layers, by tile, column group of 4 and sample
  // (float4 index ((head * tiles + tile) * 64 + column / 4) * 128 + sample); activations and
  // their gradients transposed (heads x 256 x n); dL/dout; squared errors
  float *g1, *g2, *g3;
  __nv_bfloat16 *t1, *t2, *t3;
  float *dout, *sqerr;
  int* err;
};

// z = W1 x + b1, then h = GELU(W2 GELU(z) + b2), GELU(W3 h + b3), out = W4 h + b4.  A CTA takes
// consecutive tiles of 128 samples (mostly of one head).  TRAIN: also writes what the backward
// pass needs, with the targets' squared errors and dL/dout.
template <bool TRAIN, int R>
__global__ void __launch_bounds__(kNetThreads, 1) k_forward(NetArgs a) {
  constexpr int kS = tc::kTileM / R;  // samples per tile
  extern __shared__ __align__(1024) uint8_t smem[];
  NetSmall* s = reinterpret_cast<NetSmall*>(smem + kNetA + kNetW);
  uint8_t* wsm = smem + kNetA;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int arow = 32 * (warp & 3) + lane, grp = warp >> 2;  // operand row, K chunk
  const int row = arow % kS, sub8 = arow / kS * (8 / R);     // sample, first 8 columns of its own
  const int tiles = a.n / kS, total = tiles * a.heads;
  const int t0 = (int)((long long)blockIdx.x * total / gridDim.x);
  const int t1 = (int)((long long)(blockIdx.x + 1) * total / gridDim.x);
  if (t0 >= t1) return;
  net_open(s);
  const uint32_t tm = s->tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 64 * grp + 8 * sub8;
  net_load_weights(wsm, a.wa + (size_t)(t0 / tiles) * HID * HID);
  int loaded = -1;
  uint32_t parity = 0;
  bool ok = true;
  for (int t = t0; t < t1; ++t) {
    const int head = t / tiles, b = (t % tiles) * kS + row;
    if (head != loaded) {
      __syncthreads();  // the last tile's readers
      const float* P = a.params + (size_t)head * NPARAM;
      for (int j = threadIdx.x; j < HID; j += kNetThreads) {
#pragma unroll
        for (int i = 0; i < IN; ++i)
          s->w1[j][i] = __bfloat162float(a.w1b[(size_t)head * HID * IN + j * IN + i]);
        s->w1[j][6] = P[OFF_B1 + j];
        s->b2[j] = P[OFF_B2 + j];
        s->b3[j] = P[OFF_B3 + j];
#pragma unroll
        for (int o = 0; o < OUT; ++o)
          s->w4[j][o] = __bfloat162float(a.w4b[(size_t)head * OUT * HID + o * HID + j]);
      }
      if (threadIdx.x < OUT) s->b4[threadIdx.x] = P[OFF_B4 + threadIdx.x];
      loaded = head;
      __syncthreads();
    }
    const size_t gbase = ((size_t)t * 64 + 16 * grp) * kS + row;          // slopes, float4
    const size_t tbase = ((size_t)head * HID + 64 * grp) * a.n + b;       // transposed
    // Output sums of a prediction: 16 columns in order, then pairs of such sums, pairs of pairs
    // and so on.  The tree is the same for every R, so that a point's outputs do not depend on
    // how many others are predicted with it.
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 o4 = zero4, pair4 = zero4, half4 = zero4;
    // 8 neurons: pre-activations z -> activations into the A operand (and the backward
    // pass's arrays); last: the output layer's sums instead of an operand
    auto activate = [&](const float (&z)[8], int k, float* g, __nv_bfloat16* ht, bool last) {
      const int k8 = sub8 + k;
      Act8 h;
      float sl[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float e = erff(z[q] * 0.70710678118654752f);
        h[q] = __float2bfloat16(0.5f * z[q] * (1.0f + e));
        if (TRAIN)
          sl[q] = 0.5f * (1.0f + e) + z[q] * expf(-0.5f * z[q] * z[q]) * 0.39894228040143268f;
        if (!TRAIN && last) {
          const float4 w = *reinterpret_cast<const float4*>(s->w4[64 * grp + 8 * k8 + q]);
          const float hq = __bfloat162float(h[q]);
          o4.x = fmaf(w.x, hq, o4.x);
          o4.y = fmaf(w.y, hq, o4.y);
          o4.z = fmaf(w.z, hq, o4.z);
          o4.w = fmaf(w.w, hq, o4.w);
        }
      }
      if (!last || TRAIN) net_store8<R>(smem, grp, row, k8, h);
      if (TRAIN) {
        float4* gp = reinterpret_cast<float4*>(g) + gbase + (size_t)(2 * k8) * kS;
        gp[0] = make_float4(sl[0], sl[1], sl[2], sl[3]);
        gp[kS] = make_float4(sl[4], sl[5], sl[6], sl[7]);
#pragma unroll
        for (int q = 0; q < 8; ++q) ht[tbase + (size_t)(8 * k8 + q) * a.n] = h[q];
      }
    };
    {
      float x[IN];
#pragma unroll
      for (int i = 0; i < IN; ++i) x[i] = a.x[(size_t)b * IN + i];  // any float alignment
#pragma unroll 1
      for (int k = 0; k < 8 / R; ++k) {
        float z[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float* w = s->w1[64 * grp + 8 * (sub8 + k) + q];
          const float4 u = *reinterpret_cast<const float4*>(w);
          const float4 v = *reinterpret_cast<const float4*>(w + 4);
          z[q] = fmaf(v.y, x[5], fmaf(v.x, x[4], fmaf(u.w, x[3], fmaf(u.z, x[2],
                 fmaf(u.y, x[1], fmaf(u.x, x[0], v.z))))));
        }
        activate(z, k, a.g1, a.t1, false);
      }
    }
    ok = net_product(smem, s, parity);
    parity ^= 1;
    if (!ok) break;
    net_load_weights(wsm, a.wb + (size_t)head * HID * HID);
    net_columns<R>(tm, [&](int k, const float (&v)[8]) {
      float z[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) z[q] = v[q] + s->b2[64 * grp + 8 * (sub8 + k) + q];
      activate(z, k, a.g2, a.t2, false);
    });
    ok = net_product(smem, s, parity);
    parity ^= 1;
    if (!ok) break;
    if (t + 1 < t1) net_load_weights(wsm, a.wa + (size_t)((t + 1) / tiles) * HID * HID);
    net_columns<R>(tm, [&](int k, const float (&v)[8]) {
      float z[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) z[q] = v[q] + s->b3[64 * grp + 8 * (sub8 + k) + q];
      activate(z, k, a.g3, a.t3, true);
      if (!TRAIN && (k & 1)) {  // the 16 columns of group k / 2 are done
        const int g = k >> 1;
        if (g & 1) o4 = add4(pair4, o4);
        if (g == 3) o4 = add4(half4, o4);
        if (g == 1) half4 = o4;
        if (g + 1 < 4 / R) {
          pair4 = o4;
          o4 = zero4;
        }
      }
    });
    const size_t at = (size_t)head * a.n + b;
    if (!TRAIN) {
      s->red[grp][arow] = o4;
      __syncthreads();
      if (grp == 0 && arow < kS) {
        float4 g4[kNetChunks];  // the sums of the sample's columns 64 c .. + 63
#pragma unroll
        for (int c = 0; c < kNetChunks; ++c) {
          g4[c] = s->red[c][row];
          if (R > 1) g4[c] = add4(g4[c], s->red[c][row + kS]);
          if (R == 4)
            g4[c] = add4(g4[c], add4(s->red[c][row + 2 * kS], s->red[c][row + 3 * kS]));
        }
        float* o = a.out + at * OUT;  // any float alignment
        o[0] = ((g4[0].x + g4[1].x) + (g4[2].x + g4[3].x)) + s->b4[0];
        o[1] = ((g4[0].y + g4[1].y) + (g4[2].y + g4[3].y)) + s->b4[1];
        o[2] = ((g4[0].z + g4[1].z) + (g4[2].z + g4[3].z)) + s->b4[2];
        o[3] = ((g4[0].w + g4[1].w) + (g4[2].w + g4[3].w)) + s->b4[3];
      }
    } else {
      // output `grp` of the sample, summed over the neurons in their order
      __syncthreads();
      float* red = reinterpret_cast<float*>(s->red);
      if (arow < kS) {
        float acc = 0.0f;
        for (int c = 0; c < kNetChunks; ++c)
#pragma unroll 2
          for (int k8 = 0; k8 < 8; ++k8) {
            const uint4 u = *reinterpret_cast<const uint4*>(smem + c * kNetChunkA +
                                                            tc::core_offset(row, k8));
            const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float2 h = __bfloat1622float2(h2[q]);
              acc = fmaf(s->w4[64 * c + 8 * k8 + 2 * q][grp], h.x, acc);
              acc = fmaf(s->w4[64 * c + 8 * k8 + 2 * q + 1][grp], h.y, acc);
            }
          }
        const float r = acc + s->b4[grp], e = r - a.y[(size_t)b * OUT + grp];
        a.dout[at * OUT + grp] = 2.0f * e / (float)(a.n * OUT);
        red[4 * row + grp] = e;
      }
      __syncthreads();
      if (grp == 0 && arow < kS) {
        float se = 0.0f;
#pragma unroll
        for (int o = 0; o < OUT; ++o) se += red[4 * row + o] * red[4 * row + o];
        a.sqerr[at] = se;
      }
    }
  }
  net_close(s, ok, a.err);
}

// dz3 = (W4^T dout) GELU'(z3), dz2 = (dz3 W3) GELU'(z2), dz1 = (dz2 W2) GELU'(z1), each written
// transposed (t3, t2, t1).
template <int R>
__global__ void __launch_bounds__(kNetThreads, 1) k_backward(NetArgs a) {
  constexpr int kS = tc::kTileM / R;
  extern __shared__ __align__(1024) uint8_t smem[];
  NetSmall* s = reinterpret_cast<NetSmall*>(smem + kNetA + kNetW);
  uint8_t* wsm = smem + kNetA;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int arow = 32 * (warp & 3) + lane, grp = warp >> 2;
  const int row = arow % kS, sub8 = arow / kS * (8 / R);
  const int tiles = a.n / kS;
  const int t = blockIdx.x, head = t / tiles, b = (t % tiles) * kS + row;
  net_open(s);
  const uint32_t tm = s->tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 64 * grp + 8 * sub8;
  net_load_weights(wsm, a.wa + (size_t)head * HID * HID);
  for (int j = threadIdx.x; j < HID; j += kNetThreads)
#pragma unroll
    for (int o = 0; o < OUT; ++o)
      s->w4[j][o] = __bfloat162float(a.w4b[(size_t)head * OUT * HID + o * HID + j]);
  __syncthreads();
  const size_t gbase = ((size_t)t * 64 + 16 * grp) * kS + row;
  const size_t tbase = ((size_t)head * HID + 64 * grp) * a.n + b;
  auto back = [&](const float (&v)[8], int k, const float* g, __nv_bfloat16* dzt, bool last) {
    const int k8 = sub8 + k;
    const float4* gp = reinterpret_cast<const float4*>(g) + gbase + (size_t)(2 * k8) * kS;
    const float4 u = gp[0], w = gp[kS];
    const float sl[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
    Act8 h;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      h[q] = __float2bfloat16(v[q] * sl[q]);
      dzt[tbase + (size_t)(8 * k8 + q) * a.n] = h[q];
    }
    if (!last) net_store8<R>(smem, grp, row, k8, h);
  };
  const float4 d = reinterpret_cast<const float4*>(a.dout)[(size_t)head * a.n + b];
#pragma unroll 1
  for (int k = 0; k < 8 / R; ++k) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float4 w = *reinterpret_cast<const float4*>(s->w4[64 * grp + 8 * (sub8 + k) + q]);
      v[q] = fmaf(d.w, w.w, fmaf(d.z, w.z, fmaf(d.y, w.y, fmaf(d.x, w.x, 0.0f))));
    }
    back(v, k, a.g3, a.t3, false);
  }
  bool ok = net_product(smem, s, 0);
  if (ok) {
    net_load_weights(wsm, a.wb + (size_t)head * HID * HID);
    net_columns<R>(tm, [&](int k, const float (&v)[8]) { back(v, k, a.g2, a.t2, false); });
    ok = net_product(smem, s, 1);
  }
  if (ok) {
    net_columns<R>(tm, [&](int k, const float (&v)[8]) { back(v, k, a.g1, a.t1, true); });
  }
  net_close(s, ok, a.err);
}

// Weight gradients of both 256 x 256 layers, K = the batch split over `splits` CTAs per output
// tile (2 tiles per head and layer leave most SMs idle otherwise): blockIdx.z = layer * splits
// + slice, slices summed in order by k_update.
// Two CTAs share an SM (2 x 96 KB of stages, 2 x 256 TMEM columns).
constexpr int kWgradSmem = 2 * tc::kStageBytes;
constexpr int kMaxSplits = 8;  // slices of the K = batch reduction, at most
struct WgradArgs {
  const __nv_bfloat16 *dz[2], *h[2];  // transposed, heads x 256 x B
  float* ws;                          // (layer * splits + slice) x heads x 256 x 256
  int B, splits;
  int* err;
};
__global__ void __launch_bounds__(128, 2) k_wgrad(WgradArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t bar[2];
  __shared__ uint32_t tmem_sh;
  const int warp = threadIdx.x >> 5;
  if (warp == 0) tc::tmem_alloc(&tmem_sh, tc::kTmemCols);
  if (threadIdx.x == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_sh;
  const int layer = (int)blockIdx.z / a.splits;
  GemmArgs g;
  g.A = layer ? a.dz[1] : a.dz[0];
  g.B = layer ? a.h[1] : a.h[0];
  g.strideA = g.strideB = (long long)a.B * HID;
  g.lda = g.ldb = a.B;
  g.M = g.N = g.ntile = HID;
  g.K = a.B;
  g.err = a.err;
  const bool ok = __syncthreads_and(
      tc::gemm_mainloop(g, smem, bar, tmem, (int)blockIdx.z % a.splits, a.splits));
  if (ok) {
    const int row = tc::tile_m0(g) + threadIdx.x;
    float* c = a.ws + (((size_t)blockIdx.z * gridDim.y + blockIdx.y) * HID + row) * HID;
    for (int c0 = 0; c0 < HID; c0 += 16) {
      float v[16];
      tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
      for (int q = 0; q < 16; q += 4)
        *reinterpret_cast<float4*>(c + c0 + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
    }
  } else if (threadIdx.x == 0) {
    atomicExch(a.err, 1);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_free(tmem, tc::kTmemCols);
  }
}

// The gradients that are not 256 x 256: dW4[.][j], dW1[j][.], db1[j], db2[j], db3[j] of neuron j
// and db4.  A lane per gradient, 16 per neuron, 16 neurons per block; every gradient is one
// chain s = v u + s over the batch in order, with v one of the neuron's (transposed) activations
// or gradients and u one of dout, x or 1, staged for the whole block 128 samples at a time.
// What bounds it is the chain itself, 1024 dependent multiply-adds; a thread per gradient that
// fetched both factors for each sample took 172 us of a 373 us step at batch 1024 (5 heads).
constexpr int kSgNeurons = 16, kSgBatch = 128;
__global__ void __launch_bounds__(256) k_small_grads(const float* __restrict__ dout,
                                                     const __nv_bfloat16* __restrict__ h3t,
                                                     const __nv_bfloat16* __restrict__ dz1t,
                                                     const __nv_bfloat16* __restrict__ dz2t,
                                                     const __nv_bfloat16* __restrict__ dz3t,
                                                     const float* __restrict__ x, int B,
                                                     float* grads) {
  __shared__ float su[kSgBatch][16];                                  // dout (4), x (6), 1
  __shared__ __align__(16) __nv_bfloat16 sv[kSgNeurons][5][kSgBatch + 8];  // h3, dz1, dz2, dz3, 1
  const int head = blockIdx.y, q = threadIdx.x & 15, nj = threadIdx.x >> 4;
  const int j0 = blockIdx.x * kSgNeurons, j = j0 + nj;
  // chain q of the neuron: dW4 0..3, dW1 4..9, db1..3 10..12, db4 (two neurons' last lanes)
  const int o4 = (j & 1) * 3 + q - 13;  // db4 output of lanes 13..15 of neurons 0 and 1
  const int src = q < 4 ? 0 : q < 11 ? 1 : q == 11 ? 2 : q == 12 ? 3 : 4;
  const int col = q < 10 ? q : q < 13 ? 10 : min(o4, 3);
  for (int k = threadIdx.x; k < kSgNeurons * (kSgBatch + 8); k += 256)
    sv[k / (kSgBatch + 8)][4][k % (kSgBatch + 8)] = __float2bfloat16(1.0f);
  const __nv_bfloat16* const arrays[4] = {h3t, dz1t, dz2t, dz3t};
  // staged by this thread: 8 factors u (column tc of samples tr + 16 m) and 8 samples of each of
  // its neuron's arrays, fetched while the samples before are summed
  const int tc = threadIdx.x & 15, tr = threadIdx.x >> 4;
  float ru[8];
  uint4 rv[4];
  auto fetch = [&](int b0) {
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int b = b0 + tr + 16 * m;
      ru[m] = tc < OUT ? dout[((size_t)head * B + b) * OUT + tc]
              : tc < OUT + IN ? x[(size_t)b * IN + tc - OUT] : 1.0f;
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
      rv[m] = *reinterpret_cast<const uint4*>(arrays[m] + ((size_t)head * HID + j0 + tr) * B + b0 +
                                              8 * tc);
  };
  fetch(0);
  float s = 0.0f;
  for (int b0 = 0; b0 < B; b0 += kSgBatch) {
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 8; ++m) su[tr + 16 * m][tc] = ru[m];
#pragma unroll
    for (int m = 0; m < 4; ++m) *reinterpret_cast<uint4*>(&sv[tr][m][8 * tc]) = rv[m];
    __syncthreads();
    if (b0 + kSgBatch < B) fetch(b0 + kSgBatch);
#pragma unroll 2
    for (int b = 0; b < kSgBatch; b += 8) {
      const uint4 u = *reinterpret_cast<const uint4*>(&sv[nj][src][b]);
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float2 v = __bfloat1622float2(h2[p]);
        s = fmaf(v.x, su[b + 2 * p][col], s);
        s = fmaf(v.y, su[b + 2 * p + 1][col], s);
      }
    }
  }
  float* G = grads + (size_t)head * NPARAM;
  if (q < 4) G[OFF_W4 + q * HID + j] = s;
  else if (q < 10) G[OFF_W1 + j * IN + q - 4] = s;
  else if (q < 13) G[(q == 10 ? OFF_B1 : q == 11 ? OFF_B2 : OFF_B3) + j] = s;
  else if (j < 2 && o4 < OUT) G[OFF_B4 + o4] = s;
}

struct AdamArgs {
  float lr, b1, b2, eps, bc1, bc2;
};
__device__ __forceinline__ float adam(float* params, float* m, float* v, size_t t, float g,
                                      const AdamArgs& a) {
  const float mt = fmaf(1.0f - a.b1, g, __fmul_rn(a.b1, m[t]));
  const float vt = fmaf(__fmul_rn(1.0f - a.b2, g), g, __fmul_rn(a.b2, v[t]));
  m[t] = mt;
  v[t] = vt;
  const float p = params[t] - a.lr * (mt / a.bc1) / (sqrtf(vt / a.bc2) + a.eps);
  params[t] = p;
  return p;
}

// What is done with a head's parameters, 32 x 32 tiles of W2 and W3 per block and the others in
// the last blocks: SUM: the weight gradients' slices summed in slice order into grads; ADAM: the
// update of the FP32 master parameters; CAST: the bf16 copies the kernels use (W1, W4 as they
// are, W2 and W3 also transposed, through shared memory).
struct UpdateArgs {
  float *params, *grads, *m, *v;
  const float* sqerr;  // SUM: the last block of a head also sums its squared errors, B of them
  float* loss;
  int B;
  const float* ws;
  int splits;
  __nv_bfloat16 *w1b, *w2b, *w2tb, *w3b, *w3tb, *w4b;
  AdamArgs adam;
};
constexpr int kUpdTiles = 2 * (HID / 32) * (HID / 32);
constexpr int kUpdSmall = NPARAM - 2 * HID * HID;  // the other parameters of a head
constexpr int kUpdBlocks = kUpdTiles + (kUpdSmall + 1023) / 1024;
template <bool SUM, bool ADAM, bool CAST>
__global__ void __launch_bounds__(256) k_update(UpdateArgs a) {
  __shared__ __nv_bfloat16 tile[32][34];
  const int head = blockIdx.y;
  const size_t base = (size_t)head * NPARAM;
  if (SUM && blockIdx.x == kUpdBlocks) {
    // the head's loss, in a fixed order
    __shared__ float sh[256];
    float s = 0.0f;
    for (int b = threadIdx.x; b < a.B; b += 256) s += a.sqerr[(size_t)head * a.B + b];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
      if ((int)threadIdx.x < k) sh[threadIdx.x] += sh[threadIdx.x + k];
      __syncthreads();
    }
    if (threadIdx.x == 0) a.loss[head] = sh[0] / (float)(a.B * OUT);
    return;
  }
  if ((int)blockIdx.x < kUpdTiles) {
    const int layer = blockIdx.x / (kUpdTiles / 2), k = blockIdx.x % (kUpdTiles / 2);
    const int r0 = (k / (HID / 32)) * 32, c0 = (k % (HID / 32)) * 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const size_t wo = (size_t)head * HID * HID;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = (r0 + w + 8 * q) * HID + c0 + lane;
      const size_t t = base + (layer ? OFF_W3 : OFF_W2) + e;
      float g = 0.0f;
      if (SUM) {
        const float* ws = a.ws + ((size_t)(layer * a.splits) * gridDim.y + head) * HID * HID + e;
        float part[kMaxSplits];
#pragma unroll
        for (int sl = 0; sl < kMaxSplits; ++sl)
          part[sl] = sl < a.splits ? ws[(size_t)sl * gridDim.y * HID * HID] : 0.0f;
        g = part[0];
#pragma unroll
        for (int sl = 1; sl < kMaxSplits; ++sl)
          if (sl < a.splits) g += part[sl];
        a.grads[t] = g;
      }
      const float p = ADAM ? adam(a.params, a.m, a.v, t, g, a.adam) : CAST ? a.params[t] : 0.0f;
      if (CAST) {
        const __nv_bfloat16 h = __float2bfloat16(p);
        (layer ? a.w3b : a.w2b)[wo + e] = h;
        tile[lane][w + 8 * q] = h;
      }
    }
    if (CAST) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; ++q)
        (layer ? a.w3tb : a.w2tb)[wo + (size_t)(c0 + w + 8 * q) * HID + r0 + lane] =
            tile[w + 8 * q][lane];
    }
    return;
  }
  for (int u = 0; u < 4 && (ADAM || CAST); ++u) {
    const int k = ((int)blockIdx.x - kUpdTiles) * 1024 + u * 256 + (int)threadIdx.x;
    if (k >= kUpdSmall) return;
    // the parameters in order, without W2 and W3
    const int off = k < OFF_W2 ? k : k < OFF_W2 + HID ? k + HID * HID : k + 2 * HID * HID;
    const size_t t = base + off;
    const float p =
        ADAM ? adam(a.params, a.m, a.v, t, a.grads[t], a.adam) : CAST ? a.params[t] : 0.0f;
    if (CAST) {
      if (off < OFF_B1) a.w1b[(size_t)head * HID * IN + off] = __float2bfloat16(p);
      if (off >= OFF_W4 && off < OFF_B4)
        a.w4b[(size_t)head * OUT * HID + off - OFF_W4] = __float2bfloat16(p);
    }
  }
}

// C = A . B^T in FP32 (the tensor-core GEMM with a plain store epilogue).
__global__ void __launch_bounds__(128, 1) k_gemm_f32(GemmArgs g, float* C, int ldc,
                                                      long long strideC) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t bar[2];
  __shared__ uint32_t tmem_sh;
  const int warp = threadIdx.x >> 5;
  if (warp == 0) tc::tmem_alloc(&tmem_sh, tc::kTmemCols);
  if (threadIdx.x == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_sh;
  const bool ok = __syncthreads_and(tc::gemm_mainloop(g, smem, bar, tmem, 0, 1));
  if (ok) {
    const int row = tc::tile_m0(g) + threadIdx.x;
    float* c = C + blockIdx.y * strideC + (size_t)row * ldc + tc::tile_n0(g);
    for (int c0 = 0; c0 < g.ntile; c0 += 16) {
      float v[16];
      tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
      for (int q = 0; q < 16; ++q) c[c0 + q] = v[q];
    }
  } else if (threadIdx.x == 0) {
    atomicExch(g.err, 1);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_free(tmem, tc::kTmemCols);
  }
}

bool gemm_shape_ok(int M, int N, int K) {
  return M > 0 && N > 0 && K > 0 && M % tc::kTileM == 0 && N % 16 == 0 && N <= tc::kMaxN &&
         K % tc::kChunkK == 0;
}

}  // namespace

struct sph_mlp {
  int heads = 0, max_batch = 0, device = 0;
  int nsm = 148;  // multiprocessors of the device
  cudaStream_t stream = nullptr;  // cudaStreamLegacy
  std::vector<void*> allocs;
  float *params = nullptr, *grads = nullptr, *m = nullptr, *v = nullptr;
  __nv_bfloat16 *w1b = nullptr, *w2b = nullptr, *w2tb = nullptr, *w3b = nullptr, *w3tb = nullptr,
                *w4b = nullptr;
  // slopes GELU'(z) and the transposed activations and gradients of one batch
  float *g1 = nullptr, *g2 = nullptr, *g3 = nullptr;
  __nv_bfloat16 *h1t = nullptr, *h2t = nullptr, *h3t = nullptr, *dz1t = nullptr, *dz2t = nullptr,
                *dz3t = nullptr;
  float *dout = nullptr, *sqerr = nullptr, *loss = nullptr;
  float* ws = nullptr;  // weight-gradient slices (2 x kMaxSplits x heads x HID x HID)
  int* err = nullptr;
  long long step = 0;
};

namespace {

template <typename T>
bool mlp_alloc(sph_mlp* c, T** p, size_t n) {
  void* q = nullptr;
  if (cudaMalloc(&q, (n ? n : 1) * sizeof(T)) != cudaSuccess) return false;
  cudaMemsetAsync(q, 0, (n ? n : 1) * sizeof(T), c->stream);
  c->allocs.push_back(q);
  *p = static_cast<T*>(q);
  return true;
}

void mlp_free(sph_mlp* c) {
  if (!c) return;
  for (void* p : c->allocs) cudaFree(p);
  delete c;
}

// splitmix64: the initial weights depend only on (seed, head, tensor, index)
double uniform01(uint64_t key) {
  uint64_t z = key + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// PyTorch-style default initialisation of a linear layer: U(-1/sqrt(fan_in), +1/sqrt(fan_in))
// for weights and biases.
void init_params(std::vector<float>& P, int heads, unsigned long long seed) {
  struct T { int off, n, fan_in; };
  const T t[] = {{OFF_W1, HID * IN, IN},   {OFF_B1, HID, IN},   {OFF_W2, HID * HID, HID},
                 {OFF_B2, HID, HID},       {OFF_W3, HID * HID, HID}, {OFF_B3, HID, HID},
                 {OFF_W4, OUT * HID, HID}, {OFF_B4, OUT, HID}};
  for (int h = 0; h < heads; ++h)
    for (int k = 0; k < 8; ++k) {
      const double bound = 1.0 / std::sqrt((double)t[k].fan_in);
      for (int i = 0; i < t[k].n; ++i) {
        const uint64_t key = ((uint64_t)seed * 1000003ull + (uint64_t)h) * 1315423911ull +
                             (uint64_t)(t[k].off + i);
        P[(size_t)h * NPARAM + t[k].off + i] = (float)((2.0 * uniform01(key) - 1.0) * bound);
      }
    }
}

// Rows of the operand per sample: 4 or 2 where all tiles then still run at once.
int net_rep(const sph_mlp* c, int n) {
  const int tiles = n / tc::kTileM * c->heads;
  return 4 * tiles <= c->nsm ? 4 : 2 * tiles <= c->nsm ? 2 : 1;
}

NetArgs net_args(const sph_mlp* c, const float* x, int n) {
  NetArgs a{};
  a.x = x;
  a.params = c->params;
  a.w1b = c->w1b;
  a.w4b = c->w4b;
  a.n = n;
  a.heads = c->heads;
  a.g1 = c->g1;
  a.g2 = c->g2;
  a.g3 = c->g3;
  a.dout = c->dout;
  a.sqerr = c->sqerr;
  a.err = c->err;
  return a;
}

int wgrad_splits(int B) {
  int splits = kMaxSplits;
  while (splits > 1 && B % (tc::kChunkK * splits) != 0) splits /= 2;
  return splits;
}

UpdateArgs update_args(const sph_mlp* c, int splits, int B = 0) {
  UpdateArgs u{};
  u.sqerr = c->sqerr;
  u.loss = c->loss;
  u.B = B;
  u.params = c->params;
  u.grads = c->grads;
  u.m = c->m;
  u.v = c->v;
  u.ws = c->ws;
  u.splits = splits;
  u.w1b = c->w1b;
  u.w2b = c->w2b;
  u.w2tb = c->w2tb;
  u.w3b = c->w3b;
  u.w3tb = c->w3tb;
  u.w4b = c->w4b;
  return u;
}

// Gradients of the mean squared error of every head on B samples, but for the sum of the
// weight gradients' slices (k_update<true, ...>), whose number is returned in *splits.
template <bool TRAIN>
void forward_launch(const sph_mlp* c, const NetArgs& f, int rep) {
  const int grid = std::min(f.n / tc::kTileM * f.heads * rep, c->nsm);
  if (rep == 4) k_forward<TRAIN, 4><<<grid, kNetThreads, kNetSmem, c->stream>>>(f);
  else if (rep == 2) k_forward<TRAIN, 2><<<grid, kNetThreads, kNetSmem, c->stream>>>(f);
  else k_forward<TRAIN, 1><<<grid, kNetThreads, kNetSmem, c->stream>>>(f);
}

int backprop(sph_mlp* c, const float* x, const float* y, int B, int* splits) {
  const int rep = net_rep(c, B), tiles = B / tc::kTileM * c->heads * rep;
  NetArgs f = net_args(c, x, B);
  f.y = y;
  f.wa = c->w2b;
  f.wb = c->w3b;
  f.t1 = c->h1t;
  f.t2 = c->h2t;
  f.t3 = c->h3t;
  forward_launch<true>(c, f, rep);
  if (cudaGetLastError() != cudaSuccess) return 1;
  NetArgs r = net_args(c, x, B);
  r.wa = c->w3tb;
  r.wb = c->w2tb;
  r.t1 = c->dz1t;
  r.t2 = c->dz2t;
  r.t3 = c->dz3t;
  if (rep == 4) k_backward<4><<<tiles, kNetThreads, kNetSmem, c->stream>>>(r);
  else if (rep == 2) k_backward<2><<<tiles, kNetThreads, kNetSmem, c->stream>>>(r);
  else k_backward<1><<<tiles, kNetThreads, kNetSmem, c->stream>>>(r);
  if (cudaGetLastError() != cudaSuccess) return 1;
  // dW2 = dz2^T h1, dW3 = dz3^T h2
  WgradArgs w{};
  w.dz[0] = c->dz2t;
  w.h[0] = c->h1t;
  w.dz[1] = c->dz3t;
  w.h[1] = c->h2t;
  w.ws = c->ws;
  w.B = B;
  w.splits = *splits = wgrad_splits(B);
  w.err = c->err;
  k_wgrad<<<dim3(HID / tc::kTileM, c->heads, 2 * w.splits), 128, kWgradSmem, c->stream>>>(w);
  if (cudaGetLastError() != cudaSuccess) return 1;
  k_small_grads<<<dim3(HID / kSgNeurons, c->heads), 256, 0, c->stream>>>(
      c->dout, c->h3t, c->dz1t, c->dz2t, c->dz3t, x, B, c->grads);
  return cudaGetLastError() != cudaSuccess;
}

int cast_weights(sph_mlp* c) {
  k_update<false, false, true><<<dim3(kUpdBlocks, c->heads), 256, 0, c->stream>>>(update_args(c, 1));
  return cudaGetLastError() != cudaSuccess;
}

sph_status finish(sph_mlp* c) {
  int e = 0;
  if (cudaMemcpyAsync(&e, c->err, sizeof(int), cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
      cudaStreamSynchronize(c->stream) != cudaSuccess)
    return SPH_ERR_CUDA;
  return e ? SPH_ERR_TIMEOUT : SPH_OK;
}

bool batch_ok(const sph_mlp* c, int B) { return B > 0 && B % tc::kTileM == 0 && B <= c->max_batch; }

}  // namespace

extern "C" {

sph_status sph_tc_gemm(const void* A, const void* B, float* C, int M, int N, int K, int heads,
                       void* stream) {
  if (!A || !B || !C || heads <= 0 || !gemm_shape_ok(M, N, K)) return SPH_ERR_STATE;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(k_gemm_f32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             tc::kSmemBytes) != cudaSuccess)
      return SPH_ERR_CUDA;
    attr_set = true;
  }
  int* err = nullptr;
  if (cudaMalloc(&err, sizeof(int)) != cudaSuccess) return SPH_ERR_NOMEM;
  cudaStream_t st = (cudaStream_t)stream;
  cudaMemsetAsync(err, 0, sizeof(int), st);
  GemmArgs g;
  g.A = static_cast<const __nv_bfloat16*>(A);
  g.B = static_cast<const __nv_bfloat16*>(B);
  g.strideA = (long long)M * K;
  g.strideB = (long long)N * K;
  g.lda = K;
  g.ldb = K;
  g.M = M;
  g.N = N;
  g.K = K;
  g.ntile = N;
  g.err = err;
  k_gemm_f32<<<dim3(M / tc::kTileM, heads), 128, tc::kSmemBytes, st>>>(g, C, N, (long long)M * N);
  int h = 0;
  sph_status s = SPH_OK;
  if (cudaGetLastError() != cudaSuccess ||
      cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    s = SPH_ERR_CUDA;
  else if (h)
    s = SPH_ERR_TIMEOUT;
  cudaFree(err);
  return s;
}

int sph_mlp_num_params(void) { return NPARAM; }

sph_status sph_mlp_create(int heads, int max_batch, unsigned long long seed, int device,
                          sph_mlp** out) {
  if (!out || heads <= 0 || max_batch <= 0 || max_batch % tc::kTileM != 0) return SPH_ERR_STATE;
  *out = nullptr;
  if (cudaSetDevice(device) != cudaSuccess) return SPH_ERR_CUDA;
  sph_mlp* c = new sph_mlp;
  c->heads = heads;
  c->max_batch = max_batch;
  c->device = device;
  cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, device);
  // the legacy default stream: the caller's inputs (batches made by default-stream work,
  // e.g. a framework's allocator) are then ordered before, and their reuse after, the
  // network's kernels
  c->stream = cudaStreamLegacy;
  const size_t np = (size_t)heads * NPARAM, hh = (size_t)heads * HID * HID;
  const size_t act = (size_t)heads * max_batch * HID;
  bool ok = mlp_alloc(c, &c->params, np) && mlp_alloc(c, &c->grads, np) && mlp_alloc(c, &c->m, np) &&
            mlp_alloc(c, &c->v, np);
  ok = ok && mlp_alloc(c, &c->w1b, (size_t)heads * HID * IN) && mlp_alloc(c, &c->w2b, hh) &&
       mlp_alloc(c, &c->w2tb, hh) && mlp_alloc(c, &c->w3b, hh) && mlp_alloc(c, &c->w3tb, hh) &&
       mlp_alloc(c, &c->w4b, (size_t)heads * OUT * HID);
  for (float** p : {&c->g1, &c->g2, &c->g3}) ok = ok && mlp_alloc(c, p, act);
  for (__nv_bfloat16** p : {&c->h1t, &c->h2t, &c->h3t, &c->dz1t, &c->dz2t, &c->dz3t})
    ok = ok && mlp_alloc(c, p, act);
  ok = ok && mlp_alloc(c, &c->dout, (size_t)heads * max_batch * OUT) &&
       mlp_alloc(c, &c->sqerr, (size_t)heads * max_batch) && mlp_alloc(c, &c->loss, heads) &&
       mlp_alloc(c, &c->ws, 2 * (size_t)kMaxSplits * hh) && mlp_alloc(c, &c->err, 1);
  if (!ok) {
    mlp_free(c);
    return SPH_ERR_NOMEM;
  }
  const std::pair<const void*, int> kernels[] = {
      {(const void*)k_forward<false, 1>, kNetSmem}, {(const void*)k_forward<false, 2>, kNetSmem},
      {(const void*)k_forward<false, 4>, kNetSmem}, {(const void*)k_forward<true, 1>, kNetSmem},
      {(const void*)k_forward<true, 2>, kNetSmem},  {(const void*)k_forward<true, 4>, kNetSmem},
      {(const void*)k_backward<1>, kNetSmem},       {(const void*)k_backward<2>, kNetSmem},
      {(const void*)k_backward<4>, kNetSmem},       {(const void*)k_wgrad, kWgradSmem}};
  for (const auto& k : kernels)
    if (cudaFuncSetAttribute(k.first, cudaFuncAttributeMaxDynamicSharedMemorySize, k.second) !=
        cudaSuccess) {
      mlp_free(c);
      return SPH_ERR_CUDA;
    }
  std::vector<float> P(np);
  init_params(P, heads, seed);
  if (cudaMemcpyAsync(c->params, P.data(), np * sizeof(float), cudaMemcpyHostToDevice, c->stream) !=
          cudaSuccess ||
      cast_weights(c) || cudaStreamSynchronize(c->stream) != cudaSuccess) {
    mlp_free(c);
    return SPH_ERR_CUDA;
  }
  *out = c;
  return SPH_OK;
}

void sph_mlp_destroy(sph_mlp* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  cudaStreamSynchronize(c->stream);
  mlp_free(c);
}

sph_status sph_mlp_get_params(sph_mlp* c, float* host) {
  if (!c || !host) return SPH_ERR_STATE;
  cudaSetDevice(c->device);
  if (cudaMemcpyAsync(host, c->params, (size_t)c->heads * NPARAM * sizeof(float),
                      cudaMemcpyDeviceToHost, c->stream) != cudaSuccess)
    return SPH_ERR_CUDA;
  return finish(c);
}

sph_status sph_mlp_set_params(sph_mlp* c, const float* host) {
  if (!c || !host) return SPH_ERR_STATE;
  cudaSetDevice(c->device);
  if (cudaMemcpyAsync(c->params, host, (size_t)c->heads * NPARAM * sizeof(float),
                      cudaMemcpyHostToDevice, c->stream) != cudaSuccess ||
      cast_weights(c))
    return SPH_ERR_CUDA;
  return finish(c);
}

sph_status sph_mlp_gradients(sph_mlp* c, const float* x, const float* y, int batch,
                             float* grads_host, float* loss_host) {
  if (!c || !x || !y || !batch_ok(c, batch)) return SPH_ERR_STATE;
  cudaSetDevice(c->device);
  int splits = 1;
  if (backprop(c, x, y, batch, &splits)) return SPH_ERR_CUDA;
  k_update<true, false, false><<<dim3(kUpdBlocks + 1, c->heads), 256, 0, c->stream>>>(
      update_args(c, splits, batch));
  if (cudaGetLastError() != cudaSuccess) return SPH_ERR_CUDA;
  if (grads_host && cudaMemcpyAsync(grads_host, c->grads, (size_t)c->heads * NPARAM * sizeof(float),
                                    cudaMemcpyDeviceToHost, c->stream) != cudaSuccess)
    return SPH_ERR_CUDA;
  if (loss_host && cudaMemcpyAsync(loss_host, c->loss, (size_t)c->heads * sizeof(float),
                                   cudaMemcpyDeviceToHost, c->stream) != cudaSuccess)
    return SPH_ERR_CUDA;
  return finish(c);
}

sph_status sph_mlp_train_step(sph_mlp* c, const float* x, const float* y, int batch, float lr,
                              float* loss_host) {
  if (!c || !x || !y || !batch_ok(c, batch)) return SPH_ERR_STATE;
  cudaSetDevice(c->device);
  int splits = 1;
  if (backprop(c, x, y, batch, &splits)) return SPH_ERR_CUDA;
  c->step++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float bc1 = 1.0f - (float)std::pow((double)b1, (double)c->step);
  const float bc2 = 1.0f - (float)std::pow((double)b2, (double)c->step);
  UpdateArgs u = update_args(c, splits, batch);
  u.adam = {lr, b1, b2, 1e-8f, bc1, bc2};
  k_update<true, true, true><<<dim3(kUpdBlocks + 1, c->heads), 256, 0, c->stream>>>(u);
  if (cudaGetLastError() != cudaSuccess) return SPH_ERR_CUDA;
  if (loss_host && cudaMemcpyAsync(loss_host, c->loss, (size_t)c->heads * sizeof(float),
                                   cudaMemcpyDeviceToHost, c->stream) != cudaSuccess)
    return SPH_ERR_CUDA;
  if (!loss_host) return SPH_OK;  // asynchronous: errors surface at the next synchronising call
  return finish(c);
}

sph_status sph_mlp_predict(sph_mlp* c, const float* x, int n, float* out) {
  if (!c || !x || !out || n <= 0 || n % tc::kTileM != 0) return SPH_ERR_STATE;
  cudaSetDevice(c->device);
  NetArgs f = net_args(c, x, n);
  f.wa = c->w2b;
  f.wb = c->w3b;
  f.out = out;
  forward_launch<false>(c, f, net_rep(c, n));
  if (cudaGetLastError() != cudaSuccess) return SPH_ERR_CUDA;
  return finish(c);
}

sph_status sph_mlp_synchronize(sph_mlp* c) {
  if (!c) return SPH_ERR_STATE;
  cudaSetDevice(c->device);
  return finish(c);
}

}  // extern "C"
