// Row kernels of the FP8 linear path for sm_100a: the per-token e4m3 quantiser and the
// consumers of raw GEMM accumulators.  One group of TPR threads owns one row and keeps it in
// registers, so each element is read once and written once; loads are 128-bit, codes are
// stored 8 at a time.  All of them are HBM-bound: bytes per row are in the comments.
#include <cuda_runtime.h>

#include <type_traits>

#include "../../include/iflb200.h"
#include "launch.cuh"
#include "row_stream.cuh"
#include "rowmath.cuh"

// The file compiles as one translation unit, or as three (IFLB200_ROW_PART = 0, 1, 2) so that
// the build can run them in parallel: 0 = row_quant + dequant_rows, 1 = gated_act_quant + the
// per-tensor pack, 2 = residual_norm_quant.
#ifndef IFLB200_ROW_PART
#define IFLB200_ROW_PART -1
#endif

namespace iflb200 {

// One thread waits for the kernel before this one in the stream, the others park at the CTA
// barrier: a CTA that became resident early costs the still-running kernel next to it nothing.
__device__ __forceinline__ void row_dependency_wait() {
  if (threadIdx.x == 0) grid_dependency_wait();
  __syncthreads();
}

// Row kernels let the next kernel in the stream be scheduled as soon as their last CTAs start -- before
// their own dependency wait where the caller says so (early_trigger_for).
__device__ __forceinline__ void row_trigger() { grid_launch_dependents(); }
__device__ __forceinline__ void row_begin(int early) {
  if (early) row_trigger();
  row_dependency_wait();
  if (!early) row_trigger();
}
// The same in two parts, for kernels that have work for the time before the wait.
__device__ __forceinline__ void row_open(int early) {
  if (early) row_trigger();
}
__device__ __forceinline__ void row_enter(int early) {
  row_dependency_wait();
  if (!early) row_trigger();
}

// Holds a value in a register from here on: what a launch of a few microseconds computes from its arguments (whose first
// reads miss the constant cache) is done when the kernel before it ends, and not between the wait and the first load
// (18 expert layers 352 -> 344 us; 50 x 4096 gated on one buffer 1.90 -> 1.74 behind one another, 350 sizes 0.97 of the time).
// Not in instantiations that have no registers to spare: float32 rows with scales (row_quant_kernel: 16 x 5120 2.68 -> 2.87 us with
// them), eight planes with every operand (residual_norm_planes_kernel).
template <typename T>
__device__ __forceinline__ void keep(T*& p) {
  asm volatile("" : "+l"(p));
}
__device__ __forceinline__ void keep(int& v) { asm volatile("" : "+r"(v)); }

// CTAs have 256 threads.  A row is owned by a group of TPR threads, each holding IT chunks of 8
// elements: narrow rows share a CTA (TPR = 32 / 64 / 128, one chunk per thread), wide rows take
// the whole CTA with 1, 2, 4 or 8 chunks per thread (up to 16384 columns).  Measured on B200,
// 256-thread groups beat wider ones at every size: the two or three block-wide synchronisations
// per row are hidden by the other CTAs resident on the SM, not by more threads per row.
constexpr int kRowThreads = 256;
constexpr int kMaxWidth = kRowThreads * 8 * 8;  // 16384 columns

// --------------------------------------------------------------------------------------------
// Chunks of 8 elements.  FAST kernels are launched when every buffer obeys the 16-byte rule and
// the row width is a multiple of 8: every access is one or two 128-bit instructions and a chunk
// is either wholly inside the row or wholly outside, so there is no per-element masking.  The
// other instantiation is fully element-wise (any alignment, any width).
// --------------------------------------------------------------------------------------------
template <typename T>
struct Raw8 {  // eight elements as they sit in memory
  uint4 u;
};
template <>
struct Raw8<float> {
  float4 a, b;
};
template <typename T>
__device__ __forceinline__ Raw8<T> raw_zero() {
  Raw8<T> r;
  r.u = make_uint4(0u, 0u, 0u, 0u);
  return r;
}
template <>
__device__ __forceinline__ Raw8<float> raw_zero<float>() {
  Raw8<float> r;
  r.a = make_float4(0.f, 0.f, 0.f, 0.f);
  r.b = r.a;
  return r;
}
template <typename T>
__device__ __forceinline__ Raw8<T> raw_load(const T* p) {
  Raw8<T> r;
  r.u = *reinterpret_cast<const uint4*>(p);
  return r;
}
template <>
__device__ __forceinline__ Raw8<float> raw_load<float>(const float* p) {
  Raw8<float> r;
  r.a = *reinterpret_cast<const float4*>(p);
  r.b = *reinterpret_cast<const float4*>(p + 4);
  return r;
}
template <typename T>
__device__ __forceinline__ Raw8<T> raw_gather(const T* row_ptr, int c0, int width) {
  uint32_t w[4] = {0u, 0u, 0u, 0u};
  const uint16_t* p = reinterpret_cast<const uint16_t*>(row_ptr);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (c0 + i < width) w[i >> 1] |= (uint32_t)p[c0 + i] << (16 * (i & 1));
  Raw8<T> r;
  r.u = make_uint4(w[0], w[1], w[2], w[3]);
  return r;
}
template <>
__device__ __forceinline__ Raw8<float> raw_gather<float>(const float* row_ptr, int c0, int width) {
  float f[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = (c0 + i < width) ? row_ptr[c0 + i] : 0.0f;
  Raw8<float> r;
  r.a = make_float4(f[0], f[1], f[2], f[3]);
  r.b = make_float4(f[4], f[5], f[6], f[7]);
  return r;
}
// All loads of a row are issued through this before the first value is used, so a thread has
// every chunk in flight at once.  `on`: the chunk belongs to a live row and starts inside it.
template <bool FAST, typename T>
__device__ __forceinline__ Raw8<T> fetch(const T* row_ptr, int c0, int width, bool on) {
  if (!on) return raw_zero<T>();
  if (FAST) return raw_load<T>(row_ptr + c0);
  return raw_gather<T>(row_ptr, c0, width);
}
__device__ __forceinline__ void unpack(const Raw8<__nv_bfloat16>& r, float (&o)[8]) {
  const uint32_t w[4] = {r.u.x, r.u.y, r.u.z, r.u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    o[2 * i] = __uint_as_float(w[i] << 16);
    o[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}
__device__ __forceinline__ void unpack(const Raw8<__half>& r, float (&o)[8]) {
  const uint32_t w[4] = {r.u.x, r.u.y, r.u.z, r.u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    o[2 * i] = f.x;
    o[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void unpack(const Raw8<float>& r, float (&o)[8]) {
  o[0] = r.a.x; o[1] = r.a.y; o[2] = r.a.z; o[3] = r.a.w;
  o[4] = r.b.x; o[5] = r.b.y; o[6] = r.b.z; o[7] = r.b.w;
}
// Two elements of a 16-bit type as a packed pair.
__device__ __forceinline__ uint64_t widen2(uint32_t w, __nv_bfloat16) {
  return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}
__device__ __forceinline__ uint64_t widen2(uint32_t w, __half) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  return pack2(f.x, f.y);
}
// float32 vector operand (scales, bias, gates, norm weights) for one chunk.
template <bool FAST>
__device__ __forceinline__ void load_f32(const float* p, int c0, int width, float (&o)[8]) {
  if (FAST) {
    unpack(raw_load<float>(p + c0), o);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = (c0 + i < width) ? p[c0 + i] : 0.0f;
  }
}
// Zero the elements of a chunk that lie beyond the row end (element-wise kernels only).
template <bool FAST>
__device__ __forceinline__ void mask_tail(float (&v)[8], int c0, int width) {
  if (!FAST) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (c0 + i < width) ? v[i] : 0.0f;
  }
}
template <bool FAST>
__device__ __forceinline__ void store_codes(uint8_t* row_ptr, int c0, int width, const float (&v)[8], float inv) {
  float s[8];
  const uint64_t inv2 = pack2(inv, inv);
#pragma unroll
  for (int i = 0; i < 8; i += 2) unpack2(mul2(pack2(v[i], v[i + 1]), inv2), s[i], s[i + 1]);
  const uint32_t lo = cvt_e4m3x4(s[0], s[1], s[2], s[3]);
  const uint32_t hi = cvt_e4m3x4(s[4], s[5], s[6], s[7]);
  if (FAST) {
    *reinterpret_cast<uint2*>(row_ptr + c0) = make_uint2(lo, hi);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c0 + i < width) row_ptr[c0 + i] = (uint8_t)(((i < 4 ? lo : hi) >> (8 * (i & 3))) & 0xFF);
  }
}
template <bool FAST>
__device__ __forceinline__ void store_out(void* base, int dtype, int64_t row_off, int c0, int width,
                                          const float (&v)[8]) {
  if (dtype == IFLB200_F32) {
    float* o = reinterpret_cast<float*>(base) + row_off + c0;
    if (FAST) {
      *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
      *reinterpret_cast<float4*>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c0 + i < width) o[i] = v[i];
    }
    return;
  }
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    w[i] = (dtype == IFLB200_BF16) ? (f32_to_bf16_bits(v[2 * i]) | (f32_to_bf16_bits(v[2 * i + 1]) << 16))
                                   : (f32_to_f16_bits(v[2 * i]) | (f32_to_f16_bits(v[2 * i + 1]) << 16));
  uint16_t* o = reinterpret_cast<uint16_t*>(base) + row_off + c0;
  if (FAST) {
    *reinterpret_cast<uint4*>(o) = make_uint4(w[0], w[1], w[2], w[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c0 + i < width) o[i] = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
  }
}
template <typename T>
__host__ __device__ constexpr int dtype_of();
template <>
__host__ __device__ constexpr int dtype_of<float>() { return IFLB200_F32; }
template <>
__host__ __device__ constexpr int dtype_of<__nv_bfloat16>() { return IFLB200_BF16; }
template <>
__host__ __device__ constexpr int dtype_of<__half>() { return IFLB200_F16; }

// --------------------------------------------------------------------------------------------
// Reductions over the TPR threads of one row (TPR a multiple of 32; rows never share a warp).
// `slot` is a per-reduction shared array of kRowThreads/32 floats.
// --------------------------------------------------------------------------------------------
template <int TPR, bool IS_MAX>
__device__ __forceinline__ float row_reduce(float v, float* slot) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float other = __shfl_xor_sync(0xFFFFFFFFu, v, o);
    v = IS_MAX ? max_f32(v, other) : __fadd_rn(v, other);
  }
  if (TPR > 32) {
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) slot[warp] = v;
    __syncthreads();
    constexpr int WPR = TPR / 32;
    const int first = (warp / WPR) * WPR;
    float r = slot[first];
#pragma unroll
    for (int i = 1; i < WPR; ++i) r = IS_MAX ? max_f32(r, slot[first + i]) : __fadd_rn(r, slot[first + i]);
    v = r;
  }
  return v;
}

// Resident CTAs per SM the compiler must leave room for (register cap): the block-wide
// synchronisations of one row are hidden by the other CTAs on the SM.
template <int IT>
__host__ __device__ constexpr int row_min_blocks() {
  return IT <= 2 ? 3 : 2;
}
// residual_norm_quant: three CTAs per SM for up to three chunks per thread (85 registers; capping
// at 64 for a fourth CTA spills and was measured slower: 7.7 against 4.9 us at 816 x 2048).
template <int IT>
__host__ __device__ constexpr int resnorm_min_blocks() {
  return IT <= 3 ? 3 : 2;
}

// --------------------------------------------------------------------------------------------
// row_quant: 2K (bf16 in) + K (codes out) + 4 bytes per row.
// --------------------------------------------------------------------------------------------
constexpr int kMaxMirrors = 7;  // copies of a result in the buffers of the other GPUs of a group of up to eight

struct RowQuantArgs {
  int early;  // see row_begin
  const void* x;
  int64_t ld_x;
  int M, K, iters;
  const float* row;
  const float* col;
  const float* bias;
  int gelu;
  uint8_t* q;
  int64_t ld_q;
  float* qs;
  // Column-sharded rows (tensor parallel): phase 1 writes the shard's row maximum to `amax` and
  // stops; phase 2 takes the row maximum from `amax` (after an all-reduce-max over the shards)
  // instead of its own, so the codes equal those of the unsharded row.  0: one pass.  Phase 3 is
  // phase 2 that also leaves amax[m] at zero (the maxima came from a GEMM epilogue's atomicMax,
  // which needs the words to start at zero the next time).
  int phase;
  float* amax;
  // phase 1 only: further copies of the row maxima (the other GPUs' slots for this rank, peer-mapped)
  float* amax_mirror[kMaxMirrors];
  int mirrors;
};

__device__ __forceinline__ void write_row_max(const RowQuantArgs& a, int m, float amax) {
  a.amax[m] = amax;
#pragma unroll
  for (int k = 0; k < kMaxMirrors; ++k)
    if (k < a.mirrors) a.amax_mirror[k][m] = amax;
}

// PLAIN: no prologue.  The row then stays in registers as loaded (4 registers per 8 elements)
// and is widened twice, once for the maximum and once for the cast, which keeps enough CTAs
// resident to cover the HBM latency.
template <typename XT, int TPR, int IT, bool PLAIN, bool FAST>
__global__ void __launch_bounds__(kRowThreads, PLAIN ? (IT <= 2 ? 4 : 3) : row_min_blocks<IT>())
row_quant_kernel(const RowQuantArgs a) {
  row_open(a.early);
  __shared__ float red[kRowThreads / 32];
  const int t = threadIdx.x % TPR;
  const int m = blockIdx.x * (kRowThreads / TPR) + threadIdx.x / TPR;
  const bool live = m < a.M;
  const XT* xr = reinterpret_cast<const XT*>(a.x) + (live ? (int64_t)m * a.ld_x : 0);
  int K = a.K;
  uint8_t* qr = a.q + (live ? (int64_t)m * a.ld_q : 0);
  float* qs = a.qs + (live ? m : 0);
  if (PLAIN || sizeof(XT) == 2) { keep(K); keep(xr); keep(qr); keep(qs); }
  row_enter(a.early);  // inputs may come from the kernel before this one in the stream
  const float rs = (live && a.row) ? a.row[m] : 1.0f;

  Raw8<XT> raw[IT];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c0 = (it * TPR + t) * 8;
    raw[it] = fetch<FAST, XT>(xr, c0, K, it < a.iters && live && c0 < K);
  }
  float amax = 0.0f;
  if (PLAIN) {
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      float w[8];
      unpack(raw[it], w);
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = max_f32(amax, fabsf(w[i]));
    }
    amax = row_reduce<TPR, true>(amax, red);
    if (a.phase == 1) {
      if (live && t == 0) write_row_max(a, m, amax);
      return;
    }
    if (a.phase >= 2 && live) amax = a.amax[m];
    if (a.phase == 3) {  // every thread of the row has its copy: leave the word at zero for the next producer
      __syncthreads();
      if (live && t == 0) a.amax[m] = 0.0f;
    }
    float scale, inv;
    quant_scales(amax, scale, inv);
    if (!live) return;
    if (t == 0) *qs = scale;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int c0 = (it * TPR + t) * 8;
      if (it < a.iters && c0 < K) {
        float w[8];
        unpack(raw[it], w);
        store_codes<FAST>(qr, c0, K, w, inv);
      }
    }
    return;
  }
  float v[IT][8];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c0 = (it * TPR + t) * 8;
    unpack(raw[it], v[it]);
    if (it < a.iters && live && c0 < a.K) {
      float cs[8], bs[8];
      if (a.col) load_f32<FAST>(a.col, c0, a.K, cs);
      if (a.bias) load_f32<FAST>(a.bias, c0, a.K, bs);
      Chain8 ch(v[it]);
      if (a.row) ch.mul(rs);
      if (a.col) ch.mul(cs);
      if (a.bias) ch.add(bs);
      ch.done(v[it]);
      if (a.gelu) {
#pragma unroll
        for (int i = 0; i < 8; i += 2) gelu_tanh_ref2(v[it][i], v[it][i + 1]);
      }
      mask_tail<FAST>(v[it], c0, a.K);
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = max_f32(amax, fabsf(v[it][i]));
    }
  }
  amax = row_reduce<TPR, true>(amax, red);
  if (a.phase == 1) {
    if (live && t == 0) write_row_max(a, m, amax);
    return;
  }
  if (a.phase >= 2 && live) amax = a.amax[m];
  if (a.phase == 3) {
    __syncthreads();
    if (live && t == 0) a.amax[m] = 0.0f;
  }
  float scale, inv;
  quant_scales(amax, scale, inv);
  if (!live) return;
  if (t == 0) *qs = scale;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c0 = (it * TPR + t) * 8;
    if (it < a.iters && c0 < a.K) store_codes<FAST>(qr, c0, a.K, v[it], inv);
  }
}

// --------------------------------------------------------------------------------------------
// gated_act_quant: 4F (bf16 g,u in) + F (codes out) + 4 bytes per row.  Bound by instruction
// issue, not by HBM: ~40 instructions per element (the reference's ex2.approx / div.full chains).
// --------------------------------------------------------------------------------------------
struct GatedArgs {
  int early;  // see row_begin
  const void* gu;
  int64_t ld_gu;
  int M, F, iters;
  const float* row;
  const float* col;
  int act;
  uint8_t* q;
  int64_t ld_q;
  float* qs;
};

template <typename XT, int TPR, int IT, bool FAST>
__global__ void __launch_bounds__(kRowThreads, row_min_blocks<IT>())
gated_act_quant_kernel(const GatedArgs a) {
  row_begin(a.early);  // inputs may come from the kernel before this one in the stream
  __shared__ float red[kRowThreads / 32];
  const int t = threadIdx.x % TPR;
  const int m = blockIdx.x * (kRowThreads / TPR) + threadIdx.x / TPR;
  const bool live = m < a.M;
  const XT* gr = reinterpret_cast<const XT*>(a.gu) + (live ? (int64_t)m * a.ld_gu : 0);
  const XT* ur = gr + a.F;
  const float rs = (live && a.row) ? a.row[m] : 1.0f;

  Raw8<XT> rg[IT], ru[IT];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c0 = (it * TPR + t) * 8;
    const bool on = it < a.iters && live && c0 < a.F;
    rg[it] = fetch<FAST, XT>(gr, c0, a.F, on);
    ru[it] = fetch<FAST, XT>(ur, c0, a.F, on);
  }
  float h[IT][8];
  float amax = 0.0f;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c0 = (it * TPR + t) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) h[it][i] = 0.0f;
    if (it < a.iters && live && c0 < a.F) {
      float g[8], u[8];
      unpack(rg[it], g);
      unpack(ru[it], u);
      if (a.row) {
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          const uint64_t rs2 = pack2(rs, rs);
          unpack2(mul2(pack2(g[i], g[i + 1]), rs2), g[i], g[i + 1]);
          unpack2(mul2(pack2(u[i], u[i + 1]), rs2), u[i], u[i + 1]);
        }
      }
      if (a.col) {
        float cg[8], cu[8];
        load_f32<FAST>(a.col, c0, a.F, cg);
        load_f32<FAST>(a.col + a.F, c0, a.F, cu);
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          unpack2(mul2(pack2(g[i], g[i + 1]), pack2(cg[i], cg[i + 1])), g[i], g[i + 1]);
          unpack2(mul2(pack2(u[i], u[i + 1]), pack2(cu[i], cu[i + 1])), u[i], u[i + 1]);
        }
      }
      if (a.act == IFLB200_ACT_GELU_TANH) {
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          gelu_tanh_ref2(g[i], g[i + 1]);
          unpack2(mul2(pack2(u[i], u[i + 1]), pack2(g[i], g[i + 1])), h[it][i], h[it][i + 1]);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) h[it][i] = __fmul_rn(u[i], silu_ref(g[i]));
      }
      mask_tail<FAST>(h[it], c0, a.F);
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = max_f32(amax, fabsf(h[it][i]));
    }
  }
  amax = row_reduce<TPR, true>(amax, red);
  float scale, inv;
  quant_scales(amax, scale, inv);
  if (!live) return;
  if (t == 0) a.qs[m] = scale;
  uint8_t* qr = a.q + (int64_t)m * a.ld_q;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c0 = (it * TPR + t) * 8;
    if (it < a.iters && c0 < a.F) store_codes<FAST>(qr, c0, a.F, h[it], inv);
  }
}

// The same for few rows (a skinny decoder layer: 50 x 4096): no bytes to speak of, a launch is round trips to L2 and the
// instructions of one row, fetched cold.  So a row has a thread for every four columns (eight, sixteen beyond 4096, 8192), every
// load -- gate, up, their column scales, the row scale -- is issued before the first use, and the code is one
// activation's: 50 x 4096 2.48 -> 1.91 us behind one another, 18 expert layers 418 -> 403; over 50 sizes and both
// activations 0.79 of the time.  Two or four CTAs a row as a cluster took 0.4 us longer than one.
constexpr int kGatedFewThreads = 1024;

template <typename XT, int ACT, int Q>
__global__ void __launch_bounds__(kGatedFewThreads) gated_act_quant_few_kernel(const GatedArgs a) {
  row_open(a.early);
  __shared__ float red[kGatedFewThreads / 32];
  const int m = blockIdx.x, step = blockDim.x * 4, c0 = threadIdx.x * 4;
  int F = a.F;
  const XT* gr = reinterpret_cast<const XT*>(a.gu) + (int64_t)m * a.ld_gu + c0;
  const XT* ur = gr + F;
  const float *col = a.col ? a.col + c0 : nullptr, *row = a.row ? a.row + m : nullptr;
  uint8_t* q = a.q + (int64_t)m * a.ld_q + c0;
  float* qs = a.qs + m;
  keep(F); keep(gr); keep(ur); keep(col); keep(row); keep(q); keep(qs);
  row_enter(a.early);  // inputs may come from the kernel before this one in the stream
  uint2 rg[Q], ru[Q];
  float4 cg[Q], cu[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    cg[i] = cu[i] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);  // an absent scale is a factor of 1
    rg[i] = ru[i] = make_uint2(0u, 0u);
    if (c0 + i * step < F) {
      rg[i] = *reinterpret_cast<const uint2*>(gr + i * step);
      ru[i] = *reinterpret_cast<const uint2*>(ur + i * step);
      if (col) {
        cg[i] = *reinterpret_cast<const float4*>(col + i * step);
        cu[i] = *reinterpret_cast<const float4*>(col + F + i * step);
      }
    }
  }
  const float rs = row ? *row : 1.0f;
  const uint64_t rs2 = pack2(rs, rs);
  float h[Q][4], amax = 0.0f;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    uint64_t g[2] = {widen2(rg[i].x, XT()), widen2(rg[i].y, XT())}, u[2] = {widen2(ru[i].x, XT()), widen2(ru[i].y, XT())};
    g[0] = mul2(mul2(g[0], rs2), pack2(cg[i].x, cg[i].y));
    g[1] = mul2(mul2(g[1], rs2), pack2(cg[i].z, cg[i].w));
    u[0] = mul2(mul2(u[0], rs2), pack2(cu[i].x, cu[i].y));
    u[1] = mul2(mul2(u[1], rs2), pack2(cu[i].z, cu[i].w));
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (ACT == IFLB200_ACT_GELU_TANH) {
        g[j] = gelu_tanh_ref2(g[j]);
      } else {
        float x, y;
        unpack2(g[j], x, y);
        g[j] = pack2(silu_ref(x), silu_ref(y));
      }
      unpack2(mul2(u[j], g[j]), h[i][2 * j], h[i][2 * j + 1]);
    }
    if (c0 + i * step < F) amax = max_abs_f32(max_abs_f32(amax, h[i][0], h[i][1]), h[i][2], h[i][3]);
  }
  amax = warp_max_abs_f32(amax);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = warp_max_abs_f32((threadIdx.x & 31) < blockDim.x / 32 ? red[threadIdx.x & 31] : 0.0f);
  float scale, inv;
  quant_scales(amax, scale, inv);
  if (threadIdx.x == 0) *qs = scale;
#pragma unroll
  for (int i = 0; i < Q; ++i)
    if (c0 + i * step < F)
      *reinterpret_cast<uint32_t*>(q + i * step) =
          cvt_e4m3x4(__fmul_rn(h[i][0], inv), __fmul_rn(h[i][1], inv), __fmul_rn(h[i][2], inv), __fmul_rn(h[i][3], inv));
}

// --------------------------------------------------------------------------------------------
// dequant_rows: 2D in + out bytes per row; flat, one chunk per thread.
// --------------------------------------------------------------------------------------------
struct DequantArgs {
  const void* x;
  int64_t ld_x;
  int M, D;
  const float* row;
  const float* col;
  const float* bias;
  void* y;
  int y_dtype;
  int64_t ld_y;
};

template <typename XT, bool FAST>
__global__ void __launch_bounds__(256) dequant_rows_kernel(const DequantArgs a) {
  row_dependency_wait();  // inputs may come from the kernel before this one in the stream
  row_trigger();
  const int m = blockIdx.y;
  const int c0 = (blockIdx.x * 256 + threadIdx.x) * 8;
  if (c0 >= a.D) return;
  const XT* xr = reinterpret_cast<const XT*>(a.x) + (int64_t)m * a.ld_x;
  float v[8], cs[8], bs[8];
  unpack(fetch<FAST, XT>(xr, c0, a.D, true), v);
  if (a.col) load_f32<FAST>(a.col, c0, a.D, cs);
  if (a.bias) load_f32<FAST>(a.bias, c0, a.D, bs);
  const float rs = a.row ? a.row[m] : 1.0f;
  Chain8 ch(v);
  if (a.row) ch.mul(rs);
  if (a.col) ch.mul(cs);
  if (a.bias) ch.add(bs);
  ch.done(v);
  store_out<FAST>(a.y, a.y_dtype, (int64_t)m * a.ld_y, c0, a.D, v);
}

// --------------------------------------------------------------------------------------------
// residual_norm_quant: (f32 residual) 2D delta + 4D res in, 4D res + D codes out, + 4 bytes.
// --------------------------------------------------------------------------------------------
struct ResNormArgs {
  int early;  // see row_begin
  void* res;
  int64_t ld_res;
  int M, D, iters;
  const __nv_bfloat16* delta;
  int64_t ld_delta;
  // the delta as fp32 partial sums of a K-split GEMM, [dsplits][M][ld_delta] (delta is null then): summed in
  // split order and rounded to bf16, the raw accumulator's rounding point
  const float* dpart;
  int dsplits;
  const float* drow;
  const float* dcol;
  const float* bias;
  const float* gate;
  int write_res;
  int layernorm;
  const float* weight;
  const float* beta;
  const float* mod_scale;
  const float* mod_shift;
  const int32_t* mod_index;
  float eps;
  uint8_t* q;
  int64_t ld_q;
  float* qs;
  void* y;
  int y_dtype;
  int64_t ld_y;
  // partial-sum form only: further copies of the codes and row scales (same row stride as q), the
  // other GPUs' replicas of the next block's input, written from the same registers
  uint8_t* q_mirror[kMaxMirrors];
  float* qs_mirror[kMaxMirrors];
  int mirrors;
};

// Whether a call is what the PLAIN instantiations below hold (the residual is float32 or bfloat16, any delta).
static inline bool resnorm_plain(const ResNormArgs& a) {
  return a.drow && a.dcol && a.write_res && a.q && !(a.bias || a.gate || a.layernorm || a.weight || a.beta || a.mod_scale || a.y || a.mirrors);
}

template <typename RT>
__device__ __forceinline__ float round_through(float x);
template <>
__device__ __forceinline__ float round_through<float>(float x) { return x; }
template <>
__device__ __forceinline__ float round_through<__nv_bfloat16>(float x) {
  return __bfloat162float(__float2bfloat16_rn(x));
}

// PART: the delta arrives as fp32 planes of a K-split GEMM (a.dpart) instead of a raw bf16 accumulator; an
// instantiation of its own, so that the ordinary one keeps its registers.
// PLAIN: a scaled delta, RMS norm, codes -- what a decoder layer asks for (resnorm_plain).  A launch over a few hundred rows
// fetches its instructions cold and holds the registers of its longest path, so this instantiation has no other
// (816 x 2048 4.60 -> 4.39 us, 1100 x 2048 6.96 -> 4.43).
template <typename RT, int TPR, int IT, bool FAST, bool PART = false, bool PLAIN = false>
__global__ void __launch_bounds__(kRowThreads, PART ? 2 : resnorm_min_blocks<IT>())
residual_norm_quant_kernel(const ResNormArgs a) {
  row_begin(a.early);  // inputs may come from the kernel before this one in the stream
  __shared__ float red[3][kRowThreads / 32];
  const int t = threadIdx.x % TPR;
  const int m = blockIdx.x * (kRowThreads / TPR) + threadIdx.x / TPR;
  const bool live = m < a.M;
  RT* rr = reinterpret_cast<RT*>(a.res) + (live ? (int64_t)m * a.ld_res : 0);
  const __nv_bfloat16* dr = PLAIN || a.delta ? a.delta + (live ? (int64_t)m * a.ld_delta : 0) : nullptr;
  const float* dp = PART ? a.dpart + (live ? (int64_t)m * a.ld_delta : 0) : nullptr;
  const int64_t dp_plane = (int64_t)a.M * a.ld_delta;
  const int64_t mofs = (!PLAIN && live && a.mod_index) ? (int64_t)a.mod_index[m] * a.D : 0;
  const float drs = (live && (PLAIN || a.drow)) ? a.drow[m] : 1.0f;
  const float fD = (float)a.D;

  Raw8<RT> rres[IT];
  Raw8<__nv_bfloat16> rdel[IT];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c0 = (it * TPR + t) * 8;
    const bool on = it < a.iters && live && c0 < a.D;
    rres[it] = fetch<FAST, RT>(rr, c0, a.D, on);
    rdel[it] = fetch<FAST, __nv_bfloat16>(dr, c0, a.D, on && (PLAIN || dr != nullptr) && !PART);
  }
  float x[IT][8];
  float sum = 0.0f, sumsq = 0.0f;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c0 = (it * TPR + t) * 8;
    unpack(rres[it], x[it]);
    if (it < a.iters && live && c0 < a.D) {
      if (PLAIN || dr || PART) {
        float d[8], cs[8], bs[8], gs[8];
        if constexpr (PART) {
          // four planes in flight together, added in split order
          constexpr int kGroup = 4;
#pragma unroll
          for (int i = 0; i < 8; ++i) d[i] = 0.0f;
#pragma unroll 1
          for (int s0 = 0; s0 < a.dsplits; s0 += kGroup) {
            float e[kGroup][8];
#pragma unroll
            for (int sp = 0; sp < kGroup; ++sp)
              if (s0 + sp < a.dsplits) load_f32<FAST>(dp + (s0 + sp) * dp_plane, c0, a.D, e[sp]);
#pragma unroll
            for (int sp = 0; sp < kGroup; ++sp) {
              if (s0 + sp < a.dsplits) {
#pragma unroll
                for (int i = 0; i < 8; ++i) d[i] = (s0 + sp == 0) ? e[sp][i] : __fadd_rn(d[i], e[sp][i]);
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) d[i] = __bfloat162float(__float2bfloat16_rn(d[i]));
        } else {
          unpack(rdel[it], d);
        }
        if (PLAIN || a.dcol) load_f32<FAST>(a.dcol, c0, a.D, cs);
        if (!PLAIN && a.bias) load_f32<FAST>(a.bias, c0, a.D, bs);
        if (!PLAIN && a.gate) load_f32<FAST>(a.gate + mofs, c0, a.D, gs);
        Chain8 ch(d);
        if (PLAIN || a.drow) ch.mul(drs);
        if (PLAIN || a.dcol) ch.mul(cs);
        if (!PLAIN && a.bias) ch.add(bs);
        if (!PLAIN && a.gate) ch.mul(gs);
        ch.add(x[it]);  // x + d, contracted with d's last multiply when there is one
        ch.done(x[it]);
        if (PLAIN || a.write_res) {
#pragma unroll
          for (int i = 0; i < 8; ++i) x[it][i] = round_through<RT>(x[it][i]);
        }
        mask_tail<FAST>(x[it], c0, a.D);
        if (PLAIN || a.write_res) store_out<FAST>(a.res, dtype_of<RT>(), (int64_t)m * a.ld_res, c0, a.D, x[it]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (!PLAIN) sum = __fadd_rn(sum, x[it][i]);
        sumsq = __fmaf_rn(x[it][i], x[it][i], sumsq);
      }
    }
  }
  if (!PLAIN && a.q == nullptr && a.y == nullptr) return;  // residual update only (uniform across the CTA)

  float rstd;
  if (!PLAIN && a.layernorm) {
    const float mean = div_full(row_reduce<TPR, false>(sum, red[0]), fD);
    float sq = 0.0f;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int c0 = (it * TPR + t) * 8;
      if (it < a.iters && live && c0 < a.D) {
#pragma unroll
        for (int i = 0; i < 8; i += 2)  // x - mean == x + (-mean), two lanes per instruction
          unpack2(add2(pack2(x[it][i], x[it][i + 1]), pack2(-mean, -mean)), x[it][i], x[it][i + 1]);
        mask_tail<FAST>(x[it], c0, a.D);
#pragma unroll
        for (int i = 0; i < 8; ++i) sq = __fmaf_rn(x[it][i], x[it][i], sq);
      }
    }
    const float var = div_full(row_reduce<TPR, false>(sq, red[1]), fD);
    rstd = rsqrt_approx_ftz(__fadd_rn(var, a.eps));
  } else {
    const float var = div_full(row_reduce<TPR, false>(sumsq, red[1]), fD);
    rstd = rsqrt_approx_ftz(__fadd_rn(var, a.eps));
  }

  float amax = 0.0f;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c0 = (it * TPR + t) * 8;
    if (it < a.iters && live && c0 < a.D) {
      float ws[8], bs[8], ms[8], mh[8];
      if (!PLAIN && a.weight) load_f32<FAST>(a.weight, c0, a.D, ws);
      if (!PLAIN && a.beta) load_f32<FAST>(a.beta, c0, a.D, bs);
      if (!PLAIN && a.mod_scale) {
        load_f32<FAST>(a.mod_scale + mofs, c0, a.D, ms);
        load_f32<FAST>(a.mod_shift + mofs, c0, a.D, mh);
      }
      Chain8 ch(x[it]);
      ch.mul(rstd);
      if (!PLAIN && a.weight) ch.mul(ws);
      if (!PLAIN && a.beta) ch.add(bs);
      if (!PLAIN && a.mod_scale) {
#pragma unroll
        for (int i = 0; i < 8; i += 2) unpack2(add2(pack2(ms[i], ms[i + 1]), pack2(1.0f, 1.0f)), ms[i], ms[i + 1]);
        ch.mul(ms);
        ch.add(mh);
      }
      ch.done(x[it]);
      mask_tail<FAST>(x[it], c0, a.D);
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = max_f32(amax, fabsf(x[it][i]));
      if (!PLAIN && a.y) store_out<FAST>(a.y, a.y_dtype, (int64_t)m * a.ld_y, c0, a.D, x[it]);
    }
  }
  if (!PLAIN && a.q == nullptr) return;
  amax = row_reduce<TPR, true>(amax, red[2]);
  float scale, inv;
  quant_scales(amax, scale, inv);
  if (!live) return;
  if (t == 0) a.qs[m] = scale;
  uint8_t* qr = a.q + (int64_t)m * a.ld_q;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c0 = (it * TPR + t) * 8;
    if (it < a.iters && c0 < a.D) store_codes<FAST>(qr, c0, a.D, x[it], inv);
  }
  if constexpr (PART) {
#pragma unroll
    for (int k = 0; k < kMaxMirrors; ++k) {
      if (k < a.mirrors) {
        if (t == 0) a.qs_mirror[k][m] = scale;
        uint8_t* qm = a.q_mirror[k] + (int64_t)m * a.ld_q;
#pragma unroll
        for (int it = 0; it < IT; ++it) {
          const int c0 = (it * TPR + t) * 8;
          if (it < a.iters && c0 < a.D) store_codes<FAST>(qm, c0, a.D, x[it], inv);
        }
      }
    }
  }
}

#if IFLB200_ROW_PART == 2 || IFLB200_ROW_PART == -1
// --------------------------------------------------------------------------------------------
// residual_norm_quant for a delta that arrives as fp32 planes of a K-split GEMM (p of them: 4 p bytes per
// element where the bf16 accumulator has 2), one CTA per row.
//
// Bound by latency and by how many rows are in flight at once: a thread owns IT quads of columns 1024
// apart, so that every access of a warp is 512 contiguous bytes, all loads of the row -- residual,
// PL planes, column scales -- are issued before the first use, and the registers are held down
// so that a few hundred rows are resident together.  Eight columns a thread, chunk after chunk and plane
// group after plane group before: 50 x 1024 with eight planes 2.9 -> 2.3 us, 816 x 2048 with two 7.6 -> 5.6.
// PL: planes loaded together (further ones follow in groups of PL).
// PLAIN: the decoder layer's operands alone (resnorm_plain), in a quarter of the code and with one meeting of the row's
// warps for the sum and the maximum: 50 x 1024 with eight planes 2.42 -> 1.77 us, 816 x 2048 with two 5.59 -> 3.89, 18 expert
// layers 403 -> 381; over 250 sizes of 1 to 2000 rows 0.80 of the time, but for many bytes of planes (launch_resnorm_planes_form).
// --------------------------------------------------------------------------------------------
template <typename T>
struct Quad;
template <>
struct Quad<float> {
  float4 u;
  __device__ __forceinline__ void load(const float* p) { u = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ void widen(float (&o)[4]) const { o[0] = u.x; o[1] = u.y; o[2] = u.z; o[3] = u.w; }
};
template <>
struct Quad<__nv_bfloat16> {
  uint2 u;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { u = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ void widen(float (&o)[4]) const {
    o[0] = __uint_as_float(u.x << 16); o[1] = __uint_as_float(u.x & 0xFFFF0000u);
    o[2] = __uint_as_float(u.y << 16); o[3] = __uint_as_float(u.y & 0xFFFF0000u);
  }
};
__device__ __forceinline__ void load_quad(const float* p, float (&o)[4]) {
  Quad<float> q;
  q.load(p);
  q.widen(o);
}
__device__ __forceinline__ void store_quad(void* base, int dtype, int64_t off, const float (&v)[4]) {
  if (dtype == IFLB200_F32) {
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(base) + off) = make_float4(v[0], v[1], v[2], v[3]);
    return;
  }
  uint32_t w[2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
    w[i] = dtype == IFLB200_BF16 ? (f32_to_bf16_bits(v[2 * i]) | (f32_to_bf16_bits(v[2 * i + 1]) << 16))
                                 : (f32_to_f16_bits(v[2 * i]) | (f32_to_f16_bits(v[2 * i + 1]) << 16));
  *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(base) + off) = make_uint2(w[0], w[1]);
}

// Sum or maximum of magnitudes over the CTA; `slots` is used once per row.
template <bool IS_MAX>
__device__ __forceinline__ float row_cta_reduce(float v, float* slots) {
  if (IS_MAX) {
    v = warp_max_abs_f32(v);
  } else {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  }
  if ((threadIdx.x & 31) == 0) slots[threadIdx.x >> 5] = v;
  __syncthreads();
  const float4 a = reinterpret_cast<const float4*>(slots)[0], b = reinterpret_cast<const float4*>(slots)[1];
  if (IS_MAX) return max_f32(max_f32(max_f32(a.x, a.y), max_f32(a.z, a.w)), max_f32(max_f32(b.x, b.y), max_f32(b.z, b.w)));
  return __fadd_rn(__fadd_rn(__fadd_rn(a.x, a.y), __fadd_rn(a.z, a.w)), __fadd_rn(__fadd_rn(b.x, b.y), __fadd_rn(b.z, b.w)));
}

// Resident CTAs per SM that the registers have to leave room for: about 4 * IT * (PL + 4) live values and the
// addresses.
template <int IT, int PL>
__host__ __device__ constexpr int row_cta_min_blocks() {
  return IT * (PL + 4) <= 12 ? 4 : (IT * (PL + 4) <= 18 ? 3 : 2);
}

template <typename RT, int IT, int PL, bool PLAIN>
__global__ void __launch_bounds__(kRowThreads, row_cta_min_blocks<IT, PL>())
residual_norm_planes_kernel(const ResNormArgs a) {
  static_assert(kRowThreads == 256, "eight warps per row");
  __shared__ __align__(16) float red[3][kRowThreads / 32];
  constexpr int kStep = kRowThreads * 4;
  const int m = blockIdx.x, c = threadIdx.x * 4;
  // What is computed from the arguments ahead of the wait, for PLAIN certain to be in registers then.  The general form over up to
  // eight planes has none to spare: with these ahead it took up to 1.2 times as long (1677 x 1456 in eight 20.6 -> 23.7 us);
  // over up to four planes a group it gains by them (3770 x 392 18.9 -> 16.5, 334 x 136 in two 2.73 -> 2.39).
  constexpr bool kAhead = PLAIN || PL < 8;
  int D_kept = a.D, splits_kept = a.dsplits;
  RT* rr_kept = reinterpret_cast<RT*>(a.res) + (int64_t)m * a.ld_res + c;
  const float *dp_kept = a.dpart + (int64_t)m * a.ld_delta + c, *col_kept = a.dcol + c, *row_kept = a.drow + m;
  int64_t plane_kept = (int64_t)a.M * a.ld_delta;
  uint8_t* q_kept = a.q + (int64_t)m * a.ld_q + c;
  float *qs_kept = a.qs + m, eps_kept = a.eps;
  row_open(a.early);
  if (PLAIN) {
    keep(D_kept); keep(splits_kept); keep(rr_kept); keep(dp_kept); keep(col_kept); keep(row_kept); keep(q_kept); keep(qs_kept);
    asm volatile("" : "+l"(plane_kept), "+f"(eps_kept));
  }
  row_enter(a.early);  // inputs may come from the kernel before this one in the stream
#define KEPT(kept, value) (kAhead ? (kept) : (value))
  RT* rr = KEPT(rr_kept, reinterpret_cast<RT*>(a.res) + (int64_t)m * a.ld_res + c);
  const int64_t mofs = !PLAIN && a.mod_index ? (int64_t)a.mod_index[m] * a.D + c : c;
  const float drs = PLAIN || a.drow ? *KEPT(row_kept, a.drow + m) : 1.0f;

  Quad<RT> rres[IT];
  Quad<float> plane[PL][IT], dcol[IT];
  const float* dp = KEPT(dp_kept, a.dpart + (int64_t)m * a.ld_delta + c);
  const int64_t dp_plane = KEPT(plane_kept, (int64_t)a.M * a.ld_delta);
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    if (it * kStep + c < KEPT(D_kept, a.D)) {
      rres[it].load(rr + it * kStep);
      if (PLAIN || a.dcol) dcol[it].load(KEPT(col_kept, a.dcol + c) + it * kStep);
    }
#pragma unroll
    for (int s = 0; s < PL; ++s)
      if (s < KEPT(splits_kept, a.dsplits) && it * kStep + c < KEPT(D_kept, a.D)) plane[s][it].load(dp + s * dp_plane + it * kStep);
  }
  float x[IT][4];
  float sum = 0.0f;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int o = it * kStep;
#pragma unroll
    for (int i = 0; i < 4; ++i) x[it][i] = 0.0f;
    if (o + c < KEPT(D_kept, a.D)) {
      rres[it].widen(x[it]);
      float d[4], op[4];
      plane[0][it].widen(d);  // the planes in split order, then the raw accumulator's rounding point
#pragma unroll
      for (int s = 1; s < PL; ++s) {
        if (s < KEPT(splits_kept, a.dsplits)) {
          float e[4];
          plane[s][it].widen(e);
#pragma unroll
          for (int i = 0; i < 4; ++i) d[i] = __fadd_rn(d[i], e[i]);
        }
      }
      if (PL < 8) {
#pragma unroll 1
        for (int s0 = PL; s0 < KEPT(splits_kept, a.dsplits); s0 += PL) {
          float e[PL][4];
#pragma unroll
          for (int s = 0; s < PL; ++s)
            if (s0 + s < KEPT(splits_kept, a.dsplits)) load_quad(dp + (s0 + s) * dp_plane + o, e[s]);
#pragma unroll
          for (int s = 0; s < PL; ++s) {
            if (s0 + s < KEPT(splits_kept, a.dsplits)) {
#pragma unroll
              for (int i = 0; i < 4; ++i) d[i] = __fadd_rn(d[i], e[s][i]);
            }
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) d[i] = __bfloat162float(__float2bfloat16_rn(d[i]));
      ChainV<4> ch(d);
      if (PLAIN || a.drow) ch.mul(drs);
      if (PLAIN || a.dcol) {
        dcol[it].widen(op);
        ch.mul(op);
      }
      if (!PLAIN && a.bias) {
        load_quad(a.bias + c + o, op);
        ch.add(op);
      }
      if (!PLAIN && a.gate) {
        load_quad(a.gate + mofs + o, op);
        ch.mul(op);
      }
      ch.add(x[it]);  // x + d, contracted with d's last multiply when there is one
      ch.done(x[it]);
      if (PLAIN || a.write_res) {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[it][i] = round_through<RT>(x[it][i]);
        store_quad(KEPT((void*)rr, a.res), dtype_of<RT>(), KEPT(0, (int64_t)m * a.ld_res + c) + o, x[it]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) sum = !PLAIN && a.layernorm ? __fadd_rn(sum, x[it][i]) : __fmaf_rn(x[it][i], x[it][i], sum);
    }
  }
  if (!PLAIN && a.q == nullptr && a.y == nullptr) return;  // residual update only (uniform across the CTA)

  const float fD = (float)KEPT(D_kept, a.D);
  float amax = 0.0f;
  if (PLAIN) {  // rounding keeps the order of the |x| rstd, so that the largest |x| gives the largest of them: one meeting for both
#pragma unroll
    for (int it = 0; it < IT; ++it) amax = max_abs_f32(max_abs_f32(amax, x[it][0], x[it][1]), x[it][2], x[it][3]);
    amax = warp_max_abs_f32(amax);
    if ((threadIdx.x & 31) == 0) red[2][threadIdx.x >> 5] = amax;
  }
  sum = row_cta_reduce<false>(sum, red[0]);
  if (!PLAIN && a.layernorm) {
    const float mean = div_full(sum, fD);
    sum = 0.0f;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      if (it * kStep + c < KEPT(D_kept, a.D)) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[it][i] = __fadd_rn(x[it][i], -mean);
          sum = __fmaf_rn(x[it][i], x[it][i], sum);
        }
      }
    }
    sum = row_cta_reduce<false>(sum, red[1]);
  }
  const float rstd = rsqrt_approx_ftz(__fadd_rn(div_full(sum, fD), KEPT(eps_kept, a.eps)));
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int o = it * kStep;
    if (o + c < KEPT(D_kept, a.D)) {
      float op[4];
      ChainV<4> ch(x[it]);
      ch.mul(rstd);
      if (!PLAIN && a.weight) {
        load_quad(a.weight + c + o, op);
        ch.mul(op);
      }
      if (!PLAIN && a.beta) {
        load_quad(a.beta + c + o, op);
        ch.add(op);
      }
      if (!PLAIN && a.mod_scale) {
        load_quad(a.mod_scale + mofs + o, op);
#pragma unroll
        for (int i = 0; i < 4; ++i) op[i] = __fadd_rn(op[i], 1.0f);
        ch.mul(op);
        load_quad(a.mod_shift + mofs + o, op);
        ch.add(op);
      }
      ch.done(x[it]);
      if (!PLAIN) amax = max_abs_f32(max_abs_f32(amax, x[it][0], x[it][1]), x[it][2], x[it][3]);
      if (!PLAIN && a.y) store_quad(a.y, a.y_dtype, (int64_t)m * a.ld_y + c + o, x[it]);
    }
  }
  if (!PLAIN && a.q == nullptr) return;
  if (PLAIN) {
    const float4 lo = reinterpret_cast<const float4*>(red[2])[0], hi = reinterpret_cast<const float4*>(red[2])[1];
    amax = __fmul_rn(max_f32(max_f32(max_f32(lo.x, lo.y), max_f32(lo.z, lo.w)), max_f32(max_f32(hi.x, hi.y), max_f32(hi.z, hi.w))), rstd);
  } else {
    amax = row_cta_reduce<true>(amax, red[2]);
  }
  float scale, inv;
  quant_scales(amax, scale, inv);
  if (threadIdx.x == 0) *KEPT(qs_kept, a.qs + m) = scale;
  uint8_t* q = KEPT(q_kept, a.q + (int64_t)m * a.ld_q + c);
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    if (it * kStep + c < KEPT(D_kept, a.D)) {
#pragma unroll
      for (int i = 0; i < 4; ++i) x[it][i] = __fmul_rn(x[it][i], inv);
      const uint32_t code = cvt_e4m3x4(x[it][0], x[it][1], x[it][2], x[it][3]);
      *reinterpret_cast<uint32_t*>(q + it * kStep) = code;
#pragma unroll
      for (int k = 0; k < kMaxMirrors; ++k)
        if (!PLAIN && k < a.mirrors) *reinterpret_cast<uint32_t*>(a.q_mirror[k] + (int64_t)m * a.ld_q + c + it * kStep) = code;
    }
  }
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < kMaxMirrors; ++k)
      if (!PLAIN && k < a.mirrors) a.qs_mirror[k][m] = scale;
  }
}
#undef KEPT

// Rows of at most 8192 columns on the aligned path.  The quads form takes its further plane groups quad by quad, each
// a round trip, and that many registers let few rows be resident: it serves the widths and numbers of planes
// whose loads it has all in flight.  us, quads against rows of eight columns a thread:
//   up to 2048 columns ahead everywhere (1024, 50 rows, 8 planes 2.66 / 3.10; 2048, 816 rows, 2 planes 5.71 / 7.60);
//   to 3072 where its three rows an SM need no more waves than the other's two pairs (300 rows, 2 planes 4.58 / 5.72,
//   816 rows 7.82 / 10.49, but 500 rows 6.45 / 5.96; a wave over one or two planes is 0.6 of the other's: 1100 rows 9.97 /
//   10.78), and with seven or eight planes in one wave (816 rows 18.2 / 17.1);
//   from 4097 to 5120 with one or two planes (300 rows 8.47 / 9.02, four planes 10.8 / 10.2);
//   not elsewhere (4096, 816 rows, 8 planes 28.9 / 26.3; 8192, 500 rows, 2 / 8 planes 16.6 / 13.5 and 70.8 / 30.8).
template <typename RT, int IT, int PL>
static void launch_resnorm_planes_form(const ResNormArgs& a, cudaStream_t s) {
  if constexpr (IT <= 2) {
    // More than 32 MB of planes, five to eight of them and a wide row: the general form streams them
    // faster (measured; why was not looked into).  PLAIN against general: 500 x 2048 in eight 1.00, 600 1.05, 1000 1.09,
    // 600 x 1792 in seven 0.98, 700 1.08; under 10240 columns x planes PLAIN stays ahead (3000 x 1536 in six 0.98).
    const bool many_bytes = IT == 2 && PL == 8 && a.D * a.dsplits >= 10240 && (int64_t)a.M * a.D * a.dsplits > (1 << 23);
    if (!many_bytes && resnorm_plain(a)) {
      launch_dep(residual_norm_planes_kernel<RT, IT, PL, true>, dim3(a.M), dim3(kRowThreads), 0, s, 1, dependent_launch_for(a.M), a);
      return;
    }
  }
  launch_dep(residual_norm_planes_kernel<RT, IT, PL, false>, dim3(a.M), dim3(kRowThreads), 0, s, 1, dependent_launch_for(a.M), a);
}
template <typename RT, int TPR, int IT>
static void launch_resnorm_part_form(ResNormArgs a, cudaStream_t s) {
  constexpr int rows = kRowThreads / TPR;
  a.iters = IT;
  launch_dep(residual_norm_quant_kernel<RT, TPR, IT, true, true>, dim3((a.M + rows - 1) / rows), dim3(kRowThreads), 0, s, 1,
             dependent_launch_for(a.M), a);
}
template <typename RT>
static void launch_resnorm_planes(const ResNormArgs& a, cudaStream_t s) {
  const int quads = (a.D + 1023) / 1024, sms = device_sm_count() > 0 ? device_sm_count() : 148;
  if (quads == 1) return a.dsplits <= 4 ? launch_resnorm_planes_form<RT, 1, 4>(a, s) : launch_resnorm_planes_form<RT, 1, 8>(a, s);
  if (quads == 2)
    return a.dsplits <= 2   ? launch_resnorm_planes_form<RT, 2, 2>(a, s)
           : a.dsplits <= 4 ? launch_resnorm_planes_form<RT, 2, 4>(a, s)
                            : launch_resnorm_planes_form<RT, 2, 8>(a, s);
  if (quads == 3) {
    const int waves = (a.M + 3 * sms - 1) / (3 * sms), waves_of_pairs = (a.M + 4 * sms - 1) / (4 * sms);
    const bool ahead = a.dsplits > 6 ? waves == 1 : (a.dsplits > 2 ? waves <= waves_of_pairs : waves * 3 <= waves_of_pairs * 5);
    return ahead ? launch_resnorm_planes_form<RT, 3, 2>(a, s) : launch_resnorm_part_form<RT, 128, 3>(a, s);
  }
  if (quads == 4) return launch_resnorm_part_form<RT, kRowThreads, 2>(a, s);
  if (quads == 5 && a.dsplits <= 2) return launch_resnorm_planes_form<RT, 5, 2>(a, s);
  if (quads <= 6) return launch_resnorm_part_form<RT, kRowThreads, 3>(a, s);
  return launch_resnorm_part_form<RT, kRowThreads, 4>(a, s);
}
#endif

#if IFLB200_ROW_PART == 1 || IFLB200_ROW_PART == -1
// --------------------------------------------------------------------------------------------
// Per-tensor pack (the torch-FP8-linear recipe)
// --------------------------------------------------------------------------------------------
constexpr int kPackThreads = 256;
constexpr int kPackMaxCtas = 1024;

__device__ __forceinline__ uint32_t max_bf16_bits(const uint4& u, uint32_t best) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) best = max(best, max(w[k] & 0x7FFFu, (w[k] >> 16) & 0x7FFFu));
  return best;
}

// Maximum of |x| as an integer maximum of the bf16 magnitude bits: finite values order like
// their bits, and every NaN pattern is larger than infinity, so NaN propagates.
__global__ void __launch_bounds__(kPackThreads)
amax_partial_kernel(const uint16_t* __restrict__ x, int64_t n, uint32_t* __restrict__ partial) {
  row_dependency_wait();  // inputs may come from the kernel before this one in the stream
  row_trigger();  // never ahead of the wait: pack_kernel<true> reads x without one of its own
  __shared__ uint32_t red[kPackThreads / 32];
  uint32_t best = 0;
  const int64_t nvec = n / 8;
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const int64_t stride = (int64_t)gridDim.x * kPackThreads;
  if (vec) {
    const uint4* xv = reinterpret_cast<const uint4*>(x);
    // four loads in flight per thread (one at a time left a 4680 x 3072 tensor at 2.3 TB/s)
    for (int64_t i0 = (int64_t)blockIdx.x * kPackThreads + threadIdx.x; i0 < nvec; i0 += 4 * stride) {
      uint4 u[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) u[k] = i0 + k * stride < nvec ? xv[i0 + k * stride] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int k = 0; k < 4; ++k) best = max_bf16_bits(u[k], best);
    }
    for (int64_t i = nvec * 8 + (int64_t)blockIdx.x * kPackThreads + threadIdx.x; i < n; i += stride)
      best = max(best, (uint32_t)x[i] & 0x7FFFu);
  } else {
    for (int64_t i = (int64_t)blockIdx.x * kPackThreads + threadIdx.x; i < n; i += stride)
      best = max(best, (uint32_t)x[i] & 0x7FFFu);
  }
  best = __reduce_max_sync(0xFFFFFFFFu, best);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < kPackThreads / 32; ++i) best = max(best, red[i]);
    partial[blockIdx.x] = best;
  }
}

// n_partial > 0: dynamic scale from the partial maxima (every CTA recomputes it; CTA 0 writes
// it out).  n_partial == 0: fixed scale read from scale_in.
// ONE: dynamic, and the grid holds every element at four chunks a thread (n <= kPackOnePass).  The elements are then on their way before the
// maxima are awaited, the one read of this library's row kernels ahead of their wait: amax_partial_kernel, which is the kernel
// before, lets this one start only behind its own wait, when whatever wrote x has completed and its writes have reached
// L2.  So these loads are strong ones at GPU scope, which L2 serves: a line that L1 or the read-only path kept from an earlier
// launch cannot be the answer.  Both kernels for 2^19 elements 4.14 -> 3.48 us, 682 thousand 4.21 -> 3.57, 2^22 7.69 -> 6.80, 2^23 10.3 ->
// 8.7; with more than one pass the loads ahead were slower (2^24 15.8 -> 16.2, 2^26 71 -> 76).
__device__ __forceinline__ uint4 ld_relaxed_gpu_v4(const uint4* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
constexpr int64_t kPackOnePass = (int64_t)kPackMaxCtas * kPackThreads * 8 * 4;
template <bool ONE>
__global__ void __launch_bounds__(kPackThreads)
pack_kernel(const uint16_t* __restrict__ x, int64_t n, const uint32_t* __restrict__ partial,
            int n_partial, const float* __restrict__ scale_in, float* __restrict__ scale_out,
            uint8_t* __restrict__ q) {
  __shared__ uint32_t red[kPackThreads / 32];
  const bool vec = ((reinterpret_cast<uintptr_t>(x) & 15) == 0) && ((reinterpret_cast<uintptr_t>(q) & 7) == 0);
  const int64_t stride = (int64_t)gridDim.x * kPackThreads, first = (int64_t)blockIdx.x * kPackThreads + threadIdx.x;
  const int64_t nvec = vec ? n / 8 : 0;
  const uint4* xv = reinterpret_cast<const uint4*>(x);
  uint4 u[4];
  auto load = [&](int64_t i0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      u[k] = make_uint4(0u, 0u, 0u, 0u);
      if (i0 + k * stride < nvec) u[k] = ONE ? ld_relaxed_gpu_v4(xv + i0 + k * stride) : xv[i0 + k * stride];
    }
  };
  if (ONE) load(first);
  row_dependency_wait();  // inputs may come from the kernel before this one in the stream
  row_trigger();
  float scale;
  if (ONE || n_partial > 0) {
    uint32_t best = 0;
    for (int i = threadIdx.x; i < n_partial; i += kPackThreads) best = max(best, partial[i]);
    best = __reduce_max_sync(0xFFFFFFFFu, best);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
    __syncthreads();
    best = red[0];
#pragma unroll
    for (int i = 1; i < kPackThreads / 32; ++i) best = max(best, red[i]);
    scale = scale_of_bits(best);
    if (blockIdx.x == 0 && threadIdx.x == 0) *scale_out = scale;
  } else {
    scale = *scale_in;
  }
  // with a caller's own scale the row may hold NaN or a quotient out of range: by division
  const float r = ONE || n_partial > 0 ? reciprocal_for_pack(scale) : __uint_as_float(0x7FC00000u);
  auto store = [&](int64_t i0) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i0 + k * stride < nvec) reinterpret_cast<uint2*>(q)[i0 + k * stride] = pack_eight(u[k], scale, r);
  };
  if (ONE) {
    store(first);
  } else {
    for (int64_t i0 = first; i0 < nvec; i0 += 4 * stride) {
      load(i0);
      store(i0);
    }
  }
  for (int64_t i = nvec * 8 + first; i < n; i += stride)
    q[i] = (uint8_t)(cvt_e4m3x2(pack_one(__uint_as_float((uint32_t)x[i] << 16), scale), 0.0f) & 0xFF);
}

// Small tensors: the whole dynamic pack in one launch.  A cluster of eight CTAs (sixteen above 2^18
// elements) keeps the tensor in registers between the maximum and the cast; the maxima of the CTAs meet in
// distributed shared memory.  The two kernels above are two launches and two passes: 3.6 us up to 700 thousand elements,
// against 2.0 here at 2^16 elements, 3.2 at 2^18, 3.4 at 2^19; a cluster takes 4.3 for 680 thousand, so above
// 2^19 they stay.
constexpr int kPackClusterThreads = 1024;
constexpr int64_t kPackClusterMax = (int64_t)16 * kPackClusterThreads * 8 * 4;

template <int kPackCluster, int V>
__global__ void __cluster_dims__(kPackCluster, 1, 1) __launch_bounds__(kPackClusterThreads)
pack_cluster_kernel(const uint4* __restrict__ x, int nvec, float* __restrict__ scale_out, uint2* __restrict__ q) {
  __shared__ uint32_t red[kPackClusterThreads / 32];
  __shared__ uint32_t maxima[kPackCluster];
  const int rank = (int)cluster_ctarank();
  cluster_arrive();        // this CTA runs: its shared memory may be written from now on
  grid_dependency_wait();  // x may come from the kernel before this one in the stream
  grid_launch_dependents();
  uint4 u[V];
  uint32_t best = 0;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int i = (v * kPackCluster + rank) * kPackClusterThreads + threadIdx.x;
    u[v] = i < nvec ? x[i] : make_uint4(0u, 0u, 0u, 0u);
  }
#pragma unroll
  for (int v = 0; v < V; ++v) best = max_bf16_bits(u[v], best);
  best = __reduce_max_sync(0xFFFFFFFFu, best);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  __syncthreads();
  cluster_wait();  // every CTA of the cluster has started: a store into one that has not would be lost
  if (threadIdx.x < 32) {
    best = __reduce_max_sync(0xFFFFFFFFu, red[threadIdx.x]);
    if (threadIdx.x < kPackCluster) {
      uint32_t peer;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(smem_u32(&maxima[rank])), "r"(threadIdx.x));
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer), "r"(best) : "memory");
    }
    __syncwarp();  // the cluster barrier wants whole warps
  }
  cluster_sync_all();
  best = maxima[0];
#pragma unroll
  for (int k = 1; k < kPackCluster; ++k) best = max(best, maxima[k]);
  const float scale = scale_of_bits(best), r = reciprocal_for_pack(scale);
  if (rank == 0 && threadIdx.x == 0) *scale_out = scale;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int i = (v * kPackCluster + rank) * kPackClusterThreads + threadIdx.x;
    if (i < nvec) q[i] = pack_eight(u[v], scale, r);
  }
}

#endif  // pack kernels

// --------------------------------------------------------------------------------------------
// Host side: geometry selection and launches
// --------------------------------------------------------------------------------------------
static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
static inline bool aligned8(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7) == 0; }
static inline int esize(int dtype) { return dtype == IFLB200_F32 ? 4 : 2; }
static inline bool dtype_ok(int d) { return d == IFLB200_F32 || d == IFLB200_BF16 || d == IFLB200_F16; }

// Geometry of a row kernel: threads per row and chunks per thread (see kRowThreads above).
struct RowGeom {
  int tpr;
  int iters;
};
// experiments: force the group size (0 = choose); one definition shared by the three units
#if IFLB200_ROW_PART == 0 || IFLB200_ROW_PART == -1
int g_row_tpr_override = 0;
#else
extern int g_row_tpr_override;
#endif

static RowGeom pick_geom(int width) {
  const int chunks = (width + 7) / 8;
  int tpr = 32;
  while (tpr < kRowThreads && tpr < chunks) tpr *= 2;
  if (g_row_tpr_override && (chunks + g_row_tpr_override - 1) / g_row_tpr_override <= 8) tpr = g_row_tpr_override;
  RowGeom g;
  g.tpr = tpr;
  g.iters = (chunks + tpr - 1) / tpr;
  return g;
}

// Calls `launch(tpr_tag, it_tag)` with compile-time tags for the geometry: groups narrower than
// the CTA always hold one chunk per thread; full-CTA groups hold 1, 2, 4 or 8.
template <int V>
struct IntTag {
  static constexpr int value = V;
};
template <typename F>
static void dispatch_geom(const RowGeom& g, F&& launch) {
  if (g.iters <= 1) {
    switch (g.tpr) {
      case 32: launch(IntTag<32>{}, IntTag<1>{}); return;
      case 64: launch(IntTag<64>{}, IntTag<1>{}); return;
      case 128: launch(IntTag<128>{}, IntTag<1>{}); return;
      default: launch(IntTag<256>{}, IntTag<1>{}); return;
    }
  }
  switch (g.tpr) {  // forced narrow groups with several chunks (experiments): deepest variant
    case 32: launch(IntTag<32>{}, IntTag<8>{}); return;
    case 64: launch(IntTag<64>{}, IntTag<8>{}); return;
    case 128:
      if (g.iters <= 2) launch(IntTag<128>{}, IntTag<2>{});
      else if (g.iters == 3) launch(IntTag<128>{}, IntTag<3>{});
      else if (g.iters <= 4) launch(IntTag<128>{}, IntTag<4>{});
      else launch(IntTag<128>{}, IntTag<8>{});
      return;
    default: break;
  }
  if (g.iters <= 2) launch(IntTag<256>{}, IntTag<2>{});
  else if (g.iters == 3) launch(IntTag<256>{}, IntTag<3>{});
  else if (g.iters <= 4) launch(IntTag<256>{}, IntTag<4>{});
  else launch(IntTag<256>{}, IntTag<8>{});
}

// The element-wise (any alignment) kernels exist in one geometry only: a full-CTA group with up
// to 8 chunks per thread.
static RowGeom slow_geom(int width) {
  RowGeom g;
  g.tpr = kRowThreads;
  g.iters = ((width + 7) / 8 + kRowThreads - 1) / kRowThreads;
  return g;
}

template <typename XT>
static void launch_row_quant(RowQuantArgs a, bool fast, cudaStream_t s) {
  const bool plain = !(a.row || a.col || a.bias || a.gelu);
  if (!fast) {
    a.iters = slow_geom(a.K).iters;
    if (plain) launch_dep(row_quant_kernel<XT, kRowThreads, 8, true, false>, dim3(a.M), dim3(kRowThreads), 0, s, 1, dependent_launch_for(a.M), a);
    else launch_dep(row_quant_kernel<XT, kRowThreads, 8, false, false>, dim3(a.M), dim3(kRowThreads), 0, s, 1, dependent_launch_for(a.M), a);
    return;
  }
  const RowGeom g = pick_geom(a.K);
  a.iters = g.iters;
  const bool dep = dependent_launch_for(a.M, a.phase == 0 && (int64_t)a.M * a.K <= 1 << 24);  // see launch.cuh
  dispatch_geom(g, [&](auto tpr, auto it) {
    constexpr int TPR = decltype(tpr)::value, IT = decltype(it)::value;
    const int grid = (a.M + kRowThreads / TPR - 1) / (kRowThreads / TPR);
    if (plain) launch_dep(row_quant_kernel<XT, TPR, IT, true, true>, dim3(grid), dim3(kRowThreads), 0, s, 1, dep, a);
    else launch_dep(row_quant_kernel<XT, TPR, IT, false, true>, dim3(grid), dim3(kRowThreads), 0, s, 1, dep, a);
  });
}
template <typename XT>
static void launch_gated(GatedArgs a, bool fast, cudaStream_t s) {
  if (!fast) {
    a.iters = slow_geom(a.F).iters;
    launch_dep(gated_act_quant_kernel<XT, kRowThreads, 8, false>, dim3(a.M), dim3(kRowThreads), 0, s, 1, dependent_launch_for(a.M), a);
    return;
  }
  if constexpr (sizeof(XT) == 2) {
    // A CTA for every row at once: while each has an SM of its own, and up to three an SM for rows that are one or two quads a
    // thread.  us behind one another, this form against groups of 256 threads: 50 x 4096 1.91 / 2.48, 148 x 512 1.32 / 1.80, 148 x
    // 8192 2.71 / 3.85, 148 x 16384 4.03 / 5.88, 444 x 4096 3.70 / 3.85, 444 x 5120 4.17 / 4.63; beyond, 200 x 8192 4.65 / 4.28, 149 x
    // 6144 3.59 / 3.35, 445 x 4096 4.24 / 3.86, 600 x 4096 5.47 / 4.87 (up to 2048 columns it stays ahead: 600 x 512 1.54 / 2.19).
    const int sms = device_sm_count() > 0 ? device_sm_count() : 148, q = (a.F + 4 * kGatedFewThreads - 1) / (4 * kGatedFewThreads);
    if (g_row_tpr_override == 0 && (a.M <= sms || (a.F <= 5120 && a.M <= 3 * sms))) {
      auto few = [&](auto quads) {
        constexpr int Q = decltype(quads)::value;
        const int threads = ((a.F / 4 + Q - 1) / Q + 31) / 32 * 32;
        const bool gelu = a.act == IFLB200_ACT_GELU_TANH;
        launch_dep(gelu ? gated_act_quant_few_kernel<XT, IFLB200_ACT_GELU_TANH, Q> : gated_act_quant_few_kernel<XT, IFLB200_ACT_SILU, Q>,
                   dim3(a.M), dim3(threads), 0, s, 1, dependent_launch_for(a.M), a);
      };
      if (q <= 1) few(IntTag<1>{});
      else if (q <= 2) few(IntTag<2>{});
      else few(IntTag<4>{});
      return;
    }
  }
  const RowGeom g = pick_geom(a.F);
  a.iters = g.iters;
  dispatch_geom(g, [&](auto tpr, auto it) {
    constexpr int TPR = decltype(tpr)::value, IT = decltype(it)::value;
    const int grid = (a.M + kRowThreads / TPR - 1) / (kRowThreads / TPR);
    launch_dep(gated_act_quant_kernel<XT, TPR, IT, true>, dim3(grid), dim3(kRowThreads), 0, s, 1,
               dependent_launch_for(a.M, (int64_t)a.M * a.F <= 1 << 22), a);  // see launch.cuh
  });
}
template <typename RT>
static void launch_resnorm(ResNormArgs a, bool fast, cudaStream_t s) {
  if (!fast) {
    a.iters = slow_geom(a.D).iters;
    launch_dep(residual_norm_quant_kernel<RT, kRowThreads, 8, false>, dim3(a.M), dim3(kRowThreads), 0, s, 1, dependent_launch_for(a.M), a);
    return;
  }
  RowGeom g = pick_geom(a.D);
  // 1025..2048 columns: two rows per CTA, two chunks per thread (measured at 816 x 2048 with an
  // f32 residual: 4.9 us against 5.7 us with one row per CTA; the reference's kernel 4.4 us)
  if (g.tpr == kRowThreads && g.iters == 1 && g_row_tpr_override == 0) {
    g.tpr = 128;
    g.iters = 2;
  }
  // 2049..3072 columns: 128 threads x 3 chunks use every chunk slot (256 x 2 leaves a quarter empty)
  const int chunks = (a.D + 7) / 8;
  if (g.tpr == kRowThreads && g.iters == 2 && chunks <= 384 && g_row_tpr_override == 0) {
    g.tpr = 128;
    g.iters = 3;
  }
  a.iters = g.iters;
  dispatch_geom(g, [&](auto tpr, auto it) {
    constexpr int TPR = decltype(tpr)::value, IT = decltype(it)::value;
    const int grid = (a.M + kRowThreads / TPR - 1) / (kRowThreads / TPR);
    if constexpr (std::is_same<RT, float>::value && IT <= 3) {
      if (a.delta && resnorm_plain(a)) {
        launch_dep(residual_norm_quant_kernel<RT, TPR, IT, true, false, true>, dim3(grid), dim3(kRowThreads), 0, s, 1, dependent_launch_for(a.M), a);
        return;
      }
    }
    launch_dep(residual_norm_quant_kernel<RT, TPR, IT, true>, dim3(grid), dim3(kRowThreads), 0, s, 1, dependent_launch_for(a.M), a);
  });
}

}  // namespace iflb200

using namespace iflb200;

#if IFLB200_ROW_PART == 0 || IFLB200_ROW_PART == -1
extern "C" int iflb200_row_set_group(int threads_per_row) {
  if (threads_per_row != 0 && (threads_per_row < 32 || threads_per_row > kRowThreads ||
                               (threads_per_row & (threads_per_row - 1))))
    return IFLB200_ERR_ARG;
  iflb200::g_row_tpr_override = threads_per_row;
  return IFLB200_OK;
}

static int row_quant_impl(const void* x, int x_dtype, int64_t ld_x, int M, int K, const float* row,
                          const float* col, const float* bias, int gelu, void* q, int64_t ld_q, float* qs,
                          int phase, float* amax, void* stream, float* const* amax_mirrors = nullptr,
                          int mirrors = 0) {
  if (M < 0 || K < 0) return IFLB200_ERR_ARG;
  if (mirrors < 0 || mirrors > kMaxMirrors || (mirrors > 0 && (!amax_mirrors || phase != 1))) return IFLB200_ERR_ARG;
  if (M == 0 || K == 0) return IFLB200_OK;
  if (!x) return IFLB200_ERR_ARG;
  if (phase != 1 && (!q || !qs)) return IFLB200_ERR_ARG;
  if (phase != 0 && !amax) return IFLB200_ERR_ARG;
  if (!dtype_ok(x_dtype)) return IFLB200_ERR_DTYPE;
  if (K > kMaxWidth) return IFLB200_ERR_SHAPE;
  if (ld_x < K || (phase != 1 && ld_q < K)) return IFLB200_ERR_ARG;
  RowQuantArgs a;
  a.x = x; a.ld_x = ld_x; a.M = M; a.K = K;
  a.row = row; a.col = col; a.bias = bias; a.gelu = gelu;
  a.q = reinterpret_cast<uint8_t*>(q); a.ld_q = ld_q; a.qs = qs;
  a.phase = phase; a.amax = amax;
  a.early = early_trigger_for(reinterpret_cast<cudaStream_t>(stream));
  a.mirrors = mirrors;
  for (int k = 0; k < kMaxMirrors; ++k) {
    a.amax_mirror[k] = k < mirrors ? amax_mirrors[k] : nullptr;
    if (k < mirrors && !a.amax_mirror[k]) return IFLB200_ERR_ARG;
  }
  const bool fast = K % 8 == 0 && aligned16(x) && (ld_x * esize(x_dtype)) % 16 == 0 &&
                    (phase == 1 || (aligned8(q) && ld_q % 8 == 0)) && (!col || aligned16(col)) &&
                    (!bias || aligned16(bias));
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (fast && gelu && phase == 0 && x_dtype != IFLB200_F32 && g_row_tpr_override == 0 &&
      launch_gelu_quant_stream({x, ld_x, M, K, row, col, bias, a.q, ld_q, qs, a.early}, x_dtype == IFLB200_F16, s))
    return (int)cudaGetLastError();
  if (x_dtype == IFLB200_BF16) launch_row_quant<__nv_bfloat16>(a, fast, s);
  else if (x_dtype == IFLB200_F16) launch_row_quant<__half>(a, fast, s);
  else launch_row_quant<float>(a, fast, s);
  return (int)cudaGetLastError();
}

extern "C" int iflb200_row_quant(const void* x, int x_dtype, int64_t ld_x, int M, int K,
                                 const float* row, const float* col, const float* bias, int gelu,
                                 void* q, int64_t ld_q, float* qs, void* stream) {
  return row_quant_impl(x, x_dtype, ld_x, M, K, row, col, bias, gelu, q, ld_q, qs, 0, nullptr, stream);
}

extern "C" int iflb200_row_quant_sharded(const void* x, int x_dtype, int64_t ld_x, int M, int K,
                                         const float* row, const float* col, const float* bias, int gelu,
                                         int phase, float* amax, void* q, int64_t ld_q, float* qs,
                                         void* stream) {
  if (phase != 1 && phase != 2 && phase != 3) return IFLB200_ERR_ARG;
  return row_quant_impl(x, x_dtype, ld_x, M, K, row, col, bias, gelu, q, ld_q, qs, phase, amax, stream);
}

extern "C" int iflb200_row_max_sharded(const void* x, int x_dtype, int64_t ld_x, int M, int K, const float* row,
                                       const float* col, const float* bias, int gelu, float* amax,
                                       float* const* amax_mirrors, int mirrors, void* stream) {
  return row_quant_impl(x, x_dtype, ld_x, M, K, row, col, bias, gelu, nullptr, 0, nullptr, 1, amax, stream,
                        amax_mirrors, mirrors);
}

#endif

#if IFLB200_ROW_PART == 0 || IFLB200_ROW_PART == -1
// Quantiser pass over fp32 rows whose maxima are already known (the second half of the gated GEMM):
// no reduction, so a row is cut into pieces for separate CTAs and the pass runs as a flat elementwise
// kernel (816 x 16384: 3264 CTAs instead of 816 CTAs that each hold a whole row).
// The maxima are read, never written; `amax_zero` (another buffer, or NULL) is cleared for the
// producer after next -- clearing the buffer that is being read would race with the row's other CTAs.
// Five bytes per element, mostly from L2: a thread takes Q quads 1024 columns apart, every access of a
// warp contiguous and all of them in flight (one pair of loads per thread before: 816 x 16384 10.2 us).
template <int Q>
__global__ void __launch_bounds__(kRowThreads)
quant_from_amax_kernel(const float* __restrict__ h, int64_t ld_h, int M, int F, const float* __restrict__ amax,
                       float* __restrict__ amax_zero, uint8_t* __restrict__ q, int64_t ld_q, float* __restrict__ qs, int early) {
  row_open(early);
  const int m = blockIdx.y;
  const int c0 = blockIdx.x * (kRowThreads * 4 * Q) + threadIdx.x * 4;
  const float *src = h + (int64_t)m * ld_h + c0, *top = amax + m;
  uint8_t* dst = q + (int64_t)m * ld_q + c0;
  keep(F); keep(src); keep(top); keep(dst);
  row_enter(early);  // h and amax come from the kernel before this one in the stream
  float4 v[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i)
    if (c0 + i * kRowThreads * 4 < F) v[i] = *reinterpret_cast<const float4*>(src + i * kRowThreads * 4);
  float scale, inv;
  quant_scales(*top, scale, inv);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    qs[m] = scale;
    if (amax_zero) amax_zero[m] = 0.0f;
  }
#pragma unroll
  for (int i = 0; i < Q; ++i)
    if (c0 + i * kRowThreads * 4 < F)
      *reinterpret_cast<uint32_t*>(dst + i * kRowThreads * 4) =
          cvt_e4m3x4(__fmul_rn(v[i].x, inv), __fmul_rn(v[i].y, inv), __fmul_rn(v[i].z, inv), __fmul_rn(v[i].w, inv));
}

// The same for any alignment and width.
__global__ void __launch_bounds__(kRowThreads)
quant_from_amax_any_kernel(const float* __restrict__ h, int64_t ld_h, int M, int F, const float* __restrict__ amax,
                           float* __restrict__ amax_zero, uint8_t* __restrict__ q, int64_t ld_q, float* __restrict__ qs, int early) {
  row_begin(early);
  const int m = blockIdx.y;
  const int c0 = (blockIdx.x * kRowThreads + threadIdx.x) * 8;
  float scale, inv;
  quant_scales(amax[m], scale, inv);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    qs[m] = scale;
    if (amax_zero) amax_zero[m] = 0.0f;
  }
  if (c0 >= F) return;
  float v[8];
  load_f32<false>(h + (int64_t)m * ld_h, c0, F, v);
  store_codes<false>(q + (int64_t)m * ld_q, c0, F, v, inv);
}

extern "C" int iflb200_quant_from_amax(const float* h, int64_t ld_h, int M, int F, const float* amax, float* amax_zero,
                                       void* q, int64_t ld_q, float* qs, void* stream) {
  if (M < 0 || F < 0) return IFLB200_ERR_ARG;
  if (M == 0 || F == 0) return IFLB200_OK;
  if (!h || !amax || !q || !qs || amax_zero == amax) return IFLB200_ERR_ARG;
  if (ld_h < F || ld_q < F) return IFLB200_ERR_ARG;
  if (M > 65535) return IFLB200_ERR_SHAPE;
  const bool fast = F % 8 == 0 && aligned16(h) && (ld_h * 4) % 16 == 0 && aligned8(q) && ld_q % 8 == 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  uint8_t* codes = reinterpret_cast<uint8_t*>(q);
  auto launch = [&](auto kernel, int columns) {
    launch_dep(kernel, dim3((unsigned)((F + columns - 1) / columns), (unsigned)M), dim3(kRowThreads), 0, s, 1,
               dependent_launch_for(M, fast && (int64_t)M * F <= 1 << 23), h, ld_h, M, F, amax, amax_zero, codes, ld_q, qs, early_trigger_for(s));
  };
  // Pieces of 4096 columns where there is work for every SM, of 1024 while six of them a SM hold all, of 2048 between
  // (a piece of 1024 columns is one load a thread): us for pieces of 1024 / 2048 / 4096 columns -- 50 x 4096 1.30 / 1.30 /
  // 1.47, 150 x 4096 1.44 / 1.49 / 1.80, 500 x 4096 2.82 / 1.90 / 2.21, 150 x 13824 3.00 / 1.90 / 2.41, 2000 x 1040 4.85 /
  // 2.85 / 2.86, 816 x 16384 14.2 / 7.62 / 5.12.
  const int pieces = (F + kRowThreads * 4 - 1) / (kRowThreads * 4), sms = device_sm_count() > 0 ? device_sm_count() : 148;
  if (!fast) launch(quant_from_amax_any_kernel, kRowThreads * 8);
  else if ((int64_t)M * F >= (int64_t)1 << 21) launch(quant_from_amax_kernel<4>, kRowThreads * 16);
  else if (pieces > 1 && (int64_t)M * pieces > 6 * sms) launch(quant_from_amax_kernel<2>, kRowThreads * 8);
  else launch(quant_from_amax_kernel<1>, kRowThreads * 4);
  return (int)cudaGetLastError();
}
#endif

#if IFLB200_ROW_PART == 1 || IFLB200_ROW_PART == -1
extern "C" int iflb200_gated_act_quant(const void* gu, int gu_dtype, int64_t ld_gu, int M, int F,
                                       const float* row, const float* col, int act,
                                       void* q, int64_t ld_q, float* qs, void* stream) {
  if (M < 0 || F < 0) return IFLB200_ERR_ARG;
  if (F > 16384) return IFLB200_ERR_SHAPE;
  if (act != IFLB200_ACT_GELU_TANH && act != IFLB200_ACT_SILU) return IFLB200_ERR_ARG;
  if (M == 0 || F == 0) return IFLB200_OK;
  if (!gu || !q || !qs) return IFLB200_ERR_ARG;
  if (!dtype_ok(gu_dtype)) return IFLB200_ERR_DTYPE;
  if (ld_gu < 2 * (int64_t)F || ld_q < F) return IFLB200_ERR_ARG;
  GatedArgs a;
  a.gu = gu; a.ld_gu = ld_gu; a.M = M; a.F = F; a.row = row; a.col = col; a.act = act;
  a.q = reinterpret_cast<uint8_t*>(q); a.ld_q = ld_q; a.qs = qs;
  a.early = early_trigger_for(reinterpret_cast<cudaStream_t>(stream));
  const int es = esize(gu_dtype);
  const bool fast = F % 8 == 0 && aligned16(gu) && (ld_gu * es) % 16 == 0 && aligned8(q) && ld_q % 8 == 0 &&
                    (!col || aligned16(col));
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (gu_dtype == IFLB200_BF16) launch_gated<__nv_bfloat16>(a, fast, s);
  else if (gu_dtype == IFLB200_F16) launch_gated<__half>(a, fast, s);
  else launch_gated<float>(a, fast, s);
  return (int)cudaGetLastError();
}

#endif

#if IFLB200_ROW_PART == 0 || IFLB200_ROW_PART == -1
extern "C" int iflb200_dequant_rows(const void* x, int x_dtype, int64_t ld_x, int M, int D,
                                    const float* row, const float* col, const float* bias,
                                    void* y, int y_dtype, int64_t ld_y, void* stream) {
  if (M < 0 || D < 0) return IFLB200_ERR_ARG;
  if (M == 0 || D == 0) return IFLB200_OK;
  if (!x || !y) return IFLB200_ERR_ARG;
  if (!dtype_ok(x_dtype) || !dtype_ok(y_dtype)) return IFLB200_ERR_DTYPE;
  if (ld_x < D || ld_y < D) return IFLB200_ERR_ARG;
  if (M > 65535 * 1024) return IFLB200_ERR_SHAPE;
  DequantArgs a;
  a.x = x; a.ld_x = ld_x; a.M = M; a.D = D; a.row = row; a.col = col; a.bias = bias;
  a.y = y; a.y_dtype = y_dtype; a.ld_y = ld_y;
  const bool fast = D % 8 == 0 && aligned16(x) && (ld_x * esize(x_dtype)) % 16 == 0 && aligned16(y) &&
                    (ld_y * esize(y_dtype)) % 16 == 0 && (!col || aligned16(col)) && (!bias || aligned16(bias));
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int chunks = (D + 2047) / 2048;
  // blockIdx.y carries the row: split very tall inputs into slabs of 65535 rows.
  for (int m0 = 0; m0 < M; m0 += 65535) {
    DequantArgs b = a;
    const int rows = (M - m0 < 65535) ? (M - m0) : 65535;
    b.M = rows;
    b.x = reinterpret_cast<const char*>(x) + (int64_t)m0 * ld_x * esize(x_dtype);
    b.y = reinterpret_cast<char*>(y) + (int64_t)m0 * ld_y * esize(y_dtype);
    b.row = row ? row + m0 : nullptr;
    const dim3 grid(chunks, rows);
    if (fast) {
      const bool dep = dependent_launch_for(b.M, (int64_t)M * D <= 1 << 24);  // see launch.cuh
      if (x_dtype == IFLB200_BF16) launch_dep(dequant_rows_kernel<__nv_bfloat16, true>, dim3(grid), dim3(256), 0, s, 1, dep, b);
      else if (x_dtype == IFLB200_F16) launch_dep(dequant_rows_kernel<__half, true>, dim3(grid), dim3(256), 0, s, 1, dep, b);
      else launch_dep(dequant_rows_kernel<float, true>, dim3(grid), dim3(256), 0, s, 1, dep, b);
    } else {
      if (x_dtype == IFLB200_BF16) launch_dep(dequant_rows_kernel<__nv_bfloat16, false>, dim3(grid), dim3(256), 0, s, 1, dependent_launch_for(b.M), b);
      else if (x_dtype == IFLB200_F16) launch_dep(dequant_rows_kernel<__half, false>, dim3(grid), dim3(256), 0, s, 1, dependent_launch_for(b.M), b);
      else launch_dep(dequant_rows_kernel<float, false>, dim3(grid), dim3(256), 0, s, 1, dependent_launch_for(b.M), b);
    }
  }
  return (int)cudaGetLastError();
}

#endif

#if IFLB200_ROW_PART == 2 || IFLB200_ROW_PART == -1
static int resnorm_impl(void* res, int res_dtype, int64_t ld_res, int M, int D, const void* delta, int delta_splits,
                        int64_t ld_delta, const float* delta_row, const float* delta_col, const float* bias,
                        const float* gate, int write_res, int layernorm, const float* weight, const float* beta,
                        const float* mod_scale, const float* mod_shift, const int32_t* mod_index, float eps, void* q,
                        int64_t ld_q, float* qs, void* y, int y_dtype, int64_t ld_y, void* stream,
                        void* const* q_mirrors = nullptr, float* const* qs_mirrors = nullptr, int mirrors = 0) {
  if (M < 0 || D < 0) return IFLB200_ERR_ARG;
  if (mirrors < 0 || mirrors > kMaxMirrors || (mirrors > 0 && (!q_mirrors || !qs_mirrors || !q || !delta_splits)))
    return IFLB200_ERR_ARG;
  if (M == 0 || D == 0) return IFLB200_OK;
  if (!res) return IFLB200_ERR_ARG;
  if (res_dtype != IFLB200_F32 && res_dtype != IFLB200_BF16) return IFLB200_ERR_DTYPE;
  if (y && !dtype_ok(y_dtype)) return IFLB200_ERR_DTYPE;
  if (D > kMaxWidth) return IFLB200_ERR_SHAPE;
  if (q && !qs) return IFLB200_ERR_ARG;
  if ((mod_scale == nullptr) != (mod_shift == nullptr)) return IFLB200_ERR_ARG;
  if (ld_res < D || (delta && ld_delta < D) || (q && ld_q < D) || (y && ld_y < D)) return IFLB200_ERR_ARG;
  ResNormArgs a;
  a.res = res; a.ld_res = ld_res; a.M = M; a.D = D;
  a.delta = delta_splits ? nullptr : reinterpret_cast<const __nv_bfloat16*>(delta);
  a.dpart = delta_splits ? reinterpret_cast<const float*>(delta) : nullptr;
  a.dsplits = delta_splits;
  a.ld_delta = ld_delta;
  a.drow = delta ? delta_row : nullptr; a.dcol = delta ? delta_col : nullptr;
  a.bias = delta ? bias : nullptr; a.gate = delta ? gate : nullptr;
  a.write_res = (write_res && delta) ? 1 : 0;
  a.layernorm = layernorm; a.weight = weight; a.beta = beta;
  a.mod_scale = mod_scale; a.mod_shift = mod_shift; a.mod_index = mod_index; a.eps = eps;
  a.q = reinterpret_cast<uint8_t*>(q); a.ld_q = ld_q; a.qs = qs;
  a.y = y; a.y_dtype = y_dtype; a.ld_y = ld_y;
  a.mirrors = mirrors;
  a.early = early_trigger_for(reinterpret_cast<cudaStream_t>(stream));
  bool mirrors_ok = true;
  for (int k = 0; k < kMaxMirrors; ++k) {
    a.q_mirror[k] = k < mirrors ? reinterpret_cast<uint8_t*>(q_mirrors[k]) : nullptr;
    a.qs_mirror[k] = k < mirrors ? qs_mirrors[k] : nullptr;
    if (k < mirrors && (!a.q_mirror[k] || !a.qs_mirror[k])) return IFLB200_ERR_ARG;
    if (k < mirrors && !aligned8(a.q_mirror[k])) mirrors_ok = false;
  }
  if (!mirrors_ok) return IFLB200_ERR_ALIGN;
  const bool tables_ok = (!a.dcol || aligned16(a.dcol)) && (!a.bias || aligned16(a.bias)) &&
                         (!a.gate || aligned16(a.gate)) && (!weight || aligned16(weight)) &&
                         (!beta || aligned16(beta)) && (!mod_scale || aligned16(mod_scale)) &&
                         (!mod_shift || aligned16(mod_shift));
  const bool fast = D % 8 == 0 && aligned16(res) && (ld_res * esize(res_dtype)) % 16 == 0 &&
                    (!delta || (aligned16(delta) && (ld_delta * (delta_splits ? 4 : 2)) % 16 == 0)) &&
                    (!q || (aligned8(q) && ld_q % 8 == 0)) &&
                    (!y || (aligned16(y) && (ld_y * esize(y_dtype)) % 16 == 0)) && tables_ok;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (delta_splits) {
    if (!fast || D > 8192) return IFLB200_ERR_SHAPE;
    if (res_dtype == IFLB200_F32) launch_resnorm_planes<float>(a, s);
    else launch_resnorm_planes<__nv_bfloat16>(a, s);
    return (int)cudaGetLastError();
  }
  // one affine after the norm, or none; per-row tables, a second output and a residual that is not
  // stored stay with the one-row-per-group kernels
  const bool modulated = mod_scale != nullptr;
  if (fast && res_dtype == IFLB200_BF16 && layernorm && q && !y && !mod_index && (write_res || !delta) &&
      !(modulated && (weight || beta)) && g_row_tpr_override == 0 &&
      launch_residual_norm_stream({res, ld_res, M, D, a.delta, ld_delta, a.drow, a.dcol, a.bias, a.gate,
                                   modulated ? mod_scale : weight, modulated ? mod_shift : beta, modulated, eps, a.q, ld_q, qs, a.early}, s))
    return (int)cudaGetLastError();
  if (res_dtype == IFLB200_F32) launch_resnorm<float>(a, fast, s);
  else launch_resnorm<__nv_bfloat16>(a, fast, s);
  return (int)cudaGetLastError();
}

extern "C" int iflb200_residual_norm_quant(void* res, int res_dtype, int64_t ld_res, int M, int D,
                                           const void* delta, int64_t ld_delta,
                                           const float* delta_row, const float* delta_col,
                                           const float* bias, const float* gate, int write_res,
                                           int layernorm, const float* weight, const float* beta,
                                           const float* mod_scale, const float* mod_shift,
                                           const int32_t* mod_index, float eps,
                                           void* q, int64_t ld_q, float* qs,
                                           void* y, int y_dtype, int64_t ld_y, void* stream) {
  return resnorm_impl(res, res_dtype, ld_res, M, D, delta, 0, ld_delta, delta_row, delta_col, bias, gate, write_res,
                      layernorm, weight, beta, mod_scale, mod_shift, mod_index, eps, q, ld_q, qs, y, y_dtype, ld_y, stream);
}

extern "C" int iflb200_residual_norm_quant_partials(void* res, int res_dtype, int64_t ld_res, int M, int D,
                                                    const float* delta_partials, int splits, int64_t ld_delta,
                                                    const float* delta_row, const float* delta_col,
                                                    const float* bias, const float* gate, int write_res,
                                                    int layernorm, const float* weight, const float* beta,
                                                    const float* mod_scale, const float* mod_shift,
                                                    const int32_t* mod_index, float eps,
                                                    void* q, int64_t ld_q, float* qs,
                                                    void* y, int y_dtype, int64_t ld_y, void* stream) {
  if (!delta_partials || splits < 1 || splits > 8) return IFLB200_ERR_ARG;
  return resnorm_impl(res, res_dtype, ld_res, M, D, delta_partials, splits, ld_delta, delta_row, delta_col, bias, gate,
                      write_res, layernorm, weight, beta, mod_scale, mod_shift, mod_index, eps, q, ld_q, qs, y, y_dtype,
                      ld_y, stream);
}

extern "C" int iflb200_residual_norm_quant_peers(void* res, int res_dtype, int64_t ld_res, int M, int D,
                                                 const float* delta_partials, int splits, int64_t ld_delta,
                                                 const float* delta_row, const float* delta_col, const float* bias,
                                                 const float* gate, int write_res, int layernorm, const float* weight,
                                                 const float* beta, const float* mod_scale, const float* mod_shift,
                                                 const int32_t* mod_index, float eps, void* q, int64_t ld_q, float* qs,
                                                 void* const* q_mirrors, float* const* qs_mirrors, int mirrors,
                                                 void* stream) {
  if (!delta_partials || splits < 1 || splits > 8) return IFLB200_ERR_ARG;
  return resnorm_impl(res, res_dtype, ld_res, M, D, delta_partials, splits, ld_delta, delta_row, delta_col, bias, gate,
                      write_res, layernorm, weight, beta, mod_scale, mod_shift, mod_index, eps, q, ld_q, qs, nullptr, 0,
                      0, stream, q_mirrors, qs_mirrors, mirrors);
}

#endif

#if IFLB200_ROW_PART == 1 || IFLB200_ROW_PART == -1
static int pack_grid(int64_t n) {
  int64_t ctas = (n + (int64_t)kPackThreads * 8 * 4 - 1) / ((int64_t)kPackThreads * 8 * 4);
  if (ctas < 1) ctas = 1;
  if (ctas > kPackMaxCtas) ctas = kPackMaxCtas;
  return (int)ctas;
}

// The one-launch form where it applies.
static bool launch_pack_cluster(const void* x, int64_t n, void* q, float* scale, cudaStream_t s) {
  if (n > kPackClusterMax || n % 8 || !aligned16(x) || !aligned8(q)) return false;
  const int nvec = (int)(n / 8);
  auto xv = reinterpret_cast<const uint4*>(x);
  auto qv = reinterpret_cast<uint2*>(q);
  auto go = [&](auto kernel, int ctas) {
    launch_dep(kernel, dim3(ctas), dim3(kPackClusterThreads), 0, s, 1, dependent_launch_for(1), xv, nvec, scale, qv);
  };
  const int per_thread = (nvec + 8 * kPackClusterThreads - 1) / (8 * kPackClusterThreads);  // on eight CTAs
  if (per_thread <= 1) go(pack_cluster_kernel<8, 1>, 8);
  else if (per_thread <= 2) go(pack_cluster_kernel<8, 2>, 8);
  else if (per_thread <= 4) go(pack_cluster_kernel<8, 4>, 8);
  else {
    static bool granted[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    if (!granted[dev]) {
      if (cudaFuncSetAttribute(pack_cluster_kernel<16, 4>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return false;
      granted[dev] = true;
    }
    go(pack_cluster_kernel<16, 4>, 16);
  }
  return true;
}

extern "C" size_t iflb200_pack_workspace_bytes(int64_t n) {
  return (size_t)pack_grid(n < 0 ? 0 : n) * sizeof(uint32_t);
}

extern "C" int iflb200_dynamic_pack_bf16_e4m3(const void* x, int64_t n, void* q, float* scale,
                                              void* workspace, size_t workspace_bytes,
                                              void* stream) {
  if (n <= 0 || !x || !q || !scale) return IFLB200_ERR_ARG;
  if (!workspace || workspace_bytes < iflb200_pack_workspace_bytes(n)) return IFLB200_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(x) & 1) || (reinterpret_cast<uintptr_t>(workspace) & 3))
    return IFLB200_ERR_ALIGN;
  const int grid = pack_grid(n);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (launch_pack_cluster(x, n, q, scale, s)) return (int)cudaGetLastError();
  uint32_t* partial = reinterpret_cast<uint32_t*>(workspace);
  launch_dep(amax_partial_kernel, dim3(grid), dim3(kPackThreads), 0, s, 1, dependent_launch_for(n >> 12), reinterpret_cast<const uint16_t*>(x), n, partial);
  // (n >> 12: dependent up to 2^23 elements; above, the first kernel directly behind a GEMM took 1.01 to 1.08 times as long.)
  // The pass over the maxima is the kernel before at any size, and it is short beside a GEMM: its
  // successor starts early however large the tensor is (4680 x 3072 15.2 -> 14.9 us).
  launch_dep(n <= kPackOnePass ? pack_kernel<true> : pack_kernel<false>, dim3(grid), dim3(kPackThreads), 0, s, 1, dependent_launch_for(0),
             reinterpret_cast<const uint16_t*>(x), n, partial, grid, nullptr, scale, reinterpret_cast<uint8_t*>(q));
  return (int)cudaGetLastError();
}

extern "C" int iflb200_pack_bf16_e4m3(const void* x, int64_t n, const float* scale, void* q,
                                      void* stream) {
  if (n < 0 || !scale) return IFLB200_ERR_ARG;
  if (n == 0) return IFLB200_OK;
  if (!x || !q) return IFLB200_ERR_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  launch_dep(pack_kernel<false>, dim3(pack_grid(n)), dim3(kPackThreads), 0, s, 1, dependent_launch_for(n >> 12), reinterpret_cast<const uint16_t*>(x), n, nullptr,
                                                    0, scale, nullptr, reinterpret_cast<uint8_t*>(q));
  return (int)cudaGetLastError();
}
// --------------------------------------------------------------------------------------------
// Dynamic pack for callers that cannot allocate.
//
// The dynamic pack needs a few hundred words of scratch (one partial maximum per CTA of the first
// kernel).  Hosts that drive this library from a fixed memory plan -- an embedded control loop
// whose device memory was carved up at start-up, a C or C++ runtime that has no caching
// allocator behind it, a real-time loop that cannot afford the device-wide stall of a
// cudaMalloc -- have nowhere to get that scratch from.  For them
// the scratch lives in the library image itself: a file-scope device array, resident on every GPU
// that loads the library until the process exits (4 KB).
//
// Host code must not pass the array's name to a kernel: on the host that name is only a
// stand-in symbol, not a device address.  The address is looked up once per device with
// cudaGetSymbolAddress while that device is current, and that pointer is what the kernels get.
// --------------------------------------------------------------------------------------------
static __device__ __align__(256) uint32_t g_pack_noalloc_scratch[kPackMaxCtas];

static int pack_noalloc_scratch(uint32_t** out) {
  static uint32_t* resolved[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= 64) return IFLB200_ERR_DEVICE;
  uint32_t* p = __atomic_load_n(&resolved[dev], __ATOMIC_ACQUIRE);
  if (p == nullptr) {
    // First call on this device (which is the current one): resolve the symbol.  Two host
    // threads racing here resolve the same address; the store is idempotent.
    void* addr = nullptr;
    e = cudaGetSymbolAddress(&addr, g_pack_noalloc_scratch);
    if (e != cudaSuccess) return (int)e;
    if (addr == nullptr) return IFLB200_ERR_DEVICE;
    p = reinterpret_cast<uint32_t*>(addr);
    __atomic_store_n(&resolved[dev], p, __ATOMIC_RELEASE);
  }
  *out = p;
  return IFLB200_OK;
}

extern "C" int iflb200_dynamic_pack_bf16_e4m3_noalloc(const void* x, int64_t n, void* q, float* scale,
                                                      void* stream) {
  if (n <= 0 || !x || !q || !scale) return IFLB200_ERR_ARG;
  if (n > IFLB200_PACK_NOALLOC_MAX_ELEMENTS) return IFLB200_ERR_TOO_LARGE;
  if (reinterpret_cast<uintptr_t>(x) & 1) return IFLB200_ERR_ALIGN;
  uint32_t* partial = nullptr;
  const int st = pack_noalloc_scratch(&partial);
  if (st != IFLB200_OK) return st;
  const int grid = pack_grid(n);  // <= kPackMaxCtas words of scratch, all written before they are read
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  launch_dep(amax_partial_kernel, dim3(grid), dim3(kPackThreads), 0, s, 1, dependent_launch_for(n >> 12), reinterpret_cast<const uint16_t*>(x), n, partial);
  launch_dep(n <= kPackOnePass ? pack_kernel<true> : pack_kernel<false>, dim3(grid), dim3(kPackThreads), 0, s, 1, dependent_launch_for(0),
             reinterpret_cast<const uint16_t*>(x), n, partial, grid, nullptr, scale, reinterpret_cast<uint8_t*>(q));
  return (int)cudaGetLastError();
}
#endif

