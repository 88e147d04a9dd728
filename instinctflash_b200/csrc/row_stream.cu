// Row kernels for many rows: the GELU quantiser of a feed-forward row and the residual + norm +
// quantiser of a residual row, as persistent CTAs.
//
// With one group of threads per row (row_ops.cu) every row reads its per-column float32 operands
// again: scale and bias are 8 bytes per element beside 3 bytes of HBM traffic in the GELU quantiser,
// five vectors are 20 bytes beside 7 in the residual kernel, all through L1.  Here a CTA stays on its
// SM and walks over rows with the operands in shared memory or in registers.
#include "row_stream.cuh"

#include "../../include/iflb200.h"
#include "launch.cuh"
#include "rowmath.cuh"

namespace iflb200 {
namespace {

// Eight elements as four packed pairs (the arithmetic below is two lanes per instruction throughout;
// keeping the pairs packed between the steps saves the register moves around them).
struct Eight {
  uint64_t p[4];
};
__device__ __forceinline__ Eight widen(const uint4& u, __nv_bfloat16) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  Eight e;
#pragma unroll
  for (int i = 0; i < 4; ++i) e.p[i] = pack2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xFFFF0000u));
  return e;
}
__device__ __forceinline__ Eight widen(const uint4& u, __half) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  Eight e;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    e.p[i] = pack2(f.x, f.y);
  }
  return e;
}
// A float32 vector in shared memory (stage_vector): the first four of every eight values, then the last
// four, so that a warp's 16-byte accesses are contiguous (32 bytes apart they collide in pairs of lanes).
__device__ __forceinline__ Eight lds_f32x8(uint32_t addr, int half_bytes) {
  Eight e;
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(e.p[0]), "=l"(e.p[1]) : "r"(addr));
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(e.p[2]), "=l"(e.p[3]) : "r"(addr + half_bytes));
  return e;
}
__device__ __forceinline__ void scale(Eight& v, float f) {
  const uint64_t f2 = pack2(f, f);
#pragma unroll
  for (int i = 0; i < 4; ++i) v.p[i] = mul2(v.p[i], f2);
}
__device__ __forceinline__ void mul(Eight& v, const Eight& f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) v.p[i] = mul2(v.p[i], f.p[i]);
}
__device__ __forceinline__ void mul_add(Eight& v, const Eight& f, const Eight& c) {
#pragma unroll
  for (int i = 0; i < 4; ++i) v.p[i] = fma2(v.p[i], f.p[i], c.p[i]);
}
__device__ __forceinline__ float max_abs(const Eight& v, float m) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a, b;
    unpack2(v.p[i], a, b);
    m = max_abs_f32(m, a, b);
  }
  return m;
}
__device__ __forceinline__ void store_codes(uint8_t* p, const Eight& v, float inv) {
  const uint64_t inv2 = pack2(inv, inv);
  float s[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) unpack2(mul2(v.p[i], inv2), s[2 * i], s[2 * i + 1]);
  *reinterpret_cast<uint2*>(p) = make_uint2(cvt_e4m3x4(s[0], s[1], s[2], s[3]), cvt_e4m3x4(s[4], s[5], s[6], s[7]));
}

// 16 bytes from global to shared memory, asynchronously; every thread reads back only what it copied.
__device__ __forceinline__ void copy16_async(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ uint4 lds16(uint32_t addr) {
  uint4 u;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "r"(addr) : "memory");
  return u;
}

// Copies a float32 vector of K elements to `dst` in shared memory, `plus` added, and moves `dst` on.
__device__ __forceinline__ void stage_vector(float*& dst, const float* src, int K, float plus) {
  for (int i = threadIdx.x * 4; i < K; i += blockDim.x * 4) {
    float4 f = *reinterpret_cast<const float4*>(src + i);
    if (plus != 0.0f) f = make_float4(__fadd_rn(f.x, plus), __fadd_rn(f.y, plus), __fadd_rn(f.z, plus), __fadd_rn(f.w, plus));
    *reinterpret_cast<float4*>(dst + ((i & 4) ? K / 2 : 0) + (i >> 3) * 4) = f;
  }
  dst += K;
}

// Meeting of one group of `threads` threads (whole warps, barrier `id`) over a value per warp; `slots` are
// the group's, kMaxWarps of them, the neutral element (0) beyond its warps.
constexpr int kMaxWarps = 16;
constexpr int kMaxGroups = 12;  // one named barrier each, barrier 0 is the CTA's
template <bool IS_MAX>
__device__ __forceinline__ float group_meet(float v, float* slots, int warp, int id, int threads) {
  if (IS_MAX) {
    v = warp_max_abs_f32(v);
  } else {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  }
  if ((threadIdx.x & 31) == 0) slots[warp] = v;
  named_bar_sync(id, threads);
  const float4* q = reinterpret_cast<const float4*>(slots);
  float4 s = q[0];
  const int quads = (threads + 127) / 128;
#pragma unroll
  for (int i = 1; i < kMaxWarps / 4; ++i) {
    if (i < quads) {
      const float4 e = q[i];
      s.x = IS_MAX ? max_f32(s.x, e.x) : __fadd_rn(s.x, e.x);
      s.y = IS_MAX ? max_f32(s.y, e.y) : __fadd_rn(s.y, e.y);
      s.z = IS_MAX ? max_f32(s.z, e.z) : __fadd_rn(s.z, e.z);
      s.w = IS_MAX ? max_f32(s.w, e.w) : __fadd_rn(s.w, e.w);
    }
  }
  return IS_MAX ? max_f32(max_f32(s.x, s.y), max_f32(s.z, s.w)) : __fadd_rn(__fadd_rn(s.x, s.y), __fadd_rn(s.z, s.w));
}

// A row belongs to a group of `tg` threads with kChunks chunks of eight columns each; a CTA (one per
// SM) holds as many groups as its threads and its shared memory allow, or as many as spread the rows
// evenly over its turns.  Calls with fewer rows than there are groups are left to the other kernels,
// below that SMs would stay empty; at about one row per group the stream kernels are already ahead
// (GELU 500 x 14336 15.9 -> 11.8 us, residual 600 x 5120 14.3 -> 13.2).
constexpr int kChunks = 4;
constexpr size_t kSmemLimit = 224 * 1024;
struct StreamGeom {
  int tg = 0, groups = 0;
  size_t smem = 0;
};
StreamGeom stream_geom(int M, int K, int vectors, int row_bytes, int max_threads, int sms, int chunks = kChunks) {
  StreamGeom g;
  g.tg = ((K / 8 + chunks - 1) / chunks + 31) / 32 * 32;
  g.groups = max_threads / g.tg;
  if (g.groups > kMaxGroups) g.groups = kMaxGroups;
  const size_t fixed = (size_t)vectors * K * 4;
  while (g.groups > 0 && fixed + (size_t)g.groups * row_bytes > kSmemLimit) --g.groups;
  if (g.groups < 2 || M < g.groups * sms) {
    g.groups = 0;
    return g;
  }
  const int turns = (M + g.groups * sms - 1) / (g.groups * sms);
  g.groups = (M + turns * sms - 1) / (turns * sms);
  g.smem = fixed + (size_t)g.groups * row_bytes;
  return g;
}
template <auto kKernel, typename KArgs>
bool launch_stream(const StreamGeom& g, int sms, cudaStream_t s, const KArgs& a) {
  static bool granted[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (!granted[dev]) {
    if (cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit) != cudaSuccess) return false;
    granted[dev] = true;
  }
  launch_dep(kKernel, dim3(sms), dim3(g.tg * g.groups), g.smem, s, 1, dependent_launch_for(a.rows_of_call(), a.many()), a, g.tg);
  return true;
}

// --------------------------------------------------------------------------------------------
// GELU quantiser: q[m] = e4m3(gelu(x[m] * row[m] * col + bias) / s[m]).
//
// Bytes per element: 2 in, 1 out; two special-function operations (ex2, rcp: 16 a clock and SM) and about
// 12 issue slots, so that the special-function unit and HBM finish close together (4680 x 14336: 30 us
// each).  One row per group of threads: while one group meets at its row maximum, the others
// compute.  The row after the one being computed is on its way into a private shared-memory slot of the
// thread that will read it (cp.async; no barrier between copy and use), which keeps a row per group
// in flight without registers.  Scale and bias vectors are staged once per CTA: read from L1 for every
// row they were 8 bytes beside 3 of HBM traffic.  4680 x 14336: 106 -> 62 us, 16384 x 13824: 343 -> 183,
// the special-function unit busy for half of it.
// --------------------------------------------------------------------------------------------
template <typename XT, bool BIAS, int THREADS, int CHUNKS>
__global__ void __launch_bounds__(THREADS, 1) gelu_quant_stream_kernel(const GeluStreamArgs a, int tg) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ __align__(16) float red[2][kMaxGroups][kMaxWarps];
  const int g = threadIdx.x / tg, t = threadIdx.x - g * tg, groups = blockDim.x / tg;
  const uint32_t s_col = smem_u32(smem) + t * 16, s_bias = s_col + a.K * 4;
  const int half_bytes = a.K * 2;
  const uint32_t slot = smem_u32(smem) + a.K * (BIAS ? 8 : 4) + g * a.K * 2 + t * 16;
  const XT* x = reinterpret_cast<const XT*>(a.x) + t * 8;
  for (int i = threadIdx.x; i < 2 * kMaxGroups * kMaxWarps; i += blockDim.x) (&red[0][0][0])[i] = 0.0f;

  if (a.early) grid_launch_dependents();
  grid_dependency_wait();  // inputs may come from the kernel before this one in the stream
  if (!a.early) grid_launch_dependents();
  const int stride = gridDim.x * groups;
  int m = blockIdx.x * groups + g;
  float rs = 1.0f;
  auto fetch = [&](int row, int it) { copy16_async(slot + it * tg * 16, x + (int64_t)row * a.ld_x + it * tg * 8); };
  if (m < a.M) {
#pragma unroll
    for (int it = 0; it < CHUNKS; ++it)
      if ((it * tg + t) * 8 < a.K) fetch(m, it);
    rs = a.row[m];
  }
  copy_commit();
  float* dst = reinterpret_cast<float*>(smem);
  stage_vector(dst, a.col, a.K, 0.0f);
  if (BIAS) stage_vector(dst, a.bias, a.K, 0.0f);
  __syncthreads();

  for (int turn = 0; m < a.M; m += stride, turn ^= 1) {
    const int next = m + stride;
    const bool more = next < a.M;
    const float rs_next = more ? a.row[next] : 1.0f;
    copy_wait_all();
    Eight v[CHUNKS];
    float amax = 0.0f;
#pragma unroll
    for (int it = 0; it < CHUNKS; ++it) {
      if ((it * tg + t) * 8 < a.K) {
        v[it] = widen(lds16(slot + it * tg * 16), XT());
        if (more) fetch(next, it);  // the slot has been read by the only thread that uses it
        scale(v[it], rs);
        if (BIAS) mul_add(v[it], lds_f32x8(s_col + it * tg * 16, half_bytes), lds_f32x8(s_bias + it * tg * 16, half_bytes));
        else mul(v[it], lds_f32x8(s_col + it * tg * 16, half_bytes));
#pragma unroll
        for (int i = 0; i < 4; ++i) v[it].p[i] = gelu_tanh_ref2(v[it].p[i]);
        amax = max_abs(v[it], amax);
      }
    }
    copy_commit();
    // two arrays in turn: a warp may be one row ahead
    amax = group_meet<true>(amax, red[turn][g], t >> 5, 1 + g, tg);
    float scale_out, inv;
    quant_scales(amax, scale_out, inv);
    if (t == 0) a.qs[m] = scale_out;
    uint8_t* q = a.q + (int64_t)m * a.ld_q + t * 8;
#pragma unroll
    for (int it = 0; it < CHUNKS; ++it)
      if ((it * tg + t) * 8 < a.K) store_codes(q + it * tg * 8, v[it], inv);
    rs = rs_next;
  }
}

template <typename XT, int THREADS, int CHUNKS>
bool gelu_form(const GeluStreamArgs& a, int sms, cudaStream_t s) {
  const StreamGeom g = stream_geom(a.M, a.K, a.bias ? 2 : 1, a.K * 2, THREADS, sms, CHUNKS);
  if (g.groups == 0) return false;
  return a.bias ? launch_stream<gelu_quant_stream_kernel<XT, true, THREADS, CHUNKS>>(g, sms, s, a)
                : launch_stream<gelu_quant_stream_kernel<XT, false, THREADS, CHUNKS>>(g, sms, s, a);
}
template <typename XT>
bool gelu_width(const GeluStreamArgs& a, int sms, cudaStream_t s) {
  // two groups of 448 threads hold rows of up to 14336 columns with eight more registers a thread; wider rows are
  // faster with eight chunks on half the threads (16384 x 16384 221 -> 207 us; 16384 x 13824 is not, 183 -> 199)
  return a.K <= 14336 ? gelu_form<XT, 896, 4>(a, sms, s) : gelu_form<XT, 512, 8>(a, sms, s);
}

// --------------------------------------------------------------------------------------------
// Residual update + layer norm + quantiser of a bf16 residual stream (7 bytes per element with a
// delta, 3 without), the row kernel of the diffusion blocks:
//     res += fma(delta * drow, dcol, bias) * gate;   y = norm(res) * scale + shift;   q, s = e4m3(y)
// Bound by HBM and by the shared-memory port that delivers the vectors (20 bytes per element, 0.8 of the
// port's cycles): 16384 x 5120 217 -> 111 us (5.3 TB/s; 3 bytes per element, no vectors: 112 -> 50),
// 4680 x 3072 38 -> 23.5.
// The same structure: the residual and delta rows of the next turn are fetched into private slots, the
// five vectors are in shared memory, the three meetings of a row (mean, variance, maximum) cost the
// CTA's other groups nothing.
// --------------------------------------------------------------------------------------------
constexpr int kResNormThreads = 640, kResNormMore = 768;

template <bool DELTA, bool GATE, bool AFFINE, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) residual_norm_stream_kernel(const ResNormStreamArgs a, int tg) {
  constexpr int kVectors = (DELTA ? 2 : 0) + (GATE ? 1 : 0) + (AFFINE ? 2 : 0);
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ __align__(16) float red[3][kMaxGroups][kMaxWarps];
  const int g = threadIdx.x / tg, t = threadIdx.x - g * tg, groups = blockDim.x / tg;
  const uint32_t vec0 = smem_u32(smem) + t * 16;
  const int half_bytes = a.D * 2;
  const uint32_t s_dcol = vec0, s_bias = vec0 + a.D * 4, s_gate = vec0 + a.D * 8;
  const uint32_t s_scale = vec0 + a.D * 4 * (kVectors - 2), s_shift = s_scale + a.D * 4;
  const uint32_t slot_res = smem_u32(smem) + a.D * 4 * kVectors + g * a.D * (DELTA ? 4 : 2) + t * 16;
  const uint32_t slot_delta = slot_res + a.D * 2;
  __nv_bfloat16* res = reinterpret_cast<__nv_bfloat16*>(a.res) + t * 8;
  const float fD = (float)a.D;
  for (int i = threadIdx.x; i < 3 * kMaxGroups * kMaxWarps; i += blockDim.x) (&red[0][0][0])[i] = 0.0f;

  if (a.early) grid_launch_dependents();
  grid_dependency_wait();  // inputs may come from the kernel before this one in the stream
  if (!a.early) grid_launch_dependents();
  const int stride = gridDim.x * groups;
  int m = blockIdx.x * groups + g;
  float rs = 1.0f;
  auto fetch = [&](int row, int it) {
    copy16_async(slot_res + it * tg * 16, res + (int64_t)row * a.ld_res + it * tg * 8);
    if (DELTA) copy16_async(slot_delta + it * tg * 16, a.delta + (int64_t)row * a.ld_delta + (it * tg + t) * 8);
  };
  if (m < a.M) {
#pragma unroll
    for (int it = 0; it < kChunks; ++it)
      if ((it * tg + t) * 8 < a.D) fetch(m, it);
    if (DELTA) rs = a.drow[m];
  }
  copy_commit();
  float* dst = reinterpret_cast<float*>(smem);
  if (DELTA) {
    stage_vector(dst, a.dcol, a.D, 0.0f);
    stage_vector(dst, a.bias, a.D, 0.0f);
  }
  if (GATE) stage_vector(dst, a.gate, a.D, 0.0f);
  if (AFFINE) {
    stage_vector(dst, a.scale, a.D, a.scale_plus_one ? 1.0f : 0.0f);
    stage_vector(dst, a.shift, a.D, 0.0f);
  }
  __syncthreads();

  for (; m < a.M; m += stride) {
    const int next = m + stride;
    const bool more = next < a.M;
    const float rs_next = DELTA && more ? a.drow[next] : 1.0f;
    copy_wait_all();
    Eight x[kChunks];
    uint64_t acc = 0;
#pragma unroll
    for (int it = 0; it < kChunks; ++it) {
      if ((it * tg + t) * 8 < a.D) {
        x[it] = widen(lds16(slot_res + it * tg * 16), __nv_bfloat16());
        if (DELTA) {
          Eight d = widen(lds16(slot_delta + it * tg * 16), __nv_bfloat16());
          if (more) fetch(next, it);  // the slots have been read by the only thread that uses them
          scale(d, rs);
          mul_add(d, lds_f32x8(s_dcol + it * tg * 16, half_bytes), lds_f32x8(s_bias + it * tg * 16, half_bytes));
          if (GATE) {
            const Eight gate = lds_f32x8(s_gate + it * tg * 16, half_bytes);
#pragma unroll
            for (int i = 0; i < 4; ++i) x[it].p[i] = fma2(d.p[i], gate.p[i], x[it].p[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) x[it].p[i] = add2(x[it].p[i], d.p[i]);
          }
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {  // the residual is stored as bf16, and goes on as what was stored
            float lo, hi;
            unpack2(x[it].p[i], lo, hi);
            const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
          }
          const uint4 packed = make_uint4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<uint4*>(res + (int64_t)m * a.ld_res + it * tg * 8) = packed;
          x[it] = widen(packed, __nv_bfloat16());
        } else if (more) {
          fetch(next, it);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) acc = add2(acc, x[it].p[i]);
      }
    }
    copy_commit();
    float s0, s1;
    unpack2(acc, s0, s1);
    const float mean = div_full(group_meet<false>(__fadd_rn(s0, s1), red[0][g], t >> 5, 1 + g, tg), fD);
    const uint64_t minus = pack2(-mean, -mean);
    acc = 0;
#pragma unroll
    for (int it = 0; it < kChunks; ++it) {
      if ((it * tg + t) * 8 < a.D) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // x - mean == x + (-mean)
          x[it].p[i] = add2(x[it].p[i], minus);
          acc = fma2(x[it].p[i], x[it].p[i], acc);
        }
      }
    }
    unpack2(acc, s0, s1);
    const float var = div_full(group_meet<false>(__fadd_rn(s0, s1), red[1][g], t >> 5, 1 + g, tg), fD);
    const float rstd = rsqrt_approx_ftz(__fadd_rn(var, a.eps));
    float amax = 0.0f;
#pragma unroll
    for (int it = 0; it < kChunks; ++it) {
      if ((it * tg + t) * 8 < a.D) {
        scale(x[it], rstd);
        if (AFFINE) mul_add(x[it], lds_f32x8(s_scale + it * tg * 16, half_bytes), lds_f32x8(s_shift + it * tg * 16, half_bytes));
        amax = max_abs(x[it], amax);
      }
    }
    amax = group_meet<true>(amax, red[2][g], t >> 5, 1 + g, tg);
    float scale_out, inv;
    quant_scales(amax, scale_out, inv);
    if (t == 0) a.qs[m] = scale_out;
    uint8_t* q = a.q + (int64_t)m * a.ld_q + t * 8;
#pragma unroll
    for (int it = 0; it < kChunks; ++it)
      if ((it * tg + t) * 8 < a.D) store_codes(q + it * tg * 8, x[it], inv);
    rs = rs_next;
  }
}

template <bool DELTA, bool GATE, bool AFFINE, int THREADS>
bool resnorm_launch(const ResNormStreamArgs& a, const StreamGeom& g, int sms, cudaStream_t s) {
  return g.groups != 0 && launch_stream<residual_norm_stream_kernel<DELTA, GATE, AFFINE, THREADS>>(g, sms, s, a);
}
template <bool DELTA, bool GATE, bool AFFINE>
bool resnorm_form(const ResNormStreamArgs& a, int sms, cudaStream_t s) {
  auto geom = [&](int threads) {
    return stream_geom(a.M, a.D, (DELTA ? 2 : 0) + (GATE ? 1 : 0) + (AFFINE ? 2 : 0), a.D * (DELTA ? 4 : 2), threads, sms);
  };
  const StreamGeom g = geom(kResNormThreads);
  if constexpr (DELTA) {
    // More groups on fewer registers a thread where the rows then fill the turns better, by one row place in twenty at
    // least: 4680 x 3072 takes four turns of eight rows an SM instead of six of six, 26.9 -> 23.5 us with a gate and 24.3
    // -> 21.0 without, and of 59 other sizes none more than 2 % slower. With the same places the spills cost more (16384 x 5120 107 -> 115).
    const StreamGeom more = geom(kResNormMore);
    auto places = [&](const StreamGeom& x) { return (a.M + x.groups * sms - 1) / (x.groups * sms) * x.groups; };
    if (g.groups != 0 && more.groups > g.groups && places(more) * 20 <= places(g) * 19)
      return resnorm_launch<DELTA, GATE, AFFINE, kResNormMore>(a, more, sms, s);
  }
  return resnorm_launch<DELTA, GATE, AFFINE, kResNormThreads>(a, g, sms, s);
}

// --------------------------------------------------------------------------------------------
// QKV consumer of a diffusion block (iflb200_wan_qkv): dequantise, RMS norm of Q and K over their full
// width, rotate pairs (2j, 2j+1), store Q densely and K / V into pool rows.
//
// 2 bytes per element in, 2 out.  A group takes the parts (Q, K, V) of a row in turn; slots as above, the
// vectors of all parts (eight of D floats) stay in shared memory.  The angles of a token are
// shared by its heads and by Q and K: the group computes one sine and cosine per pair of a head, into a
// table that the first meeting of the row makes visible.  4680 x 9216: 61.6 -> 43.7 us with one
// CTA per (row, part) before, 16384 x 15360: 367 -> 232 (4.3 TB/s, issue slots 62 % busy).
// --------------------------------------------------------------------------------------------
constexpr int kWanThreads = 768;

template <typename OT>
__device__ __forceinline__ uint4 narrow(const Eight& v);
template <>
__device__ __forceinline__ uint4 narrow<__nv_bfloat16>(const Eight& v) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float lo, hi;
    unpack2(v.p[i], lo, hi);
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
template <>
__device__ __forceinline__ uint4 narrow<__half>(const Eight& v) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float lo, hi;
    unpack2(v.p[i], lo, hi);
    const __half2 h = __floats2half2_rn(lo, hi);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

template <typename OT>
__global__ void __launch_bounds__(kWanThreads, 1) wan_qkv_stream_kernel(const WanStreamArgs a, int tg) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ __align__(16) float red[2][kMaxGroups][kMaxWarps];
  const int D = a.D;
  const int g = threadIdx.x / tg, t = threadIdx.x - g * tg, groups = blockDim.x / tg;
  const int half_bytes = D * 2, step = a.bias ? 8 : 4;  // bytes of a part's vectors per column
  const uint32_t vec0 = smem_u32(smem) + t * 16;
  const uint32_t s_qn = vec0 + a.parts * D * step, s_kn = s_qn + (a.q_norm ? D * 4 : 0);
  const uint32_t slot = s_kn + (a.k_norm ? D * 4 : 0) + g * D * 2;
  // cosines, then sines, of the pairs of a head: a table per group, behind the slots
  float* cosines = reinterpret_cast<float*>(smem + (slot - t * 16 - g * D * 2 - smem_u32(smem)) + groups * D * 2) + g * a.HD;
  const int pair0 = (t * 8 % a.HD) >> 1;           // of the thread's first chunk
  const bool same_pairs = tg * 8 % a.HD == 0;      // and of all its chunks
  const __nv_bfloat16* raw = reinterpret_cast<const __nv_bfloat16*>(a.raw) + t * 8;
  for (int i = threadIdx.x; i < 2 * kMaxGroups * kMaxWarps; i += blockDim.x) (&red[0][0][0])[i] = 0.0f;

  grid_dependency_wait();  // inputs may come from the kernel before this one in the stream
  grid_launch_dependents();
  const int stride = gridDim.x * groups;
  int row = blockIdx.x * groups + g;
  auto fetch = [&](int r, int part, int it) {
    copy16_async(slot + it * tg * 16, raw + (int64_t)r * a.ld_raw + (int64_t)part * D + it * tg * 8);
  };
  // the angle of pair t of a head (tg covers the pairs): its frequency stays here, the position of the next
  // row's token is read a row ahead
  const bool rope = a.inv_freq != nullptr, turns_pair = rope && t < a.HD / 2;
  const float freq = turns_pair ? a.inv_freq[t] : 0.0f;
  const float* pos = turns_pair ? a.pos + a.sections[t] : nullptr;
  float rs = 1.0f, at = 0.0f;
  if (row < a.rows) {
#pragma unroll
    for (int it = 0; it < kChunks; ++it)
      if ((it * tg + t) * 8 < D) fetch(row, 0, it);
    if (a.row) rs = a.row[row];
    if (turns_pair) at = pos[(int64_t)(row % a.tokens) * a.ld_pos];
  }
  copy_commit();
  float* dst = reinterpret_cast<float*>(smem);
  for (int p = 0; p < a.parts; ++p) {
    stage_vector(dst, a.col + (int64_t)p * D, D, 0.0f);
    if (a.bias) stage_vector(dst, a.bias + (int64_t)p * D, D, 0.0f);
  }
  if (a.q_norm) stage_vector(dst, a.q_norm, D, 0.0f);
  if (a.k_norm) stage_vector(dst, a.k_norm, D, 0.0f);
  __syncthreads();

  int turn = 0;
  int b = 0, tok = 0;
  for (int part = 0; row < a.rows;) {
    if (part == 0) {
      b = row / a.tokens;
      tok = row - b * a.tokens;
    }
    const bool last = part + 1 == a.parts, more = !last || row + stride < a.rows;
    const int next_row = last ? row + stride : row, next_part = last ? 0 : part + 1;
    const bool norm = part == 0 ? a.q_norm != nullptr : (part == 1 && a.k_norm != nullptr);
    if (part == 0 && turns_pair) {  // for Q and K of this row
      const float ang = __fmul_rn(at, freq);
      cosines[t] = cosf(ang);
      cosines[a.HD / 2 + t] = sinf(ang);
    }
    float rs_next = rs;
    if (last && more) {
      if (a.row) rs_next = a.row[next_row];
      if (turns_pair) at = pos[(int64_t)(next_row % a.tokens) * a.ld_pos];
    }
    const uint32_t s_col = vec0 + part * D * step, s_bias = s_col + D * 4;
    copy_wait_all();
    Eight x[kChunks];
    uint64_t acc = 0;
#pragma unroll
    for (int it = 0; it < kChunks; ++it) {
      if ((it * tg + t) * 8 < D) {
        x[it] = widen(lds16(slot + it * tg * 16), __nv_bfloat16());
        if (more) fetch(next_row, next_part, it);  // the slot has been read by the only thread that uses it
        if (a.row) scale(x[it], rs);
        if (a.bias) mul_add(x[it], lds_f32x8(s_col + it * tg * 16, half_bytes), lds_f32x8(s_bias + it * tg * 16, half_bytes));
        else mul(x[it], lds_f32x8(s_col + it * tg * 16, half_bytes));
#pragma unroll
        for (int i = 0; i < 4; ++i) acc = fma2(x[it].p[i], x[it].p[i], acc);
      }
    }
    copy_commit();
    if (norm) {
      float s0, s1;
      unpack2(acc, s0, s1);
      const float sum = group_meet<false>(__fadd_rn(s0, s1), red[turn][g], t >> 5, 1 + g, tg);
      const float rstd = rsqrt_approx_ftz(__fadd_rn(div_full(sum, (float)D), a.eps));
      const uint32_t s_w = part == 0 ? s_qn : s_kn;
#pragma unroll
      for (int it = 0; it < kChunks; ++it) {
        if ((it * tg + t) * 8 < D) {
          scale(x[it], rstd);
          mul(x[it], lds_f32x8(s_w + it * tg * 16, half_bytes));
        }
      }
      turn ^= 1;
    } else if (rope && part == 0) {
      named_bar_sync(1 + g, tg);
    }
    if (rope && part < 2) {
      float4 co, si;
#pragma unroll
      for (int it = 0; it < kChunks; ++it) {
        if ((it * tg + t) * 8 < D) {
          if (it == 0 || !same_pairs) {  // the chunk lies inside one head
            const int j = it == 0 ? pair0 : ((it * tg + t) * 8 % a.HD) >> 1;
            co = *reinterpret_cast<const float4*>(cosines + j);
            si = *reinterpret_cast<const float4*>(cosines + a.HD / 2 + j);
          }
          const float c[4] = {co.x, co.y, co.z, co.w}, n[4] = {si.x, si.y, si.z, si.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            // (a, b) <- (a cos - b sin, b cos + a sin): sine products rounded, cosine products fused
            float lo, hi;
            unpack2(x[it].p[i], lo, hi);
            x[it].p[i] = fma2(x[it].p[i], pack2(c[i], c[i]), mul2(pack2(hi, lo), pack2(-n[i], n[i])));
          }
        }
      }
    }
    if (rope && last) named_bar_sync(1 + g, tg);  // the table has been read: the next row may replace it
    OT* out;
    if (part == 0) {
      out = reinterpret_cast<OT*>(a.q) + (int64_t)row * a.ld_q;
    } else {
      const int64_t place = a.slots ? a.slots[tok] : tok;
      out = part == 1 ? reinterpret_cast<OT*>(a.k) + (int64_t)b * a.sk_b + place * a.sk_s
                      : reinterpret_cast<OT*>(a.v) + (int64_t)b * a.sv_b + place * a.sv_s;
    }
#pragma unroll
    for (int it = 0; it < kChunks; ++it)
      if ((it * tg + t) * 8 < D) *reinterpret_cast<uint4*>(out + (it * tg + t) * 8) = narrow<OT>(x[it]);
    row = next_row;
    part = next_part;
    rs = rs_next;
  }
}

}  // namespace

bool launch_gelu_quant_stream(const GeluStreamArgs& a, bool half, cudaStream_t s) {
  const int sms = device_sm_count();
  if (sms == 0 || !a.row || !a.col || a.K <= 1024 || a.K > 16384) return false;
  return half ? gelu_width<__half>(a, sms, s) : gelu_width<__nv_bfloat16>(a, sms, s);
}

bool launch_residual_norm_stream(const ResNormStreamArgs& a, cudaStream_t s) {
  const int sms = device_sm_count();
  if (sms == 0 || a.D <= 1024 || a.D > 8192 || (a.scale != nullptr) != (a.shift != nullptr)) return false;
  if (!a.delta) return a.scale ? resnorm_form<false, false, true>(a, sms, s) : resnorm_form<false, false, false>(a, sms, s);
  if (!a.drow || !a.dcol || !a.bias || !a.scale) return false;
  return a.gate ? resnorm_form<true, true, true>(a, sms, s) : resnorm_form<true, false, true>(a, sms, s);
}

bool launch_wan_qkv_stream(const WanStreamArgs& a, bool half, cudaStream_t s) {
  const int sms = device_sm_count();
  if (sms == 0 || !a.col || a.D <= 1024 || a.D > 16384 || a.HD % 8) return false;
  const int vectors = a.parts * (a.bias ? 2 : 1) + (a.q_norm ? 1 : 0) + (a.k_norm ? 1 : 0);
  StreamGeom g = stream_geom(a.rows, a.D, vectors, a.D * 2 + a.HD * 4, kWanThreads, sms);
  if (g.groups == 0 || g.tg < a.HD / 2) return false;
  return half ? launch_stream<wan_qkv_stream_kernel<__half>>(g, sms, s, a) : launch_stream<wan_qkv_stream_kernel<__nv_bfloat16>>(g, sms, s, a);
}

}  // namespace iflb200
