// Merge of split-KV attention partials with the per-token e4m3 quantiser of the merged row: the
// producer of the O projection's FP8 input in the reference engines
// (instinctflash/kernels/attention.py:109-145, _attn_combine with QUANT).
//
// The attention kernel leaves, per split sp, batch b, KV head and query row r = token * GROUP + h,
// an unnormalised output vector PO (BLOCK_D floats, BLOCK_D = head_dim rounded up to a power of
// two), the running maximum PM and the running sum PL.  For one token this kernel computes, for
// every query head and every d < head_dim, in the order of the reference's source:
//     m   = max over sp of PM                       (max.f32, starting from -inf)
//     w   = ex2.approx.ftz(PM[sp] - m)
//     l   = fma(w, PL[sp], l)                       (from 0, splits in order)
//     acc = fma(w, PO[sp][d], acc)                  (from 0, splits in order)
//     out = div.full(acc, l)
// stores out in O's type (optional), and quantises the token's full row of heads * head_dim
// values with one scale: amax = max(max |out|, 1e-8), qs = div.full(amax, 448),
// code = cvt.rn.satfinite.e4m3(out * div.full(448, amax)).  The row maximum is order-independent,
// every other operation is per element, so codes and scales equal the reference's bit for bit.
//
// One CTA per (token, batch); a thread owns chunks of four consecutive d of one head.  HBM-bound:
// splits * (4 * BLOCK_D + 8) bytes in per (head, token), head_dim * (1 + sizeof(O)) bytes out.
#include <cuda_runtime.h>

#include "../../include/iflb200.h"
#include "launch.cuh"
#include "rowmath.cuh"

namespace iflb200 {

constexpr int kCombineThreads = 512;
constexpr int kCombineMaxCluster = 8;
constexpr int kCombineIters = 4;  // 512 threads x 4 chunks x 4 values = 8192 values per token row

struct CombineArgs {
  const float* po;
  const float* pm;
  const float* pl;
  void* o;
  int o_dtype;
  int64_t sob, sot, soh;
  uint8_t* q;
  int64_t ld_q;
  float* qs;
  int tokens, batch, group, heads_kv, head_dim, block_d, splits, cluster;
};

// The partials of a chunk come in groups of kGroup splits, every load of a group issued before the first is
// used: with at most kGroup = 8 splits (the engines' geometry) a token is one memory round trip.  Split by split
// it was a chain of dependent ones (50 tokens x 8 heads x 256, 8 splits: 4.5 -> 3.1 us between launches).
// Groups of four where there are tokens for two CTAs per SM, whose phases then cover each other.
// CL: a cluster of a.cluster CTAs shares a token's chunks -- for few tokens, whose CTAs would each pull hundreds of
// KB through one SM (28 tokens x 16 heads x 256, 12 splits: 7.9 us with one CTA per token) -- and the
// row maximum meets in distributed shared memory.
template <int IT, bool CL, int kGroup>
__global__ void __launch_bounds__(kCombineThreads, kGroup == 4 ? 2 : 1) attn_combine_quant_kernel(const CombineArgs a) {
  const int threads = blockDim.x;
  if (CL) cluster_arrive();  // this CTA runs: its shared memory may be written from now on
  __shared__ float red[kCombineThreads / 32];
  __shared__ float maxima[kCombineMaxCluster];
  const int t = CL ? blockIdx.x / a.cluster : blockIdx.x, b = blockIdx.y;
  const int chunks_per_head = a.head_dim / 4;
  const int heads = a.group * a.heads_kv;
  const int all = heads * chunks_per_head;
  const int share = CL ? (all + a.cluster - 1) / a.cluster : all;
  const int first = CL ? (int)cluster_ctarank() * share : 0;
  const int total = min(all, first + share);  // this CTA's chunks: [first, total)
  const int n_rows = a.tokens * a.group;
  const int64_t plane = (int64_t)a.batch * a.heads_kv * n_rows;  // rows of one split
  // where the first chunk's partials are, worked out ahead of the wait, which its divisions used to follow (708 tokens x 8 x 64, 14
  // splits 6.54 -> 5.91 us behind one another; 0.96 of the time over 41 sizes)
  const auto place = [&](int c, int& head, int& d, int64_t& row) {
    head = c / chunks_per_head;
    d = (c - head * chunks_per_head) * 4;
    const int kvh = head / a.group, h = head - kvh * a.group;
    row = ((int64_t)b * a.heads_kv + kvh) * n_rows + (int64_t)t * a.group + h;
  };
  int head0, d0;
  int64_t row0;
  place(first + threadIdx.x, head0, d0, row0);
  asm volatile("" : "+r"(head0), "+r"(d0), "+l"(row0));
  grid_dependency_wait();  // the partials come from the kernel before this one in the stream
  grid_launch_dependents();
  float out[IT][4];
  float amax = 0.0f;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c = first + it * threads + threadIdx.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) out[it][i] = 0.0f;
    if (c < total) {
      int head = head0, d = d0;
      int64_t row = row0;
      if (it > 0) place(c, head, d, row);
      const float *pm = a.pm + row, *pl = a.pl + row, *po = a.po + row * a.block_d + d;
      float gm[kGroup], gl[kGroup];
      float4 gv[kGroup];
      auto load = [&](int s0) {
#pragma unroll
        for (int j = 0; j < kGroup; ++j) {
          if (s0 + j < a.splits) {
            gm[j] = __ldg(pm + (s0 + j) * plane);
            gl[j] = __ldg(pl + (s0 + j) * plane);
            gv[j] = __ldg(reinterpret_cast<const float4*>(po + (s0 + j) * plane * a.block_d));
          }
        }
      };
      load(0);
      float m = __uint_as_float(0xFF800000u);  // -inf
#pragma unroll
      for (int j = 0; j < kGroup; ++j)
        if (j < a.splits) m = max_f32(m, gm[j]);
      for (int sp = kGroup; sp < a.splits; ++sp) m = max_f32(m, __ldg(pm + sp * plane));
      float l = 0.0f, acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      for (int s0 = 0; s0 < a.splits; s0 += kGroup) {
        if (s0 > 0) load(s0);
#pragma unroll
        for (int j = 0; j < kGroup; ++j) {
          if (s0 + j < a.splits) {
            const float w = ex2_approx_ftz(__fsub_rn(gm[j], m));
            l = __fmaf_rn(w, gl[j], l);
            acc[0] = __fmaf_rn(w, gv[j].x, acc[0]);
            acc[1] = __fmaf_rn(w, gv[j].y, acc[1]);
            acc[2] = __fmaf_rn(w, gv[j].z, acc[2]);
            acc[3] = __fmaf_rn(w, gv[j].w, acc[3]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        out[it][i] = div_full(acc[i], l);
        amax = max_f32(amax, fabsf(out[it][i]));
      }
      if (a.o) {
        const int64_t off = (int64_t)b * a.sob + (int64_t)t * a.sot + (int64_t)head * a.soh + d;
        if (a.o_dtype == IFLB200_F32) {
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.o) + off) =
              make_float4(out[it][0], out[it][1], out[it][2], out[it][3]);
        } else if (a.o_dtype == IFLB200_F16) {
          uint2 u;
          u.x = f32_to_f16_bits(out[it][0]) | (f32_to_f16_bits(out[it][1]) << 16);
          u.y = f32_to_f16_bits(out[it][2]) | (f32_to_f16_bits(out[it][3]) << 16);
          *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(a.o) + off) = u;
        } else {
          uint2 u;
          u.x = f32_to_bf16_bits(out[it][0]) | (f32_to_bf16_bits(out[it][1]) << 16);
          u.y = f32_to_bf16_bits(out[it][2]) | (f32_to_bf16_bits(out[it][3]) << 16);
          *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(a.o) + off) = u;
        }
      }
    }
  }
  if (CL) {
    __syncwarp();    // the cluster barrier wants whole warps
    cluster_wait();  // every CTA of the cluster has started: a store into one that has not would be lost
  }
  if (!a.q) return;  // merge only (uniform)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = max_f32(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int i = 1; i < kCombineThreads / 32; ++i)
    if (i < threads / 32) amax = max_f32(amax, red[i]);
  if (CL) {
    if ((int)threadIdx.x < a.cluster) {
      uint32_t peer;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(smem_u32(&maxima[cluster_ctarank()])), "r"(threadIdx.x));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(peer), "f"(amax) : "memory");
    }
    __syncwarp();
    cluster_sync_all();
    amax = maxima[0];
    for (int i = 1; i < a.cluster; ++i) amax = max_f32(amax, maxima[i]);
  }
  float scale, inv;
  quant_scales(amax, scale, inv);
  if (threadIdx.x == 0 && first == 0) a.qs[t] = scale;
  uint8_t* qr = a.q + (int64_t)t * a.ld_q;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int c = first + it * threads + threadIdx.x;
    if (c < total) {
      const int head = it == 0 ? head0 : c / chunks_per_head, d = it == 0 ? d0 : (c - head * chunks_per_head) * 4;
      *reinterpret_cast<uint32_t*>(qr + (int64_t)head * a.head_dim + d) =
          cvt_e4m3x4(__fmul_rn(out[it][0], inv), __fmul_rn(out[it][1], inv), __fmul_rn(out[it][2], inv),
                     __fmul_rn(out[it][3], inv));
    }
  }
}

}  // namespace iflb200

using namespace iflb200;

extern "C" int iflb200_attn_combine_quant(const float* po, const float* pm, const float* pl, int splits, int batch,
                                          int tokens, int heads_q, int heads_kv, int head_dim, void* o, int o_dtype,
                                          int64_t o_stride_b, int64_t o_stride_t, int64_t o_stride_h, void* q,
                                          int64_t ld_q, float* qs, void* stream) {
  if (splits < 0 || batch < 0 || tokens < 0 || heads_q <= 0 || heads_kv <= 0 || head_dim <= 0) return IFLB200_ERR_ARG;
  if (splits == 0 || batch == 0 || tokens == 0) return IFLB200_OK;
  if (!po || !pm || !pl || (!o && !q) || (q && !qs)) return IFLB200_ERR_ARG;
  if (heads_q % heads_kv || head_dim % 4 || head_dim > 512) return IFLB200_ERR_SHAPE;
  if ((int64_t)heads_q * head_dim > (int64_t)kCombineThreads * kCombineIters * 4) return IFLB200_ERR_SHAPE;
  if (q && batch != 1) return IFLB200_ERR_SHAPE;  // as the reference: the quantised row is indexed by token alone
  if (o && o_dtype != IFLB200_F32 && o_dtype != IFLB200_F16 && o_dtype != IFLB200_BF16) return IFLB200_ERR_DTYPE;
  if (q && ld_q < (int64_t)heads_q * head_dim) return IFLB200_ERR_ARG;
  const int es = (o_dtype == IFLB200_F32) ? 4 : 2;
  if ((reinterpret_cast<uintptr_t>(po) & 15) || (q && ((reinterpret_cast<uintptr_t>(q) & 3) || ld_q % 4)) ||
      (o && ((reinterpret_cast<uintptr_t>(o) % (4 * es)) || (o_stride_b * es) % (4 * es) || (o_stride_t * es) % (4 * es) ||
             (o_stride_h * es) % (4 * es))))
    return IFLB200_ERR_ALIGN;
  int block_d = 1;
  while (block_d < head_dim) block_d <<= 1;
  CombineArgs a;
  a.po = po; a.pm = pm; a.pl = pl;
  a.o = o; a.o_dtype = o_dtype; a.sob = o_stride_b; a.sot = o_stride_t; a.soh = o_stride_h;
  a.q = reinterpret_cast<uint8_t*>(q); a.ld_q = ld_q; a.qs = qs;
  a.tokens = tokens; a.batch = batch; a.group = heads_q / heads_kv; a.heads_kv = heads_kv;
  a.head_dim = head_dim; a.block_d = block_d; a.splits = splits;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int chunks = heads_q * (head_dim / 4);
  // a cluster per token while half of the GPU would stay idle and every CTA keeps a chunk per thread of four warps
  // -- unless one CTA has a token in one round of loads, which a cluster only makes longer (50 tokens x 8 heads x 256,
  // 8 splits 3.0 us against 3.4 in a cluster of two; with 16 splits 4.7 against 4.4, with 16 heads 5.7 against 4.0)
  a.cluster = 1;
  const bool one_round = chunks <= kCombineThreads && splits <= 8;
  while (!one_round && chunks > 256 && a.cluster < kCombineMaxCluster && (int64_t)tokens * batch * a.cluster * 2 <= 148 && chunks >= 256 * a.cluster) a.cluster *= 2;
  const int share = (chunks + a.cluster - 1) / a.cluster;
  const dim3 grid(tokens * a.cluster, batch), block(share <= 128 ? 128 : (share <= 256 ? 256 : kCombineThreads));
  const bool dep = dependent_launch_for(tokens);
  cudaError_t e;
  auto go = [&](auto kernel) { return launch_dep(kernel, grid, block, 0, s, a.cluster, dep, a); };
  if (a.cluster > 1) e = share <= kCombineThreads ? go(attn_combine_quant_kernel<1, true, 8>) : go(attn_combine_quant_kernel<kCombineIters, true, 8>);
  // groups of eight while every token has its SM (CTAs of 512 threads: one an SM with that many registers; 296 tokens x 8 x
  // 256, 4 / 16 splits 4.73 / 8.12 us in groups of eight, 3.47 / 6.90 in groups of four) or CTAs are small (296 tokens x 8 x
  // 64, 8 splits 2.69 / 3.16)
  else if (chunks <= kCombineThreads) e = tokens <= (block.x > 256 ? 148 : 296) ? go(attn_combine_quant_kernel<1, false, 8>) : go(attn_combine_quant_kernel<1, false, 4>);
  else if (chunks <= 2 * kCombineThreads) e = tokens <= 148 ? go(attn_combine_quant_kernel<2, false, 8>) : go(attn_combine_quant_kernel<2, false, 4>);
  else e = go(attn_combine_quant_kernel<kCombineIters, false, 4>);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
