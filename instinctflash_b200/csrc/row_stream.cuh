// Row kernels for many rows (row_stream.cu): persistent CTAs whose threads keep the same columns for
// every row, so that the per-column operands are read once per CTA instead of once per row.
// Each returns true when it has launched, false when the call is outside its range (the one-row-
// per-group kernels of row_ops.cu take it then).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace iflb200 {

struct GeluStreamArgs {
  const void* x;
  int64_t ld_x;
  int M, K;
  int rows_of_call() const { return M; }
  bool many() const { return (int64_t)M * K <= 1 << 25; }  // dependent launch beyond kDependentRows
  const float* row;
  const float* col;
  const float* bias;
  uint8_t* q;
  int64_t ld_q;
  float* qs;
  int early;  // let the next kernel be scheduled before the dependency wait
};
// x: bf16 or f16, every buffer on the 16-byte rule (codes: 8), K a multiple of 8
bool launch_gelu_quant_stream(const GeluStreamArgs& a, bool half, cudaStream_t s);

struct ResNormStreamArgs {
  void* res;
  int64_t ld_res;
  int M, D;
  int rows_of_call() const { return M; }
  bool many() const { return true; }
  const __nv_bfloat16* delta;  // or null
  int64_t ld_delta;
  const float *drow, *dcol, *bias, *gate;
  const float* scale;  // norm weight, or 1 + scale of the modulation (scale_plus_one), or null
  const float* shift;  // norm bias or modulation shift, or null
  int scale_plus_one;
  float eps;
  uint8_t* q;
  int64_t ld_q;
  float* qs;
  int early;  // let the next kernel be scheduled before the dependency wait
};
// layer norm of a bf16 residual, updated in place when there is a delta; every buffer on the 16-byte
// rule (codes: 8), D a multiple of 8
bool launch_residual_norm_stream(const ResNormStreamArgs& a, cudaStream_t s);

struct WanStreamArgs {
  const void* raw;  // bf16 [rows, parts * D]
  int64_t ld_raw;
  int rows, tokens, parts, D, HD;
  int rows_of_call() const { return rows; }
  bool many() const { return true; }
  const float *row, *col, *bias, *q_norm, *k_norm;
  float eps;
  const float *inv_freq, *pos;
  int64_t ld_pos;
  const int32_t *sections, *slots;
  void *q, *k, *v;
  int64_t ld_q, sk_b, sk_s, sv_b, sv_s;
};
// f16 (`half`) or bf16 outputs; every buffer and stride on the 16-byte rule, D and HD multiples of 8
bool launch_wan_qkv_stream(const WanStreamArgs& a, bool half, cudaStream_t s);

}  // namespace iflb200
