// Host-side kernel launch with the attributes this library uses: an optional cluster width and
// programmatic dependent launch (the kernel may be scheduled while its predecessor in the
// stream drains; every kernel launched through here calls grid_dependency_wait() before its
// first access to memory another kernel may write, but for two reads: the first weights of a GEMM of few rows
// (kEarlyWeightsMaxRows), and the elements in the one-pass pack, whose own first kernel stands before it (pack_kernel)).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace iflb200 {

// 0: plain stream order; 1 (default): dependent launch for kernels over at most kDependentRows activation rows, and up to
// kDependentRowsLong where the kernel says so (`many`); 2: always.  Measured on B200: with a few hundred rows
// (kernels of 3-50 us) early scheduling of the next kernel shortens a layer stack by 5-15 %.  Over more than 2048 rows a
// launch's share of the time is small, and what is scheduled early can be in the way of what still runs.  Time with
// dependent launch over time without it, 2049 to 16384 rows, each operator directly behind a GEMM, by elements:
//   GEMM forms                   0.94 to 1.00 (0.97 in the mean; 16384 x 5120 x 5120 0.97)
//   row quantiser                0.94 below 2^21, 0.98 at 2^23 to 2^24, 1.02 above 2^25 (up to 1.11 with few GEMM tiles)
//   GELU quantiser               0.96 below 2^22, 0.99 at 2^23 to 2^25, 1.00 above
//   dequantisation               0.98 below 2^22, 0.99 up to 2^24, 1.03 above 2^24.5
//   quantiser from row maxima    0.96 below 2^21, 0.99 at 2^23, 1.00 at 2^24, 1.09 above
//   gated quantiser              0.96 below 2^21, 0.98 up to 2^22, 1.01 at 2^23, 1.03 to 1.1 above
//   streaming layer-norm rows    0.98 at 1536 columns, 0.99 to 1.00 from 2048 on; other residual rows 1.01 to 1.07 (1024 columns)
//   residual over planes         1.11 in the mean, up to 1.27
//   streaming wan_qkv            1.00; behind itself 0.95 to 0.98
//   QKV split                    1.01, up to 1.06; behind itself up to 1.3 (64-wide heads, 3000 tokens)
//   first kernel of the pack     1.01 below 2^25, 1.06 above
extern int g_dependent_launch;
constexpr long long kDependentRows = 2048, kDependentRowsLong = 16384;
inline bool dependent_launch_for(long long rows, bool many = false) {
  return g_dependent_launch == 2 || (g_dependent_launch == 1 && rows <= (many ? kDependentRowsLong : kDependentRows));
}

// A GEMM of up to so many rows fetches its first weights ahead of its dependency wait, a larger one behind it: there the early
// fetch gains nothing (quantiser and linear at 50 sizes of 2049 to 16384 rows: 0.998 of the time without it), and it forbids a
// weight that the kernel directly before has written (contract: iflb200_gemm_fp8_raw).
constexpr int kEarlyWeightsMaxRows = 2048;

// Multiprocessors of the current device; 0 when it cannot be told.
inline int device_sm_count() {
  static int count[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (count[dev] == 0) cudaDeviceGetAttribute(&count[dev], cudaDevAttrMultiProcessorCount, dev);
  return count[dev];
}

// The node that a stream capture of `s` stands at: the last kernel captured into it.  False outside a
// capture, and where several branches meet.
struct CapturePoint {
  unsigned long long capture = 0;  // unique for the life of the process
  cudaGraphNode_t node = nullptr;
};
inline bool capture_point(cudaStream_t s, CapturePoint& at) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (s == nullptr || cudaStreamIsCapturing(s, &status) != cudaSuccess || status != cudaStreamCaptureStatusActive) return false;
  const cudaGraphNode_t* nodes = nullptr;
  const cudaGraphEdgeData* edges = nullptr;
  size_t n = 0;
  if (cudaStreamGetCaptureInfo_v3(s, &status, &at.capture, nullptr, &nodes, &edges, &n) != cudaSuccess || n != 1) return false;
  at.node = nodes[0];
  return true;
}

// The last GEMM of this library that this thread has captured.
inline thread_local CapturePoint t_captured_gemm;
inline void note_captured_gemm(cudaStream_t s) {
  CapturePoint at;
  if (g_dependent_launch != 0 && capture_point(s, at)) t_captured_gemm = at;
}

// Whether a row kernel should let its successor be scheduled before its own dependency wait, so that the
// GEMM behind it sets up and fetches weights while the kernel two ahead of it drains (50 rows: 27.7 -> 25.6 us
// per expert layer).  Only where the kernel before the row kernel is known to be one of this library's
// GEMMs, which a captured graph can tell and an eager stream cannot: a GEMM lets the row kernel start only once everything
// before the GEMM has completed, and writes accumulators, never the codes of a weight.  So the kernels still
// running when the next GEMM reads its weights are that GEMM and the row kernel, whose output they must not
// be anyway (contract: iflb200_gemm_fp8_raw).  Row kernels that followed one another and all signalled
// early would let a GEMM read a weight that a kernel any number of launches ahead is still writing.
inline int early_trigger_for(cudaStream_t s) {
  CapturePoint at;
  return g_dependent_launch != 0 && capture_point(s, at) && at.capture == t_captured_gemm.capture && at.node == t_captured_gemm.node;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dep(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              int cluster_x, bool dependent, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (cluster_x > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)cluster_x;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (dependent) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace iflb200
