// Element functions compared over all of their inputs (tests/test_gpu_exhaustive.py).
#include "rowmath.cuh"

using namespace iflb200;

// [0]: differing results, [1]: the first differing input seen, [2]: inputs compared
__device__ void differs(unsigned long long* out, unsigned long long what) {
  if (atomicAdd(out, 1ull) == 0) out[1] = what;
}

// The packed GELU against the scalar one for every float, in either lane.
__global__ void gelu_kernel(unsigned long long* out) {
  const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long n = 0;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (1ull << 32); i += step) {
    const float x = __uint_as_float((uint32_t)i), other = __uint_as_float((uint32_t)i * 2654435761u);
    const uint32_t want = __float_as_uint(gelu_tanh_ref(x));
    float lo = x, hi = other, lo2 = other, hi2 = x;
    gelu_tanh_ref2(lo, hi);
    gelu_tanh_ref2(lo2, hi2);
    if (__float_as_uint(lo) != want || __float_as_uint(hi2) != want) differs(out, i);
    ++n;
  }
  atomicAdd(out + 2, n);
}

// The pack by reciprocal and correction against the division: every maximum, every element it allows.
__global__ void pack_kernel_check(unsigned long long* out) {
  const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long n = 0;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (0x8000ull << 16); i += step) {
    const uint32_t best = (uint32_t)(i >> 16), x = (uint32_t)i & 0xFFFFu;
    if ((x & 0x7FFFu) > best) continue;
    const float scale = scale_of_bits(best);
    const uint32_t want = cvt_e4m3x2(pack_one(__uint_as_float(x << 16), scale), 0.0f) & 0xFFu;
    const uint32_t w = x | (x << 16);
    const uint2 got = pack_eight(make_uint4(w, w, w, w), scale, reciprocal_for_pack(scale));
    if (got.x != want * 0x01010101u || got.y != want * 0x01010101u) differs(out, i);
    ++n;
  }
  atomicAdd(out + 2, n);
}

extern "C" int compare_all(int what, unsigned long long* out) {
  if (what == 0) gelu_kernel<<<1184, 256>>>(out);
  else pack_kernel_check<<<1184, 256>>>(out);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? (int)e : (int)cudaDeviceSynchronize();
}
