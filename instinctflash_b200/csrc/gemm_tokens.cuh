// FP8 GEMM with the tokens on the MMA's N side, on CTA pairs (included by gemm_fp8_sm100.cu).
//
//   out[t, n] = epilogue( sum_k A[t, k] * W[n, k] )
//
// A pair works on 256 weight rows x `bt` tokens, bt any multiple of 16 up to 256: the accumulator holds the tile
// transposed, lane = weight row, column = token.  What bounds the main loop of every tile here is what one SM draws
// from L2, 64 bytes a clock: a 128-byte K step of a pair is 128 + bt/2 rows per SM and takes 2 clocks a row plus
// 25 to 60, where its MMAs take 2 bt.  So a tile is worth its rows, and a width that fits the tokens is worth
// more than a wide one: 816 tokens are four tiles of 208 (480 clocks a step) instead of four of 256 (571),
// 301 are two of 160 instead of three row blocks of 128.
//
// The epilogue reads tensor memory in the 16 x 256-bit shape, the layout of an 8 x 8 matrix fragment: a thread
// holds weight row t/4 (and t/4 + 8) of two neighbouring tokens.  Two-byte outputs are transposed by stmatrix; fp32
// ones are stored word by word, each store instruction on 32 different banks; both leave in 16-byte pieces of a row by
// ordinary stores: the TMA unit is busy with the operands, and a TMA store is read from shared memory late
// (816 x 2560 x 2048 on 144 tokens 9.3 us with TMA stores of 16 tokens, 7.5 without).
// The epilogue that came before this one, one 2-byte shared-memory store per value, took 11 200 clocks a tile of
// 256 x 208 and was what its GEMM waited for (78 200 clocks for 816 x 32768 x 2048, 53 800 without it).
#pragma once

namespace iflb200 {

enum : int { TOK_RAW = 0, TOK_DEQUANT = 1, TOK_PLANES = 2, TOK_GATED = 3 };

struct TokenParams {
  int M, N, K;          // tokens, output columns (hidden units for the gated form), K in bytes
  int bt;               // tokens of a tile
  int num_m, num_n, num_k, num_tiles, group_m;  // token tiles, weight blocks of 256 rows, K steps
  int parts;            // K ranges (planes form)
  int slots, pairs;     // ring: K slabs that fit beside the staging buffers; 1: given back two at a time
  uint32_t idesc;
  int exact;            // as GemmParams::exact
  const float* row;
  int row_stride;
  const float* col;
  int col_stride;
  const void* bias;
  int bias_dtype;
  uint8_t* out;
  int64_t ld_out, plane;  // bytes from one token to the next, from one plane to the next
  int out_dtype;
  int act;
  int evict;  // gated form: weights leave L2 first
  uint32_t* amax;
};

template <int EPI>
struct TokenLayout {
  static constexpr int kWarps = EPI == TOK_GATED ? 16 : 8;  // epilogue warps
  static constexpr int kProducers = 2;                       // per operand
  static constexpr int kThreads = 32 * (kWarps + 1 + 2 * kProducers);
  static constexpr int kStaging = EPI == TOK_RAW || EPI == TOK_GATED ? 1024 : 2048;  // per warp: a block of 16 tokens
  static constexpr int kMaxSlots = 12;
  static constexpr int kMaxBytes = 227 * 1024;
  static constexpr int kFixed = 1024 + kWarps * kStaging + (2 * kMaxSlots + 4) * 8 + 16;
  static int slab_bytes(int bt) { return BM * BK + bt / 2 * BK; }
  // One commit takes the thread that issues the MMAs about 320 clocks, the MMAs of a slab 170 for 48 tokens, 296 for 144
  // and 327 for 160: narrow tiles give the ring back two slabs at a time (301 x 2560 x 2048 on 112 tokens 6.3 -> 5.6 us),
  // wide ones slab by slab, which keeps more of it in flight (816 x 2048 x 16384 in two ranges on 208 tokens 23.1
  // and 25.0).
  static bool pairs(int bt) { return bt < 160; }
  static int slots(int bt) {
    const int n = (kMaxBytes - kFixed) / slab_bytes(bt), m = n < kMaxSlots ? n : kMaxSlots;
    return pairs(bt) ? m & ~1 : m;
  }
};

// Eight token columns twice: r[4j + {0, 1}] = weight row t/4, tokens 8j + 2 (t % 4) + {0, 1}; r[4j + {2, 3}] = row t/4 + 8.
__device__ __forceinline__ void tmem_ld_16x256b_x2(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// Thirty-two columns of the same.
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c),
               "r"(d)
               : "memory");
}
__device__ __forceinline__ void st_shared_f32(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// wait_bounded for a thread on its own.
__device__ __forceinline__ bool wait_bounded_one(uint32_t bar, uint32_t parity, volatile uint32_t* abort, uint32_t code) {
  if (mbar_try_wait(bar, parity)) return true;
  uint64_t t0 = 0;
  uint32_t spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort) return false;
    if (++spins > 2048) {
      if (t0 == 0) t0 = globaltimer_ns();
      __nanosleep(128);
      if (globaltimer_ns() - t0 > g_gemm_wait_budget_ns) {
        *abort = 1;
        atomicCAS(&g_timeout_record[0], 0u, code);
        return false;
      }
    }
  }
}

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TokenLayout<EPI>::kThreads, 1)
gemm_fp8_tc5_tokens_kernel(const __grid_constant__ CUtensorMap tm_t, const __grid_constant__ CUtensorMap tm_w,
                           const __grid_constant__ TokenParams p) {
  using L = TokenLayout<EPI>;
  constexpr int EW = L::kWarps, PARTS = EW / 4;
  constexpr uint32_t kAccStride = 256, kTmemCols = 512;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const int slots = p.slots, pairs = p.pairs;
  const uint32_t w_bytes = BM * BK, t_bytes = (uint32_t)p.bt / 2 * BK, slab_bytes = w_bytes + t_bytes;
  const uint32_t staging0 = base + slots * slab_bytes;
  const uint32_t bar0 = staging0 + EW * L::kStaging;
  auto full_bar = [&](int slot) { return bar0 + 8u * slot; };
  auto empty_bar = [&](int slot) { return bar0 + 8u * (slots + (slot >> pairs)); };
  auto tfull_bar = [&](int a) { return bar0 + 8u * (2 * slots + a); };
  auto tempty_bar = [&](int a) { return bar0 + 8u * (2 * slots + 2 + a); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + (bar0 - base) + (2 * slots + 4) * 8);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair_id = blockIdx.x >> 1;
  const int pair_stride = gridDim.x >> 1;
  const int parts = EPI == TOK_PLANES ? p.parts : 1;
  const int units = p.num_tiles * parts;
  // K ranges in whole stages of the skinny form, as in every planes form
  auto range_begin = [&](int part) { return (int)(((int64_t)((p.num_k + 3) / 4) * part) / parts) * 4; };
  auto place = [&](int unit, int& t_blk, int& w_blk) {
    const int tile = EPI == TOK_PLANES ? unit / parts : unit;
    const int band = p.group_m * p.num_n, g = tile / band;
    const int first = g * p.group_m, size = min(p.num_m - first, p.group_m), r = tile - g * band;
    t_blk = first + r % size;
    w_blk = r / size;
  };
  auto steps_of = [&](int unit, int& kb0, int& kb1) {
    kb0 = 0;
    kb1 = p.num_k;
    if constexpr (EPI == TOK_PLANES) {
      kb0 = range_begin(unit % parts);
      kb1 = min(p.num_k, range_begin(unit % parts + 1));
    }
  };

  if (threadIdx.x == 0) {
    prefetch_tensormap(&tm_w);
    prefetch_tensormap(&tm_t);
    for (int i = 0; i < slots; ++i) mbar_init(full_bar(i), 2);  // the leader's producers of the slab arm it; bytes of both CTAs complete it
    for (int i = 0; i < slots >> pairs; ++i) mbar_init(bar0 + 8u * (slots + i), 1);  // one multicast commit from the leader
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 2 * EW);  // the epilogue warps of both CTAs
    }
    tmem_slot[1] = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  __syncwarp();
  cluster_arrive_relaxed();  // (the initialisation has its own fence)
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  cluster_wait();  // barriers of both CTAs initialised before any remote signal

  // producers: warp 0 and the warps behind the epilogue's, W and T in turn
  const int producer = warp == 0 ? 0 : (warp < 2 + EW ? -1 : warp - 1 - EW);
  const bool w_producer = (producer & 1) == 0, t_producer = !w_producer;
  if (producer >= 0) {
    // ------------------------------------------------------------------ TMA producers (both CTAs)
    // Two warps for each operand, which take the slabs in turn; the weights' ahead of the dependency wait for few rows, as
    // in the other forms.
    bool waited = w_producer && p.M <= kEarlyWeightsMaxRows;
    const uint64_t policy = l2_evict_first();
    int slot = producer >> 1, skip = producer >> 1;  // skip: slabs of the other warp until this one's next
    uint32_t phase = 0;
    bool ok = true;
    uint32_t it = 0;
    for (int unit = pair_id; ok && unit < units; unit += pair_stride, ++it) {
      int t_blk, w_blk, kb0, kb1;
      place(unit, t_blk, w_blk);
      steps_of(unit, kb0, kb1);
      const int w_row = w_blk * 2 * BM + (int)rank * BM;
      const int t_row = t_blk * p.bt + (int)rank * (p.bt / 2);
      const int slabs = kb1 - kb0, taken = slabs + (slabs & pairs);
      int i = skip;
      for (; i < taken; i += L::kProducers) {
        ok = wait_bounded(empty_bar(slot), phase ^ 1, abort_flag, (1u << 24) | (1u << 16) | (it & 0xFFFF));
        if (!ok) break;
        if (elect_one()) {
          const uint32_t bar = full_bar(slot), dst = base + slot * slab_bytes;
          const int x = (kb0 + i) * BK;
          if (i < slabs) {
            if (leader) mbar_arrive_expect_tx(bar, 2u * (w_producer ? w_bytes : t_bytes));
            if (!waited) grid_dependency_wait();  // directly before the first load (see gemm_lean.cuh)
            waited = true;
            if (t_producer) tma_load_2d_pair(dst + w_bytes, &tm_t, bar & kPeerBitMask, x, t_row);
            else if constexpr (EPI == TOK_GATED) {
              if (p.evict) tma_load_4d_pair_hint(dst, &tm_w, bar & kPeerBitMask, x, 0, 0, w_row / 16, policy);
              else tma_load_4d_pair(dst, &tm_w, bar & kPeerBitMask, x, 0, 0, w_row / 16);
            }
            else tma_load_2d_pair(dst, &tm_w, bar & kPeerBitMask, x, w_row);
          } else if (leader) {
            mbar_arrive(bar);  // an odd number of slabs: nothing to load, but the slot's phases stay in step
          }
        }
        __syncwarp();
        slot += L::kProducers;
        if (slot >= slots) {
          slot -= slots;
          phase ^= 1;
        }
      }
      skip = i - taken;
    }
    if (t_producer) {  // last loads issued: the next kernel may be scheduled
      grid_dependency_wait();  // (a lane that has issued no load has not waited yet)
      grid_launch_dependents();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader only)
    // One thread runs the whole loop: votes and elections per slab took the warp about 100 clocks more.
    if (leader && elect_one()) {
      int slot = 0;
      uint32_t phase = 0;
      bool ok = true;
      uint32_t it = 0;
      const uint64_t dw0 = make_kmajor_sw128_desc(base), dt0 = make_kmajor_sw128_desc(base + w_bytes);
      for (int unit = pair_id; ok && unit < units; unit += pair_stride, ++it) {
        int kb0, kb1;
        steps_of(unit, kb0, kb1);
        const int slabs = kb1 - kb0;
        const uint32_t acc = it & 1u, acc_phase = (it >> 1) & 1u;
        ok = wait_bounded_one(tempty_bar(acc), acc_phase ^ 1, abort_flag, (2u << 24) | (2u << 16) | (it & 0xFFFF));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * kAccStride;
        if (pairs) {
          for (int i = 0; i < slabs; i += 2) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              ok = ok && wait_bounded_one(full_bar(slot + h), phase, abort_flag, (2u << 24) | (3u << 16) | (it & 0xFFFF));
              if (!ok) break;
              tc_fence_after();
              const uint64_t at = (uint64_t)(((slot + h) * slab_bytes) >> 4);
              if (i + h < slabs) {
#pragma unroll
                for (int j = 0; j < BK / 32; ++j)
                  mma_f8f6f4_pair(d_tmem, dw0 + at + 2 * j, dt0 + at + 2 * j, p.idesc, i > 0 || h > 0 || j > 0 ? 1u : 0u);
              }
            }
            if (!ok) break;
            mma_commit_pair(empty_bar(slot), 3);  // both free in both CTAs
            slot += 2;
            if (slot == slots) {
              slot = 0;
              phase ^= 1;
            }
          }
        } else {
          for (int i = 0; i < slabs; ++i) {
            ok = wait_bounded_one(full_bar(slot), phase, abort_flag, (2u << 24) | (3u << 16) | (it & 0xFFFF));
            if (!ok) break;
            tc_fence_after();
            const uint64_t at = (uint64_t)((slot * slab_bytes) >> 4);
#pragma unroll
            for (int j = 0; j < BK / 32; ++j)
              mma_f8f6f4_pair(d_tmem, dw0 + at + 2 * j, dt0 + at + 2 * j, p.idesc, i > 0 || j > 0 ? 1u : 0u);
            mma_commit_pair(empty_bar(slot), 3);  // free in both CTAs
            if (++slot == slots) {
              slot = 0;
              phase ^= 1;
            }
          }
        }
        if (!ok) break;
        mma_commit_pair(tfull_bar(acc), 3);  // accumulator complete in both CTAs
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue warps (both CTAs)
    // A warp owns 32 weight rows (its lanes of tensor memory) and every PARTS-th block of 16 tokens.
    const int quad = warp & 3;
    const int part = (warp - 2) >> 2;
    const uint32_t staging = staging0 + (uint32_t)(warp - 2) * L::kStaging;
    const int r4 = lane >> 2, c4 = lane & 3;
    bool ok = true;
    uint32_t it = 0;
    grid_dependency_wait();  // scales may come from the kernel before this one
    for (int unit = pair_id; ok && unit < units; unit += pair_stride, ++it) {
      int t_blk, w_blk;
      place(unit, t_blk, w_blk);
      const uint32_t acc = it & 1u, acc_phase = (it >> 1) & 1u;
      const int tok_base = t_blk * p.bt;
      const int n0 = EPI == TOK_GATED ? w_blk * BM + (int)rank * 64 + quad * 16 : w_blk * 2 * BM + (int)rank * BM + quad * 32;
      const int blocks = n0 < p.N ? min(p.bt, p.M - tok_base + 15) / 16 : 0;
      // This tile's per-row operands, fetched under the main loop: weight rows 8 i + t/4 of the warp's 32 (gated: gate
      // and up scale of hidden units 8 i + t/4 of its 16).  What is absent is a factor of 1 or an addend of -0, which
      // change nothing: no branch per value.
      float cs[4] = {1.0f, 1.0f, 1.0f, 1.0f}, bs[4] = {-0.0f, -0.0f, -0.0f, -0.0f};
      if constexpr (EPI == TOK_DEQUANT || EPI == TOK_GATED) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int n = EPI == TOK_GATED ? n0 + 8 * (i >> 1) + r4 : n0 + 8 * i + r4;
          if (n < p.N) {
            if (p.col) cs[i] = __ldg(p.col + (EPI == TOK_GATED ? (i & 1) * p.N + n : n * p.col_stride));
            if (EPI == TOK_DEQUANT && p.bias)
              bs[i] = p.bias_dtype == IFLB200_F32 ? __ldg(reinterpret_cast<const float*>(p.bias) + n)
                                                  : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[n]);
          }
        }
      }
      // row scales of the two token pairs this thread holds of a block
      const bool scaled = (EPI == TOK_DEQUANT || EPI == TOK_GATED) && p.row != nullptr;
      float rn[4] = {1.0f, 1.0f, 1.0f, 1.0f};
      auto row_scales = [&](int block) {
        if (!scaled || block >= blocks) return;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = min(tok_base + 16 * block + 8 * (i >> 1) + 2 * c4 + (i & 1), p.M - 1);
          rn[i] = __ldg(p.row + (int64_t)t * p.row_stride);
        }
      };
      row_scales(part);
      ok = wait_bounded(tfull_bar(acc), acc_phase, abort_flag, (3u << 24) | (4u << 16) | (it & 0xFFFF));
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_acc = tmem_base + ((uint32_t)(quad * 32) << 16) + acc * kAccStride;
      uint32_t nx[2][8];  // the next block: lanes 0..15 and 16..31 of the quadrant
      auto load = [&](int block) {
        tmem_ld_16x256b_x2(t_acc + 16 * block, nx[0]);
        tmem_ld_16x256b_x2(t_acc + (16u << 16) + 16 * block, nx[1]);
      };
      // the accumulator is free for the tile after next, where there is one: an arrival that nothing waits for would
      // reach the leader's shared memory at any time
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && unit + 2 * pair_stride < units) mbar_arrive_cluster(tempty_bar(acc), 0);
      };
      if (part < blocks) load(part);
      else release();
#pragma unroll 1
      for (int block = part; block < blocks; block += PARTS) {
        tmem_ld_wait();
        uint32_t r[2][8];
        float rs[4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          r[0][i] = nx[0][i];
          r[1][i] = nx[1][i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) rs[i] = rn[i];
        if (block + PARTS < blocks) {
          load(block + PARTS);
          row_scales(block + PARTS);
        } else {
          release();
        }
        const uint32_t dst = staging;
        __syncwarp();  // the block before this one has been read
        const int tok = tok_base + 16 * block;
        if constexpr (EPI == TOK_GATED) {
          // The gated activation of instinctflash/kernels/activation.py:26-43 in the order of epilogue_gated: gate and up
          // rows of a hidden unit are rows t/4 and t/4 + 8 of a half, so both are in this thread.
          uint64_t h[2][2];
#pragma unroll
          for (int half = 0; half < 2; ++half) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const uint32_t wg = pack_bf16x2(__uint_as_float(r[half][4 * j]), __uint_as_float(r[half][4 * j + 1]));
              const uint32_t wu = pack_bf16x2(__uint_as_float(r[half][4 * j + 2]), __uint_as_float(r[half][4 * j + 3]));
              const uint64_t r2 = pack2(rs[2 * j], rs[2 * j + 1]);
              uint64_t g = mul2(pack2(__uint_as_float(wg << 16), __uint_as_float(wg & 0xFFFF0000u)), r2);
              uint64_t u = mul2(pack2(__uint_as_float(wu << 16), __uint_as_float(wu & 0xFFFF0000u)), r2);
              g = mul2(g, pack2(cs[2 * half], cs[2 * half]));
              u = mul2(u, pack2(cs[2 * half + 1], cs[2 * half + 1]));
              if (p.act == IFLB200_ACT_GELU_TANH) {
                g = gelu_tanh_ref2(g);
              } else {
                float a, b;
                unpack2(g, a, b);
                g = pack2(silu_ref(a), silu_ref(b));
              }
              h[half][j] = mul2(u, g);
            }
          }
          // 64-byte rows of 16 hidden units, 16-byte pieces swizzled by the token pair; odd lanes store their second
          // token first, so that the 32 words of an instruction fall on 32 banks
          const bool odd = lane & 1;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const uint32_t at = dst + 128 * c4 + (((uint32_t)(2 * half + (lane >> 4)) ^ (uint32_t)c4) << 4) + (r4 & 3) * 4;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              float a, b;
              unpack2(h[half][j], a, b);
              st_shared_f32(at + 512 * j + (odd ? 64 : 0), odd ? b : a);
              st_shared_f32(at + 512 * j + (odd ? 0 : 64), odd ? a : b);
            }
          }
          // maximum of |h| per token over the eight lanes that hold it: halve the tokens, then the lanes
          float m[4];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            float a0, b0, a1, b1;
            unpack2(h[0][j], a0, b0);
            unpack2(h[1][j], a1, b1);
            m[2 * j] = max_abs_f32(0.0f, a0, a1);
            m[2 * j + 1] = max_abs_f32(0.0f, b0, b1);
          }
          const bool hi = lane & 16, mid = lane & 8;
          const float k0 = max_f32(hi ? m[2] : m[0], __shfl_xor_sync(0xFFFFFFFFu, hi ? m[0] : m[2], 16));
          const float k1 = max_f32(hi ? m[3] : m[1], __shfl_xor_sync(0xFFFFFFFFu, hi ? m[1] : m[3], 16));
          float k = max_f32(mid ? k1 : k0, __shfl_xor_sync(0xFFFFFFFFu, mid ? k0 : k1, 8));
          k = max_f32(k, __shfl_xor_sync(0xFFFFFFFFu, k, 4));
          const int t = tok + (hi ? 8 : 0) + 2 * c4 + (mid ? 1 : 0);
          if (!(lane & 4) && t < p.M) atomicMax(p.amax + t, __float_as_uint(k));
        } else {
          if constexpr (EPI == TOK_DEQUANT) {
            // ((acc * row) * col) + bias, the addition contracted with the last factor there is; with two per-tensor
            // scales (acc * (row * col)) + bias, each operation rounded
#pragma unroll
            for (int half = 0; half < 2; ++half) {
#pragma unroll
              for (int i = 0; i < 4; ++i) {  // pair i of the half: tokens 8 (i / 2).., weight row 8 (i % 2) + t/4
                const int n = 2 * half + (i & 1), j = i >> 1;
                float a = __uint_as_float(r[half][2 * i]), b = __uint_as_float(r[half][2 * i + 1]);
                if (!p.exact) {
                  const uint32_t w = pack_bf16x2(a, b);
                  a = __uint_as_float(w << 16);
                  b = __uint_as_float(w & 0xFFFF0000u);
                }
                if (p.exact == 2) {  // (scalar: the compiler contracts a packed product and sum)
                  a = __fadd_rn(__fmul_rn(a, __fmul_rn(rs[2 * j], cs[n])), bs[n]);
                  b = __fadd_rn(__fmul_rn(b, __fmul_rn(rs[2 * j + 1], cs[n])), bs[n]);
                } else {
                  const uint64_t x = pack2(a, b), r2 = pack2(rs[2 * j], rs[2 * j + 1]), c2 = pack2(cs[n], cs[n]), b2 = pack2(bs[n], bs[n]);
                  unpack2(p.col ? fma2(mul2(x, r2), c2, b2) : fma2(x, r2, b2), a, b);
                }
                r[half][2 * i] = __float_as_uint(a);
                r[half][2 * i + 1] = __float_as_uint(b);
              }
            }
          }
          if (EPI == TOK_PLANES || (EPI == TOK_DEQUANT && p.out_dtype == IFLB200_F32)) {
            // 128-byte rows of 32 columns, 16-byte pieces swizzled by the token
#pragma unroll
            for (int half = 0; half < 2; ++half) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int j = i >> 2, sub = (i >> 1) & 1, e = i & 1;
                const uint32_t chunk = (uint32_t)(4 * half + 2 * sub + (lane >> 4)) ^ (uint32_t)(2 * c4 + e);
                st_shared_f32(dst + (8 * j + 2 * c4 + e) * 128 + chunk * 16 + (r4 & 3) * 4, __uint_as_float(r[half][i]));
              }
            }
          } else {
            // 64-byte rows of 32 columns, pieces swizzled by the token pair: four 8 x 8 matrices a store, transposed on the way
            const uint32_t row = (uint32_t)(lane & 7), chunk = (uint32_t)(lane >> 3) ^ (row >> 1 & 3);
            const bool f16 = EPI == TOK_DEQUANT && p.out_dtype == IFLB200_F16;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              uint32_t v[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float a = __uint_as_float(r[i >> 1][4 * j + 2 * (i & 1)]), b = __uint_as_float(r[i >> 1][4 * j + 2 * (i & 1) + 1]);
                v[i] = f16 ? pack_f16x2(a, b) : pack_bf16x2(a, b);
              }
              stmatrix_x4_trans(dst + (8 * j + row) * 64 + chunk * 16, v[0], v[1], v[2], v[3]);
            }
          }
        }
        // the block's rows to memory, 16 bytes a lane
        __syncwarp();
        if (EPI == TOK_PLANES || (EPI == TOK_DEQUANT && p.out_dtype == IFLB200_F32)) {
          uint8_t* o = p.out + (int64_t)(tok + (lane >> 3)) * p.ld_out + (int64_t)n0 * 4 + (lane & 7) * 16;
          if constexpr (EPI == TOK_PLANES) o += (unit % parts) * p.plane;
          const bool in = n0 + 4 * (lane & 7) < p.N;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int t = 4 * i + (lane >> 3);
            const uint4 v = ld_shared_v4(dst + t * 128 + (((lane & 7) ^ (t & 7)) << 4));
            if (in && tok + t < p.M) *reinterpret_cast<uint4*>(o + 4 * i * p.ld_out) = v;
          }
        } else {
          constexpr int es = EPI == TOK_GATED ? 4 : 2;
          uint8_t* o = p.out + (int64_t)(tok + r4) * p.ld_out + (int64_t)n0 * es + c4 * 16;
          const bool in = n0 + c4 * (16 / es) < p.N;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint4 v = ld_shared_v4(dst + (8 * i + r4) * 64 + ((c4 ^ (r4 >> 1 & 3)) << 4));
            if (in && tok + 8 * i + r4 < p.M) *reinterpret_cast<uint4*>(o + 8 * i * p.ld_out) = v;
          }
        }
      }
    }
  }

  // Neither CTA leaves while its peer can still reach its shared or tensor memory: the leader's MMAs read and write the
  // peer's until the last accumulator is complete, which both CTAs' epilogue warps have waited for.  Arrivals that free an
  // accumulator have been waited for by then too; those of the last ring turn on the `empty` barriers, which nothing waits
  // for, were committed ahead of that accumulator.  The barrier orders no data, so that it need not wait for the stores
  // above.  After a timed-out wait the loads in flight get time to land.
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  cluster_arrive_relaxed();
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

}  // namespace iflb200
