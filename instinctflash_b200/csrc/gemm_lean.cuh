// The skinny FP8 GEMM: 64-wide tiles of up to 128 activation rows, one K range or split-K planes (included by
// gemm_fp8_sm100.cu).
//
// A launch over 50 rows takes 3 to 5 us, most of it latencies in a row: the kernel before it, first operands, MMAs,
// epilogue, completion.  It fetches its instructions cold, so the kernel holds nothing that such a launch does not run:
// the output kind is a template argument, and a lane stores its row straight from registers (6 KB a tile are not worth
// staging; fp32 rows of many tiles are).  With one epilogue for all output kinds, through shared memory and TMA, the last store of a 64 x 4096 x 1024
// launch was issued 2600 clocks after its last MMA; 18 expert layers over 50 rows (72 such launches) took 476 us, 417 now.
// Four K slabs of 128 bytes a stage come with one TMA instruction per operand; up to 64 rows the MMAs are 64 rows high
// (38 clocks each for 48), and row i of the accumulator lies in lane i % 16 of quadrant i / 16.
#pragma once

namespace iflb200 {

enum : int { LEAN_RAW = 0, LEAN_DEQUANT = 1, LEAN_PLANES = 2, LEAN_F32 = 3 };  // LEAN_F32: dequantised, fp32 output

// The lean form's arguments: K need not be a multiple of 128.  Stages of whole slabs come through the slab maps
// (K / 128 slabs); the stage that holds the ragged slab comes slab by slab through these, which read
// zeros past the end of a row.
struct LeanParams : GemmParams {
  CUtensorMap a_tail, w_tail;
  int full_slabs;  // K / 128
};

template <int AR>
struct LeanLayout {
  static constexpr int kSlabs = 4, kTile = 64, kStages = AR == 64 ? 3 : 2;
  static constexpr int kABytes = AR * BK * kSlabs, kWBytes = kTile * BK * kSlabs, kStageBytes = kABytes + kWBytes;
  // fp32 rows of the 128-row form on their way to memory, 32 x 128 bytes a warp
  static constexpr int kStagingOffset = kStages * kStageBytes, kStaging = AR == 128 ? 4096 : 0;
  static constexpr int kBarOffset = kStagingOffset + 8 * kStaging;
  static constexpr int kDynamic = kBarOffset + (2 * kStages + 4) * 8 + 16 + 1024;
  static constexpr int kThreads = 32 * 11;  // W producer, MMA, eight epilogue warps, A producer
};

template <int AR, int EPI>
__global__ void __launch_bounds__(LeanLayout<AR>::kThreads, 1)
gemm_fp8_tc5_lean_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                         const __grid_constant__ LeanParams p) {
  using L = LeanLayout<AR>;
  constexpr int SL = L::kSlabs, BN = L::kTile, STAGES = L::kStages, quad_rows = AR / 4;
  constexpr bool kDequant = EPI == LEAN_DEQUANT || EPI == LEAN_F32, kWide = EPI == LEAN_PLANES || EPI == LEAN_F32;
  constexpr uint32_t kTmemCols = 2 * BN;
  constexpr uint32_t kIdesc = make_idesc_e4m3_f32(AR, BN);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t bar0 = base + L::kBarOffset;
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar0 + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar0 + 8u * (2 * STAGES + 2 + a); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kBarOffset + (2 * STAGES + 4) * 8);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // K split over independent CTAs: each writes its fp32 partial sums to a plane of its own
  const int parts = EPI == LEAN_PLANES ? p.partials : 1;
  const int part = EPI == LEAN_PLANES ? (int)blockIdx.x % parts : 0;
  const int tile_first = EPI == LEAN_PLANES ? (int)blockIdx.x / parts : (int)blockIdx.x;
  const int tile_stride = EPI == LEAN_PLANES ? p.num_tiles : (int)gridDim.x;
  const int k_stages = (p.num_k + SL - 1) / SL;
  const int kb0 = (int)(((int64_t)k_stages * part) / parts) * SL;
  const int kb1 = min(p.num_k, (int)(((int64_t)k_stages * (part + 1)) / parts) * SL);

  if (threadIdx.x == 0) {
    prefetch_tensormap(&tm_w);
    prefetch_tensormap(&tm_a);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 2);  // one arrival per producer
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 8);  // one arrival per epilogue warp
    }
    tmem_slot[1] = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // As in the other forms: only the activations and the epilogue wait for the kernel before this one.
  const bool w_producer = warp == 0, a_producer = warp == 10;
  if (w_producer || a_producer) {
    // ------------------------------------------------------------------ TMA producers
    if (a_producer) grid_dependency_wait();
    const uint32_t slab_bytes = w_producer ? (uint32_t)(BN * BK) : (uint32_t)p.a_bytes;
    Ring<STAGES> ring;
    bool ok = true;
    uint32_t it = 0;
    for (int tile = tile_first; ok && tile < p.num_tiles; tile += tile_stride, ++it) {
      int m_blk, n_blk;
      tile_coords(p, tile, m_blk, n_blk);
      const int row = w_producer ? n_blk * BN : m_blk * BM;
      for (int kb = kb0; kb < kb1; kb += SL) {
        ok = wait_bounded(empty_bar(ring.stage), ring.phase ^ 1, abort_flag, (1u << 24) | (1u << 16) | (it & 0xFFFF));
        if (!ok) break;
        const int have = min(SL, kb1 - kb);
        if (elect_one()) {
          const uint32_t bar = full_bar(ring.stage), dst = base + ring.stage * L::kStageBytes + (w_producer ? L::kABytes : 0);
          if (kb + have <= p.full_slabs) {  // slabs past the end of a range are loaded and not used
            mbar_arrive_expect_tx(bar, SL * slab_bytes);
            tma_load_3d(dst, w_producer ? &tm_w : &tm_a, bar, 0, row, kb);
          } else {  // the stage of the ragged slab
            mbar_arrive_expect_tx(bar, (uint32_t)have * slab_bytes);
            for (int sl = 0; sl < have; ++sl)
              tma_load_2d(dst + sl * slab_bytes, w_producer ? &p.w_tail : &p.a_tail, bar, (kb + sl) * BK, row);
          }
        }
        __syncwarp();
        ring.arm();
        ring.advance();
        if (w_producer && it == 0 && kb == kb0 + (STAGES - 1) * SL && elect_one()) {
          // the ring is full: until its first stage is free, pull the boxes behind it towards L2
          for (int kp = kb + SL; kp < kb1 && kp < kb0 + kPrefetchSteps && kp < p.full_slabs; kp += SL)
            tma_prefetch_l2_3d(&tm_w, 0, row, kp);
        }
      }
    }
    if (a_producer) grid_launch_dependents();  // last loads issued: the next kernel may be scheduled
    ring.drain(full_bar(0));
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      uint32_t it = 0;
      for (int tile = tile_first; ok && tile < p.num_tiles; tile += tile_stride, ++it) {
        const uint32_t acc = it & 1u, acc_phase = (it >> 1) & 1u;
        ok = wait_bounded_one(tempty_bar(acc), acc_phase ^ 1, abort_flag, (2u << 24) | (2u << 16) | (it & 0xFFFF));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; kb += SL) {
          ok = wait_bounded_one(full_bar(stage), phase, abort_flag, (2u << 24) | (3u << 16) | (it & 0xFFFF));
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = base + stage * L::kStageBytes;
#pragma unroll
          for (int sl = 0; sl < SL; ++sl) {
            if (kb + sl >= kb1) break;
            // the activation slabs follow each other at the size of the box that brought them
            const uint64_t da = make_kmajor_sw128_desc(sa + sl * p.a_bytes);
            const uint64_t db = make_kmajor_sw128_desc(sa + L::kABytes + sl * BN * BK);
#pragma unroll
            for (int j = 0; j < BK / 32; ++j)
              mma_f8f6f4(d_tmem, da + 2 * j, db + 2 * j, kIdesc, (kb + sl > kb0 || j > 0) ? 1u : 0u);
          }
          mma_commit(empty_bar(stage));
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        mma_commit(tfull_bar(acc));
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue warps: 32 columns of a quadrant's rows
    const int quad = warp & 3, c0 = ((warp - 2) >> 2) * 32;
    bool ok = true;
    uint32_t it = 0;
    grid_dependency_wait();
    for (int tile = tile_first; ok && tile < p.num_tiles; tile += tile_stride, ++it) {
      int m_blk, n_blk;
      tile_coords(p, tile, m_blk, n_blk);
      const uint32_t acc = it & 1u, acc_phase = (it >> 1) & 1u;
      const int m = m_blk * BM + quad * quad_rows + lane, n0 = n_blk * BN + c0;
      const bool row_ok = lane < quad_rows && m < p.M;
      // this tile's scales and bias, fetched under the main loop: lane l holds column n0 + l; what is absent is a factor
      // of 1 or an addend of -0
      float rs = 1.0f, cs = 1.0f, bs = -0.0f;
      if constexpr (kDequant) {
        if (row_ok && p.row) rs = __ldg(p.row + (int64_t)m * p.row_stride);
        if (n0 + lane < p.N) {
          if (p.col) cs = __ldg(p.col + (int64_t)(n0 + lane) * p.col_stride);
          if (p.bias)
            bs = p.bias_dtype == IFLB200_F32 ? __ldg(reinterpret_cast<const float*>(p.bias) + n0 + lane)
                                             : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[n0 + lane]);
        }
      }
      ok = wait_bounded(tfull_bar(acc), acc_phase, abort_flag, (3u << 24) | (4u << 16) | (it & 0xFFFF));
      if (!ok) break;
      tc_fence_after();
      uint32_t r[32];
      tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(quad * 32) << 16) + acc * BN + c0, r);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_bar(acc));
      if constexpr (kDequant) {
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float a = __uint_as_float(r[i]), b = __uint_as_float(r[i + 1]);
          const float ca = __shfl_sync(0xFFFFFFFFu, cs, i), cb = __shfl_sync(0xFFFFFFFFu, cs, i + 1);
          const float ba = __shfl_sync(0xFFFFFFFFu, bs, i), bb = __shfl_sync(0xFFFFFFFFu, bs, i + 1);
          if (p.exact == 2) {  // (acc * (row * col)) + bias, each operation rounded (scalar: see gemm_tokens.cuh)
            a = __fadd_rn(__fmul_rn(a, __fmul_rn(rs, ca)), ba);
            b = __fadd_rn(__fmul_rn(b, __fmul_rn(rs, cb)), bb);
          } else {  // ((acc * row) * col) + bias, the addition contracted with the last factor there is
            if (!p.exact) {
              const uint32_t w = pack_bf16x2(a, b);
              a = __uint_as_float(w << 16);
              b = __uint_as_float(w & 0xFFFF0000u);
            }
            const uint64_t x = pack2(a, b), r2 = pack2(rs, rs), b2 = pack2(ba, bb);
            unpack2(p.col ? fma2(mul2(x, r2), pack2(ca, cb), b2) : fma2(x, r2, b2), a, b);
          }
          r[i] = __float_as_uint(a);
          r[i + 1] = __float_as_uint(b);
        }
      }
      const int valid = row_ok ? min(32, p.N - n0) : 0;  // a multiple of 16, or not positive
      if constexpr (EPI == LEAN_F32 && AR == 128) {
        // Many tiles of fp32 are bound by their stores, so whole 128-byte pieces of four rows leave at a time, through shared
        // memory (16-byte pieces swizzled by the row): 0.93 of the time of 16 bytes of 32 rows over 261 sizes
        // (1946 x 224 x 1744 8.7 -> 7.1 us); 16 columns, half of a piece, 1.05.
        const uint32_t mine = base + L::kStagingOffset + (uint32_t)(warp - 2) * L::kStaging;
        __syncwarp();  // the rows of the tile before this one have been read
#pragma unroll
        for (int j = 0; j < 8; ++j)
          st_shared_v4(mine + lane * 128 + ((j ^ (lane & 7)) << 4), make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]));
        __syncwarp();
        const int row0 = m_blk * BM + quad * 32, piece = lane & 7;
        float* o = reinterpret_cast<float*>(p.out) + (int64_t)row0 * p.ld_out + n0 + 4 * piece;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int t = 4 * i + (lane >> 3);
          const uint4 v = ld_shared_v4(mine + t * 128 + ((piece ^ (t & 7)) << 4));
          if (row0 + t < p.M && n0 + 4 * piece < p.N) *reinterpret_cast<uint4*>(o + (int64_t)t * p.ld_out) = v;
        }
      } else if constexpr (kWide) {
        float* o = reinterpret_cast<float*>(p.out) + ((EPI == LEAN_PLANES ? (int64_t)part * p.M : 0) + m) * p.ld_out + n0;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (4 * j < valid) *reinterpret_cast<uint4*>(o + 4 * j) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      } else {
        uint16_t* o = reinterpret_cast<uint16_t*>(p.out) + (int64_t)m * p.ld_out + n0;
        const bool f16 = EPI == LEAN_DEQUANT && p.out_dtype == IFLB200_F16;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float a = __uint_as_float(r[8 * j + 2 * i]), b = __uint_as_float(r[8 * j + 2 * i + 1]);
            v[i] = f16 ? pack_f16x2(a, b) : pack_bf16x2(a, b);
          }
          if (8 * j < valid) *reinterpret_cast<uint4*>(o + 8 * j) = make_uint4(v[0], v[1], v[2], v[3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace iflb200
