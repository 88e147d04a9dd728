// The skinny FP8 GEMM: 64-wide tiles of up to 128 activation rows, one K range or split-K planes (included by
// gemm_fp8_sm100.cu).
//
// A launch over 50 rows takes 3 to 5 us, most of it latencies in a row: the kernel before it, first operands, MMAs,
// epilogue, completion.  It fetches its instructions cold, so the kernel holds nothing that such a launch does not run:
// the output kind is a template argument, and the accumulator goes to memory straight from registers.  With one epilogue for all
// output kinds, through shared memory and TMA, the last store of a 64 x 4096 x 1024 launch was issued 2600 clocks after its
// last MMA.
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
  static constexpr int kBarOffset = kStages * kStageBytes;
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
  GEMM_TRACE_BEGIN();
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
  if (threadIdx.x == 0) GEMM_TRACE(2);  // barriers initialised, tensor memory allocated

  // As in the other forms: up to kEarlyWeightsMaxRows only the activations and the epilogue wait for the kernel before this one.
  const bool w_producer = warp == 0, a_producer = warp == 10;
  if (w_producer || a_producer) {
    // ------------------------------------------------------------------ TMA producers
    bool waited = w_producer && p.M <= kEarlyWeightsMaxRows;
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
          const bool whole = kb + have <= p.full_slabs;  // slabs past the end of a range are loaded and not used
          mbar_arrive_expect_tx(bar, (whole ? (uint32_t)SL : (uint32_t)have) * slab_bytes);
          // The activations' dependency wait stands directly before their first load: everything ahead of it has been
          // fetched and computed when the kernel before this one ends.  At the top of the loop it left 930 clocks from the end
          // of the wait to the load, most of it cold instructions; now 170 (18 expert layers 372 -> 351 us).
          if (!waited) {
            grid_dependency_wait();
            if (a_producer) GEMM_TRACE(3);  // the kernel before this one has completed
          }
          waited = true;
          if (whole) {
            tma_load_3d(dst, w_producer ? &tm_w : &tm_a, bar, 0, row, kb);
          } else {  // the stage of the ragged slab
            for (int sl = 0; sl < have; ++sl)
              tma_load_2d(dst + sl * slab_bytes, w_producer ? &p.w_tail : &p.a_tail, bar, (kb + sl) * BK, row);
          }
          if (a_producer && it == 0 && kb == kb0) GEMM_TRACE(14);  // first activations asked for
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
    if (a_producer) {  // last loads issued: the next kernel may be scheduled
      grid_dependency_wait();  // (a lane that has issued no load has not waited yet)
      grid_launch_dependents();
    }
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
          if (it == 0 && kb == kb0) GEMM_TRACE(4);  // first operands have landed
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
        if (it == 0) GEMM_TRACE(5);  // last MMA of the first tile issued
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue warps: 32 columns of a quadrant's rows
    // Tensor memory is read in the 16 x 256-bit shape: a thread holds two neighbouring columns of rows r4 and r4 + 8 of
    // every eight, so that four lanes write a whole 32-byte sector of a row (fp32, straight from the registers), or after
    // a 4 x 4 transpose among them 64 bytes (two-byte outputs).  A lane per row wrote half a sector at a time, and up to 64
    // rows half of the lanes held nothing: 64 x 4096 x 1024 with scales 3.68 -> 3.18 us behind one another, 50 x 1024 x 4096 in
    // eight planes 3.44 -> 3.26, 18 expert layers 381 -> 368; over 147 sizes dequantised 0.96 of the time, planes 0.95, raw 1.00.
    constexpr int kBlocks = AR / 64;  // sixteens of rows of a quadrant
    const int quad = warp & 3, c0 = ((warp - 2) >> 2) * 32;
    const int r4 = lane >> 2, c4 = lane & 3;
    bool ok = true;
    uint32_t it = 0;
    grid_dependency_wait();
    for (int tile = tile_first; ok && tile < p.num_tiles; tile += tile_stride, ++it) {
      int m_blk, n_blk;
      tile_coords(p, tile, m_blk, n_blk);
      const uint32_t acc = it & 1u, acc_phase = (it >> 1) & 1u;
      const int m0 = m_blk * BM + quad * quad_rows + r4, n0 = n_blk * BN + c0;
      // where this thread's first row goes, and the rows and columns that there are from it on
      constexpr int kEs = kWide ? 4 : 2;
      uint8_t* out = reinterpret_cast<uint8_t*>(p.out) + ((EPI == LEAN_PLANES ? (int64_t)part * p.M : 0) + m0) * p.ld_out * kEs +
                     (int64_t)(n0 + (kWide ? 2 : 8) * c4) * kEs;
      const int64_t eight_rows = 8 * p.ld_out * kEs;
      const int rows = p.M - m0, columns = p.N - n0;
      // this tile's scales and bias, fetched under the main loop; what is absent is a factor of 1 or an addend of -0
      float rs[2 * kBlocks], cs[8], bs[8];
      if constexpr (kDequant) {
#pragma unroll
        for (int i = 0; i < 2 * kBlocks; ++i) {
          const int m = m0 + 8 * i;
          rs[i] = p.row && m < p.M ? __ldg(p.row + (int64_t)m * p.row_stride) : 1.0f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int n = n0 + 8 * (i >> 1) + 2 * c4 + (i & 1);
          cs[i] = p.col && n < p.N ? __ldg(p.col + (int64_t)n * p.col_stride) : 1.0f;
          bs[i] = !p.bias || n >= p.N ? -0.0f
                  : p.bias_dtype == IFLB200_F32 ? __ldg(reinterpret_cast<const float*>(p.bias) + n)
                                                : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[n]);
        }
      }
      ok = wait_bounded(tfull_bar(acc), acc_phase, abort_flag, (3u << 24) | (4u << 16) | (it & 0xFFFF));
      if (!ok) break;
      if (warp == 2 && lane == 0 && it == 0) GEMM_TRACE(6);  // first accumulator complete
      tc_fence_after();
      uint32_t r[kBlocks][16];  // r[b][4j + 2h + e]: row 16 b + 8 h + r4, column 8 j + 2 c4 + e
      const uint32_t t_acc = tmem_base + ((uint32_t)(quad * 32) << 16) + acc * BN + c0;
#pragma unroll
      for (int b = 0; b < kBlocks; ++b) tmem_ld_16x256b_x4(t_acc + ((uint32_t)(16 * b) << 16), r[b]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_bar(acc));
#pragma unroll
      for (int b = 0; b < kBlocks; ++b) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (16 * b + 8 * h >= rows + r4) continue;  // none of the warp's
          const bool in = 16 * b + 8 * h < rows;
          uint8_t* o = out + (2 * b + h) * eight_rows;
          uint32_t v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float x = __uint_as_float(r[b][4 * j + 2 * h]), y = __uint_as_float(r[b][4 * j + 2 * h + 1]);
            if constexpr (kDequant) {
              const float rsc = rs[2 * b + h];
              if (p.exact == 2) {  // (acc * (row * col)) + bias, each operation rounded (scalar: see gemm_tokens.cuh)
                x = __fadd_rn(__fmul_rn(x, __fmul_rn(rsc, cs[2 * j])), bs[2 * j]);
                y = __fadd_rn(__fmul_rn(y, __fmul_rn(rsc, cs[2 * j + 1])), bs[2 * j + 1]);
              } else {  // ((acc * row) * col) + bias, the addition contracted with the last factor there is
                if (!p.exact) {
                  const uint32_t w = pack_bf16x2(x, y);
                  x = __uint_as_float(w << 16);
                  y = __uint_as_float(w & 0xFFFF0000u);
                }
                const uint64_t x2 = pack2(x, y), r2 = pack2(rsc, rsc), b2 = pack2(bs[2 * j], bs[2 * j + 1]);
                unpack2(p.col ? fma2(mul2(x2, r2), pack2(cs[2 * j], cs[2 * j + 1]), b2) : fma2(x2, r2, b2), x, y);
              }
            }
            if constexpr (kWide) {
              if (in && 8 * j < columns) *reinterpret_cast<float2*>(o + 32 * j) = make_float2(x, y);
            } else {
              v[j] = EPI == LEAN_DEQUANT && p.out_dtype == IFLB200_F16 ? pack_f16x2(x, y) : pack_bf16x2(x, y);
            }
          }
          if constexpr (!kWide) {
            // lane c4 of four hands over its columns of the other lanes' eights and ends up with eight columns of its own
            const bool odd = c4 & 1, high = c4 & 2;
            const uint32_t s0 = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[0] : v[1], 1), s1 = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[2] : v[3], 1);
            const uint32_t w0 = odd ? s0 : v[0], w1 = odd ? v[1] : s0, w2 = odd ? s1 : v[2], w3 = odd ? v[3] : s1;
            const uint32_t u0 = __shfl_xor_sync(0xFFFFFFFFu, high ? w0 : w2, 2), u1 = __shfl_xor_sync(0xFFFFFFFFu, high ? w1 : w3, 2);
            if (in && 8 * c4 < columns)
              *reinterpret_cast<uint4*>(o) = high ? make_uint4(u0, u1, w2, w3) : make_uint4(w0, w1, u0, u1);
          }
        }
      }
    }
    if (warp == 2 && lane == 0) GEMM_TRACE(7);  // last store issued
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
    if (lane == 0) GEMM_TRACE(9);  // all roles done
  }
}

}  // namespace iflb200
