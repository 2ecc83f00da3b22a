// Implicit-GEMM convolution for problems of up to one wave of tiles: 64 x 32 or 64 x 64 output tiles, one per CTA.
//
// What bounds a call with few tiles is one CTA's walk over Kgemm while other SMs idle, and the cost of the launch around it.
// Cutting Kgemm between CTAs would shorten the walk, but would make the order of summation, and so the last bit, depend on
// the batch size; it stays whole here. A step of the walk is bound by issuing copies -- ~140 cycles each, whatever their
// size -- so a stage holds two 128-byte k-steps, and B (and A, where a 1x1 convolution makes it a plain matrix) comes in one
// copy for both. 2048 -> 512 channels on one 7x7 image 8.3 -> 5.1 us, 64 x 1000 x 2048 product 8.7 -> 5.3.
//
// Not persistent, no double buffering: with one tile per CTA there is nothing to overlap. What is left is kept short: 100 KB
// of shared memory and 64 TMEM columns at most, so that the next launch's CTAs come up beside this one's; the weights' first
// k-steps are prefetched into L2 before the previous kernel on the stream has ended; bias and residual are fetched while the
// accumulator is being computed. 1x1 64->64 on one 56x56 image 3.5 -> 2.6 us.
#pragma once
#include "conv2d_sm100.cuh"

namespace tb200 {

constexpr int kSmallM = 64;
constexpr int kSmallThreads = 192;     // warp 0 TMA, warp 1 MMA, warps 2..5 epilogue
constexpr int kSmallMaxStages = 4;
constexpr int kSmallRingBytes = 96 * 1024;

// a stage: the two k-steps' rows of A, then the two k-steps' rows of B
__host__ __device__ constexpr int small_stage_bytes(int bn) { return 2 * (kSmallM + bn) * kStageKBytes; }
__host__ __device__ constexpr int small_stages(int bn) { return kSmallRingBytes / small_stage_bytes(bn); }
__host__ __device__ constexpr int small_smem_bytes(int bn, int stages) {
  return 1024 + stages * small_stage_bytes(bn) + 256;
}

// M = 64 accumulators use 16 of the 32 TMEM lanes of each epilogue warp: row i of the tile is lane 32 * (i / 16) + i % 16.
template <typename OutT, int BN>
__global__ void __launch_bounds__(kSmallThreads, 2)
conv2d_small_sm100_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                          const __grid_constant__ ConvKernelArgs args) {
  using namespace ptx;
  constexpr uint32_t kAStep = kSmallM * kStageKBytes, kBStep = BN * kStageKBytes;   // one k-step of each operand
  constexpr uint32_t kABytes = 2 * kAStep;
  constexpr uint32_t kStageBytes = kABytes + 2 * kBStep;
  constexpr int kVec = 16 / sizeof(OutT);
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = __shfl_sync(0xffffffffu, (smem_u32(smem_raw) + 1023u) & ~1023u, 0);
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const int num_stages = args.num_stages;
  const uint32_t bar_off = static_cast<uint32_t>(num_stages) * kStageBytes;
  const uint32_t bar_base = smem_base + bar_off;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kSmallMaxStages + s); };
  const uint32_t tfull_bar = bar_base + 8u * (2 * kSmallMaxStages);
  const uint32_t tmem_slot = tfull_bar + 8u;
  volatile uint32_t* tmem_slot_p = reinterpret_cast<volatile uint32_t*>(smem_gen + bar_off + 8u * (2 * kSmallMaxStages + 1));
  volatile uint32_t* abort_p = tmem_slot_p + 1;

  const int k_steps = args.total_chunks;             // 128-byte chunks only
  const int k_stages = (k_steps + 1) / 2;
  const int m_tile = static_cast<int>(blockIdx.x) / args.num_n_tiles;
  const int n_base = (static_cast<int>(blockIdx.x) - m_tile * args.num_n_tiles) * BN;
  const int m0 = args.m_begin + m_tile * kSmallM;

  if (threadIdx.x == 0) {
    for (int s = 0; s < num_stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(tfull_bar, 1);
    *abort_p = 0u;
    fence_mbar_init();
    prefetch_tmap(&tmap_x);
    prefetch_tmap(&tmap_w);
    // a hint only: whatever an earlier kernel still writes there is read after griddep_wait below
    for (int i = 0; i < min(k_stages, num_stages) && args.b_prefetch; ++i) {
      if (args.b_n_groups > 0) tma_prefetch_3d(&tmap_w, n_base, 2 * i * args.chunk_elems, 0);
      else tma_prefetch_3d(&tmap_w, 0, n_base, 2 * i);
    }
  }
  if (warp == 1) {
    tmem_alloc<BN>(tmem_slot);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot_p, 0);
  // see the general kernel for the order of the two and for the modes
  if (args.pdl_mode == 1) {
    griddep_wait();
    griddep_launch_dependents();
  } else {
    griddep_launch_dependents();
    if (args.pdl_mode != 2) griddep_wait();
  }

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (uniform control flow, one lane issues)
    const uint32_t issue = elect_one_lane();
    const int t = m0 / args.Wo;
    const int w_start = (m0 - t * args.Wo) * args.stride_w - args.pad_w;
    const int img0 = t / args.Ho;
    const int h_start = (t - img0 * args.Ho) * args.stride_h - args.pad_h;
    int c_coord = 0, k_coord = args.b_k0, tap_coord = 0, tap_s = 0;
    uint32_t off_w = 0, off_h = 0;
    // B two k-steps at a time: {0, n, chunk} of an [N][K] matrix, or {n, k, 0} of a row-major [K][N] one
    const bool n_major = args.b_n_groups > 0;
    const int b_c0 = n_major ? n_base : 0, b_d1 = n_major ? 2 * args.chunk_elems : 0, b_d2 = n_major ? 0 : 2;
    int b_c1 = n_major ? 0 : n_base, b_c2 = 0;
    int stage = 0, issued = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int it = 0; it < k_stages; ++it) {
      if (issued == args.test_producer_stop) break;   // test hook: go silent, leave normally
      if (it >= num_stages && !mbar_wait_bounded_uniform(empty_bar(stage), phase ^ 1u, abort_p, args.wait_limit)) {
        if (issue) report_error(args, abort_p, kErrProducerWait, static_cast<uint32_t>(it));
        ok = false;
        break;
      }
      const uint32_t full = full_bar(stage);
      const uint32_t a_dst = smem_base + static_cast<uint32_t>(stage) * kStageBytes;
      const uint32_t b_dst = a_dst + kABytes;
      const uint32_t steps = 2 * it + 1 < k_steps ? 2u : 1u;     // an odd last k-step has its stage to itself
      mbar_arrive_expect_tx_if(issue, full, (args.a_steps2 ? 2u : steps) * kAStep + (args.b_steps2 ? 2u : steps) * kBStep);
      // both k-steps in one copy; past the last one it reads zeros
      if (args.a_steps2) tma_load_3d_if(issue, a_dst, &tmap_x, full, 0, m0, 2 * it);
      if (args.b_steps2) {
        tma_load_3d_if(issue, b_dst, &tmap_w, full, b_c0, b_c1, b_c2);
        b_c1 += b_d1;
        b_c2 += b_d2;
      }
      if (!args.a_steps2 || !args.b_steps2) {
        for (uint32_t u = 0; u < steps; ++u) {
          if (!args.a_steps2)
            tma_load_im2col_4d_if(issue, a_dst + u * kAStep, &tmap_x, full, c_coord, w_start, h_start, img0,
                                  static_cast<uint16_t>(off_w), static_cast<uint16_t>(off_h));
          if (!args.b_steps2) tma_load_3d_if(issue, b_dst + u * kBStep, &tmap_w, full, k_coord, tap_coord, n_base);
          k_coord += args.chunk_elems;
          c_coord += args.chunk_elems;
          if (c_coord == args.C) {
            c_coord = 0;
            k_coord += args.b_jump_s;
            tap_coord += args.b_tap_step;
            off_w += args.dil_w;
            if (++tap_s == args.S) {
              tap_s = 0;
              off_w = 0;
              off_h += args.dil_h;
              k_coord += args.b_jump_r;
            }
          }
        }
      }
      ++issued;
      if (++stage == num_stages) { stage = 0; phase ^= 1u; }
    }
    // never leave with copies in flight into this CTA's shared memory
    if (ok) {
      const int pending = issued < num_stages ? issued : num_stages;
      if (issued < num_stages) { stage = 0; phase = 1u; }   // the oldest filled stage; its first release has parity 0
      for (int i = 0; i < pending; ++i) {
        if (!mbar_wait_bounded_uniform(empty_bar(stage), phase ^ 1u, abort_p, args.wait_limit)) break;
        if (++stage == num_stages) { stage = 0; phase ^= 1u; }
      }
    } else {
      const long long t0 = clock64();
      while (clock64() - t0 < 2000000LL) { __nanosleep(1000); }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (uniform control flow, one lane issues)
    const uint32_t issue = elect_one_lane();
    constexpr bool kTf32 = OutTraits<OutT>::kTf32;
    const uint32_t desc_hi = ((args.a_sbo >> 4) & 0x3FFFu) | (1u << 14) | ((args.swizzle_mode & 7u) << 29);
    uint32_t a_k[4], b_k[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a_k[k] = __shfl_sync(0xffffffffu, ((smem_base + args.a_mma_off[k]) >> 4) | (((args.a_lbo >> 4) & 0x3FFFu) << 16), 0);
      b_k[k] = __shfl_sync(0xffffffffu, ((smem_base + kABytes + args.b_mma_off[k]) >> 4) | (((args.b_lbo >> 4) & 0x3FFFu) << 16), 0);
    }
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    bool stage_ready = false;
    for (int it = 0; it < k_stages; ++it) {
      if (!stage_ready && !mbar_wait_bounded_uniform(full_bar(stage), phase, abort_p, args.wait_limit)) {
        if (issue) report_error(args, abort_p, kErrMmaWaitFull, static_cast<uint32_t>(it));
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t a_off = static_cast<uint32_t>(stage) * (kStageBytes >> 4), b_off = a_off;
      const uint32_t empty = empty_bar(stage);
      if (++stage == num_stages) { stage = 0; phase ^= 1u; }
      if (2 * it + 1 < k_steps) {               // the stage's first k-step of two
        if (it == 0)
          mma_step4<kTf32, false>(tmem_base, a_k[0] + a_off, a_k[1] + a_off, a_k[2] + a_off, a_k[3] + a_off, b_k[0] + b_off,
                                  b_k[1] + b_off, b_k[2] + b_off, b_k[3] + b_off, desc_hi, args.idesc, issue);
        else
          mma_step4<kTf32, true>(tmem_base, a_k[0] + a_off, a_k[1] + a_off, a_k[2] + a_off, a_k[3] + a_off, b_k[0] + b_off,
                                 b_k[1] + b_off, b_k[2] + b_off, b_k[3] + b_off, desc_hi, args.idesc, issue);
        a_off += kAStep >> 4;
        b_off += kBStep >> 4;
      }
      bool next_ready;
      if (k_steps == 1)
        next_ready = mma_stage4_probe<kTf32, false>(tmem_base, a_k[0] + a_off, a_k[1] + a_off, a_k[2] + a_off, a_k[3] + a_off,
                                                    b_k[0] + b_off, b_k[1] + b_off, b_k[2] + b_off, b_k[3] + b_off, desc_hi,
                                                    args.idesc, empty, full_bar(stage), phase, issue);
      else
        next_ready = mma_stage4_probe<kTf32, true>(tmem_base, a_k[0] + a_off, a_k[1] + a_off, a_k[2] + a_off, a_k[3] + a_off,
                                                   b_k[0] + b_off, b_k[1] + b_off, b_k[2] + b_off, b_k[3] + b_off, desc_hi,
                                                   args.idesc, empty, full_bar(stage), phase, issue);
      stage_ready = __all_sync(0xffffffffu, next_ready);
    }
    if (ok && issue) mma_commit(tfull_bar);
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue: one pixel per lane, lanes 0..15
    const int quarter = warp & 3;
    const int m = m0 + quarter * 16 + lane;
    const bool row_ok = lane < 16 && m < args.M;
    OutT* __restrict__ out = static_cast<OutT*>(args.out);
    const OutT* res = static_cast<const OutT*>(args.residual);
    const int pq = m / args.Wo;
    const int wo = m - pq * args.Wo;
    const int img = pq / args.Ho;
    const int ho = pq - img * args.Ho;
    out += img * args.out_sn + ho * args.out_sh + wo * args.out_sw;
    if (res != nullptr) res += img * args.res_sn + ho * args.res_sh + wo * args.res_sw;
    const bool rows = args.out_rows != 0;            // channel-contiguous output and residual
    constexpr int kBlocks = BN / 32;
    constexpr int kChunks = 32 / kVec;               // 16-byte chunks of 32 columns
    float bias_l[kBlocks];
    uint4 res_c[kBlocks][kChunks];
#pragma unroll
    for (int h = 0; h < kBlocks; ++h) {
      const int n = n_base + h * 32 + lane;
      bias_l[h] = 0.0f;
      if (args.bias != nullptr && n < args.K_out)
        bias_l[h] = args.bias_is_f32 ? static_cast<const float*>(args.bias)[n]
                                     : OutTraits<OutT>::to_f(static_cast<const OutT*>(args.bias)[n]);
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        res_c[h][c] = make_uint4(0u, 0u, 0u, 0u);
        const int col = n_base + h * 32 + c * kVec;
        if (rows && res != nullptr && row_ok && col < args.K_out) {
          if (args.res_vec == 16) {
            res_c[h][c] = *reinterpret_cast<const uint4*>(res + col);
          } else {
            OutT* e = reinterpret_cast<OutT*>(&res_c[h][c]);
#pragma unroll
            for (int j = 0; j < kVec; ++j)
              if (col + j < args.K_out) e[j] = res[col + j];
          }
        }
      }
    }
    const bool ready = mbar_wait_bounded_uniform(tfull_bar, 0u, abort_p, 2 * args.wait_limit);
    if (!ready) {
      if (lane == 0) report_error(args, abort_p, kErrEpilogueWait, blockIdx.x);
    } else {
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < kBlocks; ++h) {
        const int n_first = n_base + h * 32;
        if (n_first >= args.K_out) break;            // warp-uniform
        uint32_t v[32];
        tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + h * 32, v);
        tmem_ld_wait();
        float f[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]) + __shfl_sync(0xffffffffu, bias_l[h], j);
        if (!rows) {
          store_strided32<OutT>(args, f, res != nullptr ? res + n_first * args.res_sc : nullptr, out + n_first * args.out_sc,
                                args.K_out - n_first, row_ok, lane);
          continue;
        }
        uint4 packed[kChunks];
        if (args.act == kActRelu) {
          finish32<OutT, true>(f, res_c[h], res != nullptr, packed);
        } else {
          if (res != nullptr) {
#pragma unroll
            for (int c = 0; c < kChunks; ++c) add16<OutT>(f + c * kVec, res_c[h][c]);
          }
          apply_act32<sizeof(OutT) == 2>(f, args.act);
          finish32<OutT, false>(f, res_c[h], false, packed);
        }
        if (row_ok) {
#pragma unroll
          for (int c = 0; c < kChunks; ++c) {
            const int col = n_first + c * kVec;
            if (col >= args.K_out) break;
            if (args.out_vec == 16) {
              *reinterpret_cast<uint4*>(out + col) = packed[c];
            } else {
              const OutT* e = reinterpret_cast<const OutT*>(&packed[c]);
#pragma unroll
              for (int j = 0; j < kVec; ++j)
                if (col + j < args.K_out) out[col + j] = e[j];
            }
          }
        }
      }
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<BN>(tmem_base);
  }
  if (args.pdl_mode == 2) griddep_wait();   // do not complete before the launch in front of this one has
}

}  // namespace tb200
