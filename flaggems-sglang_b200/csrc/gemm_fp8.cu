// Grouped expert GEMMs for FP8 (e4m3) weights with one fp32 scale per 128x128 block and
// activations quantised per token and 128-wide group.
//
// The hardware's block-scaled MMA wants power-of-two scales per 32 elements, not fp32 scales
// per 128, so the scaling is done on the CUDA cores: every 128-wide slice of the reduction
// (one pipeline stage = one swizzle row of FP8) is multiplied into a fresh partial
// accumulator in tensor memory (4 x tcgen05.mma.kind::f8f6f4, K = 32 each); the promotion
// warps read it back, scale it by a_scale[token, slice] * w_scale[row block, slice] and add it
// to accumulators they keep in registers, while the MMA thread is already filling the other
// partial buffer.  Weight rows sit on the MMA's M side, the token block (16/32/64) on N, so
// the promotion costs 2*BT FMAs per thread and slice.
//
// A tile is two 128-row weight blocks that share the token block:
//   mode 0: gate rows n0.. and up rows I+n0..; tail = SiLU*mul, rounding to the 16-bit type,
//           dynamic 1x128 quantisation (the 128 lanes are exactly one group) -> e4m3 + scale.
//   mode 1: rows n0.. and n0+128.. of the down projection; tail = routing weight and
//           red.global.add.f32 into the combine buffer (K may be split across CTAs).
// Blocks of 128 tokens run in a launch of their own kind (moe_gemm_fp8_mixed_kernel, below).
//
// Warps of these kernels: TMA producer, MMA issuer (owns tensor memory), four promotion warps per group of up
// to 32 tokens (one group for blocks of 16 and 32, two for blocks of 64), and a
// loader warp that prepares the next tile's per-token tables (output row, routing weight,
// activation scales by bulk copy, weight scales) in double-buffered shared memory, so that no
// global-memory latency sits between two tiles of the promotion warps.
#include "gemm_route.cuh"
#include "gemm_sched.cuh"

namespace b200moe {

namespace {

constexpr int kMaxKB = 64;  // 128-wide reduction slices per tile whose scales are staged in shared memory
__host__ __device__ constexpr int fp8_threads(int ng) { return 7 * 32 + (ng - 1) * 128; }

// A CTA's share of a launch: tiles cta, cta + c.grid_eff, ... of c.total.
struct Fp8Part {
  Ctrl c;
  int cta;
  const int* off;   // [E+1] blocks of this share before expert e
  const int* blk;   // [E+1] blocks before expert e
  int rows;         // padded rows of a block
};
__device__ __forceinline__ TileCoord part_tile(int id, const Fp8Part& p, const GemmArgs& a, int tile_n) {
  TileCoord t = decode_tile(id, p.c, p.off, a.E, 1, a.num_nt, a.kblocks, tile_n);
  t.row0 = (p.blk[t.e] + t.row0 - p.off[t.e]) * p.rows;
  return t;
}

// NG = promotion groups; group g owns token columns [g * BT / NG, (g + 1) * BT / NG)
// MIXED: part of a launch with two kinds of tiles (moe_gemm_fp8_mixed_kernel), which hands over its share and the tensor memory
template <int MODE, int BT, int NG, bool MIXED>
__device__ __forceinline__ void weights_on_m(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const GemmArgs& a, uint8_t* smem,
                                             const int stages, Fp8Part& part, uint32_t tmem_base) {
  constexpr int W_BYTES = 2 * kTileBytes;
  constexpr int X_BYTES = BT * kStageKBytes;
  constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
  constexpr int PCOLS = 2 * BT;  // columns of one partial accumulator (both row blocks)
  constexpr int NPB = (512 / PCOLS) >= 4 ? 4 : 2;  // partial accumulators in flight
  uint8_t* ctrl_base = smem + static_cast<size_t>(stages) * STAGE_BYTES;
  float* s_xs = reinterpret_cast<float*>(ctrl_base);                    // [2][kMaxKB][BT] activation scales
  float* s_ws = s_xs + 2 * kMaxKB * BT;                                 // [2][2][kMaxKB] weight scales
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(s_ws + 2 * 2 * kMaxKB);
  uint64_t* bar_empty = bar_full + stages;
  uint64_t* bar_pfull = bar_empty + stages;
  uint64_t* bar_pempty = bar_pfull + 4;
  uint64_t* bar_sfull = bar_pempty + 4;   // per-tile tables ready
  uint64_t* bar_sempty = bar_sfull + 2;   // per-tile tables released
  uint64_t* bar_meet = bar_sempty + 2;    // [NG] meeting point of a promotion group's four warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_meet + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* s_col_row = reinterpret_cast<int*>(tmem_slot + 4);               // [2][128]
  float* s_col_gam = reinterpret_cast<float*>(s_col_row + 2 * 128);     // [2][128]
  float* s_red = s_col_gam + 2 * 128;                                   // [2][NG][4][64]
  // [2][128] mode 1: base of each token's output row
  unsigned long long* s_col_ptr = reinterpret_cast<unsigned long long*>(s_red + 2 * 2 * 4 * 64);
  const RowTables rt = row_tables(s_col_ptr + 2 * 128, a.E);            // own tables, or only the blocks' starts
  int* s_blk_off = rt.blk;                                              // [E+1]
  constexpr int CPT = BT / NG;                                          // token columns per promotion thread

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const bool own = !MIXED && BT <= 32 && a.route.own != 0, early = own && a.route.early != 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int s = 0; s < 4; ++s) {
      mbar_init(smem_u32(&bar_pfull[s]), 1);
      mbar_init(smem_u32(&bar_pempty[s]), 4 * NG);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bar_sfull[s]), 1);
      mbar_init(smem_u32(&bar_sempty[s]), 4 * NG);
      mbar_init(smem_u32(&bar_meet[s]), 4);
    }
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    prefetch_tmap(&tm_w);
    prefetch_tmap(&tm_x);
  }
  if constexpr (!MIXED) {
    if (warp == 1) {
      tmem_alloc(smem_u32(tmem_slot), static_cast<uint32_t>(a.tmem_cols));
      tmem_relinquish();
    }
    // everything above touched only shared / tensor memory and kernel parameters
    if (!early) griddep_wait();
    griddep_launch_dependents();
    if (own) count_slots(a.route, a.P, a.E, BT, rt);
    else
      for (int e = threadIdx.x; e <= a.E; e += blockDim.x) s_blk_off[e] = a.blk_off[e];
    tc_fence_before();
  }
  __syncthreads();
  if constexpr (!MIXED) {
    tc_fence_after();
    tmem_base = *tmem_slot;
    part.c = make_ctrl(a, own ? s_blk_off[a.E] : a.meta[0], MODE == 1);
    part.cta = blockIdx.x;
    part.off = part.blk = s_blk_off;
    part.rows = BT;
  }
  const Ctrl& c = part.c;
  const bool active = part.cta < c.grid_eff;
  constexpr int kTileN = (MODE == 0) ? kTileRows : 2 * kTileRows;  // output rows advanced per n-tile
  // row offset of the second weight block inside the expert
  const int second_off = (MODE == 0) ? a.up_row_off : kTileRows;

  if (active && warp == 0 && elect_one()) {
    // =============================== TMA producer ===============================
    int stage = 0;
    uint32_t phase = 0;
    long long issued = 0;
    bool ok = true;
    auto load_weights = [&](const TileCoord& t, int kb, int s) {
      const uint32_t full = smem_u32(&bar_full[s]);
      const uint32_t sw = smem_u32(smem + static_cast<size_t>(s) * STAGE_BYTES);
      const int k0 = kb * kStageKBytes;  // one byte per element
      mbar_arrive_expect_tx(full, static_cast<uint32_t>(STAGE_BYTES));
      tma_load_3d(sw, &tm_w, full, k0, t.n0, t.e);
      tma_load_3d(sw + kTileBytes, &tm_w, full, k0, second_off + t.n0, t.e);  // rows past the expert zero-fill
    };
    // the ring's first round of weights, before the activations may be read
    int ahead = 0;
    if (early) {
      for (int tile = part.cta; ahead < stages && tile < c.total; tile += c.grid_eff) {
        const TileCoord t = part_tile(tile, part, a, kTileN);
        for (int kb = t.kb0; ahead < stages && kb < t.kb1; ++kb, ++ahead) load_weights(t, kb, ahead);
      }
      griddep_wait();
    }
    for (int tile = part.cta; ok && tile < c.total; tile += c.grid_eff) {
      const TileCoord t = part_tile(tile, part, a, kTileN);
      for (int kb = t.kb0; kb < t.kb1; ++kb) {
        if (issued >= ahead) {
          if (!mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1, abort_flag, DEV_TIMEOUT_PRODUCER)) {
            ok = false;
            break;
          }
          load_weights(t, kb, stage);
        }
        tma_load_2d(smem_u32(smem + static_cast<size_t>(stage) * STAGE_BYTES) + W_BYTES, &tm_x, smem_u32(&bar_full[stage]),
                    kb * kStageKBytes, t.row0);
        ++issued;
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    if (!ok) {
      const int n = static_cast<int>(issued < stages ? issued : stages);
      for (int i = 1; i <= n; ++i) {
        int s = stage - i;
        uint32_t ph = phase;
        if (s < 0) {
          s += stages;
          ph ^= 1;
        }
        mbar_wait_brief(smem_u32(&bar_full[s]), ph);
      }
    }
  } else if (active && warp == 1 && elect_one()) {
    // =============================== MMA issuer =================================
    const uint32_t idesc = make_idesc(0u /* e4m3 */, kTileRows, static_cast<uint32_t>(BT));
    int stage = 0;
    uint32_t phase = 0, j = 0;  // j counts reduction slices over the whole launch
    bool ok = true;
    for (int tile = part.cta; ok && tile < c.total; tile += c.grid_eff) {
      const TileCoord t = part_tile(tile, part, a, kTileN);
      for (int kb = t.kb0; kb < t.kb1; ++kb, ++j) {
        const uint32_t pb = j % NPB;
        if (!mbar_wait(smem_u32(&bar_full[stage]), phase, abort_flag, DEV_TIMEOUT_MMA) ||
            !mbar_wait(smem_u32(&bar_pempty[pb]), ((j / NPB) & 1u) ^ 1u, abort_flag, DEV_TIMEOUT_MMA)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d0 = tmem_base + pb * PCOLS;
        const uint32_t sw = smem_u32(smem + static_cast<size_t>(stage) * STAGE_BYTES);
        const uint64_t dw = smem_desc_k_sw128(sw);
        const uint64_t du = smem_desc_k_sw128(sw + kTileBytes);
        const uint64_t dx = smem_desc_k_sw128(sw + W_BYTES);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          tc_mma_f8(d0, dw + 2 * k, dx + 2 * k, idesc, k > 0 ? 1u : 0u);
          tc_mma_f8(d0 + BT, du + 2 * k, dx + 2 * k, idesc, k > 0 ? 1u : 0u);
        }
        tc_commit(smem_u32(&bar_empty[stage]));
        tc_commit(smem_u32(&bar_pfull[pb]));
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (active && warp == 6) {
    // =============================== per-tile table loader ======================
    griddep_wait();
    const int kb_total = a.kblocks;
    int iter = 0;
    for (int tile = part.cta; tile < c.total; tile += c.grid_eff, ++iter) {
      const TileCoord t = part_tile(tile, part, a, kTileN);
      const int buf = iter & 1;
      if (!mbar_wait(smem_u32(&bar_sempty[buf]), ((iter >> 1) & 1) ^ 1, abort_flag, DEV_TIMEOUT_EPILOGUE)) {
        // the scales in flight land before the CTA leaves
        for (int i = 1; i <= 2 && i <= iter; ++i) mbar_wait_brief(smem_u32(&bar_sfull[(iter - i) & 1]), ((iter - i) >> 1) & 1);
        break;
      }
      const int nkb = t.kb1 - t.kb0;
      for (int r = 0; r < BT; r += 32) {
        const int slot = rows_slot(a, rt, BT, t.e, t.row0 + r, BT < 32 ? BT : 32), cidx = r + lane;
        if (cidx >= BT) continue;
        const bool valid = slot >= 0;
        const bool pairs = MIXED && MODE == 1 && a.out_pairs != nullptr;      // the output row is the pair's own slot
        const int orow = valid ? (MODE == 1 && !pairs ? slot / a.topk : slot) : -1;
        s_col_row[buf * 128 + cidx] = orow;
        s_col_gam[buf * 128 + cidx] = rows_weight(a, rt, BT, t.e, t.row0 + r, slot);
        if (MODE == 1 && valid)
          s_col_ptr[buf * 128 + cidx] = reinterpret_cast<unsigned long long>(
              pairs ? out_row_base(a, a.out_pairs, orow, static_cast<size_t>(a.N) * 2)
                    : out_row_base(a, a.out, orow, static_cast<size_t>(a.ld_out) * sizeof(float)));
      }
      const int nb0 = t.n0 / 128, nb1 = (second_off + t.n0) / 128;
      const float* ws0 = a.w_scale + (static_cast<size_t>(t.e) * a.w_scale_rows + nb0) * kb_total + t.kb0;
      const float* ws1 = a.w_scale + (static_cast<size_t>(t.e) * a.w_scale_rows + nb1) * kb_total + t.kb0;
      const bool second_ok = nb1 < a.w_scale_rows;
      float* ws_t = s_ws + buf * 2 * kMaxKB;
      for (int i = lane; i < nkb; i += 32) {
        ws_t[i] = __ldg(ws0 + i);
        ws_t[kMaxKB + i] = second_ok ? __ldg(ws1 + i) : 0.f;
      }
      __syncwarp();
      const uint32_t sfull = smem_u32(&bar_sfull[buf]);
      if (lane == 0) mbar_arrive_expect_tx(sfull, static_cast<uint32_t>(nkb * BT * 4));
      __syncwarp();
      // one bulk copy per reduction slice: BT consecutive activation scales
      for (int i = lane; i < nkb; i += 32)
        bulk_copy_g2s(smem_u32(s_xs + (buf * kMaxKB + i) * BT),
                      a.x_scale + static_cast<size_t>(t.kb0 + i) * a.ld_xscale + t.row0, BT * 4, sfull);
    }
  } else if (active && warp >= 2 && warp != 6 && warp < fp8_threads(NG) / 32) {
    // =============================== promotion + tail ===========================
    griddep_wait();
    const int grp = warp < 6 ? 0 : 1;               // promotion group
    const int gw = warp < 6 ? warp - 2 : warp - 7;  // warp inside the group
    const int quad = warp & 3;                      // TMEM lane quadrant (each group covers all four)
    const int ep_tid = gw * 32 + lane;
    const int lrow = quad * 32 + lane;
    const int cb = grp * CPT;                       // first token column of this thread
    const bool w_on_input = (a.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0;
    uint32_t j = 0;
    uint32_t meet_phase = 0;
    int iter = 0;
    bool ok = true;
    for (int tile = part.cta; ok && tile < c.total; tile += c.grid_eff, ++iter) {
      const TileCoord t = part_tile(tile, part, a, kTileN);
      const int buf = iter & 1;
      const int* col_row = s_col_row + buf * 128 + cb;
      const float* col_gam = s_col_gam + buf * 128 + cb;
      const float* xs_t = s_xs + buf * kMaxKB * BT;
      const float* ws_t = s_ws + buf * 2 * kMaxKB;
      if (!mbar_wait(smem_u32(&bar_sfull[buf]), (iter >> 1) & 1, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;

      float acc0[CPT], acc1[CPT];
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        acc0[i] = 0.f;
        acc1[i] = 0.f;
      }

      constexpr int CH = (CPT < 32 || CPT > 32 && NG > 1) ? 16 : 32;  // columns drained from tensor memory per step
      for (int kb = t.kb0; kb < t.kb1; ++kb, ++j) {
        const float w0 = ws_t[kb - t.kb0];
        const float w1 = ws_t[kMaxKB + kb - t.kb0];
        const float4* sx = reinterpret_cast<const float4*>(xs_t + (kb - t.kb0) * BT + cb);
        const uint32_t pb = j % NPB;
        if (!mbar_wait(smem_u32(&bar_pfull[pb]), (j / NPB) & 1u, abort_flag, DEV_TIMEOUT_EPILOGUE)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + pb * PCOLS + cb;
#pragma unroll
        for (int c0 = 0; c0 < CPT; c0 += CH) {
          float g[CH], u[CH];
          if constexpr (CH == 32) tmem_ld32x2_wait(taddr + c0, taddr + BT + c0, g, u);
          else tmem_ld16x2_wait(taddr + c0, taddr + BT + c0, g, u);
#pragma unroll
          for (int q = 0; q < CH / 4; ++q) {
            const float4 s4 = sx[c0 / 4 + q];
            const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              acc0[c0 + 4 * q + i] = fmaf(g[4 * q + i], sv[i] * w0, acc0[c0 + 4 * q + i]);
              acc1[c0 + 4 * q + i] = fmaf(u[4 * q + i], sv[i] * w1, acc1[c0 + 4 * q + i]);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_pempty[pb]));
      }
      if (!ok) break;

      const int n = t.n0 + lrow;
      if (MODE == 0) {
        // activation, rounding to the 16-bit type, then one 1x128 group per (token, tile):
        // warp maxima by redux on the bit patterns (non-negative floats order like integers),
        // one thread per token turns the four warp maxima into the scale and its reciprocal.
        float* red = s_red + (buf * 2 + grp) * 4 * 64;
        // per-expert bias of this thread's gate row and up / linear row, and the clamped swiglu: the
        // rarer tail, kept out of the plain one
        const bool ext = a.bias != nullptr || a.activation == B200MOE_ACT_SWIGLU_OAI;
        float bg = 0.f, bu = 0.f;
        if (a.bias != nullptr && n < a.N) {
          bg = __ldg(a.bias + static_cast<size_t>(t.e) * 2 * a.N + n);
          bu = __ldg(a.bias + static_cast<size_t>(t.e) * 2 * a.N + a.N + n);
        }
        if (ext) {
#pragma unroll
          for (int i = 0; i < CPT; ++i) {
            acc0[i] += bg;
            acc1[i] += bu;
          }
          act_mul_array<__nv_bfloat16, true>(acc0, acc1, w_on_input, false, act_params(a), [&](int i) { return col_gam[i]; });
        } else {
          act_mul_array<__nv_bfloat16, false>(acc0, acc1, w_on_input, false, act_params(a), [&](int i) { return col_gam[i]; });
        }
        const bool bf = a.dtype == B200MOE_DTYPE_BF16;
#pragma unroll
        for (int i = 0; i < CPT; ++i) {
          acc0[i] = bf ? __bfloat162float(__float2bfloat16_rn(acc0[i])) : __half2float(__float2half_rn(acc0[i]));
          const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(acc0[i])));
          if (lane == 0) red[gw * 64 + i] = __uint_as_float(m);
        }
        if (!warps_meet(smem_u32(&bar_meet[grp]), meet_phase, lane, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;
        if (ep_tid < CPT) {
          const float amax = fmaxf(fmaxf(red[ep_tid], red[64 + ep_tid]), fmaxf(red[128 + ep_tid], red[192 + ep_tid]));
          const float sc = __fdiv_rn(fmaxf(amax, 1e-10f), 448.0f);
          a.out_scale[static_cast<size_t>(t.n0 / 128) * a.ld_xscale + t.row0 + cb + ep_tid] = sc;
          red[ep_tid] = __fdiv_rn(1.0f, sc);
        }
        if (!warps_meet(smem_u32(&bar_meet[grp]), meet_phase, lane, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;
        uint8_t* outq = a.out_q + static_cast<size_t>(t.row0 + cb) * a.ld_out + n;
#pragma unroll
        for (int i = 0; i < CPT; ++i) {
          outq[static_cast<size_t>(i) * a.ld_out] =
              static_cast<uint8_t>(__nv_cvt_float_to_fp8(acc0[i] * red[i], __NV_SATFINITE, __NV_E4M3));
        }
      } else {
        const unsigned long long* col_ptr = s_col_ptr + buf * 128 + cb;
        const bool second = n + kTileRows < a.N;
        float b0 = 0.f, b1 = 0.f;      // bias of the two output columns; the first reduction split carries it
        if (a.bias != nullptr && t.kb0 == 0) {
          if (n < a.N) b0 = __ldg(a.bias + static_cast<size_t>(t.e) * a.N + n);
          if (second) b1 = __ldg(a.bias + static_cast<size_t>(t.e) * a.N + n + kTileRows);
        }
        if (MIXED && a.out_pairs != nullptr) {
          // the pair's row, weighted and rounded to the 16-bit type; a warp stores 64 contiguous bytes of it
          const bool bf = a.dtype == B200MOE_DTYPE_BF16;
          auto half_bits = [&](float v) -> uint16_t {
            return bf ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
          };
#pragma unroll
          for (int i = 0; i < CPT; ++i) {
            const int orow = col_row[i];
            if (orow < 0) continue;
            const float gam = w_on_input ? 1.0f : col_gam[i];
            uint16_t* out = reinterpret_cast<uint16_t*>(col_ptr[i]) + n;
            out[0] = half_bits((acc0[i] + b0) * gam);
            if (second) out[kTileRows] = half_bits((acc1[i] + b1) * gam);
            if (n == 0) mark_pair_valid(a, orow);
          }
        } else {
#pragma unroll
          for (int i = 0; i < CPT; ++i) {
            const int orow = col_row[i];
            if (orow >= 0) {
              const float gam = w_on_input ? 1.0f : col_gam[i];
              float* out = reinterpret_cast<float*>(col_ptr[i]) + n;   // the token's row, here or on its owner
              atomicAdd(out, (acc0[i] + b0) * gam);
              if (second) atomicAdd(out + kTileRows, (acc1[i] + b1) * gam);
            }
          }
        }
      }
      // the tables of this tile may now be overwritten
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_sempty[buf]));
    }
  }

  // ---- teardown
  tc_fence_before();
  __syncthreads();
  if (!MIXED && warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, static_cast<uint32_t>(a.tmem_cols));
  }
  if (threadIdx.x == 0 && *abort_flag != 0) atomicCAS(a.status, 0, *abort_flag);
}

template <int MODE, int BT, int NG>
__global__ void __launch_bounds__(fp8_threads(NG), 1)
moe_gemm_fp8_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                    const GemmArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  Fp8Part part;
  weights_on_m<MODE, BT, NG, false>(tm_w, tm_x, a, smem, a.stages, part, 0);
}

// ------------------------------------------------------------------------------------------
// Tokens-on-M variant for 128-token blocks (prefill-sized batches).
//
// With many tokens per expert the token block goes on the M side (128 rows) and 256 weight rows on the N side:
// four MMAs per 128-wide reduction slice instead of sixteen.  An accumulator row is then a
// token, so the activation scale is one scalar per thread and slice, the weight scale one
// scalar per 128 columns; two promotion groups split the 256 columns (gate columns
// [64g, 64g+64) with the matching up columns for mode 0, columns [128g, 128g+128) for mode 1)
// and keep 128 accumulators per thread.  The 1x128 quantisation group of a token is the 64
// activations of its thread in group 0 plus the 64 of its thread in group 1: the two partial
// maxima meet in shared memory, no shuffles.
//
// What bounds it, from the CTAs' cycles at 4096 tokens (256 experts, zipf-skewed) with and without parts of the work: the
// promotion, about 970 cycles per slice in the gate/up projection and 800 in the down projection against 512 for the
// slice's MMAs, and the tail that nothing overlaps (11400 and 5300 cycles per tile: the accumulators fill the registers
// and the two partial buffers all of tensor memory).  With a third of the operand loads left out the cycles stay and the
// clock rises by 9 %: in a train of calls the board is at its power cap.  Alone, with operands that stay in shared
// memory, the same promotion takes 696 cycles per slice, its tensor-memory reads 513.
// Kept off that path: the tile's coordinates (decoded by the table warp), the activation scales (a ring filled per slice, which
// also frees the room of a fourth stage).  A warp whose 32 rows are all padding keeps in step with the others and promotes
// nothing, which leaves the board's power to the rest.
// Tried and slower: sixteen promotion warps, 32-column reads, scalar FMAs, partial buffers released by halves, hot and
// cold experts' tiles interleaved on every CTA.
// warps 0-3: TMA, MMA, tables, idle; warps 4-11: promotion.  Launched with 168 registers a thread; the first four warps
// give some up for the promotion, within 12 * 168: 72 and 216 in mode 0, where the other roles spill with less (their
// spills cost the whole tile 10 %), 56 and 224 in mode 1, whose promotion does with less.
constexpr int kThreadsFp8TokM = 12 * 32;
constexpr int kXsSlots = 8;                                       // ring of activation scales, one slot per slice

#ifdef B200MOE_STALL_STATS
__device__ unsigned long long g_stall_fp8[16];
#define STALL_ADD8(slot, v) atomicAdd(&g_stall_fp8[slot], v)
#else
#define STALL_ADD8(slot, v) ((void)0)
#endif

// 32 bytes of one thread, a whole sector.
__device__ __forceinline__ void st_global_v8(uint8_t* p, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
               "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

template <int MODE>
__device__ __forceinline__ void tokens_on_m(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const GemmArgs& a, uint8_t* smem,
                                            const Fp8Part& part, const uint32_t tmem_base) {
  constexpr int BT = 128;
  constexpr int W_BYTES = 2 * kTileBytes;
  constexpr int X_BYTES = BT * kStageKBytes;
  constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
  constexpr int PCOLS = 256;
  const int stages = a.stages;

  const int KBS = a.kblocks;   // reduction slices of a whole row: size of the per-tile weight-scale tables
  uint8_t* ctrl_base = smem + static_cast<size_t>(stages) * STAGE_BYTES;
  float* s_xs = reinterpret_cast<float*>(ctrl_base);                    // [kXsSlots][128] activation scales
  float* s_ws = s_xs + kXsSlots * BT;                                   // [2][2][KBS] weight scales
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(s_ws + 2 * 2 * KBS);
  uint64_t* bar_empty = bar_full + stages;
  uint64_t* bar_pfull = bar_empty + stages;
  uint64_t* bar_pempty = bar_pfull + 2;
  uint64_t* bar_sfull = bar_pempty + 2;
  uint64_t* bar_sempty = bar_sfull + 2;
  uint64_t* bar_meet8 = bar_sempty + 2;         // both groups: the halves of a quantisation group's maximum
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_meet8 + 1);
  int* s_tile = reinterpret_cast<int*>(bar_meet8 + 3);                  // [2][8] expert, row0, n0, kb0, kb1 of a tile
  int* s_col_row = s_tile + 16;               // [2][128] output row of each token
  float* s_col_gam = reinterpret_cast<float*>(s_col_row + 2 * 128);     // [2][128]
  float* s_red = s_col_gam + 2 * 128;                                   // mode 0: [2][2][128] partial group maxima
  // [2][128] mode 1: base of each row's output row
  unsigned long long* s_col_ptr = reinterpret_cast<unsigned long long*>(s_red + (MODE == 0 ? 2 * 2 * 128 : 0));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bar_pfull[s]), 1);
      mbar_init(smem_u32(&bar_pempty[s]), 8);
      mbar_init(smem_u32(&bar_sfull[s]), 1);
      mbar_init(smem_u32(&bar_sempty[s]), 8);
    }
    mbar_init(smem_u32(bar_meet8), 8);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    prefetch_tmap(&tm_w);
    prefetch_tmap(&tm_x);
  }
  __syncthreads();

  const Ctrl& c = part.c;
  const bool active = part.cta < c.grid_eff;
  constexpr int kTileN = (MODE == 0) ? kTileRows : 2 * kTileRows;
  const int second_off = (MODE == 0) ? a.up_row_off : kTileRows;

  if (warp < 4) {
    if (MODE == 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (active && warp == 0 && elect_one()) {
      // =============================== TMA producer ===============================
      int stage = 0;
      uint32_t phase = 0;
      long long issued = 0;
      uint32_t jx = 0;     // slices issued over the whole launch
      bool ok = true;
      unsigned long long w_empty = 0;
      const long long role_t0 = clock64();
      for (int tile = part.cta; ok && tile < c.total; tile += c.grid_eff) {
        const TileCoord t = part_tile(tile, part, a, kTileN);
        for (int kb = t.kb0; kb < t.kb1; ++kb) {
          if (!mbar_wait_t(smem_u32(&bar_empty[stage]), phase ^ 1, abort_flag, DEV_TIMEOUT_PRODUCER, w_empty)) {
            ok = false;
            break;
          }
          // The slice's activation scales go to a ring of their own, which the promotion warps read once the slice's
          // MMAs are done (these wait for the whole stage, scales included).  The slot is free: this stage's last MMA has
          // finished, and it was issued after the promotion of the slice two before it, which is at most
          // stages + 2 <= kXsSlots slices back.
          const uint32_t xs_slot = jx % kXsSlots;
          ++jx;
          const uint32_t full = smem_u32(&bar_full[stage]);
          mbar_arrive_expect_tx(full, static_cast<uint32_t>(STAGE_BYTES + BT * 4));
          bulk_copy_g2s(smem_u32(s_xs + xs_slot * BT), a.x_scale + static_cast<size_t>(kb) * a.ld_xscale + t.row0, BT * 4, full);
          const uint32_t sw = smem_u32(smem + static_cast<size_t>(stage) * STAGE_BYTES);
          const int k0 = kb * kStageKBytes;
          tma_load_3d(sw, &tm_w, full, k0, t.n0, t.e);
          tma_load_3d(sw + kTileBytes, &tm_w, full, k0, second_off + t.n0, t.e);
          tma_load_2d(sw + W_BYTES, &tm_x, full, k0, t.row0);
          ++issued;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      STALL_ADD8(0, w_empty);
      STALL_ADD8(8, static_cast<unsigned long long>(clock64() - role_t0));
      if (!ok) {
        const int n = static_cast<int>(issued < stages ? issued : stages);
        for (int i = 1; i <= n; ++i) {
          int s = stage - i;
          uint32_t ph = phase;
          if (s < 0) {
            s += stages;
            ph ^= 1;
          }
          mbar_wait_brief(smem_u32(&bar_full[s]), ph);
        }
      }
    } else if (active && warp == 1 && elect_one()) {
      // =============================== MMA issuer =================================
      const uint32_t idesc = make_idesc(0u /* e4m3 */, kTileRows, 256u);
      int stage = 0;
      uint32_t phase = 0, j = 0;
      bool ok = true;
      unsigned long long w_full = 0, w_pempty = 0;
      const long long role_t0 = clock64();
      for (int tile = part.cta; ok && tile < c.total; tile += c.grid_eff) {
        int kb0 = 0, kb1 = a.kblocks;
        if (c.split > 1) {       // only the slice count matters here
          const TileCoord t = part_tile(tile, part, a, kTileN);
          kb0 = t.kb0;
          kb1 = t.kb1;
        }
        for (int kb = kb0; kb < kb1; ++kb, ++j) {
          const uint32_t pb = j & 1u;
          if (!mbar_wait_t(smem_u32(&bar_full[stage]), phase, abort_flag, DEV_TIMEOUT_MMA, w_full) ||
              !mbar_wait_t(smem_u32(&bar_pempty[pb]), ((j >> 1) & 1u) ^ 1u, abort_flag, DEV_TIMEOUT_MMA, w_pempty)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d0 = tmem_base + pb * PCOLS;
          const uint32_t sw = smem_u32(smem + static_cast<size_t>(stage) * STAGE_BYTES);
          const uint64_t dw = smem_desc_k_sw128(sw);             // 256 weight rows: N side
          const uint64_t dx = smem_desc_k_sw128(sw + W_BYTES);   // 128 token rows: M side
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma_f8(d0, dx + 2 * k, dw + 2 * k, idesc, k > 0 ? 1u : 0u);
          tc_commit(smem_u32(&bar_empty[stage]));
          tc_commit(smem_u32(&bar_pfull[pb]));
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      STALL_ADD8(1, w_pempty);
      STALL_ADD8(2, w_full);
      STALL_ADD8(9, static_cast<unsigned long long>(clock64() - role_t0));
    } else if (active && warp == 2) {
      // =============================== per-tile table loader ======================
      const int kb_total = a.kblocks;
      int iter = 0;
      for (int tile = part.cta; tile < c.total; tile += c.grid_eff, ++iter) {
        const TileCoord t = part_tile(tile, part, a, kTileN);
        const int buf = iter & 1;
        if (!mbar_wait(smem_u32(&bar_sempty[buf]), ((iter >> 1) & 1) ^ 1, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;
        const int nkb = t.kb1 - t.kb0;
        for (int cidx = lane; cidx < BT; cidx += 32) {
          const int slot = a.sorted_ids[t.row0 + cidx];
          const bool valid = slot >= 0 && slot < a.P;
          // mode 1: output row = token, or the pair's own slot when rows are stored per pair
          const int orow = valid ? ((MODE == 1 && a.out_pairs == nullptr) ? slot / a.topk : slot) : -1;
          s_col_row[buf * 128 + cidx] = orow;
          s_col_gam[buf * 128 + cidx] = valid ? a.row_gamma[t.row0 + cidx] : 0.f;
          if (MODE == 1 && valid)
            s_col_ptr[buf * 128 + cidx] = reinterpret_cast<unsigned long long>(
                a.out_pairs != nullptr ? out_row_base(a, a.out_pairs, orow, static_cast<size_t>(a.N) * 2)
                                       : out_row_base(a, a.out, orow, static_cast<size_t>(a.ld_out) * sizeof(float)));
        }
        const int nb0 = t.n0 / 128, nb1 = (second_off + t.n0) / 128;
        const float* ws0 = a.w_scale + (static_cast<size_t>(t.e) * a.w_scale_rows + nb0) * kb_total + t.kb0;
        const float* ws1 = a.w_scale + (static_cast<size_t>(t.e) * a.w_scale_rows + nb1) * kb_total + t.kb0;
        const bool second_ok = nb1 < a.w_scale_rows;
        float* ws_t = s_ws + buf * 2 * KBS;
        for (int i = lane; i < nkb; i += 32) {
          ws_t[i] = __ldg(ws0 + i);
          ws_t[KBS + i] = second_ok ? __ldg(ws1 + i) : 0.f;
        }
        if (lane == 0) {
          int* ti = s_tile + buf * 8;
          ti[0] = t.e;
          ti[1] = t.row0;
          ti[2] = t.n0;
          ti[3] = t.kb0;
          ti[4] = t.kb1;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_sfull[buf]));
      }
    }
  } else {
    if (MODE == 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    if (active) {
      // =============================== promotion + tail ===========================
      const int grp = warp < 8 ? 0 : 1;
      const int quad = warp & 3;
      const int lrow = quad * 32 + lane;  // token row inside the block = TMEM lane
      const bool w_on_input = (a.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0;
      // columns of this thread: mode 0 -> gate [64g, 64g+64) and up [128+64g, ..+64); mode 1 -> [128g, 128g+128)
      const uint32_t colA = (MODE == 0) ? 64u * grp : 128u * grp;
      const uint32_t colB = (MODE == 0) ? 128u + 64u * grp : 128u * grp + 64u;
      uint32_t j = 0;
      uint32_t meet8_phase = 0;
      int iter = 0;
      bool ok = true;
      unsigned long long w_pfull = 0, w_sfull = 0, t_tail = 0;
      const long long role_t0 = clock64();
      for (int tile = part.cta; ok && tile < c.total; tile += c.grid_eff, ++iter) {
        const int buf = iter & 1;
        const float* ws_t = s_ws + buf * 2 * KBS;
        if (!mbar_wait_t(smem_u32(&bar_sfull[buf]), (iter >> 1) & 1, abort_flag, DEV_TIMEOUT_EPILOGUE, w_sfull)) break;
        const int* ti = s_tile + buf * 8;      // decoded by the table warp, off this critical path
        const TileCoord t = {ti[0], ti[1], ti[2], ti[3], ti[4]};
        const int orow = s_col_row[buf * 128 + lrow];
        const float gam = s_col_gam[buf * 128 + lrow];
        const bool idle = !__any_sync(0xffffffffu, orow >= 0);   // 32 padding rows: keep in step, promote and store nothing

        // running sums stay packed two to a 64-bit register for the whole reduction
        unsigned long long pA[32], pB[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          pA[i] = 0ull;
          pB[i] = 0ull;
        }
        for (int kb = t.kb0; kb < t.kb1; ++kb, ++j) {
          const uint32_t pb = j & 1u;
          if (!mbar_wait_t(smem_u32(&bar_pfull[pb]), (j >> 1) & 1u, abort_flag, DEV_TIMEOUT_EPILOGUE, w_pfull)) {
            ok = false;
            break;
          }
          if (idle) {
            __syncwarp();      // every lane has seen this phase: two slices on, the barrier has the same parity again
            if (lane == 0) mbar_arrive(smem_u32(&bar_pempty[pb]));
            continue;
          }
          tc_fence_after();
          const uint32_t xs_slot = j % kXsSlots;
          const float sx = s_xs[xs_slot * BT + lrow];
          // mode 0: A columns belong to the first weight block, B columns to the second;
          // mode 1: group g works entirely inside weight block g
          const float fA = sx * ws_t[(MODE == 0 ? 0 : grp * KBS) + kb - t.kb0];
          const float fB = sx * ws_t[(MODE == 0 ? KBS : grp * KBS) + kb - t.kb0];
          const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + pb * PCOLS;
          // Packed f32x2 FMAs, 16 columns at a time.  They run at half the rate of scalar ones, so the FMA pipe is
          // as busy, but they leave the MMA thread's scheduler twice the issue slots (with scalar FMAs the MMAs of a
          // slice took 684 cycles instead of 516).  Wider reads spill: the accumulators alone take 128 registers.
          const unsigned long long fA2 = pack_f32x2(fA, fA), fB2 = pack_f32x2(fB, fB);
#pragma unroll
          for (int c0 = 0; c0 < 64; c0 += 16) {
            uint32_t g[16];
            tmem_ld16_wait_u32(taddr + colA + c0, g);
#pragma unroll
            for (int i = 0; i < 8; ++i) ffma2_packed(pA[c0 / 2 + i], g[2 * i], g[2 * i + 1], fA2);
            tmem_ld16_wait_u32(taddr + colB + c0, g);
#pragma unroll
            for (int i = 0; i < 8; ++i) ffma2_packed(pB[c0 / 2 + i], g[2 * i], g[2 * i + 1], fB2);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_pempty[pb]));
        }
        if (!ok) break;
        const long long tail_t0 = clock64();
        if (idle) {
          if (MODE == 0 && !warps_meet(smem_u32(bar_meet8), meet8_phase, lane, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_sempty[buf]));
          continue;
        }
        float accA[64], accB[64];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          unpack_f32x2(pA[i], accA[2 * i], accA[2 * i + 1]);
          unpack_f32x2(pB[i], accB[2 * i], accB[2 * i + 1]);
        }

        if (MODE == 1 && a.bias != nullptr && t.kb0 == 0) {
          // bias of columns n0 + 128 grp + [0, 128): accA holds the first 64, accB the next 64
          const float* bo = a.bias + static_cast<size_t>(t.e) * a.N + t.n0 + 128 * grp;
#pragma unroll
          for (int i = 0; i < 64; ++i) {
            accA[i] += (t.n0 + 128 * grp + i < a.N) ? __ldg(bo + i) : 0.f;
            accB[i] += (t.n0 + 128 * grp + 64 + i < a.N) ? __ldg(bo + 64 + i) : 0.f;
          }
        }
        if (MODE == 0) {
          // 64 activations of this token; the other 64 of its quantisation group live in the
          // same lane of the other promotion group
          float amax = 0.f;
          const bool ext = a.bias != nullptr || a.activation == B200MOE_ACT_SWIGLU_OAI;
          if (a.bias != nullptr) {
            // gate columns n0 + 64 grp + i and the matching up / linear columns of the same expert
            const float* bgp = a.bias + static_cast<size_t>(t.e) * 2 * a.N + t.n0 + 64 * grp;
#pragma unroll
            for (int i = 0; i < 64; ++i) {
              const bool in = t.n0 + 64 * grp + i < a.N;
              accA[i] += in ? __ldg(bgp + i) : 0.f;
              accB[i] += in ? __ldg(bgp + a.N + i) : 0.f;
            }
          }
          if (ext) act_mul_array<__nv_bfloat16, true>(accA, accB, w_on_input, false, act_params(a), [&](int) { return gam; });
          else act_mul_array<__nv_bfloat16, false>(accA, accB, w_on_input, false, act_params(a), [&](int) { return gam; });
          const bool bf = a.dtype == B200MOE_DTYPE_BF16;
#pragma unroll
          for (int i = 0; i < 64; i += 2) {
            const float2 v = bf ? __bfloat1622float2(__floats2bfloat162_rn(accA[i], accA[i + 1]))
                                : __half22float2(__floats2half2_rn(accA[i], accA[i + 1]));
            accA[i] = v.x;
            accA[i + 1] = v.y;
            amax = fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y)));
          }
          float* red = s_red + buf * 2 * 128;
          red[grp * 128 + lrow] = amax;
          if (!warps_meet(smem_u32(bar_meet8), meet8_phase, lane, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;
          amax = fmaxf(red[lrow], red[128 + lrow]);
          const float sc = __fdiv_rn(fmaxf(amax, 1e-10f), 448.0f);
          const float inv = __fdiv_rn(1.0f, sc);
          const int r = t.row0 + lrow;
          if (grp == 0) a.out_scale[static_cast<size_t>(t.n0 / 128) * a.ld_xscale + r] = sc;
          uint32_t pk[16];
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            // two values per conversion instruction
            const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(accA[4 * q] * inv, accA[4 * q + 1] * inv),
                                                         __NV_SATFINITE, __NV_E4M3);
            const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(accA[4 * q + 2] * inv, accA[4 * q + 3] * inv),
                                                         __NV_SATFINITE, __NV_E4M3);
            pk[q] = lo | (hi << 16);
          }
          uint8_t* dst = a.out_q + static_cast<size_t>(r) * a.ld_out + t.n0 + 64 * grp;
          st_global_v8(dst, pk);
          st_global_v8(dst + 32, pk + 8);
        } else if (a.out_pairs != nullptr) {
          // The pair's row, weighted and rounded to the 16-bit type.  A thread owns 128 contiguous columns of one row and
          // stores them as whole sectors straight from its registers.  (Turning them in shared memory so that a store
          // covers eight rows made the tail 4700 cycles of a 20000-cycle tile: 4096 tokens 3205 -> 3065 us.)
          const float scale = w_on_input ? 1.0f : gam;
          const bool bf = a.dtype == B200MOE_DTYPE_BF16;
          if (orow >= 0) {
            uint8_t* dst = reinterpret_cast<uint8_t*>(s_col_ptr[buf * 128 + lrow]) + (t.n0 + 128 * grp) * 2;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const float* src = (q < 4 ? accA : accB) + 16 * (q & 3);
              uint32_t w[8];
#pragma unroll
              for (int b = 0; b < 8; ++b) {
                const float lo = src[2 * b] * scale, hi = src[2 * b + 1] * scale;
                if (bf) {
                  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
                  w[b] = *reinterpret_cast<uint32_t*>(&v);
                } else {
                  __half2 v = __floats2half2_rn(lo, hi);
                  w[b] = *reinterpret_cast<uint32_t*>(&v);
                }
              }
              if (t.n0 + 128 * grp < a.N) st_global_v8(dst + 32 * q, w);
            }
          }
          if (orow >= 0 && t.n0 == 0 && grp == 0) mark_pair_valid(a, orow);
        } else if (orow >= 0) {
          const float scale = w_on_input ? 1.0f : gam;
          float* out = reinterpret_cast<float*>(s_col_ptr[buf * 128 + lrow]) + t.n0 + 128 * grp;
          if (t.n0 + 128 * grp < a.N) {
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              asm volatile("red.global.v4.f32.add [%0], {%1, %2, %3, %4};" ::"l"(out + 4 * q), "f"(accA[4 * q] * scale),
                           "f"(accA[4 * q + 1] * scale), "f"(accA[4 * q + 2] * scale), "f"(accA[4 * q + 3] * scale)
                           : "memory");
              asm volatile("red.global.v4.f32.add [%0], {%1, %2, %3, %4};" ::"l"(out + 64 + 4 * q),
                           "f"(accB[4 * q] * scale), "f"(accB[4 * q + 1] * scale), "f"(accB[4 * q + 2] * scale),
                           "f"(accB[4 * q + 3] * scale)
                           : "memory");
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_sempty[buf]));
        t_tail += static_cast<unsigned long long>(clock64() - tail_t0);
      }
      if (threadIdx.x == 4 * 32) {
        STALL_ADD8(5, w_pfull);
        STALL_ADD8(6, w_sfull);
        STALL_ADD8(7, t_tail);
        STALL_ADD8(11, static_cast<unsigned long long>(clock64() - role_t0));
      }
    }
  }

  // ---- teardown (the launch frees tensor memory)
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0) atomicCAS(a.status, 0, *abort_flag);
}

// ------------------------------------------------------------------------------------------
// Prefill-sized batches: one launch for both kinds of blocks.  Routing of many-expert layers is skewed: of 4096 tokens' 397
// blocks of 128 on 256 experts, 107 hold at most 16 tokens.  Such a cold block's time is its expert's weights' way from
// HBM, a hot one's is the promotion; one kind after the other, as the experts come, leaves either idle.  So some CTAs
// take the hot blocks (tokens on M) and the rest the cold ones (weights on M, 16 tokens on N, which also spares the
// MMAs of 112 padding rows), in proportion to what they cost.  The rows lie in the same blocks of 128 for both.
// us per call in a train, all blocks with tokens on M / mixed, in turn on one board: 130 tokens 556 / 501, 200: 676 / 588,
// 300: 810 / 676, 1024: 1398 / 1202, 2048: 1966 / 1752, 4096: 3010 / 2795.
constexpr int kColdRows = 16;
// Cycles of a 128-wide reduction slice and of a tile's tail, from the CTAs' times at 4096 tokens: hot tiles 65800 (gate/up, 56
// slices) and 18000 cycles (down, 16), 40000 and 13500 with a quarter of the promotion, cold ones 31800 and 11800.
// A constant for the cold slice is the model's weak point: it is the time of the slice's weights on their way from HBM, 525
// cycles here, where the launch draws 3 TB/s, and 950 at 200 to 300 tokens, where it draws all there is and both kinds of
// CTAs wait for it.  Gate/up takes 600 for it (4096 tokens: 2800 us with 525, 2750 with 600, 2766 with 680).  When
// the last hot and the last cold CTA finish, us, gate/up and down, 256 experts of 7168 x 2048, zipf: 300 tokens 343 / 395
// and 213 / 200 (at HBM's rate, however they are divided), 1024: 589 / 612 and 363 / 343, 2048: 932 / 915 and 553 / 522,
// 4096: 1592 / 1576 and 950 / 877.  Tried and slower: hot blocks rated by the groups of 32 rows they promote (3 % over ten
// layers), and divisions rated by whole tiles on top (3.5 %).
template <int MODE>
struct MixedCost {
  static constexpr float kHotSlice = MODE == 0 ? 970.f : 800.f, kHotTail = MODE == 0 ? 11400.f : 5300.f;
  static constexpr float kColdSlice = MODE == 0 ? 600.f : 580.f, kColdTail = 2500.f;
};

__host__ __device__ __forceinline__ size_t mixed_table_bytes(int E) {
  return (3 * static_cast<size_t>(E + 1) * 4 + 16 + sizeof(Fp8Part) + 1023) & ~static_cast<size_t>(1023);
}

template <int MODE>
__global__ void __launch_bounds__(kThreadsFp8TokM, 1)
moe_gemm_fp8_mixed_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                          const __grid_constant__ CUtensorMap tm_xc, const GemmArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  // tables behind the larger of the two kinds' shared memory (whose addresses then need no offset: the promotion has no
  // register left for one)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + a.table_off);
  Fp8Part* s_part = reinterpret_cast<Fp8Part*>(tmem_slot + 4);
  int* s_blk = reinterpret_cast<int*>(s_part + 1);      // [E+1] blocks before expert e
  int* s_hot = s_blk + (a.E + 1);                       // [E+1] hot blocks before expert e
  int* s_cold = s_hot + (a.E + 1);                      // [E+1] cold ones
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512u);
    tmem_relinquish();
  }
  griddep_wait();
  griddep_launch_dependents();
  if (warp == 0) {
    unsigned long long run = 0;      // running sums: hot blocks below, cold ones above
    for (int e0 = 0; e0 < a.E; e0 += 32) {
      const int e = e0 + lane;
      int first = 0, n = 0;
      bool cold = false;
      if (e < a.E) {
        first = a.blk_off[e];
        n = a.blk_off[e + 1] - first;
        cold = n == 1 && a.sorted_ids[first * 128 + kColdRows] == a.P;      // an expert's rows stand in front of its padding
        s_blk[e] = first;
        if (e == a.E - 1) s_blk[a.E] = first + n;
      }
      unsigned long long v = cold ? 1ull << 32 : static_cast<unsigned long long>(n);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      if (e < a.E) {
        s_hot[e + 1] = static_cast<int>(run + v);
        s_cold[e + 1] = static_cast<int>((run + v) >> 32);
      }
      run += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) s_hot[0] = s_cold[0] = 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  int hot = s_hot[a.E], cold = s_cold[a.E];
  const int grid = gridDim.x;
  // A few cold blocks among hot ones that hold little more go with them: around 20 to 25 slots per expert, flat routing, the
  // division leaves the cold CTAs behind (us, divided / all hot: 64 experts of 2048 x 1408, average 20 163 / 154, 25 175 / 155;
  // 128 of 2048 x 768, 25 189 / 175; 32 of 7168 x 2048, 20 308 / 294).  Among full hot blocks it gains whatever their number
  // (256 of 7168 x 2048, zipf, 8192 tokens 4850 / 5080).  A launch of one CTA cannot be divided: its hot blocks take the cold
  // ones with them.
  if ((cold * 4 < hot && a.P <= 32 * hot) || (grid == 1 && hot > 0)) {
    __syncthreads();
    for (int e = threadIdx.x; e <= a.E; e += blockDim.x) {
      s_hot[e] += s_cold[e];
      s_cold[e] = 0;
    }
    hot += cold;
    cold = 0;
    __syncthreads();
  }
  int split = 1;
  if (MODE == 1 && !(a.flags & B200MOE_FLAG_NO_SPLIT_K)) split = pick_split((hot + cold) * a.num_nt, a.kblocks, grid, a.max_split);
  const int units = a.num_nt * split;
  const float slices = static_cast<float>(a.kblocks) / split;
  using Cost = MixedCost<MODE>;
  const float hot_cost = hot * (slices * Cost::kHotSlice + Cost::kHotTail);
  const float cold_cost = cold * (slices * Cost::kColdSlice + Cost::kColdTail);
  int cold_ctas = 0;
  if (cold > 0) {
    cold_ctas = static_cast<int>(grid * cold_cost / (hot_cost + cold_cost) + 0.5f);
    cold_ctas = hot > 0 ? max(1, min(grid - 1, cold_ctas)) : grid;
  }
  const bool cold_cta = static_cast<int>(blockIdx.x) < cold_ctas;
  if (threadIdx.x == 0) {
    Fp8Part part;
    part.cta = cold_cta ? blockIdx.x : blockIdx.x - cold_ctas;
    part.off = cold_cta ? s_cold : s_hot;
    part.blk = s_blk;
    part.rows = 128;
    part.c = spread_tiles(cold_cta ? cold : hot, units, split, cold_cta ? cold_ctas : grid - cold_ctas, a.flags);
    *s_part = part;
  }
  if (cold_cta) weights_on_m<MODE, kColdRows, 1, true>(tm_w, tm_xc, a, smem, a.stages_cold, *s_part, tmem_base);
  else tokens_on_m<MODE>(tm_w, tm_x, a, smem, *s_part, tmem_base);
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512u);
  }
}

size_t fp8_stage_bytes(int bt) { return 2 * static_cast<size_t>(kTileBytes) + static_cast<size_t>(bt) * kStageKBytes; }
size_t fp8_ctrl_bytes(const GemmArgs& a, int bt) {
  return 2 * static_cast<size_t>(kMaxKB) * bt * 4 + 2 * 2 * kMaxKB * 4 + 512 /*barriers*/ + 2 * 128 * 8 +
         2 * 2 * 4 * 64 * 4 + 2 * 128 * 8 +
         (a.route.own ? route_table_bytes(a.E, a.P) : static_cast<size_t>(a.E + 1) * 4) + 64;
}
size_t fp8_tokm_ctrl_bytes(const GemmArgs& a) {
  return kXsSlots * 128 * 4 + 2 * 2 * static_cast<size_t>(a.kblocks) * 4 +
         512 /*barriers, tile words*/ + 2 * 2 * 128 * 4 +
         (a.mode == 0 ? 2 * 2 * 128 * 4 : 2 * 128 * 8) + 64;
}

template <int MODE>
int launch_fp8_mixed(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const CUtensorMap& tm_xc, const GemmArgs& a, int num_sms,
                     cudaStream_t stream) {
  const size_t hot = static_cast<size_t>(a.stages) * (3 * kTileBytes) + fp8_tokm_ctrl_bytes(a);
  const size_t cold = a.stages_cold * fp8_stage_bytes(kColdRows) + fp8_ctrl_bytes(a, kColdRows);
  GemmArgs g = a;
  g.table_off = static_cast<int>(((hot > cold ? hot : cold) + 1023) & ~static_cast<size_t>(1023));
  const size_t smem = 1024 + g.table_off + mixed_table_bytes(a.E);
  if (smem > kSmemLimit) return B200MOE_ERR_TOO_LARGE;
  if (cudaFuncSetAttribute(moe_gemm_fp8_mixed_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kSmemLimit)) != cudaSuccess)
    return B200MOE_ERR_CUDA;
  note_launch(MODE == 0 ? "moe_gemm_fp8_mixed_kernel<gate/up>" : "moe_gemm_fp8_mixed_kernel<down>");
  cudaError_t err = launch_kernel(moe_gemm_fp8_mixed_kernel<MODE>, dim3(num_sms), dim3(kThreadsFp8TokM), smem, stream,
                                  a.pdl != 0, tm_w, tm_x, tm_xc, g);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

template <int MODE, int BT, int NG>
int launch_fp8(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const GemmArgs& a, int num_sms,
               cudaStream_t stream) {
  const size_t smem = 1024 + static_cast<size_t>(a.stages) * fp8_stage_bytes(a.BT) + fp8_ctrl_bytes(a, a.BT);
  if (smem > kSmemLimit) return B200MOE_ERR_TOO_LARGE;
  if (cudaFuncSetAttribute(moe_gemm_fp8_kernel<MODE, BT, NG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kSmemLimit)) != cudaSuccess)
    return B200MOE_ERR_CUDA;
  note_launch(MODE == 0 ? "moe_gemm_fp8_kernel<gate/up>" : "moe_gemm_fp8_kernel<down>");
  cudaError_t err = launch_kernel(moe_gemm_fp8_kernel<MODE, BT, NG>, dim3(num_sms), dim3(fp8_threads(NG)), smem,
                                  stream, a.pdl != 0, tm_w, tm_x, a);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

}  // namespace

#ifdef B200MOE_STALL_STATS
extern "C" int b200moe_debug_stalls_fp8(unsigned long long* out16, int reset) {
  if (cudaMemcpyFromSymbol(out16, g_stall_fp8, sizeof(unsigned long long) * 16) != cudaSuccess) return -1;
  if (reset) {
    unsigned long long z[16] = {0};
    cudaMemcpyToSymbol(g_stall_fp8, z, sizeof(z));
  }
  return 0;
}
#endif

void gemm_plan_fp8(GemmArgs* a) {
  if (a->BT != 128) a->orient = 0;
  const int tile_n = (a->mode == 0) ? kTileRows : 2 * kTileRows;
  a->num_nt = (a->N + tile_n - 1) / tile_n;
  a->kblocks = (a->K + 127) / 128;
  const int pcols = 2 * a->BT;                       // one partial: two row blocks
  const int cols = ((512 / pcols) >= 4 ? 4 : 2) * pcols;
  int tc = 32;
  while (tc < cols) tc <<= 1;
  a->tmem_cols = tc;
  a->acc_stages = 2;
  int st = static_cast<int>((kSmemLimit - 1024 - fp8_ctrl_bytes(*a, a->BT)) / fp8_stage_bytes(a->BT));
  if (a->orient == 1) {   // tokens on M, 128-token blocks
    a->tmem_cols = 512;
    const size_t room = kSmemLimit - 2048 - mixed_table_bytes(a->E);
    st = static_cast<int>((room - fp8_tokm_ctrl_bytes(*a)) / (3 * kTileBytes));
    if (st > kXsSlots - 2) st = kXsSlots - 2;
    a->stages_cold = static_cast<int>((room - fp8_ctrl_bytes(*a, kColdRows)) / fp8_stage_bytes(kColdRows));
  }
  if (st > 10) st = 10;
  if (st < 2) st = 2;
  a->stages = st;
  if (a->max_split <= 0) a->max_split = 16;
}

int launch_gemm_fp8(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const CUtensorMap& tm_xc, const GemmArgs& a, int num_sms,
                    cudaStream_t stream) {
  if (a.wmode != B200MOE_W_FP8_BLOCK) return B200MOE_ERR_BAD_ARG;
  if (a.K % 128 != 0 || a.N % 128 != 0 || a.K / 128 > kMaxKB) return B200MOE_ERR_UNSUPPORTED;
  if (a.orient == 1 && a.BT == 128)
    return a.mode == 0 ? launch_fp8_mixed<0>(tm_w, tm_x, tm_xc, a, num_sms, stream)
                       : launch_fp8_mixed<1>(tm_w, tm_x, tm_xc, a, num_sms, stream);
#define B200MOE_FP8_CASE(bt, ng)                                                          \
  case bt:                                                                                \
    return a.mode == 0 ? launch_fp8<0, bt, ng>(tm_w, tm_x, a, num_sms, stream)            \
                       : launch_fp8<1, bt, ng>(tm_w, tm_x, a, num_sms, stream);
  switch (a.BT) {
    B200MOE_FP8_CASE(16, 1)
    B200MOE_FP8_CASE(32, 1)
    B200MOE_FP8_CASE(64, 2)
    default:
      return B200MOE_ERR_BAD_ARG;
  }
#undef B200MOE_FP8_CASE
}

}  // namespace b200moe
