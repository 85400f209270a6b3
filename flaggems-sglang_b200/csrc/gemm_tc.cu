// Grouped expert GEMMs on the sm_100a tensor cores (tcgen05.mma, accumulators in
// tensor memory, operands staged by TMA into a shared-memory ring).
//
// One persistent CTA per SM, eight warps:
//   warp 0      one thread issues the TMA loads (weight tile(s) + token block per stage)
//   warp 1      one thread issues the MMAs and the commits; the warp owns the TMEM allocation
//   warps 2-5   epilogue: tcgen05.ld the accumulator, apply the fused tail, store
//   warp 6      mode 0 of a call that sorts its slots itself (gemm_route.cuh): copies the token rows into the ring
//   warp 7      looks up the next tile's slots and routing weights
//
// mode 0 (gate/up): per stage a 128-row gate tile and the matching 128-row up tile; two
//   accumulators, so that lane i of TMEM holds gate[n0+i] and up[n0+i] for every token of
//   the block and the activation needs no data exchange.
// mode 1 (down):    one 128-row tile; the reduction may be split over CTAs; the epilogue
//   multiplies by the routing weight and adds into the fp32 combine buffer with
//   red.global.add.f32 (which also merges the top-k experts of a token).
// 16-bit weights run here up to 25 tokens per expert; above that gemm_tc2.cu takes over.
//
// What bounds it: HBM.  Between its first full stage and its last commit the kernel reads its weights at 7.0 - 7.2 TB/s (32
// tokens of the 128-expert layer: 98 us for 703 MB, then 45 us for 352 MB), so what is left of a call is the time in front of
// the first stage (7 us from the start of mode 0: 2 to count the slots, 4 for the first weights), between the two kernels (3.5
// us, their first weights in flight) and behind the last.
//
// Every wait is bounded; on a time-out the CTA raises an abort flag, all roles leave their
// loops, the status word is set, TMEM is freed and the kernel returns.
#include "gemm_route.cuh"
#include "gemm_sched.cuh"

namespace b200moe {

namespace {

constexpr int kTcThreads = 256;
constexpr int kCopyLag = 2;

// Weight rows on the MMA's M side, a block of 16..256 tokens on its N side; mode 0 stages the gate and the up tile.
// EXT: per-expert bias and the clamped swiglu in the epilogues (separate instantiations, so
// that the plain kernels keep their shorter epilogue loops).
template <int MODE, typename T, bool EXT>
__global__ void __launch_bounds__(kTcThreads, 1)
moe_gemm_tc_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                   const GemmArgs a) {

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  constexpr int W_BYTES = (MODE == 0 ? 2 : 1) * kTileBytes;
  const int BT = a.BT;
  const int x_bytes = BT * kStageKBytes;
  const int stage_bytes = W_BYTES + x_bytes;
  const int stages = a.stages;

  uint8_t* ctrl_base = smem + static_cast<size_t>(stages) * stage_bytes;
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(ctrl_base);
  uint64_t* bar_empty = bar_full + stages;
  uint64_t* bar_tfull = bar_empty + stages;
  uint64_t* bar_tempty = bar_tfull + 2;
  uint64_t* bar_sfull = bar_tempty + 2;   // [2] slots and weights of a tile are in place
  uint64_t* bar_sempty = bar_sfull + 2;   // [2] ... and have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_sempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* s_col_row = reinterpret_cast<int*>(tmem_slot + 4);               // [2][BT]
  float* s_col_gam = reinterpret_cast<float*>(s_col_row + 2 * BT);      // [2][BT]
  const RowTables rt = row_tables(s_col_gam + 2 * BT, a.E);             // own tables, or only the blocks' starts
  int* s_blk_off = rt.blk;                                              // [E+1]

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;

  const bool own = a.route.own != 0, early = own && a.route.early != 0;
  const bool copier = MODE == 0 && own;
  const bool tables = MODE == 1 || (a.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0;   // the epilogue needs slots or weights

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), copier ? 2 : 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bar_tfull[s]), 1);
      mbar_init(smem_u32(&bar_tempty[s]), 4);
      mbar_init(smem_u32(&bar_sfull[s]), 1);
      mbar_init(smem_u32(&bar_sempty[s]), 4);
    }
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    prefetch_tmap(&tm_w);
    prefetch_tmap(&tm_x);
  }
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
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const Ctrl c = make_ctrl(a, own ? s_blk_off[a.E] : a.meta[0], MODE == 1);
  const int cols_per_acc = (MODE == 0 ? 2 : 1) * BT;
  const bool active = static_cast<int>(blockIdx.x) < c.grid_eff;

  if (active && warp == 0 && elect_one()) {
    // =============================== TMA producer ===============================
    int stage = 0;
    uint32_t phase = 0;
    long long issued = 0;
    bool ok = true;
    auto load_weights = [&](const TileCoord& t, int kb, int s) {
      const uint32_t full = smem_u32(&bar_full[s]);
      const uint32_t sw = smem_u32(smem + static_cast<size_t>(s) * stage_bytes);
      const int k0 = kb * (kStageKBytes / static_cast<int>(sizeof(T)));
      mbar_arrive_expect_tx(full, static_cast<uint32_t>(copier ? W_BYTES : stage_bytes));
      tma_load_3d(sw, &tm_w, full, k0, t.n0, t.e);
      if (MODE == 0) tma_load_3d(sw + kTileBytes, &tm_w, full, k0, a.up_row_off + t.n0, t.e);
    };
    // the ring's first round of weights, before the activations may be read
    int ahead = 0;
    if (early) {
      for (int tile = blockIdx.x; ahead < stages && tile < c.total; tile += c.grid_eff) {
        const TileCoord t = decode_tile(tile, c, s_blk_off, a.E, BT, a.num_nt, a.kblocks, kTileRows);
        for (int kb = t.kb0; ahead < stages && kb < t.kb1; ++kb, ++ahead) load_weights(t, kb, ahead);
      }
      griddep_wait();
    }
    for (int tile = blockIdx.x; ok && tile < c.total; tile += c.grid_eff) {
      const TileCoord t = decode_tile(tile, c, s_blk_off, a.E, BT, a.num_nt, a.kblocks, kTileRows);
      for (int kb = t.kb0; kb < t.kb1; ++kb) {
        if (issued >= ahead) {
          if (!mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1, abort_flag, DEV_TIMEOUT_PRODUCER)) {
            ok = false;
            break;
          }
          load_weights(t, kb, stage);
        }
        if (!copier)
          tma_load_2d(smem_u32(smem + static_cast<size_t>(stage) * stage_bytes) + W_BYTES, &tm_x, smem_u32(&bar_full[stage]),
                      kb * (kStageKBytes / static_cast<int>(sizeof(T))), t.row0);
        ++issued;
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    if (!ok) {
      // let the copies still in flight land before the CTA goes away
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
    const uint32_t fmt = (a.dtype == B200MOE_DTYPE_BF16) ? 1u : 0u;
    const uint32_t idesc = make_idesc(fmt, kTileRows, static_cast<uint32_t>(BT));
    constexpr int kSteps = kStageKBytes / 32;  // MMAs per stage and accumulator
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < c.total; tile += c.grid_eff) {
      const TileCoord t = decode_tile(tile, c, s_blk_off, a.E, BT, a.num_nt, a.kblocks, kTileRows);
      if (!mbar_wait(smem_u32(&bar_tempty[acc]), acc_phase ^ 1, abort_flag, DEV_TIMEOUT_MMA)) break;
      tc_fence_after();
      const uint32_t d0 = tmem_base + static_cast<uint32_t>(acc * cols_per_acc);
      for (int kb = t.kb0; kb < t.kb1; ++kb) {
        if (!mbar_wait(smem_u32(&bar_full[stage]), phase, abort_flag, DEV_TIMEOUT_MMA)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sw = smem_u32(smem + static_cast<size_t>(stage) * stage_bytes);
        const uint64_t dw = smem_desc_k_sw128(sw);
        const uint64_t dx = smem_desc_k_sw128(sw + W_BYTES);
#pragma unroll
        for (int k = 0; k < kSteps; ++k) {
          const uint32_t accum = (kb > t.kb0 || k > 0) ? 1u : 0u;
          // advancing 32 bytes inside the 128-byte swizzle atom = +2 in 16-byte units
          tc_mma_f16(d0, dw + 2 * k, dx + 2 * k, idesc, accum);
          if (MODE == 0) {
            const uint64_t du = smem_desc_k_sw128(sw + kTileBytes);
            tc_mma_f16(d0 + static_cast<uint32_t>(BT), du + 2 * k, dx + 2 * k, idesc, accum);
          }
        }
        tc_commit(smem_u32(&bar_empty[stage]));
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) break;
      tc_commit(smem_u32(&bar_tfull[acc]));
      if (++acc == a.acc_stages) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  } else if (active && warp == 7) {
    // =============================== a tile's slots and routing weights =========
    // (by the epilogue warps themselves, with a scan over 1608 slots per tile, the down projection of the 128-expert layer
    // took 84 us instead of 61)
    griddep_wait();
    if (tables) {
      int iter = 0;
      for (int tile = blockIdx.x; tile < c.total; tile += c.grid_eff, ++iter) {
        const TileCoord t = decode_tile(tile, c, s_blk_off, a.E, BT, a.num_nt, a.kblocks, kTileRows);
        const int buf = iter & 1;
        if (!mbar_wait(smem_u32(&bar_sempty[buf]), ((iter >> 1) & 1) ^ 1, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;
        for (int r = 0; r < BT; r += 32) {
          const int slot = rows_slot(a, rt, BT, t.e, t.row0 + r, min(32, BT - r));
          const float weight = rows_weight(a, rt, BT, t.e, t.row0 + r, slot);
          if (r + lane < BT) {
            s_col_row[buf * BT + r + lane] = slot >= 0 ? (MODE == 1 ? slot / a.topk : slot) : -1;
            s_col_gam[buf * BT + r + lane] = weight;
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_sfull[buf]));
      }
    }
  } else if (MODE == 0 && warp == 6) {
    // =============================== token rows (own) ===========================
    if (copier && active) {
      auto rows = [&](auto rc) {
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        const size_t row_bytes = static_cast<size_t>(a.K) * sizeof(T);
        for (int tile = blockIdx.x; ok && tile < c.total; tile += c.grid_eff) {
          const TileCoord t = decode_tile(tile, c, s_blk_off, a.E, BT, a.num_nt, a.kblocks, kTileRows);
          rc.block(a, rt, t.e, t.row0, row_bytes);
          for (int kb = t.kb0; kb < t.kb1; ++kb) {
            if (!mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1, abort_flag, DEV_TIMEOUT_PRODUCER)) {
              ok = false;
              break;
            }
            rc.copy(smem_u32(smem + static_cast<size_t>(stage) * stage_bytes) + W_BYTES, static_cast<size_t>(kb) * kStageKBytes,
                    row_bytes);
            rc.commit(smem_u32(&bar_full[stage]));
            if (++stage == stages) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
        rc.drain();
      };
      if (BT == 16) rows(RowCopier<16, kCopyLag>());
      else rows(RowCopier<32, kCopyLag>());
    }
  } else if (warp >= 2 && warp < 6) {
    // =============================== epilogue ===================================
    griddep_wait();
    if (MODE == 0) clear_combine_buffer(a, threadIdx.x - 64, 128);
    const int quad = warp & 3;                  // TMEM lane quadrant this warp may read
    const int lrow = quad * 32 + lane;          // accumulator row (TMEM lane)
    const bool w_on_input = (a.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0;
    const bool mimic = (a.flags & B200MOE_FLAG_MIMIC_ROUNDING) != 0;
    const bool round_pair = mimic && c.split == 1;
    const ActParams ap = act_params(a);
    const bool has_bias = EXT && a.bias != nullptr;
    int acc = 0, iter = 0;
    uint32_t acc_phase = 0;
    for (int tile = blockIdx.x; active && tile < c.total; tile += c.grid_eff, ++iter) {
      const TileCoord t = decode_tile(tile, c, s_blk_off, a.E, BT, a.num_nt, a.kblocks, kTileRows);
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) +
                             static_cast<uint32_t>(acc * cols_per_acc);
      // ---- accumulator row = weight row: one output column (token) at a time
      const int buf = iter & 1;
      int* col_row = s_col_row + buf * BT;
      float* col_gam = s_col_gam + buf * BT;
      if (tables && !mbar_wait(smem_u32(&bar_sfull[buf]), (iter >> 1) & 1, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;
      if (!mbar_wait(smem_u32(&bar_tfull[acc]), acc_phase, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;
      tc_fence_after();
      const int n = t.n0 + lrow;
      const bool n_ok = n < a.N;
      if (MODE == 0) {
        T* out = reinterpret_cast<T*>(a.out) + static_cast<size_t>(t.row0) * a.ld_out + n;
        float bgate = 0.f, bup = 0.f;
        if (has_bias && n_ok) {
          bgate = __ldg(a.bias + static_cast<size_t>(t.e) * 2 * a.N + n);
          bup = __ldg(a.bias + static_cast<size_t>(t.e) * 2 * a.N + a.N + n);
        }
#pragma unroll 1
        for (int c0 = 0; c0 < BT; c0 += 16) {
          float g[16], u[16];
          tmem_ld16x2_wait(taddr + c0, taddr + BT + c0, g, u);
          if (has_bias) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              g[j] += bgate;
              u[j] += bup;
            }
          }
          act_mul_array<T, EXT>(g, u, w_on_input, mimic, ap, [&](int j) { return col_gam[c0 + j]; });
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (n_ok) out[static_cast<size_t>(c0 + j) * a.ld_out] = from_f32<T>(g[j]);
        }
      } else {
        float* out = reinterpret_cast<float*>(a.out) + n;
        const float bout = (has_bias && n_ok && t.kb0 == 0) ? __ldg(a.bias + static_cast<size_t>(t.e) * a.N + n) : 0.f;
#pragma unroll 1
        for (int c0 = 0; c0 < BT; c0 += 16) {
          float v[16];
          tmem_ld16_wait(taddr + c0, v);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int orow = col_row[c0 + j];
            if (orow >= 0 && n_ok) {
              float y = v[j] + bout;
              if (!w_on_input) y *= col_gam[c0 + j];
              if (round_pair) y = to_f32<T>(from_f32<T>(y));
              atomicAdd(out + static_cast<size_t>(orow) * a.ld_out, y);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&bar_tempty[acc]));
        if (tables) mbar_arrive(smem_u32(&bar_sempty[buf]));
      }
      if (++acc == a.acc_stages) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }

  // ---- teardown (every thread, aborted or not)
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, static_cast<uint32_t>(a.tmem_cols));
  }
  if (threadIdx.x == 0 && *abort_flag != 0) atomicCAS(a.status, 0, *abort_flag);
}

}  // namespace

static size_t stage_bytes_of(const GemmArgs& a) {
  return static_cast<size_t>(a.mode == 0 ? 2 : 1) * kTileBytes + static_cast<size_t>(a.BT) * kStageKBytes;
}

static size_t ctrl_bytes_of(const GemmArgs& a) {
  return 768 /*barriers*/ + 2 * static_cast<size_t>(a.BT) * 8 +
         (a.route.own ? route_table_bytes(a.E, a.P) : static_cast<size_t>(a.E + 1) * 4) + 64;
}

void gemm_plan(GemmArgs* a) {
  a->num_nt = (a->N + kTileRows - 1) / kTileRows;
  a->kblocks = (a->K + 63) / 64;
  const int cols = (a->mode == 0 ? 2 : 1) * a->BT;
  a->acc_stages = (2 * cols <= 512) ? 2 : 1;
  int need = a->acc_stages * cols;
  int tc = 32;
  while (tc < need) tc <<= 1;
  a->tmem_cols = tc;
  int st = static_cast<int>((kSmemLimit - 1024 - ctrl_bytes_of(*a)) / stage_bytes_of(*a));
  if (st > 10) st = 10;
  if (st < 2) st = 2;
  a->stages = st;
  if (a->max_split <= 0) a->max_split = 16;
}

size_t gemm_smem_bytes(const GemmArgs& a) {
  return 1024 + static_cast<size_t>(a.stages) * stage_bytes_of(a) + ctrl_bytes_of(a);
}

template <int MODE, typename T, bool EXT>
static int launch_one(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const GemmArgs& a, int num_sms,
                      cudaStream_t stream) {
  const size_t smem = gemm_smem_bytes(a);
  if (smem > kSmemLimit) return B200MOE_ERR_TOO_LARGE;
  cudaError_t err = cudaFuncSetAttribute(moe_gemm_tc_kernel<MODE, T, EXT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kSmemLimit));
  if (err != cudaSuccess) return B200MOE_ERR_CUDA;
  note_launch(MODE == 0 ? "moe_gemm_tc_kernel<gate/up>" : "moe_gemm_tc_kernel<down>");
  err = launch_kernel(moe_gemm_tc_kernel<MODE, T, EXT>, dim3(num_sms), dim3(kTcThreads), smem, stream, a.pdl != 0, tm_w, tm_x,
                      a);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

template <typename T, bool EXT>
static int launch_typed(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const GemmArgs& a, int num_sms,
                        cudaStream_t stream) {
  return a.mode == 0 ? launch_one<0, T, EXT>(tm_w, tm_x, a, num_sms, stream)
                     : launch_one<1, T, EXT>(tm_w, tm_x, a, num_sms, stream);
}

int launch_gemm_tc(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const GemmArgs& a, int num_sms,
                   cudaStream_t stream) {
  if (a.BT < 16 || a.BT > kMaxBT || a.BT % 16 != 0) return B200MOE_ERR_BAD_ARG;
  if (a.wmode != B200MOE_W_16BIT) return B200MOE_ERR_UNSUPPORTED;
  const bool ext = a.bias != nullptr || a.activation == B200MOE_ACT_SWIGLU_OAI;
  if (a.dtype == B200MOE_DTYPE_BF16)
    return ext ? launch_typed<__nv_bfloat16, true>(tm_w, tm_x, a, num_sms, stream)
               : launch_typed<__nv_bfloat16, false>(tm_w, tm_x, a, num_sms, stream);
  return ext ? launch_typed<__half, true>(tm_w, tm_x, a, num_sms, stream)
             : launch_typed<__half, false>(tm_w, tm_x, a, num_sms, stream);
}

}  // namespace b200moe
