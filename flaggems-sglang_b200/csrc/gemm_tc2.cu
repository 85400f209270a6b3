// 16-bit grouped expert GEMMs on CTA pairs (tcgen05.mma.cta_group::2) for token blocks of 128 and more.
//
// Two CTAs of a cluster share one tile of 256 weight rows x N tokens, N = 32..256 in steps of 32: weights sit
// on the instruction's M side (each CTA stages its 128 rows), the tokens on its N side (each CTA
// stages half of them), the leader CTA issues one MMA for the pair.  Both operands are then read from
// shared memory once per pair, and N follows the tokens an expert really has: its rows are padded to 32 and
// dealt out evenly over ceil(rows / max) tiles, where a kernel with tokens on the M side pays for whole
// blocks of 128 (two experts of eight with 250 tokens on average hold more than 256: 25 % of that kernel's
// MMAs were padding).  Every launch picks `max` from the tokens at hand (see rate_max_granules).
//
//   mode 0 (gate/up):  a CTA's 128 rows are 64 gate rows and the 64 matching up rows; the pair
//                      covers 128 columns of the intermediate.
//   mode 1 (down):     128 rows of the down projection per CTA.
//
// A stage is two TMA loads per CTA whatever the tile: the gate and up rows are one box of a 4-D view
// [experts][gate | up][rows][K], and there is a token map for every half tile of 16..128 rows.  With
// the same bytes in four smaller boxes the producer thread set the pace (4096 tokens of the
// Mixtral-shaped layer, first GEMM: 1.77 ms, 1.34 ms with two loads issued behind elect.sync).
//
// An accumulator lane is a weight row, i.e. an output column, so the epilogue turns 16 tokens at a time in
// shared memory and then stores 16 bytes of a token per thread, contiguous over the lanes of a warp.
// In mode 0 gate and up rows alternate (the box puts row i of both halves next to each other), so the two
// values of a column sit in neighbouring lanes: each lane trades half of its tokens with its
// neighbour and turns finished 16-bit activations.  Turning fp32 gate and up values first cost four times
// the shared-memory traffic and, at K = 1280, more time than the tile's MMAs.
//
// No load here has the cluster-multicast qualifier: every CTA loads its own operands with plain
// tiled TMA loads.  Only tcgen05.commit is multicast (to the same barrier in both CTAs).
// Synchronisation between the two CTAs:
//   * operands staged: the loads of BOTH CTAs complete on the leader's `full` barrier (the
//     cta_group::2 form of the tiled load lets the completion go to the peer CTA's barrier), and the
//     leader alone announces the bytes of both.  Bytes of the second CTA may be counted before they
//     are announced; the phase cannot end without the leader's arrival.  (An arrive.expect_tx by the
//     second CTA on the leader's barrier, a release at cluster scope per stage, held its loads back
//     so far that the pair ran at half speed.)
//   * stage free / accumulator ready: tcgen05.commit of the leader, multicast to both CTAs;
//   * accumulator drained: the epilogue warps of both CTAs arrive on the leader's `tempty`.
// Asking for the weights in L2 ahead of the ring (cp.async.bulk.prefetch.tensor, 4 to 32 stages) was slower
// at every size: 807 us without, 843 to 978 us with, at 1000 tokens of the Mixtral-shaped layer.
//
// What bounds it, from cycle counters around the waits:
//   4096 tokens of the Mixtral-shaped layer: the tensor pipe, 476 cycles per stage for about 470 of MMA, at the clock that the
//     board's power cap leaves (1.15 - 1.25 GHz; 2.41 - 2.46 ms against 2.65 - 2.70 for 128-token blocks on single CTAs);
//   1000 tokens: 403 - 459 cycles per stage for about 350 of MMA, in a train of calls and after a pause; the weights' way from
//     HBM is the nearest other limit (739 - 765 us, 833 - 873 before);
//   K = 1280 (1280 x 3072 x 64 experts, 2048 tokens): the activation epilogue in the first GEMM, whose warps wait only 5 % of the
//     time for a tile and hold the accumulators for 13 % of the MMA thread's; HBM in the second (496 - 500 us with
//     routing, 707 before).
//
// Every wait is bounded (common.cuh); the cluster barriers at start and end are reached by every
// thread whatever happened in between.
#include "gemm_turn.cuh"

namespace b200moe {

namespace {

constexpr int kPairThreads = 320;       // TMA producer, MMA issuer, two epilogue groups of four warps
constexpr int kGran = 32;               // tokens: padding of an expert's rows and step of N
constexpr int kMaxGran = 8;             // N <= 256
constexpr int kMaxStages2 = 10;

// Shared memory: token tables, barriers, granule and tile prefixes of the experts, turning buffers, then the operand
// ring (1024-byte aligned).
constexpr size_t kTc2TableBytes = kTurnTableBytes + 512;
__host__ __device__ __forceinline__ size_t tc2_turn_offset(int E) {
  return (kTc2TableBytes + 2 * static_cast<size_t>(E + 1) * 4 + 127) & ~static_cast<size_t>(127);
}
__host__ __device__ __forceinline__ size_t tc2_fixed_bytes(int E, int mode, bool pairs) {
  return (tc2_turn_offset(E) + turn_bytes(mode, pairs) + 1023) & ~static_cast<size_t>(1023);
}
// operand bytes of one 64-k stage in one CTA: 128 weight rows and half of up to n tokens
__host__ __device__ __forceinline__ int tc2_stage_bytes(int n) { return kTileBytes + n / 2 * kStageKBytes; }

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t mapa_u32(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Tiled loads into this CTA's shared memory whose completion is counted on a barrier that may live
// in the peer CTA (cluster address).  No multicast: one destination.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* m, uint32_t bar_cluster, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
      "[%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* m, uint32_t bar_cluster, int c0, int c1,
                                                 int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, "
      "%5}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap* m, uint32_t bar_cluster, int c0, int c1,
                                                 int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, "
      "%5, %6}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Arrive on the barrier at this shared-memory offset in BOTH CTAs once the pair's MMAs issued so far are done.
__device__ __forceinline__ void tc_commit2(uint32_t bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(mask)
               : "memory");
}
__device__ __forceinline__ void tc_mma2_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Cycles of a 64-k stage of a tile with g granules: four MMAs of N / 2 cycles, or the time the stage's
// operands take from L2 at about 80 bytes per clock and SM, whichever is longer.
__device__ __forceinline__ float stage_cost(int g) {
  return fmaxf(64.f * g, 200.f + 24.f * g) + 16.f;
}

template <int MODE, typename T, bool EXT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
moe_gemm_tc2_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ PairTokenMaps tm_x,
                    const GemmArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  int* s_slot = reinterpret_cast<int*>(smem);                              // [2 groups][2][256]
  float* s_gam = reinterpret_cast<float*>(s_slot + 4 * 256);               // [2 groups][2][256]
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(s_gam + 4 * 256);       // leader: both CTAs' operands are staged
  uint64_t* bar_empty = bar_full + kMaxStages2;
  uint64_t* bar_tfull = bar_empty + kMaxStages2;
  uint64_t* bar_tempty = bar_tfull + 2;          // leader: both CTAs' epilogues have drained the accumulator
  uint64_t* bar_meet = bar_tempty + 2;           // [2] the four warps of an epilogue group
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_meet + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* s_nmax = reinterpret_cast<int*>(tmem_slot + 2);                     // tokens of the widest tile
  float* s_rate = reinterpret_cast<float*>(tmem_slot + 4);                 // [6]
  int* s_gran = reinterpret_cast<int*>(smem + kTc2TableBytes);             // [E+1]
  int* s_tile = s_gran + (a.E + 1);                                        // [E+1]
  uint8_t* s_turn = smem + tc2_turn_offset(a.E);                           // [2 groups][2][16 tokens][pitch]
  const size_t fixed = tc2_fixed_bytes(a.E, MODE, a.out_pairs != nullptr);
  uint8_t* ring = smem + fixed;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages2; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);     // the leader announces the bytes of both CTAs
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bar_tfull[s]), 1);
      mbar_init(smem_u32(&bar_tempty[s]), 16);
      mbar_init(smem_u32(&bar_meet[s]), 4);
    }
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    prefetch_tmap(&tm_w);
  }
  // barriers of both CTAs exist before either side signals the other
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    tmem_alloc2(smem_u32(tmem_slot), 512u);
    tmem_relinquish2();
  }
  griddep_wait();
  griddep_launch_dependents();
  for (int e = threadIdx.x; e <= a.E; e += blockDim.x) s_gran[e] = a.blk_off[e];
  __syncthreads();
  const int num_nt = a.num_nt;
  const int npairs = static_cast<int>(gridDim.x) >> 1;
  if (warp < 6) {
    const float r = rate_max_granules(kMaxGran - warp, s_gran, a.E, num_nt, npairs, lane, stage_cost);
    if (lane == 0) s_rate[warp] = r;
  }
  __syncthreads();
  if (warp == 0) {
    int best = 0;
    for (int w = 1; w < 6; ++w)
      if (s_rate[w] < s_rate[best]) best = w;
    const int cap = a.BT / kGran;     // a caller that fixes the token block bounds the tile with it
    const int maxg = min(kMaxGran - best, cap);
    const int widest = plan_row_tiles(maxg, s_gran, a.E, s_tile, lane);
    if (lane == 0) *s_nmax = widest * kGran;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  constexpr int kTileN = (MODE == 1) ? 256 : 128;
  const int stage_bytes = tc2_stage_bytes(*s_nmax);
  const int stages = min(kMaxStages2, static_cast<int>((kSmemLimit - 1024 - fixed) / stage_bytes));
  const int tiles = s_tile[a.E] * num_nt;
  const int split = (MODE == 1 && !(a.flags & B200MOE_FLAG_NO_SPLIT_K)) ? pick_split(tiles, a.kblocks, npairs, a.max_split) : 1;
  const int total = tiles * split;
  const int pair_id = static_cast<int>(blockIdx.x) >> 1;
  const RowTiles grid = {s_tile, s_gran, a.E, num_nt, split, a.kblocks, kTileN, kGran};
  auto tile_at = [&](int id) { return row_tile_at(id, grid); };

  if (warp == 0 && elect_one()) {
    // =============================== TMA producer (every CTA, its own operands) ===================
    int stage = 0;
    uint32_t phase = 0;
    long long issued = 0;
    bool ok = true;
    constexpr int kKElems = kStageKBytes / static_cast<int>(sizeof(T));
    constexpr int kRowsPerCta = MODE == 0 ? 64 : 128;
    for (int tile = pair_id; ok && tile < total; tile += npairs) {
      const RowTile t = tile_at(tile);
      const int wrow = t.n0 + kRowsPerCta * static_cast<int>(rank);
      const int half = t.n >> 1;
      const int xrow = t.row0 + static_cast<int>(rank) * half;
      const CUtensorMap* mx = &tm_x.m[half / 16 - 1];
      for (int kb = t.kb0; kb < t.kb1; ++kb) {
        if (!mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1, abort_flag, DEV_TIMEOUT_PRODUCER)) {
          ok = false;
          break;
        }
        const uint32_t full = mapa_u32(smem_u32(&bar_full[stage]), 0);   // the leader's barrier
        const uint32_t sw = smem_u32(ring + static_cast<size_t>(stage) * stage_bytes);
        const int k0 = kb * kKElems;
        if (leader)
          mbar_arrive_expect_tx(smem_u32(&bar_full[stage]), static_cast<uint32_t>(2 * kTileBytes + t.n * kStageKBytes));
        if (MODE == 0) tma_load_4d_pair(sw, &tm_w, full, k0, 0, wrow, t.e);
        else tma_load_3d_pair(sw, &tm_w, full, k0, wrow, t.e);
        tma_load_2d_pair(sw + kTileBytes, mx, full, k0, xrow);
        ++issued;
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    if (!ok) {
      // let the copies still in flight land before the CTA goes away: the leader sees them on its
      // barriers; the second CTA, whose completions are counted elsewhere, simply waits a while
      if (leader) {
        const int n = static_cast<int>(issued < stages ? issued : stages);
        for (int i = 1; i <= n; ++i) {
          int s2 = stage - i;
          uint32_t ph = phase;
          if (s2 < 0) {
            s2 += stages;
            ph ^= 1;
          }
          mbar_wait_brief(smem_u32(&bar_full[s2]), ph);
        }
      } else {
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 20000ull) {
        }
      }
    }
  } else if (warp == 1 && leader && elect_one()) {
    // =============================== MMA issuer (leader CTA, for the pair) ========================
    const uint32_t fmt = (a.dtype == B200MOE_DTYPE_BF16) ? 1u : 0u;
    constexpr int kSteps = kStageKBytes / 32;
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0;
    bool ok = true;
    for (int tile = pair_id; ok && tile < total; tile += npairs) {
      const RowTile t = tile_at(tile);
      const uint32_t idesc = make_idesc(fmt, 256u, static_cast<uint32_t>(t.n));
      if (!mbar_wait(smem_u32(&bar_tempty[acc]), acc_phase ^ 1, abort_flag, DEV_TIMEOUT_MMA)) break;
      tc_fence_after();
      const uint32_t d0 = tmem_base + static_cast<uint32_t>(acc * 256);
      for (int kb = t.kb0; kb < t.kb1; ++kb) {
        if (!mbar_wait(smem_u32(&bar_full[stage]), phase, abort_flag, DEV_TIMEOUT_MMA)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sw = smem_u32(ring + static_cast<size_t>(stage) * stage_bytes);
        const uint64_t dw = smem_desc_k_sw128(sw);                 // this CTA's weight rows: the M side
        const uint64_t dx = smem_desc_k_sw128(sw + kTileBytes);    // this CTA's half of the tokens: the N side
#pragma unroll
        for (int k = 0; k < kSteps; ++k) tc_mma2_f16(d0, dw + 2 * k, dx + 2 * k, idesc, (kb > t.kb0 || k > 0) ? 1u : 0u);
        tc_commit2(smem_u32(&bar_empty[stage]));
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) break;
      tc_commit2(smem_u32(&bar_tfull[acc]));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  } else if (warp >= 2) {
    // =============================== epilogue (every CTA, its own 128 weight rows) ================
    TurnEpilogue<MODE, T, EXT> ep(a, s_turn, s_slot, s_gam, bar_meet, abort_flag, warp - 2, warp, lane,
                                  (MODE == 0 ? 64 : 128) * static_cast<int>(rank), split);
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = pair_id; tile < total; tile += npairs) {
      const RowTile t = tile_at(tile);
      if (!ep.load_tables(t)) break;
      if (!mbar_wait(smem_u32(&bar_tfull[acc]), acc_phase, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(ep.quad * 32) << 16) + static_cast<uint32_t>(acc * 256);
      if (!ep.run(t, taddr, [&] {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(mapa_u32(smem_u32(&bar_tempty[acc]), 0));
          }))
        break;
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }

  // ---- teardown (every thread of both CTAs, aborted or not): neither CTA may leave while the other
  // can still signal its barriers or read its shared memory
  tc_fence_before();
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc2(tmem_base, 512u);
  }
  if (threadIdx.x == 0 && *abort_flag != 0) atomicCAS(a.status, 0, *abort_flag);
}

int g_tc2_pairs_seen = 0;   // resident CTA pairs found for the last launch (diagnostics)

// How many CTA pairs of this kernel the device keeps resident at once.  The kernel is persistent with
// a static tile assignment, so a grid with even one pair more than that would run its last pairs as a
// second wave and take twice as long.
template <int MODE, typename T, bool EXT>
int max_resident_pairs(int num_sms) {
  static const int resident = [] {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = kSmemLimit;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, moe_gemm_tc2_kernel<MODE, T, EXT>, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = 0;
    }
    return n;
  }();
  const int half = num_sms / 2;
  const int n = resident > 0 ? resident : half - 2;     // conservative guess where the query fails
  return n < half ? n : half;
}

template <int MODE, typename T, bool EXT>
int launch_tc2(const CUtensorMap& tm_w, const PairTokenMaps& tm_x, const GemmArgs& a, int num_sms, cudaStream_t stream) {
  if (cudaFuncSetAttribute(moe_gemm_tc2_kernel<MODE, T, EXT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kSmemLimit)) != cudaSuccess)
    return B200MOE_ERR_CUDA;
  const int pairs = max_resident_pairs<MODE, T, EXT>(num_sms);
  if (pairs <= 0) return B200MOE_ERR_UNSUPPORTED;
  g_tc2_pairs_seen = pairs;
  note_launch(MODE == 0 ? "moe_gemm_tc2_kernel<gate/up>" : "moe_gemm_tc2_kernel<down>");
  cudaError_t err = launch_kernel(moe_gemm_tc2_kernel<MODE, T, EXT>, dim3(2 * pairs), dim3(kPairThreads), kSmemLimit, stream,
                                  a.pdl != 0, tm_w, tm_x, a);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

template <typename T, bool EXT>
int launch_typed(const CUtensorMap& tm_w, const PairTokenMaps& tm_x, const GemmArgs& a, int num_sms, cudaStream_t stream) {
  return a.mode == 0 ? launch_tc2<0, T, EXT>(tm_w, tm_x, a, num_sms, stream)
                     : launch_tc2<1, T, EXT>(tm_w, tm_x, a, num_sms, stream);
}

}  // namespace

int gemm_tc2_resident_pairs() { return g_tc2_pairs_seen; }

// The pair kernel keeps two prefixes over the experts in shared memory and needs a few stages beside them.
bool gemm_tc2_ok(int E, int num_sms) {
  return num_sms >= 6 && kSmemLimit - 1024 - tc2_fixed_bytes(E, 1, false) >= 3 * static_cast<size_t>(tc2_stage_bytes(256));
}

// a->BT: upper bound of the tokens per tile (a multiple of 32)
void gemm_plan_tc2(GemmArgs* a) {
  const int tile_n = (a->mode == 1) ? 256 : kTileRows;
  a->num_nt = (a->N + tile_n - 1) / tile_n;
  a->kblocks = (a->K + 63) / 64;
  a->acc_stages = 2;
  a->tmem_cols = 512;
  if (a->max_split <= 0) a->max_split = 16;
}

int launch_gemm_tc2(const CUtensorMap& tm_w, const PairTokenMaps& tm_x, const GemmArgs& a, int num_sms,
                    cudaStream_t stream) {
  if (a.wmode != B200MOE_W_16BIT || a.BT < kGran || a.BT % kGran != 0) return B200MOE_ERR_UNSUPPORTED;
  const bool ext = a.bias != nullptr || a.activation == B200MOE_ACT_SWIGLU_OAI;
  if (a.dtype == B200MOE_DTYPE_BF16)
    return ext ? launch_typed<__nv_bfloat16, true>(tm_w, tm_x, a, num_sms, stream)
               : launch_typed<__nv_bfloat16, false>(tm_w, tm_x, a, num_sms, stream);
  return ext ? launch_typed<__half, true>(tm_w, tm_x, a, num_sms, stream)
             : launch_typed<__half, false>(tm_w, tm_x, a, num_sms, stream);
}

}  // namespace b200moe
