// Grouped expert GEMMs for int4 (AWQ, group 128, zero points) weights and fp16 activations.
//
// A tile is 128 weight rows on the MMA's M side (mode 0: 64 gate rows and the matching up rows, alternating; mode 1:
// 128 rows of the down projection) x N tokens.  The packed nibbles of one quantisation group (128 k) arrive by TMA,
// conversion warps expand them to fp16 and write them straight into tensor memory (tcgen05.st), from where the MMA
// takes its A operand: the expanded weights never touch shared memory, which carries only the packed
// rows and the tokens.  (Expanding into shared memory moved 104 KiB per 64 k through it for 512 cycles of MMA.)
//
// Two variants of the same kernel (GemmArgs::w4_var):
//   NT = 0       any number of tokens per tile (16..192, dealt out evenly over an expert's tiles); the operand is
//                (q - zero) * scale, rounded once to fp16, and the reduction accumulates in tensor memory.
//   NT = 16, 32  decode: a tile is one block of NT tokens; the operand is the exact integer q - zero, each group's
//                sum goes into a partial accumulator of its own and is added as acc += scale * sum in fp32 by the
//                promotion warps.  Weights and activations are then exact up to the fp32 sums.
//                NT = 16 expands nothing: a masked nibble already is the fp16 subnormal q * 2^-24, and eight more MMAs per
//                group add -zero (times the same 2^-24) against every k.  The schedulers, which all roles
//                share, then see 7 instructions per eight weights instead of 9, none of them half-precision arithmetic
//                (Mixtral-shaped layer, us, expanded / unexpanded: 2 tokens 111.8 / 102.8, 4: 164.7 / 156.7, 16: 222 / 219).
//                At NT = 32 the extra MMAs are the longer path (64 tokens 269 / 285).
//
// Packed rows and tokens have rings of their own: the packed rows of a group are needed a conversion (about 900 cycles)
// earlier than its tokens, and at 192 tokens only three stages of tokens fit.  The MMA thread works on units of one (NT =
// 0) or two groups and commits once per unit to one barrier, on which the token producer, the conversion warps and
// the promotion warps all wait; with three commits and three waits per group that thread set the pace at decode.
//
// What bounds it, from cycle counters around every wait on the Mixtral-shaped layer (8 experts, top-2):
//   2048 tokens  the MMAs: a unit of the first GEMM takes 894 cycles, 704 of them MMAs of 176 tokens; its thread waits 9 %
//                of the time for operands and 10 % for tokens, never for an accumulator.  The conversion keeps the same pace
//                (1786 cycles per group and set, two sets) and waits 23 % of the time for a free operand slot.
//   32 tokens    no single role.  A unit takes 1047 cycles in the first GEMM and 1273 in the second, where HBM needs 770; the
//                MMA thread spends about 650 issuing its 32 MMAs of 16 tokens, and waits 19 % of the time for operands, 10 %
//                for tokens and 9 % for partial accumulators (second GEMM: 25 %, whose tails add 16 tokens to the combine
//                buffer with atomics).  A conversion set is busy about 1000 cycles per group of its own.
// us per call on one board: 2 tokens 124, 4: 158, 16: 215, 32: 222, 64: 258, 256: 368, 600: 552, 2048: 1423 (integer MMAs on
// three byte planes up to 32 tokens, above them 128-token blocks on the M side with the nibbles expanded into shared memory:
// 144, 178, 237, 244, 365, 494, 939, 2027).
//
// Decode calls sort their slots in here (gemm_route.cuh) behind a launch that gathers the rows; the packed rows and their
// conversion start before those are there.  (Fetching the rows from here was slower: gather4 loads take about 80 cycles each,
// four rows of 128 bytes, and set the pace of a unit, 32 tokens 205 -> 233 us; a copying warp waits for a proxy fence per unit, 217.)
// A lane looks one row's slot and weight up and tells the others: one after the other they cost a tile two memory latencies
// per row (32 tokens 205 -> 200).
//
// Warps: 0 packed rows, 1 MMA, 2 tokens, from 4 on the conversion (two or three sets of four warps), then the epilogue or
// promotion (one or two groups of four).
#include "gemm_route.cuh"
#include "gemm_turn.cuh"

namespace b200moe {

namespace {

constexpr int kPackedRowBytes = 64;                              // 128 k (one group) of one weight row
constexpr int kPackedBytes = kTileRows * kPackedRowBytes;        // 8 KiB per group
constexpr int kMaxStagesX = 8;
constexpr int kDone = 8;                                         // ring of unit-complete barriers
constexpr int kGranW4 = 16;                                      // tokens: padding of an expert's rows and step of N
constexpr int kMaxGranW4 = 12;                                   // N <= 192: two accumulators and two operand stages fit

// Per variant: groups per unit, packed stages (of a unit each), slots of scale / zero words (one per group).  A slot is
// refilled once the packed stage `kPacked` units before it has been read; the promotion may then be as far back as the packed
// stages, the groups in conversion, and the units whose operands or partial sums are in flight.
template <int NT>
struct W4Geo {
  static constexpr int kGroups = NT > 0 ? 2 : 1;
  static constexpr int kPacked = NT > 0 ? 8 : 4;
  static constexpr int kWords = NT > 0 ? 48 : 16;
  static constexpr int kPartials = NT == 16 ? 4 : 2;      // units (NT = 0: tiles) whose accumulators are in flight
  // NT = 16: the nibbles go in as they are and the zero points as an operand of their own (8 columns a group)
  static constexpr bool kZeroMma = NT == 16;
  static constexpr int kSlots = NT == 16 ? 2 : 3;         // NT > 0: units whose operands are in flight
  static constexpr int kSlotCols = kGroups * (kZeroMma ? 72 : 64);   // tensor-memory columns of a unit's operands
  // Conversion sets: at decode a group's conversion takes one set about 1000 cycles, most of them latency, and HBM
  // delivers a group every 380.  One promotion group holds all 16 tokens of a block.
  static constexpr int kSets = NT > 0 ? 3 : 2;
  static constexpr int kTailGroups = NT == 16 ? 1 : 2;
  static constexpr int kThreads = (4 + 4 * kSets + 4 * kTailGroups) * 32;
  static constexpr size_t kPackedStage = kGroups * static_cast<size_t>(kPackedBytes);
  static constexpr size_t kTableBytes = kWords * kTileRows * 4 + (NT == 0 ? kTurnTableBytes : 0) + 768;
};
static_assert(W4Geo<16>::kWords >= 2 * W4Geo<16>::kPacked + W4Geo<16>::kSets + 2 * (3 + W4Geo<16>::kPartials + 1), "scale word ring");

template <int NT>
__host__ __device__ __forceinline__ size_t w4_turn_offset(int E) {
  // prefixes over the experts: granules and tiles, which at decode are the same
  return (W4Geo<NT>::kTableBytes + (NT > 0 ? 1 : 2) * static_cast<size_t>(E + 1) * 4 + 127) & ~static_cast<size_t>(127);
}
// own_slots: slots of a decode call that sorts them itself (its tables stand in the place of the prefixes), or 0
template <int NT>
__host__ __device__ __forceinline__ size_t w4_fixed_bytes(int E, int mode, bool pairs, int own_slots = 0) {
  return (((NT > 0 && own_slots > 0 ? W4Geo<NT>::kTableBytes + route_table_bytes(E, own_slots)
                                    : w4_turn_offset<NT>(E) + (NT == 0 ? turn_bytes(mode, pairs) : 0)) + 1023) & ~static_cast<size_t>(1023)) +
         W4Geo<NT>::kPacked * W4Geo<NT>::kPackedStage;
}
// tokens of one unit: swizzle atoms of 64 k
__host__ __device__ __forceinline__ int w4_token_bytes(int n, int groups) { return n * 256 * groups; }

// Cycles per group of a tile with g granules: eight MMAs of N / 2 cycles, or the conversion.
__device__ __forceinline__ float w4_cost(int g) { return fmaxf(64.f * g, 320.f) + 30.f; }

__device__ __forceinline__ void tmem_st8_same(uint32_t taddr, uint32_t v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr), "r"(v) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Eight packed weights (element 2i in nibble i, element 2i+1 in nibble 4+i) -> four fp16 pairs of q - zero, exact:
// w & 0x000F000F | 0x64006400 reads as the pair (1024 + q), less (1024 + zero); w & 0x00F000F0 | 0x64006400 as (1024 +
// 16 q), times 1/16 less (64 + zero).  SCALED: times the scale, rounded once.
template <bool SCALED>
__device__ __forceinline__ void expand8(uint32_t w, __half2 zero1024, __half2 mzero64, __half2 scale, uint32_t* out) {
  const __half2 sixteenth = __float2half2_rn(0.0625f);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    uint32_t lo = (w & 0x000F000Fu) | 0x64006400u, hi = (w & 0x00F000F0u) | 0x64006400u;
    __half2 a = __hsub2(*reinterpret_cast<__half2*>(&lo), zero1024);
    __half2 b = __hfma2(*reinterpret_cast<__half2*>(&hi), sixteenth, mzero64);
    if (SCALED) {
      a = __hmul2(a, scale);
      b = __hmul2(b, scale);
    }
    out[2 * i] = *reinterpret_cast<uint32_t*>(&a);
    out[2 * i + 1] = *reinterpret_cast<uint32_t*>(&b);
    w >>= 8;
  }
}

template <int MODE, bool EXT, int NT>
__global__ void __launch_bounds__(W4Geo<NT>::kThreads, 1)
moe_gemm_w4_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_sz,
                   const __grid_constant__ W4TokenMaps tm_x, const GemmArgs a) {
  using T = __half;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  using G = W4Geo<NT>;
  constexpr int GP = G::kGroups;
  uint32_t* s_sz = reinterpret_cast<uint32_t*>(smem);                        // [kWords][128] scale | 1024 + zero
  int* s_slot = reinterpret_cast<int*>(s_sz + G::kWords * kTileRows);        // NT = 0: token tables of the turning epilogue
  float* s_gam = reinterpret_cast<float*>(s_slot + 4 * kTurnMaxTok);
  uint64_t* bar_wfull = reinterpret_cast<uint64_t*>(NT == 0 ? reinterpret_cast<int*>(s_gam + 4 * kTurnMaxTok) : s_slot);
  uint64_t* bar_wempty = bar_wfull + G::kPacked;
  uint64_t* bar_xfull = bar_wempty + G::kPacked;
  uint64_t* bar_dq = bar_xfull + kMaxStagesX;       // [4] operand stage written
  uint64_t* bar_done = bar_dq + 4;                  // [kDone] the MMAs of a unit have finished
  uint64_t* bar_tfull = bar_done + kDone;           // [2] NT = 0: accumulator of a tile complete
  uint64_t* bar_tempty = bar_tfull + 2;             // [4] accumulator or partial sums read
  uint64_t* bar_meet = bar_tempty + 4;              // [2] the four warps of an epilogue group
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_meet + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* s_nmax = reinterpret_cast<int*>(tmem_slot + 2);
  float* s_rate = reinterpret_cast<float*>(tmem_slot + 4);                   // [6]
  int* s_gran = reinterpret_cast<int*>(smem + G::kTableBytes);               // [E+1] granules (NT > 0: blocks) before e
  int* s_tile = NT > 0 ? s_gran : s_gran + (a.E + 1);                        // [E+1] tiles before e
  uint8_t* s_turn = smem + w4_turn_offset<NT>(a.E);
  const bool own = NT > 0 && a.route.own != 0, early = own && a.route.early != 0;
  const RowTables rt = row_tables(s_gran, a.E);
  const size_t fixed = w4_fixed_bytes<NT>(a.E, MODE, a.out_pairs != nullptr, own ? a.P : 0);
  uint8_t* packed = smem + fixed - G::kPacked * G::kPackedStage;
  uint8_t* tokens = smem + fixed;

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < G::kPacked; ++s) {
      mbar_init(smem_u32(&bar_wfull[s]), 1);
      mbar_init(smem_u32(&bar_wempty[s]), 4 * GP);
    }
    for (int s = 0; s < kMaxStagesX; ++s) mbar_init(smem_u32(&bar_xfull[s]), 1);
    for (int s = 0; s < kDone; ++s) mbar_init(smem_u32(&bar_done[s]), 1);
    for (int s = 0; s < 4; ++s) {
      mbar_init(smem_u32(&bar_dq[s]), 4 * GP);
      mbar_init(smem_u32(&bar_tempty[s]), 4 * G::kTailGroups);
    }
    for (int s = 0; s < 2; ++s) mbar_init(smem_u32(&bar_tfull[s]), 1);
    for (int s = 0; s < 2; ++s) mbar_init(smem_u32(&bar_meet[s]), 4);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    prefetch_tmap(&tm_w);
    prefetch_tmap(&tm_sz);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512u);
    tmem_relinquish();
  }
  if (!early) griddep_wait();
  griddep_launch_dependents();
  if (NT > 0 && own) count_slots(a.route, a.P, a.E, NT, rt);
  else
    for (int e = threadIdx.x; e <= a.E; e += blockDim.x) s_gran[e] = a.blk_off[e];
  __syncthreads();
  const int num_nt = a.num_nt;
  if (NT == 0) {
    constexpr int kTry[6] = {12, 10, 8, 6, 5, 4};
    if (warp < 6) {
      const float r = rate_max_granules(kTry[warp], s_gran, a.E, num_nt, gridDim.x, lane, w4_cost);
      if (lane == 0) s_rate[warp] = r;
    }
    __syncthreads();
    if (warp == 0) {
      int best = 0;
      for (int w = 1; w < 6; ++w)
        if (s_rate[w] < s_rate[best]) best = w;
      int maxg = kTry[0];
#pragma unroll
      for (int w = 1; w < 6; ++w)
        if (w == best) maxg = kTry[w];
      const int widest = plan_row_tiles(min(maxg, a.BT / kGranW4), s_gran, a.E, s_tile, lane);
      if (lane == 0) *s_nmax = widest * kGranW4;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  constexpr int kTileN = MODE == 0 ? 64 : 128;        // output columns per tile
  const int nmax = NT > 0 ? NT : *s_nmax;
  const int token_bytes = w4_token_bytes(nmax, GP);
  const int stages = min(kMaxStagesX, static_cast<int>((kSmemLimit - 1024 - fixed) / token_bytes));
  const int tiles = s_tile[a.E] * num_nt;
  const int split = (MODE == 1 && !(a.flags & B200MOE_FLAG_NO_SPLIT_K)) ? pick_split(tiles, a.kblocks, gridDim.x, a.max_split) : 1;
  const int total = tiles * split;
  const RowTiles grid = {s_tile, s_gran, a.E, num_nt, split, a.kblocks, kTileN, NT > 0 ? NT : kGranW4};
  // tensor memory: accumulators first, then the operand stages
  const int acc_cols = NT > 0 ? GP * NT : nmax;
  const uint32_t a_col0 = static_cast<uint32_t>(G::kPartials * acc_cols);
  const int slots_a = NT > 0 ? G::kSlots : min(4, (512 - 2 * nmax) / 64);
  const int first = blockIdx.x, stride = gridDim.x;
  // units of this CTA over the whole launch; a lane takes a tile (every thread taking all of them one after the other
  // cost the second GEMM of a decode call 8 us before its first load)
  int units = 0;
  if (split == 1) {
    units = first < total ? ((total - first + stride - 1) / stride) * a.kblocks : 0;
  } else {
    for (int tile = first + lane * stride; tile < total; tile += 32 * stride) {
      const RowTile t = row_tile_at(tile, grid);
      units += t.kb1 - t.kb0;
    }
    units = __reduce_add_sync(0xffffffffu, units);
  }
  // The MMAs of unit u have finished.  Nobody falls a whole ring behind: the MMA thread needs every waiter's
  // product (tokens, operands, free partial sums) within fewer units than the ring has barriers.
  auto wait_done = [&](int u, int code) -> bool {
    return u < 0 || mbar_wait(smem_u32(&bar_done[u % kDone]), (u / kDone) & 1, abort_flag, code);
  };

  if (warp == 0) {
    if (elect_one()) {
      // =============================== packed rows and their scale / zero words ===
      int u = 0;
      bool ok = true;
      const int kgroups = a.K / 128;
      for (int tile = first; ok && tile < total; tile += stride) {
        const RowTile t = row_tile_at(tile, grid);
        // (the second group of an odd reduction's last unit lies past the rows: zeros, like its tokens)
        for (int kb = t.kb0; kb < t.kb1; ++kb, ++u) {
          const int ws = u % G::kPacked;
          if (!mbar_wait(smem_u32(&bar_wempty[ws]), ((u / G::kPacked) & 1) ^ 1, abort_flag, DEV_TIMEOUT_PRODUCER)) {
            ok = false;
            break;
          }
          const uint32_t full = smem_u32(&bar_wfull[ws]);
          const uint32_t spk = smem_u32(packed + ws * G::kPackedStage);
          mbar_arrive_expect_tx(full, static_cast<uint32_t>(GP * (kPackedBytes + kTileRows * 4)));
          if (MODE == 0) tma_load_4d(spk, &tm_w, full, kb * GP * kPackedRowBytes, 0, t.n0, t.e);
          else tma_load_3d(spk, &tm_w, full, kb * GP * kPackedRowBytes, t.n0, t.e);
          tma_load_3d(smem_u32(s_sz + (u * GP % G::kWords) * kTileRows), &tm_sz, full, t.n0, 0, t.e * kgroups + kb * GP);
        }
      }
      if (!ok)       // let the copies still in flight land before the CTA goes away
        for (int i = 1; i <= G::kPacked && i <= u; ++i)
          mbar_wait_brief(smem_u32(&bar_wfull[(u - i) % G::kPacked]), ((u - i) / G::kPacked) & 1);
    }
  } else if (warp == 2) {
    if (elect_one()) {
      // =============================== tokens =====================================
      griddep_wait();       // (the packed rows and their conversion need not wait for the activations)
      int u = 0;
      bool ok = true;
      for (int tile = first; ok && tile < total; tile += stride) {
        const RowTile t = row_tile_at(tile, grid);
        const CUtensorMap* mx = NT > 0 ? &tm_x.m[0] : &tm_x.m[t.n / 16 - 1];
        for (int kb = t.kb0; kb < t.kb1; ++kb, ++u) {
          if (!wait_done(u - stages, DEV_TIMEOUT_PRODUCER)) {
            ok = false;
            break;
          }
          const uint32_t full = smem_u32(&bar_xfull[u % stages]);
          mbar_arrive_expect_tx(full, static_cast<uint32_t>(w4_token_bytes(t.n, GP)));
          tma_load_3d(smem_u32(tokens + static_cast<size_t>(u % stages) * token_bytes), mx, full, 0, t.row0, kb * 2 * GP);
        }
      }
      if (!ok)
        for (int i = 1; i <= stages && i <= u; ++i)
          mbar_wait_brief(smem_u32(&bar_xfull[(u - i) % stages]), ((u - i) / stages) & 1);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // =============================== MMA issuer =================================
      int stage = 0, slot = 0, acc = 0, u = 0;
      uint32_t phase = 0, ophase = 0, acc_phase = 0;
      bool ok = true;
      // one unit: operands of GP groups against n tokens; group g accumulates at d + g * n (NT > 0: afresh)
      auto unit_mma = [&](uint32_t d, int n, bool fresh) -> bool {
        if (!mbar_wait(smem_u32(&bar_xfull[stage]), phase, abort_flag, DEV_TIMEOUT_MMA) ||
            !mbar_wait(smem_u32(&bar_dq[slot]), ophase, abort_flag, DEV_TIMEOUT_MMA))
          return false;
        tc_fence_after();
        const uint32_t idesc = make_idesc(0u, kTileRows, static_cast<uint32_t>(n));
        const uint32_t a0 = tmem_base + a_col0 + static_cast<uint32_t>(slot) * G::kSlotCols;
        const uint64_t dx = smem_desc_k_sw128(smem_u32(tokens + static_cast<size_t>(stage) * token_bytes));
        const uint64_t atom = static_cast<uint64_t>(n * 128) >> 4;
#pragma unroll
        for (int g = 0; g < GP; ++g) {
          const uint32_t dg = d + static_cast<uint32_t>(g * n);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            tc_mma_f16_ts(dg, a0 + 64u * g + 8 * k, dx + (2 * g + (k >> 2)) * atom + 2 * (k & 3), idesc,
                          (!fresh || k > 0) ? 1u : 0u);
          if (G::kZeroMma) {       // the zero points: the same 16 columns of -zero against every 16 k of the tokens
#pragma unroll
            for (int k = 0; k < 8; ++k)
              tc_mma_f16_ts(dg, a0 + 64u * GP + 8u * g, dx + (2 * g + (k >> 2)) * atom + 2 * (k & 3), idesc, 1u);
          }
        }
        tc_commit(smem_u32(&bar_done[u % kDone]));
        ++u;
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
        if (++slot == slots_a) {
          slot = 0;
          ophase ^= 1;
        }
        return true;
      };
      if (NT > 0) {
        while (u < units) {
          if (!mbar_wait(smem_u32(&bar_tempty[acc]), acc_phase ^ 1, abort_flag, DEV_TIMEOUT_MMA)) break;
          if (!unit_mma(tmem_base + static_cast<uint32_t>(acc * acc_cols), NT, true)) break;
          if (++acc == G::kPartials) {
            acc = 0;
            acc_phase ^= 1;
          }
        }
      } else {
        for (int tile = first; ok && tile < total; tile += stride) {
          const RowTile t = row_tile_at(tile, grid);
          if (!mbar_wait(smem_u32(&bar_tempty[acc]), acc_phase ^ 1, abort_flag, DEV_TIMEOUT_MMA)) break;
          for (int kb = t.kb0; ok && kb < t.kb1; ++kb)
            ok = unit_mma(tmem_base + static_cast<uint32_t>(acc * acc_cols), t.n, kb == t.kb0);
          if (!ok) break;
          tc_commit(smem_u32(&bar_tfull[acc]));
          if (++acc == 2) {
            acc = 0;
            acc_phase ^= 1;
          }
        }
      }
    }
  } else if (warp >= 4 && warp < 4 + 4 * G::kSets) {
    // =============================== nibbles -> fp16 in tensor memory ============
    // the sets take groups in turn; a thread owns the row in its own TMEM lane
    const int set = (warp - 4) >> 2, quad = warp & 3;
    const int row = quad * 32 + lane;
    // the packed rows are staged with the swizzle of their width: 16-byte chunk c of row r sits at chunk c ^ (r & 7) of
    // its 128 bytes (two groups) or c ^ ((r >> 1) & 3) of its 64, which spreads the rows over all banks
    const int sw = GP == 2 ? (row & 7) : ((row >> 1) & 3);
    const int word = MODE == 0 ? (row & 1) * 64 + (row >> 1) : row;    // gate words first, then the up words
    for (int g = set; g < units * GP; g += G::kSets) {
      const int u = g / GP, ws = u % G::kPacked;
      if (!mbar_wait(smem_u32(&bar_wfull[ws]), (u / G::kPacked) & 1, abort_flag, DEV_TIMEOUT_MMA)) break;
      const uint4* prow = reinterpret_cast<const uint4*>(packed + ws * G::kPackedStage + row * (GP * kPackedRowBytes));
      const uint32_t szv = s_sz[(g % G::kWords) * kTileRows + word];
      uint4 v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) v[c] = prow[(4 * (g % GP) + c) ^ sw];
      const __half2 sc = __half2half2(__ushort_as_half(static_cast<unsigned short>(szv & 0xFFFFu)));
      const __half2 zp = __half2half2(__ushort_as_half(static_cast<unsigned short>(szv >> 16)));
      const __half2 mz = __hsub2(__float2half2_rn(960.f), zp);       // -(64 + zero)
      const uint32_t dst = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + a_col0 +
                           static_cast<uint32_t>(u % slots_a) * G::kSlotCols + static_cast<uint32_t>(g % GP) * 64u;
      // As much as the registers hold is converted before the wait for a free operand stage: with two stages (192
      // tokens) the time from there to the MMA would otherwise add to every second unit.
      constexpr int kBefore = NT == 0 ? 2 : 1;
      uint32_t o[2][32];
      auto convert = [&](int b) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint32_t w[4] = {v[2 * b + c].x, v[2 * b + c].y, v[2 * b + c].z, v[2 * b + c].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (!G::kZeroMma) {
              expand8<NT == 0>(w[q], zp, mz, sc, o[b] + 16 * c + 4 * q);
            } else {
#pragma unroll
              for (int i = 0; i < 4; ++i) o[b][16 * c + 4 * q + i] = (w[q] >> (4 * i)) & 0x000F000Fu;
            }
          }
        }
      };
#pragma unroll
      for (int b = 0; b < kBefore; ++b) convert(b);
      // The loads of the rows are issued here, but nothing needs their data before the operands are stored, and the next
      // rows are written by another proxy (TMA), which the arrival alone does not hold back: at 176-192 tokens a tile, where
      // the MMAs and the token loads take all of shared memory's bandwidth, one refill in about 10^5 overtook the loads of
      // some lanes of a warp.  The fence orders them (2048 tokens 1415 -> 1432 us, 32 tokens 222 -> 224).
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_wempty[ws]));
      if (!wait_done(u - slots_a, DEV_TIMEOUT_MMA)) break;
      tc_fence_after();
      tmem_st32(dst, o[0]);
      if (kBefore == 1) convert(1);
      tmem_st32(dst + 32, o[1]);
      if (G::kZeroMma) {
        const uint32_t z = 0x8000u | ((szv >> 16) & 0x3FFu);       // -zero as a subnormal, like the nibbles
        tmem_st8_same(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + a_col0 +
                          static_cast<uint32_t>(u % slots_a) * G::kSlotCols + 64u * GP + static_cast<uint32_t>(g % GP) * 8u,
                      z | (z << 16));
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_dq[u % slots_a]));
    }
  } else if (warp < 4) {
    // idle
  } else if (NT == 0) {
    // =============================== epilogue: turn and store ====================
    TurnEpilogue<MODE, T, EXT> ep(a, s_turn, s_slot, s_gam, bar_meet, abort_flag, warp - 4 - 4 * G::kSets, warp, lane, 0, split);
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = first; tile < total; tile += stride) {
      const RowTile t = row_tile_at(tile, grid);
      if (!ep.load_tables(t)) break;
      if (!mbar_wait(smem_u32(&bar_tfull[acc]), acc_phase, abort_flag, DEV_TIMEOUT_EPILOGUE)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(ep.quad * 32) << 16) + static_cast<uint32_t>(acc * acc_cols);
      if (!ep.run(t, taddr, [&] {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_tempty[acc]));
          }))
        break;
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  } else {
    // =============================== promotion + tail ============================
    griddep_wait();
    constexpr int HT = NT > 0 ? NT / G::kTailGroups : 16;         // tokens per thread
    const int grp = (warp - 4 - 4 * G::kSets) >> 2, quad = warp & 3;
    const int row = quad * 32 + lane;
    const int word = MODE == 0 ? (row & 1) * 64 + (row >> 1) : row;
    const bool w_on_input = (a.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0;
    const bool mimic = (a.flags & B200MOE_FLAG_MIMIC_ROUNDING) != 0;
    const bool round_pair = mimic && split == 1;
    const bool has_bias = EXT && a.bias != nullptr;
    const ActParams ap = act_params(a);
    const bool odd = (lane & 1) != 0;
    int acc = 0, u = 0;
    bool ok = true;
    for (int tile = first; ok && tile < total; tile += stride) {
      const RowTile t = row_tile_at(tile, grid);
      const int r0 = t.row0 + grp * HT;
      // output row and routing weight of this group's tokens, fetched ahead of the reduction (uniform over the warp)
      int orow[HT];
      float gam[HT];
      if (MODE == 1 || w_on_input) {      // a lane looks one row up and tells the others
        const int slot = rows_slot(a, rt, NT, t.e, r0, HT);
        const float weight = rows_weight(a, rt, NT, t.e, r0, slot);
        const int token = slot >= 0 ? slot / a.topk : -1;
#pragma unroll
        for (int i = 0; i < HT; ++i) {
          orow[i] = __shfl_sync(0xffffffffu, token, i);
          gam[i] = __shfl_sync(0xffffffffu, weight, i);
        }
      }
      float sum[HT];
#pragma unroll
      for (int i = 0; i < HT; ++i) sum[i] = 0.f;
      for (int kb = t.kb0; kb < t.kb1; ++kb, ++u) {
        if (!wait_done(u, DEV_TIMEOUT_EPILOGUE)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(acc * acc_cols + grp * HT);
        // the groups' scales landed with the packed rows, before the conversion that these MMAs waited for
        const uint32_t sz0 = s_sz[(2 * u % G::kWords) * kTileRows + word];
        const uint32_t sz1 = s_sz[((2 * u + 1) % G::kWords) * kTileRows + word];
        float v[HT], w[HT];
        tmem_ld16x2_wait(taddr, taddr + NT, v, w);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_tempty[acc]));
        constexpr float kUnit = G::kZeroMma ? 16777216.f : 1.f;     // the operands are integers times 2^-24
        const float s0 = kUnit * __half2float(__ushort_as_half(static_cast<unsigned short>(sz0 & 0xFFFFu)));
        const float s1 = kUnit * __half2float(__ushort_as_half(static_cast<unsigned short>(sz1 & 0xFFFFu)));
#pragma unroll
        for (int i = 0; i < HT; ++i) sum[i] = fmaf(s1, w[i], fmaf(s0, v[i], sum[i]));
        if (++acc == G::kPartials) acc = 0;
      }
      if (!ok) break;
      if (MODE == 0) {
        // even lanes hold gate values and finish the even tokens, odd lanes hold up values and finish the odd ones
        const int col = t.n0 + quad * 16 + (lane >> 1);
        float bias0 = 0.f, bias1 = 0.f;
        if (has_bias) {
          bias0 = __ldg(a.bias + static_cast<size_t>(t.e) * 2 * a.N + col);
          bias1 = __ldg(a.bias + static_cast<size_t>(t.e) * 2 * a.N + a.N + col);
        }
        float g[HT / 2], u[HT / 2];
#pragma unroll
        for (int i = 0; i < HT / 2; ++i) {
          const float other = __shfl_xor_sync(0xffffffffu, odd ? sum[2 * i] : sum[2 * i + 1], 1);
          g[i] = (odd ? other : sum[2 * i]) + bias0;
          u[i] = (odd ? sum[2 * i + 1] : other) + bias1;
        }
        act_mul_array<T, EXT>(g, u, w_on_input, mimic, ap, [&](int i) { return odd ? gam[2 * i + 1] : gam[2 * i]; });
        T* out = reinterpret_cast<T*>(a.out) + static_cast<size_t>(r0 + (odd ? 1 : 0)) * a.ld_out + col;
#pragma unroll
        for (int i = 0; i < HT / 2; ++i) out[static_cast<size_t>(2 * i) * a.ld_out] = from_f32<T>(g[i]);
      } else {
        const int col = t.n0 + row;
        const float bias0 = (has_bias && t.kb0 == 0) ? __ldg(a.bias + static_cast<size_t>(t.e) * a.N + col) : 0.f;
        float* out = reinterpret_cast<float*>(a.out) + col;
#pragma unroll
        for (int i = 0; i < HT; ++i) {
          if (orow[i] < 0) continue;
          float y = (sum[i] + bias0) * (w_on_input ? 1.0f : gam[i]);
          if (round_pair) y = to_f32<T>(from_f32<T>(y));
          atomicAdd(out + static_cast<size_t>(orow[i]) * a.ld_out, y);
        }
      }
    }
  }

  // ---- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512u);
  }
  if (threadIdx.x == 0 && *abort_flag != 0) atomicCAS(a.status, 0, *abort_flag);
}

template <int MODE, bool EXT, int NT>
int launch_w4(const CUtensorMap& tm_w, const CUtensorMap& tm_sz, const W4TokenMaps& tm_x, const GemmArgs& a, int num_sms,
              cudaStream_t stream) {
  if (cudaFuncSetAttribute(moe_gemm_w4_kernel<MODE, EXT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kSmemLimit)) != cudaSuccess)
    return B200MOE_ERR_CUDA;
  note_launch(MODE == 0 ? "moe_gemm_w4_kernel<gate/up>" : "moe_gemm_w4_kernel<down>");
  cudaError_t err = launch_kernel(moe_gemm_w4_kernel<MODE, EXT, NT>, dim3(num_sms), dim3(W4Geo<NT>::kThreads), kSmemLimit, stream,
                                  a.pdl != 0, tm_w, tm_sz, tm_x, a);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

template <int MODE, bool EXT>
int launch_mode(const CUtensorMap& tm_w, const CUtensorMap& tm_sz, const W4TokenMaps& tm_x, const GemmArgs& a, int num_sms,
                cudaStream_t stream) {
  // a field of its own decides: the tables and tensor maps are laid out for one of the variants, and a tile bound of 16 or
  // 32 tokens is not a decode block of that size
  if (a.w4_var) return launch_w4<MODE, EXT, 0>(tm_w, tm_sz, tm_x, a, num_sms, stream);
  if (a.BT == 16) return launch_w4<MODE, EXT, 16>(tm_w, tm_sz, tm_x, a, num_sms, stream);
  if (a.BT == 32) return launch_w4<MODE, EXT, 32>(tm_w, tm_sz, tm_x, a, num_sms, stream);
  return B200MOE_ERR_UNSUPPORTED;
}

}  // namespace

// The prefixes over the experts beside at least two stages of tokens.
bool gemm_w4_ok(int E) {
  return kSmemLimit - 1024 >= w4_fixed_bytes<0>(E, 1, false) + 2 * static_cast<size_t>(w4_token_bytes(kMaxGranW4 * kGranW4, 1)) &&
         kSmemLimit - 1024 >= w4_fixed_bytes<32>(E, 1, false) + 2 * static_cast<size_t>(w4_token_bytes(32, 2));
}

// Tables of a call whose GEMMs sort its P slots themselves, beside as many stages of tokens as they leave at least.
bool gemm_w4_own_ok(int E, int P, int BT) {
  const size_t fixed = BT == 16 ? w4_fixed_bytes<16>(E, 1, false, P) : w4_fixed_bytes<32>(E, 1, false, P);
  return kSmemLimit - 1024 >= fixed + 3 * static_cast<size_t>(w4_token_bytes(BT, 2));
}

// a->BT: 16 or 32 (decode blocks); with a->w4_var the upper bound of the tokens per tile
void gemm_plan_w4(GemmArgs* a) {
  const int tile_n = a->mode == 0 ? 64 : 128;
  a->num_nt = (a->N + tile_n - 1) / tile_n;
  // reduction unit: one quantisation group, two for decode blocks
  a->kblocks = a->w4_var ? a->K / 128 : (a->K + 255) / 256;
  if (a->max_split <= 0) a->max_split = 16;
}

int launch_gemm_w4(const CUtensorMap& tm_w, const CUtensorMap& tm_sz, const W4TokenMaps& tm_x, const GemmArgs& a,
                   int num_sms, cudaStream_t stream) {
  if (a.wmode != B200MOE_W_INT4_AWQ || a.dtype != B200MOE_DTYPE_FP16 || a.K % 128 != 0 || a.N % 128 != 0 || a.BT < 16)
    return B200MOE_ERR_UNSUPPORTED;
  const bool ext = a.bias != nullptr || a.activation == B200MOE_ACT_SWIGLU_OAI;
  if (a.mode == 0)
    return ext ? launch_mode<0, true>(tm_w, tm_sz, tm_x, a, num_sms, stream)
               : launch_mode<0, false>(tm_w, tm_sz, tm_x, a, num_sms, stream);
  return ext ? launch_mode<1, true>(tm_w, tm_sz, tm_x, a, num_sms, stream)
             : launch_mode<1, false>(tm_w, tm_sz, tm_x, a, num_sms, stream);
}

}  // namespace b200moe
