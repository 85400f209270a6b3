// Shared by the kernels that keep weight rows on the M side and a variable number of tokens on the N side
// (gemm_tc2.cu, gemm_w4.cu): token tiles that follow the experts' rows, and the epilogue that turns an accumulator
// (lane = weight row) into rows of the output.
#pragma once
#include "gemm_sched.cuh"

namespace b200moe {

__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
  asm volatile("red.global.v4.f32.add [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}

// ---------------------------------------------------------------- token tiles
// An expert's rows are padded to a granule and dealt out evenly over ceil(granules / max) tiles.
struct RowTile {
  int e;         // expert
  int n0;        // first weight row (mode 0: of the gate rows)
  int row0, n;   // padded rows of the tile
  int kb0, kb1;  // reduction range in stages
};
struct RowTiles {
  const int* tile;   // [E+1] token tiles before expert e
  const int* gran;   // [E+1] granules before expert e
  int E, num_nt, split, kblocks, tile_n, gran_rows;
};

// Tile `id` in expert-major, n-tile, reduction split, token tile order.
__device__ __forceinline__ RowTile row_tile_at(int id, const RowTiles& r) {
  int lo = 0, hi = r.E;
  const int u = r.num_nt * r.split;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (r.tile[mid] * u <= id) lo = mid; else hi = mid;
  }
  RowTile t;
  t.e = lo;
  const int nt_e = r.tile[lo + 1] - r.tile[lo];
  const int local = id - r.tile[lo] * u;
  const int tt = local % nt_e;
  const int rest = local / nt_e;
  const int s = rest % r.split;
  const int g = r.gran[lo + 1] - r.gran[lo];
  const int g0 = tt * g / nt_e, g1 = (tt + 1) * g / nt_e;
  t.n0 = (rest / r.split) * r.tile_n;
  t.row0 = (r.gran[lo] + g0) * r.gran_rows;
  t.n = (g1 - g0) * r.gran_rows;
  t.kb0 = 0;
  t.kb1 = r.kblocks;
  if (r.split > 1) {      // (32 bits: see decode_tile)
    t.kb0 = static_cast<int>(static_cast<unsigned>(s) * static_cast<unsigned>(r.kblocks) / static_cast<unsigned>(r.split));
    t.kb1 = static_cast<int>(static_cast<unsigned>(s + 1) * static_cast<unsigned>(r.kblocks) / static_cast<unsigned>(r.split));
  }
  return t;
}

// Estimated length of a launch that puts up to maxg granules into a tile, for choosing maxg: (sum of the tiles' costs)
// / workers + half the longest tile (a static round-robin ends that much later than a perfect split on average).
// Wide tiles re-read the weights least; narrower ones fill the last wave of a launch with few tiles.  cost(g): one
// stage of a tile with g granules.  Called by a whole warp; the result is in every lane.
template <typename Cost>
__device__ __forceinline__ float rate_max_granules(int maxg, const int* s_gran, int E, int num_nt, int workers, int lane,
                                                   Cost cost) {
  float sum = 0.f, longest = 0.f;
  for (int e = lane; e < E; e += 32) {
    const int g = s_gran[e + 1] - s_gran[e];
    if (g > 0) {
      const int t = (g + maxg - 1) / maxg;
      const int lo = g / t, rem = g - lo * t;
      sum += (t - rem) * cost(lo) + rem * cost(lo + 1);
      longest = fmaxf(longest, cost(rem > 0 ? lo + 1 : lo));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    longest = fmaxf(longest, __shfl_xor_sync(0xffffffffu, longest, o));
  }
  return sum * num_nt / workers + 0.5f * longest;
}

// Prefix of the token tiles per expert (s_tile[0..E]); called by a whole warp, returns the granules of the widest tile.
__device__ __forceinline__ int plan_row_tiles(int maxg, const int* s_gran, int E, int* s_tile, int lane) {
  int run = 0, widest = 1;
  for (int e0 = 0; e0 < E; e0 += 32) {
    const int e = e0 + lane;
    const int g = e < E ? s_gran[e + 1] - s_gran[e] : 0;
    const int t = (g + maxg - 1) / maxg;
    if (t > 0) widest = max(widest, (g + t - 1) / t);
    int v = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (e < E) s_tile[e + 1] = run + v;
    run += __shfl_sync(0xffffffffu, v, 31);
  }
  if (lane == 0) s_tile[0] = 0;
  return __reduce_max_sync(0xffffffffu, widest);
}

// ---------------------------------------------------------------- turning epilogue
// Two groups of four warps take turns at steps of 16 tokens.  A step is turned in shared memory (two buffers per
// group) and stored with 16 bytes of one token per thread.
//   mode 0: gate and up rows alternate over the lanes, 64 activations per token and CTA
//   mode 1: 128 output columns per token and CTA: 16-bit pair rows, or fp32 sums added to the combine buffer
constexpr int kTurnTok = 16;
constexpr int kTurnMaxTok = 256;     // tokens per tile that the token tables hold

// Bytes per token in a turning buffer: 64 activations, 128 pair-row values (both 16-bit) or 128 fp32 sums, and
// a pad that keeps the rows 16-byte aligned and spreads them over the banks.
__host__ __device__ __forceinline__ int turn_pitch(int mode, bool pairs) { return mode == 0 ? 160 : (pairs ? 272 : 528); }
__host__ __device__ __forceinline__ size_t turn_bytes(int mode, bool pairs) {
  return 4 * kTurnTok * static_cast<size_t>(turn_pitch(mode, pairs));
}
constexpr size_t kTurnTableBytes = 2 * 2 * kTurnMaxTok * 8;    // [2 groups][2 tiles][256] slot and weight

template <int MODE, typename T, bool EXT>
struct TurnEpilogue {
  const GemmArgs& a;
  uint8_t* turn;            // [2 groups][2][16 tokens][pitch]
  int* slot_tab;            // [2 groups][2][256]
  float* gam_tab;           // [2 groups][2][256]
  uint32_t meet;            // barrier of this thread's group (four warps)
  volatile int* abort_flag;
  int grp, quad, gt, lane;  // group, TMEM lane quadrant of the warp, thread inside the group
  int cta_col;              // first column of this CTA inside the tile
  int pitch;
  bool w_on_input, mimic, round_pair, has_bias;
  ActParams ap;
  uint32_t meet_phase;
  int par, step_no;

  __device__ __forceinline__ TurnEpilogue(const GemmArgs& args, uint8_t* s_turn, int* s_slot, float* s_gam, uint64_t* bar_meet,
                                          volatile int* abort, int ewarp, int warp, int lane_, int cta_col_, int split)
      : a(args), turn(s_turn), slot_tab(s_slot), gam_tab(s_gam), abort_flag(abort), grp(ewarp >> 2), quad(warp & 3),
        gt((ewarp & 3) * 32 + lane_), lane(lane_), cta_col(cta_col_), pitch(turn_pitch(MODE, args.out_pairs != nullptr)),
        w_on_input((args.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0),
        mimic((args.flags & B200MOE_FLAG_MIMIC_ROUNDING) != 0),
        round_pair((args.flags & B200MOE_FLAG_MIMIC_ROUNDING) != 0 && split == 1), has_bias(EXT && args.bias != nullptr),
        ap(act_params(args)), meet_phase(0), par(0), step_no(0) {
    meet = smem_u32(&bar_meet[grp]);
  }
  __device__ __forceinline__ bool meets() { return warps_meet(meet, meet_phase, lane, abort_flag, DEV_TIMEOUT_EPILOGUE); }

  // The tile's slots and routing weights; before the wait for its accumulator.
  __device__ __forceinline__ bool load_tables(const RowTile& t) {
    if (MODE == 0 && !w_on_input) return true;
    int* slots = slot_tab + (grp * 2 + par) * kTurnMaxTok;
    float* gams = gam_tab + (grp * 2 + par) * kTurnMaxTok;
    for (int i = gt; i < t.n; i += 128) {
      const int slot = a.sorted_ids[t.row0 + i];
      const bool valid = slot >= 0 && slot < a.P;
      slots[i] = valid ? slot : -1;
      gams[i] = valid ? a.row_gamma[t.row0 + i] : 0.f;
    }
    return meets();      // they are read before a step's meeting
  }

  // taddr: first column of the accumulator in this warp's lanes; release() is called by every warp once it
  // has read its last part of it.
  template <typename Release>
  __device__ __forceinline__ bool run(const RowTile& t, uint32_t taddr, Release release) {
    const int* slots = slot_tab + (grp * 2 + par) * kTurnMaxTok;
    const float* gams = gam_tab + (grp * 2 + par) * kTurnMaxTok;
    par ^= 1;
    const int steps = t.n / kTurnTok;
    // mode 0: output column of this lane pair; mode 1: of this lane
    const int lcol = cta_col + ((MODE == 0) ? quad * 16 + (lane >> 1) : quad * 32 + lane);
    float bias0 = 0.f, bias1 = 0.f;
    if (has_bias && t.n0 + lcol < a.N) {
      if (MODE == 0) {
        bias0 = __ldg(a.bias + static_cast<size_t>(t.e) * 2 * a.N + t.n0 + lcol);
        bias1 = __ldg(a.bias + static_cast<size_t>(t.e) * 2 * a.N + a.N + t.n0 + lcol);
      } else if (t.kb0 == 0) {      // the first reduction split carries the bias
        bias0 = __ldg(a.bias + static_cast<size_t>(t.e) * a.N + t.n0 + lcol);
      }
    }
    if (grp >= steps) {
      release();
      return true;
    }
    for (int st = grp; st < steps; st += 2, ++step_no) {
      float v[16];
      tmem_ld16_wait(taddr + st * kTurnTok, v);
      if (st + 2 >= steps) release();
      uint8_t* buf = turn + static_cast<size_t>((grp * 2 + (step_no & 1)) * kTurnTok) * pitch;
      if (MODE == 0) {
        // even lanes hold gate values and finish the even tokens, odd lanes hold up values and finish the odd ones
        const bool odd = (lane & 1) != 0;
        float g[8], u[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float other = __shfl_xor_sync(0xffffffffu, odd ? v[2 * j] : v[2 * j + 1], 1);
          g[j] = (odd ? other : v[2 * j]) + bias0;
          u[j] = (odd ? v[2 * j + 1] : other) + bias1;
        }
        act_mul_array<T, EXT>(g, u, w_on_input, mimic, ap, [&](int j) { return gams[st * kTurnTok + 2 * j + (odd ? 1 : 0)]; });
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<T*>(buf + (2 * j + (odd ? 1 : 0)) * pitch + (quad * 16 + (lane >> 1)) * 2) = from_f32<T>(g[j]);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float scale = w_on_input ? 1.0f : gams[st * kTurnTok + j];
          v[j] = (v[j] + bias0) * scale;
        }
        if (a.out_pairs != nullptr) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            *reinterpret_cast<T*>(buf + j * pitch + (quad * 32 + lane) * 2) = from_f32<T>(v[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            *reinterpret_cast<float*>(buf + j * pitch + (quad * 32 + lane) * 4) =
                round_pair ? to_f32<T>(from_f32<T>(v[j])) : v[j];
        }
      }
      // one meeting per step: a warp that writes this buffer again, two steps on, has met the others
      // once more in between, after they had finished reading it
      if (!meets()) return false;
      if (MODE == 0) {
        const int tk = gt >> 3, ch = gt & 7;        // 16 tokens x 8 chunks of 16 bytes
        const int col = t.n0 + cta_col + ch * 8;
        if (col < a.N)
          *reinterpret_cast<uint4*>(reinterpret_cast<T*>(a.out) +
                                    static_cast<size_t>(t.row0 + st * kTurnTok + tk) * a.ld_out + col) =
              *reinterpret_cast<const uint4*>(buf + tk * pitch + ch * 16);
      } else if (a.out_pairs != nullptr) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int tk = q * 8 + (gt >> 4), ch = gt & 15;     // 16 tokens x 16 chunks
          const int slot = slots[st * kTurnTok + tk];
          const int col = t.n0 + cta_col + ch * 8;
          if (slot >= 0 && col < a.N) {
            *reinterpret_cast<uint4*>(reinterpret_cast<T*>(a.out_pairs) + static_cast<size_t>(slot) * a.N + col) =
                *reinterpret_cast<const uint4*>(buf + tk * pitch + ch * 16);
            if (col == 0) a.pair_valid[slot] = 1;
          }
        }
      } else {
        const int col = t.n0 + cta_col + lane * 4;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int tk = q * 4 + (gt >> 5);
          const int slot = slots[st * kTurnTok + tk];
          if (slot < 0 || col >= a.N) continue;
          const float4 y = *reinterpret_cast<const float4*>(buf + tk * pitch + lane * 16);
          red_add_v4(reinterpret_cast<float*>(a.out) + static_cast<size_t>(slot / a.topk) * a.ld_out + col, y.x, y.y, y.z, y.w);
        }
      }
    }
    return true;
  }
};

}  // namespace b200moe
