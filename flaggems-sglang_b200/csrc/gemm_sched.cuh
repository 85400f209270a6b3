// Tile scheduler shared by the grouped GEMM kernels: constants of the pipeline, the split
// of the work into (expert, token block, n-tile, k-split) units and the decode of a unit id.
#pragma once
#include "gemm.cuh"

namespace b200moe {

constexpr int kTileRows = 128;           // weight rows per MMA (the instruction's M)
constexpr int kStageKBytes = 128;        // bytes of the reduction dim per stage row (one swizzle atom)
constexpr int kTileBytes = kTileRows * kStageKBytes;  // 16 KiB
constexpr int kMaxBT = 256;
// 227 KiB.  A kernel is always allowed the same amount, whatever a call needs: the setting is shared by all host threads,
// and one that lowered it would make another thread's launch fail.
constexpr size_t kSmemLimit = 232448;

struct Ctrl {
  int nblocks;
  int units_per_block;  // num_nt (* split)
  int split;
  int total;
  int grid_eff;
};

// Called by whole warps.  A lane rates one split; with the rates one after the other the two divisions of each stood in the
// way of a launch's first loads for 2 us (reductions of 224 steps, up to 16 splits).
__device__ __forceinline__ int pick_split(int tiles, int kblocks, int grid, int max_split) {
  const int smax = min(max_split, max(1, kblocks / 4));
  int best = 1;
  float best_eff = -1.f;
  for (int s0 = 1; s0 <= smax; s0 += 32) {
    const int total = tiles * (s0 + static_cast<int>(threadIdx.x & 31));
    const int waves = (total + grid - 1) / grid;
    const float eff = static_cast<float>(total) / static_cast<float>(waves * grid);
    for (int i = 0; i < 32 && s0 + i <= smax; ++i) {
      const float e = __shfl_sync(0xffffffffu, eff, i);
      if (e > best_eff + 0.04f) {
        best_eff = e;
        best = s0 + i;
      }
    }
  }
  return best;
}

struct TileCoord {
  int e;      // expert
  int row0;   // first padded row of the token block
  int n0;     // first weight row inside the expert
  int kb0, kb1;  // k-block range
};

__device__ __forceinline__ TileCoord decode_tile(int id, const Ctrl& c, const int* s_blk_off, int E,
                                                 int BT, int num_nt, int kblocks, int tile_n) {
  // largest e with blk_off[e] * units <= id
  int lo = 0, hi = E;
  const int u = c.units_per_block;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (s_blk_off[mid] * u <= id) lo = mid; else hi = mid;
  }
  TileCoord t;
  t.e = lo;
  const int first = s_blk_off[lo];
  const int nb = s_blk_off[lo + 1] - first;
  const int local = id - first * u;
  const int b = local % nb;
  const int rest = local / nb;
  const int s = rest % c.split;
  const int nt = rest / c.split;
  t.row0 = (first + b) * BT;
  t.n0 = nt * tile_n;
  t.kb0 = 0;
  t.kb1 = kblocks;
  if (c.split > 1) {      // (32 bits: the reduction has at most 2^20 steps, the split is at most 1024)
    t.kb0 = static_cast<int>(static_cast<unsigned>(s) * static_cast<unsigned>(kblocks) / static_cast<unsigned>(c.split));
    t.kb1 = static_cast<int>(static_cast<unsigned>(s + 1) * static_cast<unsigned>(kblocks) / static_cast<unsigned>(c.split));
  }
  return t;
}

// Fused tail of the gate/up projection.
//   SiLU / GELU (the reference's plain op, fused_moe.py:198-206): optional routing weight on the
//   two projections, optional rounding of both to the 16-bit type (as the reference stores
//   them), activation(gate) * up.
//   B200MOE_ACT_SWIGLU_OAI (the reference's bias variant fuses its dependency's swiglu into
//   GEMM-1, fused_moe.py:258-298): gate clamped from above, linear clamped to [-limit, limit],
//   s = g / (1 + exp(-alpha * g)), result s * (linear + 1); the routing weight, if it goes on
//   the input side, multiplies the result.
struct ActParams {
  int activation;
  float alpha, limit;
};
// EXT = false compiles the SiLU / GELU tail only: the epilogues are bound by their instruction
// count, so the plain kernels must not carry the extra tests.
template <typename T, bool EXT = false>
__device__ __forceinline__ float act_mul(float g, float u, bool w_on_input, float gam, bool mimic,
                                         const ActParams& p) {
  if (EXT && p.activation == B200MOE_ACT_SWIGLU_OAI) {
    if (p.limit > 0.f) {
      g = fminf(g, p.limit);
      u = fminf(fmaxf(u, -p.limit), p.limit);
    }
    const float s = __fdividef(g, 1.0f + __expf(-p.alpha * g));
    const float r = fmaf(s, u, s);
    return w_on_input ? r * gam : r;
  }
  if (w_on_input) {
    g *= gam;
    u *= gam;
  }
  if (mimic) {
    g = to_f32<T>(from_f32<T>(g));
    u = to_f32<T>(from_f32<T>(u));
  }
  const float s = (p.activation == B200MOE_ACT_SILU) ? __fdividef(g, 1.0f + __expf(-g)) : gelu_f32(g);
  return s * u;
}
// The same tail over an array, results in g.  Every test is outside the loops: with a branch per element
// the exponential and the division of one element could not overlap those of the next, and that latency
// set the pace of the epilogues (1400 cycles for eight elements of a thread in the pair kernel).
// gam(i) is the routing weight of element i; it is only called where the weight goes on the input.
template <typename T, bool EXT, int N, typename Gam>
__device__ __forceinline__ void act_mul_array(float (&g)[N], const float (&u0)[N], bool w_on_input, bool mimic,
                                              const ActParams& p, Gam gam) {
  if (EXT && p.activation == B200MOE_ACT_SWIGLU_OAI) {
#pragma unroll
    for (int i = 0; i < N; ++i) g[i] = act_mul<T, EXT>(g[i], u0[i], false, 1.f, false, p);
    if (w_on_input) {
#pragma unroll
      for (int i = 0; i < N; ++i) g[i] *= gam(i);
    }
    return;
  }
  float u[N];
#pragma unroll
  for (int i = 0; i < N; ++i) u[i] = u0[i];
  if (w_on_input) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float w = gam(i);
      g[i] *= w;
      u[i] *= w;
    }
  }
  if (mimic) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      g[i] = to_f32<T>(from_f32<T>(g[i]));
      u[i] = to_f32<T>(from_f32<T>(u[i]));
    }
  }
  if (p.activation == B200MOE_ACT_SILU) {
#pragma unroll
    for (int i = 0; i < N; ++i) g[i] = __fdividef(g[i], 1.0f + __expf(-g[i])) * u[i];
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) g[i] = gelu_f32(g[i]) * u[i];
  }
}
__device__ __forceinline__ ActParams act_params(const GemmArgs& a) {
  ActParams p;
  p.activation = a.activation;
  p.alpha = a.act_alpha;
  p.limit = a.act_limit;
  return p;
}

// `nblocks` blocks of `units` tiles each over `ctas` CTAs, evenly: with w waves, ceil(total / w) CTAs do w tiles each.
__device__ __forceinline__ Ctrl spread_tiles(int nblocks, int units, int split, int ctas, int flags) {
  Ctrl c;
  c.nblocks = nblocks;
  c.split = split;
  c.units_per_block = units;
  c.total = nblocks * units;
  const int waves = ctas > 0 ? (c.total + ctas - 1) / ctas : 0;
  c.grid_eff = waves > 0 ? (c.total + waves - 1) / waves : 1;
  if (flags & B200MOE_FLAG_NO_GRID_BALANCE) c.grid_eff = ctas;
  return c;
}

// Work decomposition for one launch; identical in every thread of every CTA.
__device__ __forceinline__ Ctrl make_ctrl(const GemmArgs& a, int nblocks, bool may_split) {
  int split = 1;
  if (may_split && !(a.flags & B200MOE_FLAG_NO_SPLIT_K)) split = pick_split(nblocks * a.num_nt, a.kblocks, gridDim.x, a.max_split);
  return spread_tiles(nblocks, a.num_nt * split, split, gridDim.x, a.flags);
}

}  // namespace b200moe
