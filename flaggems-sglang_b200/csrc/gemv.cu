// Matrix-vector kernels for calls with a handful of (token, choice) pairs: see gemv.cuh.
#include "gemm_sched.cuh"
#include "gemv.cuh"

namespace b200moe {
namespace {

constexpr int kUpThreads = 256;     // 8 warps, one output column (gate row + up row) per warp at a time
constexpr int kDownThreads = 512;   // 16 warps, two output elements per warp at a time
constexpr int kChunk = 256;         // elements of one warp-wide 16-byte load

// streaming 16-byte load: the weights are read once, keep them out of L1
__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p));
  return v;
}

template <typename T>
__device__ __forceinline__ void unpack2(uint32_t w, float& lo, float& hi);
template <>
__device__ __forceinline__ void unpack2<__nv_bfloat16>(uint32_t w, float& lo, float& hi) {
  lo = __uint_as_float(w << 16);
  hi = __uint_as_float(w & 0xffff0000u);
}
template <>
__device__ __forceinline__ void unpack2<__half>(uint32_t w, float& lo, float& hi) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  lo = f.x;
  hi = f.y;
}

// Token rows and activations are staged in shared memory as fp32 in two planes: elements 0..3 of
// every run of eight in the first half of the row, elements 4..7 in the second.  A lane that holds
// eight consecutive weights (one 16-byte load) then reads two float4 whose addresses are
// consecutive across the lanes of the warp: no bank conflicts.
__device__ __forceinline__ int plane_index(int k, int n) {
  return ((k >> 2) & 1) * (n >> 1) + ((k >> 3) << 2) + (k & 3);
}

// acc + sum of eight 16-bit weights (elements k .. k+7, k a multiple of 8) times the staged row
template <typename T>
__device__ __forceinline__ float dot8(const uint4& w, const float* row, int k, int n, float acc) {
  const float4 x0 = *reinterpret_cast<const float4*>(row + (k >> 1));
  const float4 x1 = *reinterpret_cast<const float4*>(row + (n >> 1) + (k >> 1));
  float a, b;
  unpack2<T>(w.x, a, b);
  acc = fmaf(a, x0.x, acc);
  acc = fmaf(b, x0.y, acc);
  unpack2<T>(w.y, a, b);
  acc = fmaf(a, x0.z, acc);
  acc = fmaf(b, x0.w, acc);
  unpack2<T>(w.z, a, b);
  acc = fmaf(a, x1.x, acc);
  acc = fmaf(b, x1.y, acc);
  unpack2<T>(w.w, a, b);
  acc = fmaf(a, x1.z, acc);
  acc = fmaf(b, x1.w, acc);
  return acc;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename T>
__device__ __forceinline__ void load4_f32(const T* p, float (&v)[4]) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  unpack2<T>(raw.x, v[0], v[1]);
  unpack2<T>(raw.y, v[2], v[3]);
}

// A warp: the lane of an expert places its run of sorted rows; 128 experts' counts are fetched at a time.  (Each thread walking
// the counts by itself, both launches of one token from a graph: 128 experts of 2048 x 768 34.7 us against 23.1, 256 of
// 512 x 256 36.3 against 13.1.)
__device__ __forceinline__ void place_sorted_rows(const int* hist, const int* topk_indx, const float* gate_scal, int P, int E,
                                                  int* s_e, float* s_gam) {
  const int lane = threadIdx.x & 31;
  int run = 0;
  for (int e0 = lane; e0 - lane < E; e0 += 128) {
    int n[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) n[u] = e0 + 32 * u < E ? max(0, min(P, __ldcg(hist + e0 + 32 * u))) : 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (e0 - lane + 32 * u >= E) break;
      int end = n[u];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += v;
      }
      for (int q = run + end - n[u]; q < min(P, run + end); ++q) {
        const int slot = __ldcg(topk_indx + q);
        if (slot >= 0 && slot < P) {
          s_e[slot] = e0 + 32 * u;
          s_gam[slot] = __ldcg(gate_scal + q);
        }
      }
      __syncwarp();
      run += __shfl_sync(0xffffffffu, end, 31);
    }
  }
}

// Local expert and routing weight of every pair, into shared memory (P <= kGemvMaxPairs).  From
// topk_ids / topk_weights (with an optional global -> local map), or from the routing triple
// hist[E] / topk_indx[P] / gate_scal[P] (sorted row -> pair slot, weights in sorted order).
// Called by every thread of the CTA; the caller synchronises before reading the tables.
// The down kernels call it before they wait for the up kernel: the routing input was complete before that one started, but
// the reads go to L2, as those of gemm_route.cuh do, so that no line an earlier kernel left in this SM's L1 is taken for it.
// TRIPLE: the kernel is also launched with a routing triple.
template <bool TRIPLE = true>
__device__ __forceinline__ void stage_routing(const GemvArgs& a, int* s_e, float* s_gam) {
  const int P = a.M * a.topk;
  const int p = threadIdx.x;
  if (!TRIPLE || a.hist == nullptr) {
    if (p < P) {
      long long id = a.ids_i64 ? __ldcg(reinterpret_cast<const long long*>(a.topk_ids) + p)
                               : static_cast<long long>(__ldcg(reinterpret_cast<const int*>(a.topk_ids) + p));
      if (a.expert_map != nullptr) id = (id >= 0 && id < a.n_global) ? __ldcg(a.expert_map + id) : -1;
      s_e[p] = (id >= 0 && id < a.E) ? static_cast<int>(id) : -1;
      s_gam[p] = __ldcg(a.topk_w + p);
    }
    return;
  }
  if (p < P) s_e[p] = -1;
  __syncthreads();
  if (threadIdx.x < 32) place_sorted_rows(a.hist, a.topk_indx, a.gate_scal, P, a.E, s_e, s_gam);
}

// ------------------------------------------------------------------------------------------
// act[p][i] = activation(w1[e_p][i] . x_t, w1[e_p][I + i] . x_t) in the 16-bit type
// U: 256-element chunks of each row that a lane keeps in flight.  4 by default (8 halves the resident
// CTAs and measured 10 % slower); 5 or 6 when that is the whole row, so that a row of 1280 or 1536
// elements does not need a second, nearly empty pass.
// U = 2 where its six CTAs an SM give every column a warp of its own in one wave and three would not (launch_gemv_up); from ids
// only, since 40 registers a thread leave none for the placing of a triple's rows.
template <typename T, int U>
__global__ void __launch_bounds__(kUpThreads, U == 2 ? 6 : 1)
moe_gemv_up_kernel(const GemvArgs a) {
  extern __shared__ __align__(16) uint8_t gemv_smem[];
  const int P = a.M * a.topk;
  float* s_x = reinterpret_cast<float*>(gemv_smem);                 // [M][H], two planes per row
  int* s_e = reinterpret_cast<int*>(s_x + static_cast<size_t>(a.M) * a.H);
  float* s_gam = reinterpret_cast<float*>(s_e + kGemvMaxPairs);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  griddep_wait();
  griddep_launch_dependents();
  stage_routing<U != 2>(a, s_e, s_gam);
  const T* x = reinterpret_cast<const T*>(a.x);
  const int quads = a.H >> 2;
  for (int i = threadIdx.x; i < a.M * quads; i += kUpThreads) {
    const int t = i / quads, k = (i - t * quads) << 2;
    float v[4];
    load4_f32<T>(x + static_cast<size_t>(t) * a.H + k, v);
    *reinterpret_cast<float4*>(s_x + static_cast<size_t>(t) * a.H + plane_index(k, a.H)) =
        make_float4(v[0], v[1], v[2], v[3]);
  }
  __syncthreads();

  const bool w_on_input = (a.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0;
  const bool mimic = (a.flags & B200MOE_FLAG_MIMIC_ROUNDING) != 0;
  const bool ext = a.b1 != nullptr || a.activation == B200MOE_ACT_SWIGLU_OAI;
  ActParams ap;
  ap.activation = a.activation;
  ap.alpha = a.alpha;
  ap.limit = a.limit;
  T* act = reinterpret_cast<T*>(a.act);
  const T* w1 = reinterpret_cast<const T*>(a.w1);

  const int total = P * a.I;
  const int warps = gridDim.x * (kUpThreads / 32);
  // consecutive columns go to different SMs, so every SM streams the same share
  for (int c = warp * gridDim.x + blockIdx.x; c < total; c += warps) {
    const int p = c / a.I, i = c - p * a.I;
    const int e = s_e[p];
    if (e < 0) {
      if (lane == 0) act[c] = from_f32<T>(0.f);
      continue;
    }
    const float* xs = s_x + static_cast<size_t>(p / a.topk) * a.H;
    const T* wg = w1 + (static_cast<size_t>(e) * 2 * a.I + i) * a.H;
    const T* wu = wg + static_cast<size_t>(a.I) * a.H;
    float ag = 0.f, au = 0.f;
    for (int k0 = lane * 8; k0 < a.H; k0 += U * kChunk) {
      uint4 gq[U], uq[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int k = k0 + q * kChunk;
        if (k < a.H) {
          gq[q] = ldg_stream(wg + k);
          uq[q] = ldg_stream(wu + k);
        }
      }
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int k = k0 + q * kChunk;
        if (k < a.H) {
          ag = dot8<T>(gq[q], xs, k, a.H, ag);
          au = dot8<T>(uq[q], xs, k, a.H, au);
        }
      }
    }
    ag = warp_sum(ag);
    au = warp_sum(au);
    if (lane == 0) {
      if (a.b1 != nullptr) {
        ag += __ldg(a.b1 + static_cast<size_t>(e) * 2 * a.I + i);
        au += __ldg(a.b1 + static_cast<size_t>(e) * 2 * a.I + a.I + i);
      }
      const float av = ext ? act_mul<T, true>(ag, au, w_on_input, s_gam[p], mimic, ap)
                           : act_mul<T>(ag, au, w_on_input, s_gam[p], mimic, ap);
      act[c] = from_f32<T>(av);
    }
  }
}

// ------------------------------------------------------------------------------------------
// out[t][h] = cast(routed_scaling * sum_j gamma_j * (w2[e_j][h] . act[p_j] + b2[e_j][h]))
// One warp per pair of output elements (h, h + 1) of a token: the two weight rows share every read
// of the staged activations.
template <typename T>
__global__ void __launch_bounds__(kDownThreads)
moe_gemv_down_kernel(const GemvArgs a) {
  extern __shared__ __align__(16) uint8_t gemv_smem[];
  const int P = a.M * a.topk;
  float* s_act = reinterpret_cast<float*>(gemv_smem);               // [P][I], two planes per row
  int* s_e = reinterpret_cast<int*>(s_act + static_cast<size_t>(P) * a.I);
  float* s_gam = reinterpret_cast<float*>(s_e + kGemvMaxPairs);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool w_on_input = (a.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0;
  const bool no_combine = (a.flags & B200MOE_FLAG_NO_COMBINE) != 0;
  // per-pair results are needed one by one when each is rounded or stored by itself; otherwise the
  // routing weight is folded into the staged activations and one running sum covers all pairs
  const bool by_pair = no_combine || a.round_pair != 0;

  const T* w2 = reinterpret_cast<const T*>(a.w2);
  const int nch = (a.I + kChunk - 1) / kChunk;
  T* out = reinterpret_cast<T*>(a.out);
  const int half_h = a.H >> 1;
  const int tasks = a.M * half_h;
  // With fewer tasks than warps, S = a.down_split warps share a task: each takes a contiguous share
  // of the (pair, chunk) slots, the partial sums meet in shared memory and are added in a fixed order.
  const int S = by_pair ? 1 : a.down_split;
  const int grp = warp / S, sub = warp - grp * S;
  const int groups = gridDim.x * ((kDownThreads / 32) / S);
  const int Q = a.topk * nch;
  const int share = (Q + S - 1) / S;
  const int q_lo = sub * share, q_hi = min(Q, q_lo + share);
  float* s_part = s_gam + kGemvMaxPairs;                            // [2 buffers][16 warps][2]

  // a run: eight (pair, chunk) slots of two rows, 16 loads of 16 bytes in flight per lane
  struct Run {
    uint4 wa[8], wb[8];
    int kk[8], pp[8];
  };
  auto load_run = [&](Run& r, int t, int h, int q0, int& j, int& ch) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int p = t * a.topk + j;
      const int k = ch * kChunk + lane * 8;
      const int e = (q0 + u < q_hi) ? s_e[p] : -1;
      const bool on = e >= 0 && k < a.I;
      r.kk[u] = on ? k : -1;
      r.pp[u] = p;
      if (on) {
        const T* wr = w2 + (static_cast<size_t>(e) * a.H + h) * a.I + k;
        r.wa[u] = ldg_stream(wr);
        r.wb[u] = ldg_stream(wr + a.I);
      }
      if (++ch == nch) {
        ch = 0;
        ++j;
      }
    }
  };

  // The routing tables and the weights do not depend on the up kernel: they are read before waiting
  // for it, and when the layer is small (several warps per task: the kernel is a few memory round
  // trips long) the first run of this warp's first task is put in flight as well.  With one warp per
  // task the early loads only take bandwidth from the up kernel's tail (Mixtral-shaped layer at M = 1:
  // 127 us with, 123 us without).
  stage_routing(a, s_e, s_gam);
  __syncthreads();
  Run r;                       // one register buffer: the prefetched run is consumed in place
  const int task0 = grp * gridDim.x + blockIdx.x;
  bool have_pre = false;
  int pre_j = 0, pre_ch = 0;
  if (!by_pair && S > 1 && task0 < tasks && q_lo < q_hi) {
    const int t = task0 / half_h, h = (task0 - t * half_h) << 1;
    pre_j = q_lo / nch;
    pre_ch = q_lo - pre_j * nch;
    load_run(r, t, h, q_lo, pre_j, pre_ch);
    have_pre = true;
  }
  griddep_wait();
  griddep_launch_dependents();
  const T* act = reinterpret_cast<const T*>(a.act);
  const int quads = a.I >> 2;
  for (int i = threadIdx.x; i < P * quads; i += kDownThreads) {
    const int p = i / quads, k = (i - p * quads) << 2;
    const float fold = (by_pair || w_on_input) ? 1.0f : s_gam[p];
    float v[4];
    load4_f32<T>(act + static_cast<size_t>(p) * a.I + k, v);
    *reinterpret_cast<float4*>(s_act + static_cast<size_t>(p) * a.I + plane_index(k, a.I)) =
        make_float4(v[0] * fold, v[1] * fold, v[2] * fold, v[3] * fold);
  }
  __syncthreads();

  int iter = 0;
  for (int task = task0; task < tasks; task += groups, ++iter) {
    const int t = task / half_h, h = (task - t * half_h) << 1;
    if (!by_pair) {
      float acc0 = 0.f, acc1 = 0.f;
      int j = q_lo / nch, ch = q_lo - j * nch;
      for (int q0 = q_lo; q0 < q_hi; q0 += 8) {
        if (have_pre) {
          j = pre_j;
          ch = pre_ch;
          have_pre = false;
        } else {
          load_run(r, t, h, q0, j, ch);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (r.kk[u] >= 0) {
            const float* av = s_act + static_cast<size_t>(r.pp[u]) * a.I;
            acc0 = dot8<T>(r.wa[u], av, r.kk[u], a.I, acc0);
            acc1 = dot8<T>(r.wb[u], av, r.kk[u], a.I, acc1);
          }
        }
      }
      acc0 = warp_sum(acc0);
      acc1 = warp_sum(acc1);
      if (S > 1) {
        float* part = s_part + (iter & 1) * 2 * (kDownThreads / 32);
        if (lane == 0) {
          part[2 * warp] = acc0;
          part[2 * warp + 1] = acc1;
        }
        named_bar_sync(1 + grp, 32 * S);   // the S warps of this task (same trip counts: no warp can be missing)
        if (sub == 0 && lane == 0) {
          acc0 = 0.f;
          acc1 = 0.f;
          for (int w = 0; w < S; ++w) {
            acc0 += part[2 * (warp + w)];
            acc1 += part[2 * (warp + w) + 1];
          }
        }
      }
      if (sub == 0 && lane == 0) {
        if (a.b2 != nullptr) {
          for (int jb = 0; jb < a.topk; ++jb) {
            const int p = t * a.topk + jb;
            if (s_e[p] >= 0) {
              const float gam = w_on_input ? 1.0f : s_gam[p];
              acc0 = fmaf(__ldg(a.b2 + static_cast<size_t>(s_e[p]) * a.H + h), gam, acc0);
              acc1 = fmaf(__ldg(a.b2 + static_cast<size_t>(s_e[p]) * a.H + h + 1), gam, acc1);
            }
          }
        }
        out[static_cast<size_t>(t) * a.H + h] = from_f32<T>(acc0 * a.routed_scaling);
        out[static_cast<size_t>(t) * a.H + h + 1] = from_f32<T>(acc1 * a.routed_scaling);
      }
    } else {
      float sum0 = 0.f, sum1 = 0.f;
      for (int jb = 0; jb < a.topk; ++jb) {
        const int p = t * a.topk + jb;
        const int e = s_e[p];
        float y0 = 0.f, y1 = 0.f;
        if (e >= 0) {
          const T* wr = w2 + (static_cast<size_t>(e) * a.H + h) * a.I;
          const float* av = s_act + static_cast<size_t>(p) * a.I;
          float acc0 = 0.f, acc1 = 0.f;
          for (int k0 = lane * 8; k0 < a.I; k0 += 4 * kChunk) {
            uint4 wa[4], wb[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (k0 + q * kChunk < a.I) {
                wa[q] = ldg_stream(wr + k0 + q * kChunk);
                wb[q] = ldg_stream(wr + a.I + k0 + q * kChunk);
              }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int k = k0 + q * kChunk;
              if (k < a.I) {
                acc0 = dot8<T>(wa[q], av, k, a.I, acc0);
                acc1 = dot8<T>(wb[q], av, k, a.I, acc1);
              }
            }
          }
          acc0 = warp_sum(acc0);
          acc1 = warp_sum(acc1);
          if (a.b2 != nullptr) {
            acc0 += __ldg(a.b2 + static_cast<size_t>(e) * a.H + h);
            acc1 += __ldg(a.b2 + static_cast<size_t>(e) * a.H + h + 1);
          }
          y0 = w_on_input ? acc0 : acc0 * s_gam[p];
          y1 = w_on_input ? acc1 : acc1 * s_gam[p];
          if (a.round_pair) {
            y0 = to_f32<T>(from_f32<T>(y0));
            y1 = to_f32<T>(from_f32<T>(y1));
          }
        }
        if (no_combine) {
          if (lane == 0) {
            out[static_cast<size_t>(p) * a.H + h] = from_f32<T>(y0);
            out[static_cast<size_t>(p) * a.H + h + 1] = from_f32<T>(y1);
          }
        } else {
          sum0 += y0;
          sum1 += y1;
        }
      }
      if (!no_combine && lane == 0) {
        out[static_cast<size_t>(t) * a.H + h] = from_f32<T>(sum0 * a.routed_scaling);
        out[static_cast<size_t>(t) * a.H + h + 1] = from_f32<T>(sum1 * a.routed_scaling);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// The same where a CTA's share of the down weights fits in shared memory (eight pairs of a 2048 x 768 layer: 14 rows of every
// pair, 172 KB).  It comes as one bulk copy per pair, issued before the wait for the up kernel, all of it in flight at once and
// without registers (the kernel above holds two thirds of it in flight, and a third round trip remains).  What is left is one
// pass over shared memory, which wants many warps: 128 / 256 / 512 threads took 24.5 / 20.4 / 19.0 us for both launches.
// From a graph, weights cold, both launches, us with the kernel above / with this one: 2048 x 768 with 1 pair 8.9 / 7.05,
// 6: 17.9 / 16.4, 8: 19.9 / 19.0; 1024 x 512 with 4 8.7 / 8.0, 8: 11.3 / 11.2; 512 x 256 with 8 14.3 / 6.6; 2048 x 384 with 16
// 34.2 / 21.6 (share_wins has the calls where the other one is ahead).
// What bounds it now: its bytes from HBM (75 MB at 2048 x 768: 11.5 us), the routing's round trip in front of the first
// loads, and the dependent launch between the two.
constexpr int kShareThreads = 512;
constexpr int kShareRows = 16;               // rows per CTA at most: one sum each in a lane's registers
constexpr size_t kShareBytes = 190 * 1024;   // leaves the up kernel three CTAs of up to 10 KB each

__host__ __device__ __forceinline__ int share_rows(int H, int ctas) { return (H + ctas - 1) / ctas; }
__host__ __device__ __forceinline__ size_t share_bytes(int P, int rows, int I) {
  return static_cast<size_t>(P) * (rows + 1) * I * 2;
}

// (a form without the routing triple: with the code that places its rows the sums' loop gets other registers, 15.3 us against
// 14.6 for 1 pair of 2048 x 4096)
template <typename T, bool TRIPLE>
__global__ void __launch_bounds__(kShareThreads)
moe_gemv_down_share_kernel(const GemvArgs a) {
  extern __shared__ __align__(128) uint8_t gemv_smem[];
  __shared__ __align__(8) uint64_t bar[kGemvMaxPairs];
  __shared__ int s_e[kGemvMaxPairs];
  __shared__ float s_gam[kGemvMaxPairs];
  __shared__ float s_val[kGemvMaxPairs][kShareRows];
  __shared__ volatile int abort_flag;
  const int P = a.M * a.topk;
  const int R = share_rows(a.H, gridDim.x);
  const int h0 = min(a.H, static_cast<int>(blockIdx.x) * R), rows = min(R, a.H - h0);
  T* s_w = reinterpret_cast<T*>(gemv_smem);                         // [P][rows][I]
  T* s_act = s_w + static_cast<size_t>(P) * rows * a.I;             // [P][I]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < kGemvMaxPairs) mbar_init(smem_u32(&bar[threadIdx.x]), 1);
  if (threadIdx.x == 0) {
    abort_flag = 0;
    fence_mbar_init();
  }
  // neither the routing input nor the weights depend on the up kernel
  stage_routing<TRIPLE>(a, s_e, s_gam);
  fence_proxy_async_smem();
  __syncthreads();
  const uint32_t bytes = static_cast<uint32_t>(rows) * a.I * 2;
  if (threadIdx.x < P && s_e[threadIdx.x] >= 0 && rows > 0) {
    const int p = threadIdx.x;
    mbar_arrive_expect_tx(smem_u32(&bar[p]), bytes);
    bulk_copy_g2s(smem_u32(s_w + static_cast<size_t>(p) * rows * a.I),
                  reinterpret_cast<const T*>(a.w2) + (static_cast<size_t>(s_e[p]) * a.H + h0) * a.I, bytes, smem_u32(&bar[p]));
  }
  griddep_wait();
  griddep_launch_dependents();
  const uint4* act = reinterpret_cast<const uint4*>(a.act);
  for (int i = threadIdx.x; i < P * a.I / 8; i += kShareThreads) reinterpret_cast<uint4*>(s_act)[i] = act[i];
  __syncthreads();
  // four rows of a pair at a time: their sums are independent, and one exchange adds all four over the lanes
  bool ok = true;
  const int groups = (rows + 3) / 4;
  for (int u = warp; u < P * groups; u += kShareThreads / 32) {
    const int p = u / groups, r0 = (u - p * groups) * 4;
    if (s_e[p] < 0) continue;                  // nothing reads its sums
    if (!mbar_wait(smem_u32(&bar[p]), 0, &abort_flag, DEV_TIMEOUT_PRODUCER)) {
      ok = false;
      break;
    }
    const T* w[4];
    float acc[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      w[r] = s_w + (static_cast<size_t>(p) * rows + min(r0 + r, rows - 1)) * a.I;
      acc[r] = 0.f;
    }
#pragma unroll 2
    for (int k = lane * 8; k < a.I; k += kChunk) {
      const uint4 av = *reinterpret_cast<const uint4*>(s_act + static_cast<size_t>(p) * a.I + k);
      float x[8];
      unpack2<T>(av.x, x[0], x[1]);
      unpack2<T>(av.y, x[2], x[3]);
      unpack2<T>(av.z, x[4], x[5]);
      unpack2<T>(av.w, x[6], x[7]);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint4 wv = *reinterpret_cast<const uint4*>(w[r] + k);
        const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float lo, hi;
          unpack2<T>(ww[q], lo, hi);
          acc[r] = fmaf(hi, x[2 * q + 1], fmaf(lo, x[2 * q], acc[r]));
        }
      }
    }
    // lanes 0-7 end with row 0, 8-15 with row 1, and so on
    const bool up16 = (lane & 16) != 0, up8 = (lane & 8) != 0;
    const float c0 = (up16 ? acc[2] : acc[0]) + __shfl_xor_sync(0xffffffffu, up16 ? acc[0] : acc[2], 16);
    const float c1 = (up16 ? acc[3] : acc[1]) + __shfl_xor_sync(0xffffffffu, up16 ? acc[1] : acc[3], 16);
    float v = (up8 ? c1 : c0) + __shfl_xor_sync(0xffffffffu, up8 ? c0 : c1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int r = r0 + (lane >> 3);
    if ((lane & 7) == 0 && r < rows) s_val[p][r] = v;
  }
  if (!ok && lane == 0) {
    atomicCAS(a.status, 0, static_cast<int>(abort_flag));
    // no thread leaves before the barrier below: the copies in flight land first
    for (int p = 0; p < P; ++p)
      if (s_e[p] >= 0) mbar_wait_brief(smem_u32(&bar[p]), 0);
  }
  __syncthreads();
  // a thread adds a token's pairs for one row, in their order
  const bool w_on_input = (a.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0, no_combine = (a.flags & B200MOE_FLAG_NO_COMBINE) != 0;
  T* out = reinterpret_cast<T*>(a.out);
  for (int i = threadIdx.x; i < a.M * rows; i += kShareThreads) {
    const int t = i / rows, r = i - t * rows, h = h0 + r;
    float sum = 0.f;
    for (int j = 0; j < a.topk; ++j) {
      const int p = t * a.topk + j, e = s_e[p];
      float y = 0.f;
      if (e >= 0) {
        y = s_val[p][r];
        if (a.b2 != nullptr) y += __ldg(a.b2 + static_cast<size_t>(e) * a.H + h);
        if (!w_on_input) y *= s_gam[p];
        if (a.round_pair) y = to_f32<T>(from_f32<T>(y));
      }
      if (no_combine) out[static_cast<size_t>(p) * a.H + h] = from_f32<T>(y);
      sum += y;
    }
    if (!no_combine) out[static_cast<size_t>(t) * a.H + h] = from_f32<T>(sum * a.routed_scaling);
  }
}

// ==========================================================================================
// int4 (AWQ) weights: the same two launches on integer dot products.
//
// The activations become integers: per 128-k group
// a power-of-two scale f = 2^(e-18) for a group maximum in [2^e, 2^(e+1)) and the exact integers
// v = rint(x / f), |v| < 2^19, as three signed byte planes v = p0 + 256 p1 + 65536 p2.  A packed
// word holds eight weights; `w & 0x0F0F0F0F` and `(w >> 4) & 0x0F0F0F0F` are their raw nibbles as
// unsigned bytes in the order (0, 4, 1, 5) and (2, 6, 3, 7), the planes are staged in that order,
// and one dp4a per plane and half word gives exact sums S = S0 + 256 S1 + 65536 S2.  Per 32-k
// segment (one 16-byte load of a lane, inside one quantisation group):
// acc += (s f) * float(S - z * sum(v)), s and z the group's scale and zero point of the row.
// One instruction per weight instead of a conversion and a multiply-add for each.

__device__ __forceinline__ int dp4a_u8_s8(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// A row of K staged bytes per plane is kept in two halves: bytes 0..15 of every run of 32 in the
// first, bytes 16..31 in the second, so that the two 16-byte reads of a lane (its 32 k) are
// contiguous across the warp.
__device__ __forceinline__ int half_index(int o, int K) { return ((o >> 4) & 1) * (K >> 1) + ((o >> 5) << 4) + (o & 15); }

struct StagedW4 {
  uint8_t* planes;   // [rows][3][K]
  float* f;          // [rows][K / 128] group scale (routing weight folded in where asked)
  int* vsum;         // [rows][K / 32] sum of the integers of every 32-k segment
};

// fp16 rows -> planes, scales and segment sums; one warp per (row, group).  fold[row] multiplies the stored scale (nullptr: 1).
__device__ __forceinline__ void stage_w4(const __half* src, int rows, int K, const StagedW4& st, const float* fold,
                                         int nthreads) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = K >> 7;
  for (int w = warp; w < rows * groups; w += nthreads >> 5) {
    const int r = w / groups, g = w - r * groups;
    float v[4];
    load4_f32<__half>(src + static_cast<size_t>(r) * K + g * 128 + lane * 4, v);
    const float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    const unsigned int mb = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
    const int ex = static_cast<int>(mb >> 23) - 127;
    const float mult = (mb == 0u) ? 0.f : __uint_as_float(static_cast<unsigned int>(127 + 18 - ex) << 23);
    const float f = (mb == 0u) ? 1.0f : __uint_as_float(static_cast<unsigned int>(127 + ex - 18) << 23);
    uint32_t pk[3] = {0u, 0u, 0u};
    int part = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int q = __float2int_rn(v[i] * mult);
      const int b0 = (q << 24) >> 24;
      const int q1 = (q - b0) >> 8;
      const int b1 = (q1 << 24) >> 24;
      const int b2 = (q1 - b1) >> 8;
      pk[0] |= static_cast<uint32_t>(b0 & 0xFF) << (8 * i);
      pk[1] |= static_cast<uint32_t>(b1 & 0xFF) << (8 * i);
      pk[2] |= static_cast<uint32_t>(b2 & 0xFF) << (8 * i);
      part += q;
    }
    // an even lane holds elements 0..3 of its run of eight, the odd neighbour 4..7; stored order
    // is (0, 4, 1, 5 | 2, 6, 3, 7)
    uint8_t* dst = st.planes + static_cast<size_t>(r) * 3 * K + half_index(g * 128 + lane * 4, K);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const uint32_t other = __shfl_xor_sync(0xffffffffu, pk[p], 1);
      const uint32_t word = (lane & 1) ? __byte_perm(pk[p], other, 0x3726) : __byte_perm(pk[p], other, 0x5140);
      *reinterpret_cast<uint32_t*>(dst + p * K) = word;
    }
    part += __shfl_xor_sync(0xffffffffu, part, 1);
    part += __shfl_xor_sync(0xffffffffu, part, 2);
    part += __shfl_xor_sync(0xffffffffu, part, 4);
    if ((lane & 7) == 0) st.vsum[r * (K >> 5) + g * 4 + (lane >> 3)] = part;
    if (lane == 0) st.f[r * groups + g] = f * (fold != nullptr ? fold[r] : 1.0f);
  }
}

// exact integer dot of the 32 nibbles of one 16-byte load with the staged integers of its 32 k
__device__ __forceinline__ int dot32_w4(const uint4& w, const uint8_t* row_planes, int k, int K) {
  const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
  uint32_t lo[4], hi[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    lo[r] = ww[r] & 0x0F0F0F0Fu;
    hi[r] = (ww[r] >> 4) & 0x0F0F0F0Fu;
  }
  int s[3];
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const uint4 xa = *reinterpret_cast<const uint4*>(row_planes + p * K + (k >> 1));
    const uint4 xb = *reinterpret_cast<const uint4*>(row_planes + p * K + (K >> 1) + (k >> 1));
    int acc = dp4a_u8_s8(lo[0], xa.x, 0);
    acc = dp4a_u8_s8(hi[0], xa.y, acc);
    acc = dp4a_u8_s8(lo[1], xa.z, acc);
    acc = dp4a_u8_s8(hi[1], xa.w, acc);
    acc = dp4a_u8_s8(lo[2], xb.x, acc);
    acc = dp4a_u8_s8(hi[2], xb.y, acc);
    acc = dp4a_u8_s8(lo[3], xb.z, acc);
    acc = dp4a_u8_s8(hi[3], xb.w, acc);
    s[p] = acc;
  }
  return s[0] + (s[1] << 8) + (s[2] << 16);
}

// acc + (s f) * float(S - z * sum(v)) for the segment at k; c is the scale word of the row and the
// segment's group (fp16 scale | fp16(1024 + zero) << 16).  The words of a row lie one table row
// apart ([E][K/128][rows]), so the callers load them together with the weights, not here.
__device__ __forceinline__ float seg_w4(const uint4& w, const uint8_t* row_planes, const float* f, const int* vsum,
                                        uint32_t c, int k, int K, float acc) {
  const float s = __half2float(__ushort_as_half(static_cast<unsigned short>(c & 0xFFFFu)));
  const int z = static_cast<int>((c >> 16) & 0x3FFu);
  const int S = dot32_w4(w, row_planes, k, K) - z * vsum[k >> 5];
  return fmaf(s * f[k >> 7], static_cast<float>(S), acc);
}

constexpr int kSeg = 32 * 32;   // k covered by one warp-wide 16-byte load of packed nibbles

__device__ __forceinline__ StagedW4 carve_w4(uint8_t* base, int rows, int K) {
  StagedW4 st;
  st.planes = base;
  st.f = reinterpret_cast<float*>(base + static_cast<size_t>(rows) * 3 * K);
  st.vsum = reinterpret_cast<int*>(st.f + rows * (K >> 7));
  return st;
}
size_t staged_w4_bytes(int rows, int K) {
  return static_cast<size_t>(rows) * (3 * K + (K >> 7) * 4 + (K >> 5) * 4);
}

// (capping the registers for three resident CTAs instead of two was slower: 74 us vs 69 us at M = 1)
__global__ void __launch_bounds__(kUpThreads)
moe_gemv_w4_up_kernel(const GemvArgs a) {
  extern __shared__ __align__(16) uint8_t gemv_smem[];
  const int P = a.M * a.topk;
  const StagedW4 st = carve_w4(gemv_smem, a.M, a.H);
  int* s_e = st.vsum + a.M * (a.H >> 5);
  float* s_gam = reinterpret_cast<float*>(s_e + kGemvMaxPairs);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  griddep_wait();
  griddep_launch_dependents();
  stage_routing(a, s_e, s_gam);
  stage_w4(reinterpret_cast<const __half*>(a.x), a.M, a.H, st, nullptr, kUpThreads);
  __syncthreads();

  const bool w_on_input = (a.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0;
  const bool mimic = (a.flags & B200MOE_FLAG_MIMIC_ROUNDING) != 0;
  const bool ext = a.b1 != nullptr || a.activation == B200MOE_ACT_SWIGLU_OAI;
  ActParams ap;
  ap.activation = a.activation;
  ap.alpha = a.alpha;
  ap.limit = a.limit;
  __half* act = reinterpret_cast<__half*>(a.act);
  const uint8_t* w1 = reinterpret_cast<const uint8_t*>(a.w1);
  const uint32_t* sz1 = reinterpret_cast<const uint32_t*>(a.w1_sz);
  const size_t rows = 2 * static_cast<size_t>(a.I);      // weight rows (and scale words per group) of an expert
  const int G = a.H >> 7;

  // (Two register buffers with the next item's loads in flight while the current one is multiplied
  // were tried: 89 us against 69 us for the Mixtral-shaped layer at M = 1.)
  const int total = P * a.I;
  const int warps = gridDim.x * (kUpThreads / 32);
  for (int c = warp * gridDim.x + blockIdx.x; c < total; c += warps) {
    const int p = c / a.I, i = c - p * a.I;
    const int e = s_e[p];
    if (e < 0) {
      if (lane == 0) act[c] = __float2half_rn(0.f);
      continue;
    }
    const int t = p / a.topk;
    const uint8_t* xp = st.planes + static_cast<size_t>(t) * 3 * a.H;
    const float* xf = st.f + t * G;
    const int* xv = st.vsum + t * (a.H >> 5);
    const uint8_t* wg = w1 + (static_cast<size_t>(e) * rows + i) * (a.H >> 1);
    const uint8_t* wu = wg + static_cast<size_t>(a.I) * (a.H >> 1);
    const uint32_t* szg = sz1 + static_cast<size_t>(e) * G * rows + i;
    const uint32_t* szu = szg + a.I;
    float ag = 0.f, au = 0.f;
    for (int k0 = lane * 32; k0 < a.H; k0 += 4 * kSeg) {
      uint4 gq[4], uq[4];
      uint32_t cg[4], cu[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = k0 + q * kSeg;
        if (k < a.H) {
          gq[q] = ldg_stream(wg + (k >> 1));
          uq[q] = ldg_stream(wu + (k >> 1));
          cg[q] = __ldg(szg + static_cast<size_t>(k >> 7) * rows);
          cu[q] = __ldg(szu + static_cast<size_t>(k >> 7) * rows);
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = k0 + q * kSeg;
        if (k < a.H) {
          ag = seg_w4(gq[q], xp, xf, xv, cg[q], k, a.H, ag);
          au = seg_w4(uq[q], xp, xf, xv, cu[q], k, a.H, au);
        }
      }
    }
    ag = warp_sum(ag);
    au = warp_sum(au);
    if (lane == 0) {
      if (a.b1 != nullptr) {
        ag += __ldg(a.b1 + static_cast<size_t>(e) * 2 * a.I + i);
        au += __ldg(a.b1 + static_cast<size_t>(e) * 2 * a.I + a.I + i);
      }
      const float av = ext ? act_mul<__half, true>(ag, au, w_on_input, s_gam[p], mimic, ap)
                           : act_mul<__half>(ag, au, w_on_input, s_gam[p], mimic, ap);
      act[c] = __float2half_rn(av);
    }
  }
}

__global__ void __launch_bounds__(kDownThreads)
moe_gemv_w4_down_kernel(const GemvArgs a) {
  extern __shared__ __align__(16) uint8_t gemv_smem[];
  const int P = a.M * a.topk;
  const StagedW4 st = carve_w4(gemv_smem, P, a.I);
  int* s_e = st.vsum + P * (a.I >> 5);
  float* s_gam = reinterpret_cast<float*>(s_e + kGemvMaxPairs);
  float* s_fold = s_gam + kGemvMaxPairs;
  float* s_part = s_fold + kGemvMaxPairs;                           // [2 buffers][16 warps][2]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool w_on_input = (a.flags & B200MOE_FLAG_WEIGHT_ON_INPUT) != 0;
  const bool no_combine = (a.flags & B200MOE_FLAG_NO_COMBINE) != 0;
  const bool by_pair = no_combine || a.round_pair != 0;

  griddep_wait();
  griddep_launch_dependents();
  stage_routing(a, s_e, s_gam);
  __syncthreads();
  if (threadIdx.x < P) s_fold[threadIdx.x] = (by_pair || w_on_input) ? 1.0f : s_gam[threadIdx.x];
  __syncthreads();
  stage_w4(reinterpret_cast<const __half*>(a.act), P, a.I, st, s_fold, kDownThreads);
  __syncthreads();

  const uint8_t* w2 = reinterpret_cast<const uint8_t*>(a.w2);
  const uint32_t* sz2 = reinterpret_cast<const uint32_t*>(a.w2_sz);
  const size_t rows = static_cast<size_t>(a.H);
  const int G = a.I >> 7;
  const int nch = (a.I + kSeg - 1) / kSeg;
  __half* out = reinterpret_cast<__half*>(a.out);
  const int half_h = a.H >> 1;
  const int tasks = a.M * half_h;
  const int S = by_pair ? 1 : a.down_split;
  const int grp = warp / S, sub = warp - grp * S;
  const int groups = gridDim.x * ((kDownThreads / 32) / S);
  int iter = 0;
  for (int task = grp * gridDim.x + blockIdx.x; task < tasks; task += groups, ++iter) {
    const int t = task / half_h, h = (task - t * half_h) << 1;
    if (!by_pair) {
      // (pair, segment) flattened: four slots of two 16-byte loads (and their scale words) in flight
      const int Q = a.topk * nch;
      float acc0 = 0.f, acc1 = 0.f;
      int j = 0, ch = 0;
      for (int q0 = 0; q0 < Q; q0 += 4) {
        if (S > 1 && ((q0 >> 2) % S) != sub) {
          ch += 4;
          while (ch >= nch) {
            ch -= nch;
            ++j;
          }
          continue;
        }
        uint4 wa[4], wb[4];
        uint2 cc[4];
        int kk[4], pp[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int p = t * a.topk + j;
          const int k = ch * kSeg + lane * 32;
          const int e = (q0 + u < Q) ? s_e[p] : -1;
          const bool on = e >= 0 && k < a.I;
          kk[u] = on ? k : -1;
          pp[u] = p;
          if (on) {
            const uint8_t* wr = w2 + ((static_cast<size_t>(e) * rows + h) * a.I + k) / 2;
            wa[u] = ldg_stream(wr);
            wb[u] = ldg_stream(wr + (a.I >> 1));
            // rows h and h + 1 (h even) are neighbours in the scale table: one 8-byte load
            cc[u] = __ldg(reinterpret_cast<const uint2*>(sz2 + (static_cast<size_t>(e) * G + (k >> 7)) * rows + h));
          }
          if (++ch == nch) {
            ch = 0;
            ++j;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (kk[u] >= 0) {
            const int p = pp[u];
            const uint8_t* xp = st.planes + static_cast<size_t>(p) * 3 * a.I;
            acc0 = seg_w4(wa[u], xp, st.f + p * G, st.vsum + p * (a.I >> 5), cc[u].x, kk[u], a.I, acc0);
            acc1 = seg_w4(wb[u], xp, st.f + p * G, st.vsum + p * (a.I >> 5), cc[u].y, kk[u], a.I, acc1);
          }
        }
      }
      acc0 = warp_sum(acc0);
      acc1 = warp_sum(acc1);
      if (S > 1) {
        float* part = s_part + (iter & 1) * 2 * (kDownThreads / 32);
        if (lane == 0) {
          part[2 * warp] = acc0;
          part[2 * warp + 1] = acc1;
        }
        named_bar_sync(1 + grp, 32 * S);
        if (sub == 0 && lane == 0) {
          acc0 = 0.f;
          acc1 = 0.f;
          for (int w = 0; w < S; ++w) {
            acc0 += part[2 * (warp + w)];
            acc1 += part[2 * (warp + w) + 1];
          }
        }
      }
      if (sub == 0 && lane == 0) {
        if (a.b2 != nullptr) {
          for (int jb = 0; jb < a.topk; ++jb) {
            const int p = t * a.topk + jb;
            if (s_e[p] >= 0) {
              const float gam = w_on_input ? 1.0f : s_gam[p];
              acc0 = fmaf(__ldg(a.b2 + static_cast<size_t>(s_e[p]) * a.H + h), gam, acc0);
              acc1 = fmaf(__ldg(a.b2 + static_cast<size_t>(s_e[p]) * a.H + h + 1), gam, acc1);
            }
          }
        }
        out[static_cast<size_t>(t) * a.H + h] = __float2half_rn(acc0 * a.routed_scaling);
        out[static_cast<size_t>(t) * a.H + h + 1] = __float2half_rn(acc1 * a.routed_scaling);
      }
    } else {
      float sum0 = 0.f, sum1 = 0.f;
      for (int jb = 0; jb < a.topk; ++jb) {
        const int p = t * a.topk + jb;
        const int e = s_e[p];
        float y0 = 0.f, y1 = 0.f;
        if (e >= 0) {
          const uint8_t* wr = w2 + ((static_cast<size_t>(e) * rows + h) * a.I) / 2;
          const uint32_t* sz = sz2 + static_cast<size_t>(e) * G * rows + h;
          const uint8_t* xp = st.planes + static_cast<size_t>(p) * 3 * a.I;
          float acc0 = 0.f, acc1 = 0.f;
          for (int k0 = lane * 32; k0 < a.I; k0 += 4 * kSeg) {
            uint4 wa[4], wb[4];
            uint2 cc[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (k0 + q * kSeg < a.I) {
                wa[q] = ldg_stream(wr + ((k0 + q * kSeg) >> 1));
                wb[q] = ldg_stream(wr + ((a.I + k0 + q * kSeg) >> 1));
                cc[q] = __ldg(reinterpret_cast<const uint2*>(sz + static_cast<size_t>((k0 + q * kSeg) >> 7) * rows));
              }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int k = k0 + q * kSeg;
              if (k < a.I) {
                acc0 = seg_w4(wa[q], xp, st.f + p * G, st.vsum + p * (a.I >> 5), cc[q].x, k, a.I, acc0);
                acc1 = seg_w4(wb[q], xp, st.f + p * G, st.vsum + p * (a.I >> 5), cc[q].y, k, a.I, acc1);
              }
            }
          }
          acc0 = warp_sum(acc0);
          acc1 = warp_sum(acc1);
          if (a.b2 != nullptr) {
            acc0 += __ldg(a.b2 + static_cast<size_t>(e) * a.H + h);
            acc1 += __ldg(a.b2 + static_cast<size_t>(e) * a.H + h + 1);
          }
          y0 = w_on_input ? acc0 : acc0 * s_gam[p];
          y1 = w_on_input ? acc1 : acc1 * s_gam[p];
          if (a.round_pair) {
            y0 = __half2float(__float2half_rn(y0));
            y1 = __half2float(__float2half_rn(y1));
          }
        }
        if (no_combine) {
          if (lane == 0) {
            out[static_cast<size_t>(p) * a.H + h] = __float2half_rn(y0);
            out[static_cast<size_t>(p) * a.H + h + 1] = __float2half_rn(y1);
          }
        } else {
          sum0 += y0;
          sum1 += y1;
        }
      }
      if (!no_combine && lane == 0) {
        out[static_cast<size_t>(t) * a.H + h] = __float2half_rn(sum0 * a.routed_scaling);
        out[static_cast<size_t>(t) * a.H + h + 1] = __float2half_rn(sum1 * a.routed_scaling);
      }
    }
  }
}

size_t routing_smem() { return kGemvMaxPairs * 12 + 2 * 2 * (kDownThreads / 32) * 4 + 64; }   // tables + partial sums

// resident CTAs per SM times SMs, but no more CTAs per SM than the work has warps for: the grid
// stays a multiple of the SM count, so every SM streams the same share of the weights
template <typename K>
unsigned grid_for(K kernel, size_t smem, int threads, long long items, int num_sms) {
  // the query takes longer than a launch: this thread's last answers are kept (all devices are sm_100a: one answer fits all)
  struct Known {
    const void* kernel;
    size_t smem;
    int per_sm;
  };
  static thread_local Known known[8] = {};
  const void* id = reinterpret_cast<const void*>(kernel);
  Known& k = known[(reinterpret_cast<uintptr_t>(id) >> 4) & 7];
  if (k.kernel != id || k.smem != smem) {
    int n = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess || n < 1) n = 1;
    k = {id, smem, n};
  }
  int per_sm = k.per_sm;
  const long long warps_per_cta = threads / 32;
  const long long need_per_sm = (items + warps_per_cta * num_sms - 1) / (warps_per_cta * num_sms);
  if (per_sm > need_per_sm) per_sm = static_cast<int>(need_per_sm < 1 ? 1 : need_per_sm);
  return static_cast<unsigned>(per_sm) * static_cast<unsigned>(num_sms);
}

// Warps that share an output task of the down kernel.  With few output elements (short hidden size) several do, so that every
// SM still has 16 warps' worth of loads in flight.
int down_split(const GemvArgs& a, int num_sms) {
  const long long tasks = static_cast<long long>(a.M) * (a.H / 2);
  const long long all_warps = static_cast<long long>(num_sms) * (kDownThreads / 32);
  int split = 1;
  while (split < 8 && tasks * split * 2 <= all_warps) split *= 2;
  return split;
}

// Does the share of the down weights fit?  (The rows are 16-byte pieces for the bulk copy: I is a multiple of 8.)
bool share_fits(const GemvArgs& a, int num_sms) {
  const int P = a.M * a.topk, rows = share_rows(a.H, num_sms);
  return !a.w4 && P <= kGemvMaxPairs && rows <= kShareRows && share_bytes(P, rows, a.I) <= kShareBytes;
}
// ... and is that kernel the faster one?  The other one puts a warp's first eight 256-element slots in flight before it waits, too,
// and multiplies them from its registers.  With six slots a warp that is all of them, and enough of them (96 KB an SM) to keep HBM
// busy (both launches from a graph, us, this one / share): 4 pairs of 2048 x 768 12.3 / 12.75, 12 of 1024 x 512 13.1 / 14.2,
// 3 of 768 x 2048 11.5 / 12.0, 2 of 2048 x 1408 11.9 / 12.3, 3 of 2048 x 1024 12.45 / 12.65, 4 of 2304 x 640 12.9 / 13.3.
// With eight slots it goes either way (5 pairs of 2304 x 640 14.2 / 15.7, 4 of 2048 x 1024 15.7 / 14.4), with five too (10
// of 1024 x 512 12.3 / 12.9, 3 of 2048 x 768 11.4 / 11.0); with fewer or more, and where a task has one warp, the share
// kernel is ahead.
bool share_wins(const GemvArgs& a, int num_sms) {
  const bool by_pair = (a.flags & B200MOE_FLAG_NO_COMBINE) != 0 || a.round_pair != 0;     // the other one prefetches nothing then
  const int split = down_split(a, num_sms), slots = a.topk * ((a.I + kChunk - 1) / kChunk);
  return by_pair || split == 1 || (slots + split - 1) / split != 6;
}
// Every kernel may have 48 KB, its static shared memory among them, without being told; above that always the same limit
// (see kSmemLimit).
template <typename K>
bool allow_smem(K kernel, size_t smem, size_t limit) {
  return smem <= 44 * 1024 ||
         cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(limit)) == cudaSuccess;
}
template <typename K>
int launch_up(K kernel, const GemvArgs& a, int num_sms, cudaStream_t stream, bool pdl) {
  const size_t smem = gemv_up_smem(a);
  if (!allow_smem(kernel, smem, kSmemLimit)) return B200MOE_ERR_CUDA;
  const unsigned grid = grid_for(kernel, smem, kUpThreads, static_cast<long long>(a.M) * a.topk * a.I, num_sms);
  note_launch(a.w4 ? "moe_gemv_w4_up_kernel<gate/up>" : "moe_gemv_up_kernel<gate/up>");
  return launch_kernel(kernel, dim3(grid), dim3(kUpThreads), smem, stream, pdl, a) == cudaSuccess ? B200MOE_OK
                                                                                                  : B200MOE_ERR_CUDA;
}
template <typename K>
int launch_down(K kernel, const GemvArgs& a, int num_sms, cudaStream_t stream, bool pdl) {
  const size_t smem = gemv_down_smem(a);
  if (!allow_smem(kernel, smem, kSmemLimit)) return B200MOE_ERR_CUDA;
  GemvArgs b = a;
  const long long tasks = static_cast<long long>(a.M) * (a.H / 2);
  b.down_split = down_split(a, num_sms);
  const unsigned grid = grid_for(kernel, smem, kDownThreads, tasks * b.down_split, num_sms);
  note_launch(a.w4 ? "moe_gemv_w4_down_kernel<down>" : "moe_gemv_down_kernel<down>");
  return launch_kernel(kernel, dim3(grid), dim3(kDownThreads), smem, stream, pdl, b) == cudaSuccess ? B200MOE_OK
                                                                                                    : B200MOE_ERR_CUDA;
}

template <typename K>
int launch_share(K kernel, const GemvArgs& a, int num_sms, cudaStream_t stream, bool pdl) {
  const size_t smem = share_bytes(a.M * a.topk, share_rows(a.H, num_sms), a.I);
  if (!allow_smem(kernel, smem, kShareBytes)) return B200MOE_ERR_CUDA;
  note_launch("moe_gemv_down_share_kernel<down>");
  return launch_kernel(kernel, dim3(num_sms), dim3(kShareThreads), smem, stream, pdl, a) == cudaSuccess ? B200MOE_OK
                                                                                                       : B200MOE_ERR_CUDA;
}

}  // namespace

size_t gemv_up_smem(const GemvArgs& a) {
  return (a.w4 ? staged_w4_bytes(a.M, a.H) : static_cast<size_t>(a.M) * a.H * 4) + routing_smem();
}
size_t gemv_down_smem(const GemvArgs& a) {
  return (a.w4 ? staged_w4_bytes(a.M * a.topk, a.I) : static_cast<size_t>(a.M) * a.topk * a.I * 4) + routing_smem();
}
bool gemv_fits(const GemvArgs& a) {
  return a.M * a.topk <= kGemvMaxPairs && gemv_up_smem(a) + 1024 <= kSmemLimit && gemv_down_smem(a) + 1024 <= kSmemLimit;
}

int launch_gemv_up(const GemvArgs& a, int num_sms, cudaStream_t stream, bool pdl) {
  if (!gemv_fits(a)) return B200MOE_ERR_UNSUPPORTED;
  if (a.w4) return launch_up(moe_gemv_w4_up_kernel, a, num_sms, stream, pdl);
  const int chunks = (a.H + kChunk - 1) / kChunk;
  // A warp per column in one wave: more columns than the three CTAs an SM of the kernels below seat, up to five.  Both launches,
  // us, the kernel below / with six CTAs an SM, columns per seat in front: 2048 elements 3.03 16.6 / 17.8, 3.24 15.6 / 15.0, 3.46
  // 15.8 / 15.0, 3.9 16.6 / 16.5, 4.3 17.3 / 17.05, 4.76 17.7 / 17.9; 1024 3.03 10.7 / 11.05, 3.24 11.3 / 11.2, 4.3 12.2 / 11.8;
  // 512 3.46 8.75 / 8.2; 2304 3.46 17.95 / 16.4.  Just above three the second wave is a few columns that are over soon, at five
  // six CTAs an SM are full as well.  A row that five chunks cover stays ahead in its single pass (1280 4.3 15.15 / 15.65), one that
  // six cover up to four columns a seat (1536 3.9 15.6 / 17.1, 4.3 15.0 / 14.4).  With four tokens' rows staged six CTAs no
  // longer fit (19.2 / 20.5).
  const long long columns = static_cast<long long>(a.M) * a.topk * a.I, seats = static_cast<long long>(num_sms) * (kUpThreads / 32);
  if (share_fits(a, num_sms) && a.hist == nullptr && a.M <= 2 && chunks != 5 &&
      10 * columns > (chunks == 6 ? 40 : 31) * seats && 10 * columns <= 48 * seats)
    return a.dtype == B200MOE_DTYPE_BF16 ? launch_up(moe_gemv_up_kernel<__nv_bfloat16, 2>, a, num_sms, stream, pdl)
                                         : launch_up(moe_gemv_up_kernel<__half, 2>, a, num_sms, stream, pdl);
  const bool bf = a.dtype == B200MOE_DTYPE_BF16;
  if (chunks == 5)
    return bf ? launch_up(moe_gemv_up_kernel<__nv_bfloat16, 5>, a, num_sms, stream, pdl)
              : launch_up(moe_gemv_up_kernel<__half, 5>, a, num_sms, stream, pdl);
  if (chunks == 6)
    return bf ? launch_up(moe_gemv_up_kernel<__nv_bfloat16, 6>, a, num_sms, stream, pdl)
              : launch_up(moe_gemv_up_kernel<__half, 6>, a, num_sms, stream, pdl);
  return bf ? launch_up(moe_gemv_up_kernel<__nv_bfloat16, 4>, a, num_sms, stream, pdl)
            : launch_up(moe_gemv_up_kernel<__half, 4>, a, num_sms, stream, pdl);
}
int launch_gemv_down(const GemvArgs& a, int num_sms, cudaStream_t stream, bool pdl) {
  if (!gemv_fits(a)) return B200MOE_ERR_UNSUPPORTED;
  if (a.w4) return launch_down(moe_gemv_w4_down_kernel, a, num_sms, stream, pdl);
  if (share_fits(a, num_sms) && share_wins(a, num_sms)) {
    const bool bf = a.dtype == B200MOE_DTYPE_BF16;
    if (a.hist != nullptr)
      return bf ? launch_share(moe_gemv_down_share_kernel<__nv_bfloat16, true>, a, num_sms, stream, pdl)
                : launch_share(moe_gemv_down_share_kernel<__half, true>, a, num_sms, stream, pdl);
    return bf ? launch_share(moe_gemv_down_share_kernel<__nv_bfloat16, false>, a, num_sms, stream, pdl)
              : launch_share(moe_gemv_down_share_kernel<__half, false>, a, num_sms, stream, pdl);
  }
  return a.dtype == B200MOE_DTYPE_BF16 ? launch_down(moe_gemv_down_kernel<__nv_bfloat16>, a, num_sms, stream, pdl)
                                       : launch_down(moe_gemv_down_kernel<__half>, a, num_sms, stream, pdl);
}

}  // namespace b200moe
