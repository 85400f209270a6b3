// Routing / alignment kernels: stable counting sort of the (token, expert) slots by
// expert with warp-match ranking and shared-memory counters.  Integer work only;
// every output is deterministic (no atomics decide an order).
#include "align.cuh"

namespace b200moe {

namespace {

constexpr int kAlignThreads = 1024;
constexpr int kAhead = 8;   // iterations of 32 slots whose ids are fetched together

__device__ __forceinline__ int load_id(const void* ids, int is64, int i) {
  return is64 ? static_cast<int>(reinterpret_cast<const long long*>(ids)[i])
              : reinterpret_cast<const int*>(ids)[i];
}

// Exclusive scan of one int per thread over the whole CTA (blockDim.x <= 1024).
// Returns the exclusive prefix; *total receives the sum.  scratch: 33 ints.
__device__ __forceinline__ int block_exclusive_scan(int v, int* scratch, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += t;
  }
  if (lane == 31) scratch[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int w = (lane < (blockDim.x >> 5)) ? scratch[lane] : 0;
    int winc = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, winc, d);
      if (lane >= d) winc += t;
    }
    scratch[lane] = winc - w;
    if (lane == 31) scratch[32] = winc;
  }
  __syncthreads();
  int res = inc - v + scratch[warp];
  *total = scratch[32];
  __syncthreads();
  return res;
}

// Largest e in [0, n) with offs[e] <= x, for a non-decreasing offs[0..n].
__device__ __forceinline__ int upper_expert(const int* offs, int n, int x) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (offs[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

// The kernels below run as ONE cluster of 1..8 CTAs (the whole grid): CTA c owns the contiguous slots
// [c * per, (c + 1) * per), the CTAs' counts meet through distributed shared memory, and stability follows from
// ordering by (CTA, warp, lane).  One CTA pushed every store through one SM's memory pipe (77 us at 32768 slots), and
// two launches of 32 CTAs with the counts in global memory took 47 us there.
__device__ __forceinline__ int cluster_rank() {
  int r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// the int at this CTA's shared-memory address `p`, read in CTA `rank` of the cluster
__device__ __forceinline__ int ld_cluster(const int* p, int rank) {
  uint32_t a;
  int v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}

struct GroupSmem {
  int* cnt;    // [nwarps][E] slots of each warp
  int* tot;    // [E] slots of this CTA (read by the other CTAs)
  int* hist;   // [E] slots of all CTAs
  int* base;   // [E+1] padded start row of each expert
  int* mine;   // [E] first row of this CTA's slots
  int* scan;   // 33
};
__device__ __forceinline__ GroupSmem group_smem(int* smem, int nwarps, int E) {
  GroupSmem g;
  g.cnt = smem;
  g.tot = g.cnt + nwarps * E;
  g.hist = g.tot + E;
  g.base = g.hist + E;
  g.mine = g.base + (E + 1);
  g.scan = g.mine + E;
  return g;
}
size_t group_smem_bytes(int nwarps, int E) {
  return (static_cast<size_t>(nwarps) * E + 4 * static_cast<size_t>(E) + 1 + 40) * sizeof(int);
}

// Core: stable grouping of P slots by expert.  `ids` are expert ids (mapped to local experts when
// map != nullptr); slots with an id outside [0, E) are dropped.  Each expert's group starts at a
// multiple of `block`.  place(slot, pos, pre[slot]) records a placement; `pre` (optional, [P]) is a
// per-slot value fetched alongside the ids; dropped[slot] (optional) becomes -1 for a dropped slot.  Called by every
// thread of every CTA; the caller ends with cluster_wait() (the CTAs' counts are read by their peers).
template <typename Place>
__device__ __forceinline__ void group_by_expert(const void* ids, int is64, const int* map, int map_len, int P, int E,
                                                int block, const GroupSmem& g, int nwarps, const float* pre, Place place,
                                                int* dropped = nullptr) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rank = cluster_rank(), nctas = gridDim.x;
  for (int i = threadIdx.x; i < nwarps * E; i += blockDim.x) g.cnt[i] = 0;
  __syncthreads();

  // contiguous, 32-aligned shares of the slots per CTA and, inside it, per counting warp
  const int per = ((P + nctas - 1) / nctas + 31) & ~31;
  const int cta_begin = min(P, rank * per), cta_end = min(P, cta_begin + per);
  const int seg = ((cta_end - cta_begin + nwarps - 1) / nwarps + 31) & ~31;
  const int begin = cta_begin + warp * seg;
  const int end = min(cta_end, begin + seg);

  // Both passes fetch the ids of kAhead iterations before they rank them: one dependent global
  // load per 32 slots would otherwise set the pace.  A share that fits keeps them for the second pass.
  auto fetch = [&](int i) -> int {
    int e = -1;
    if (i < end) {
      e = load_id(ids, is64, i);
      if (map != nullptr && e >= 0) e = (e < map_len) ? map[e] : -1;
      if (e < 0 || e >= E) e = -1;
    }
    return e;
  };
  int ev[kAhead];
  if (warp < nwarps) {
    for (int i0 = begin; i0 < end; i0 += 32 * kAhead) {
#pragma unroll
      for (int u = 0; u < kAhead; ++u) ev[u] = fetch(i0 + 32 * u + lane);
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (i0 + 32 * u >= end) break;
        const int e = ev[u];
        unsigned m = __match_any_sync(0xffffffffu, e);
        if (e >= 0 && (m & ((1u << lane) - 1)) == 0) g.cnt[warp * E + e] += __popc(m);
        __syncwarp();
      }
    }
  }
  __syncthreads();

  // per expert: this CTA's total and the exclusive prefix over its counting warps
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int run = 0;
    for (int w = 0; w < nwarps; ++w) {
      const int t = g.cnt[w * E + e];
      g.cnt[w * E + e] = run;
      run += t;
    }
    g.tot[e] = run;
  }
  cluster_arrive();
  cluster_wait();

  // totals and the slots of the CTAs before this one; padded starts by an exclusive scan over the
  // experts (chunks of blockDim.x experts)
  int carry = 0;
  for (int e0 = 0; e0 < E; e0 += blockDim.x) {
    const int e = e0 + threadIdx.x;
    int total = 0, before = 0;
    if (e < E) {
      for (int c = 0; c < nctas; ++c) {
        const int t = ld_cluster(g.tot + e, c);
        if (c < rank) before += t;
        total += t;
      }
      g.hist[e] = total;
    }
    int sum;
    const int ex = block_exclusive_scan((total + block - 1) / block * block, g.scan, &sum);
    if (e < E) {
      g.base[e] = carry + ex;
      g.mine[e] = carry + ex + before;
    }
    carry += sum;
  }
  if (threadIdx.x == 0) g.base[E] = carry;
  cluster_arrive();       // the peers' counts have been read; the caller waits before it leaves
  __syncthreads();

  if (warp < nwarps) {
    const bool kept = end - begin <= 32 * kAhead;
    for (int i0 = begin; i0 < end; i0 += 32 * kAhead) {
      float wv[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int i = i0 + 32 * u + lane;
        if (!kept) ev[u] = fetch(i);
        wv[u] = (pre != nullptr && i < end) ? pre[i] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (i0 + 32 * u >= end) break;
        const int i = i0 + 32 * u + lane;
        const int e = ev[u];
        unsigned m = __match_any_sync(0xffffffffu, e);
        const int r = __popc(m & ((1u << lane) - 1));
        int cur = 0;
        if (e >= 0) cur = g.cnt[warp * E + e];
        __syncwarp();
        if (e >= 0) {
          place(i, g.mine[e] + cur + r, wv[u]);
          if (r == 0) g.cnt[warp * E + e] = cur + __popc(m);
        } else if (dropped != nullptr && i < end) {
          dropped[i] = -1;
        }
        __syncwarp();
      }
    }
  }
}

__global__ void __launch_bounds__(kAlignThreads)
align_block_kernel(const void* ids, int is64, const int* map, int map_len, const float* weights, int P, int E,
                   int block, int cap, int nwarps, int* sorted_ids, int* expert_ids, int* num_post_pad,
                   float* row_gamma, int* blk_off, int* meta, int* slot_row, const FlagWait fw) {
  extern __shared__ int smem[];
  griddep_wait();             // the tables written below may still be read by the kernels of the previous call
  griddep_launch_dependents();
  wait_for_peers(fw);
  const GroupSmem g = group_smem(smem, nwarps, E);
  group_by_expert(ids, is64, map, map_len, P, E, block, g, nwarps, row_gamma != nullptr ? weights : nullptr,
                  [&](int slot, int pos, float w) {
                    sorted_ids[pos] = slot;
                    if (row_gamma != nullptr) row_gamma[pos] = w;
                    if (slot_row != nullptr) slot_row[slot] = pos;
                  },
                  slot_row);

  // padding of every expert's group, then the unused tail of the tables
  const int lane = threadIdx.x & 31;
  const int tid = cluster_rank() * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
  const int rows = g.base[E];
  for (int e = tid >> 5; e < E; e += nthreads >> 5)
    for (int r = g.base[e] + g.hist[e] + lane; r < g.base[e + 1]; r += 32) {
      sorted_ids[r] = P;
      if (row_gamma != nullptr) row_gamma[r] = 0.f;
    }
  for (int r = rows + tid; r < cap; r += nthreads) {
    sorted_ids[r] = P;
    if (row_gamma != nullptr) row_gamma[r] = 0.f;
  }
  const int nblk_cap = (cap + block - 1) / block;
  const int nblk = rows / block;
  for (int b = tid; b < nblk_cap; b += nthreads) expert_ids[b] = b < nblk ? upper_expert(g.base, E + 1, b * block) : -1;
  if (blk_off != nullptr)
    for (int e = tid; e <= E; e += nthreads) blk_off[e] = g.base[e] / block;
  if (tid == 0) {
    num_post_pad[0] = rows;
    if (meta != nullptr) {
      meta[0] = nblk;
      meta[1] = rows;
    }
  }
  cluster_wait();
}

// Internal tables from the reference's routing triple: hist[E], topk_indx[P]
// (sorted row -> slot), gate_scal[P] (sorted row order).  Every CTA scans hist by itself and fills its share of the
// padded rows (one CTA took 19 us at 16384 slots).
__global__ void __launch_bounds__(kAlignThreads)
align_from_routing_kernel(const int* hist, const int* topk_indx, const float* gate_scal, int P, int E,
                          int block, int cap, int* sorted_ids, float* row_gamma, int* blk_off,
                          int* meta) {
  extern __shared__ int smem[];
  int* s_base = smem;             // E + 1 padded starts
  int* s_raw = s_base + (E + 1);  // E + 1 raw starts
  int* s_scan = s_raw + (E + 1);  // 33
  griddep_wait();
  griddep_launch_dependents();
  int carry_p = 0, carry_r = 0;
  for (int e0 = 0; e0 < E; e0 += blockDim.x) {
    int e = e0 + threadIdx.x;
    int h = (e < E) ? hist[e] : 0;
    int total;
    int ex = block_exclusive_scan((h + block - 1) / block * block, s_scan, &total);
    if (e < E) s_base[e] = carry_p + ex;
    carry_p += total;
    ex = block_exclusive_scan(h, s_scan, &total);
    if (e < E) s_raw[e] = carry_r + ex;
    carry_r += total;
  }
  if (threadIdx.x == 0) {
    s_base[E] = carry_p;
    s_raw[E] = carry_r;
  }
  __syncthreads();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
  for (int r = tid; r < cap; r += nthreads) {
    int slot = P;
    float w = 0.f;
    if (r < carry_p) {
      const int e = upper_expert(s_base, E + 1, r);
      const int q = s_raw[e] + (r - s_base[e]);
      if (q < s_raw[e + 1] && q < P) {
        slot = topk_indx[q];
        w = gate_scal[q];
      }
    }
    sorted_ids[r] = slot;
    row_gamma[r] = w;
  }
  for (int e = tid; e <= E; e += nthreads) blk_off[e] = s_base[e] / block;
  if (tid == 0) {
    meta[0] = carry_p / block;
    meta[1] = carry_p;
  }
}

// top-k -> the reference's routing tables.  A token's experts are put in ascending order (stable): the place
// of column j is the number of columns that precede it, so each slot finds its own with k reads
// of its token's ids.  Grouping by expert needs no sorted ids: within an expert the order is by token, and by column
// where a token names an expert twice, in either numbering.
__global__ void __launch_bounds__(kAlignThreads)
routing_from_topk_kernel(const float* weights, const void* ids, int is64, int M, int k, int E,
                         int max_tiles, int nwarps, int* expt_indx, int* topk_indx, int* gate_indx,
                         float* gate_scal, int* hist, int* token_offs_raw, int* token_offs_pad,
                         int* block_pid_map) {
  extern __shared__ int smem[];
  const GroupSmem g = group_smem(smem, nwarps, E);
  const int P = M * k;
  griddep_wait();
  griddep_launch_dependents();
  auto sorted_slot = [&](int i) {
    const int t0 = i / k * k;
    const int e = load_id(ids, is64, i);
    int rank = 0;
    for (int j = t0; j < t0 + k; ++j) {
      const int ej = load_id(ids, is64, j);
      rank += (ej < e) || (ej == e && j < i);
    }
    return t0 + rank;
  };
  const int crank = cluster_rank(), nctas = gridDim.x;
  const int tid = crank * blockDim.x + threadIdx.x, nthreads = nctas * blockDim.x;
  for (int i = tid; i < P; i += nthreads) expt_indx[sorted_slot(i)] = load_id(ids, is64, i);

  group_by_expert(ids, is64, nullptr, 0, P, E, 1, g, nwarps, weights, [&](int i, int pos, float w) {
    const int slot = sorted_slot(i);
    topk_indx[pos] = slot;
    gate_indx[slot] = pos;
    gate_scal[pos] = w;
  });
  for (int e = tid; e < E; e += nthreads) hist[e] = g.hist[e];
  for (int e = tid; e <= E; e += nthreads) token_offs_raw[e] = g.base[e];
  __syncthreads();

  // padded block tables for block sizes 16, 32, 64, 128, dealt out over the CTAs
  int* s_off = g.cnt;     // E + 1 first blocks (the counters and totals behind them are no longer needed here)
  cluster_wait();         // ... nor by the peers
  for (int v = crank; v < 4; v += nctas) {
    const int bm = 16 << v;
    int carry = 0;
    for (int e0 = 0; e0 < E; e0 += blockDim.x) {
      const int e = e0 + threadIdx.x;
      const int tiles = (e < E) ? (g.hist[e] + bm - 1) / bm : 0;
      int total;
      const int ex = block_exclusive_scan(tiles, g.scan, &total);
      if (e < E) {
        s_off[e] = carry + ex;
        token_offs_pad[v * (E + 1) + e] = carry + ex;
      }
      carry += total;
    }
    if (threadIdx.x == 0) {
      s_off[E] = carry;
      token_offs_pad[v * (E + 1) + E] = carry;
    }
    __syncthreads();
    for (int b = threadIdx.x; b < max_tiles; b += blockDim.x) {
      int w = -1;
      if (b < carry) {
        const int e = upper_expert(s_off, E + 1, b);
        w = ((b - s_off[e]) << 16) + e;
      }
      block_pid_map[v * max_tiles + b] = w;
    }
    __syncthreads();
  }
}

int pick_warps(int E) {
  int nw = 32;
  while (nw > 1 && static_cast<size_t>(nw) * E * 4 > 40 * 1024) nw >>= 1;
  return nw;
}

// CTAs of the cluster: one while a CTA's 32 warps hold a few rounds of slots at most
int pick_ctas(int P) { return P < 1024 ? 1 : 8; }

// Experts a grouping launch takes; pick_warps keeps its tables below kMaxGroupSmem up to there.
constexpr int kMaxGroupExperts = 3061;
constexpr size_t kMaxGroupSmem = 96 * 1024;

// Shared memory of a grouping launch; above 48 KiB (from 613 experts on, depending on the warps that count) the
// kernel has to be told.  Always the same limit: two threads may launch with different sizes.
template <typename Kernel>
int group_smem_for(Kernel* kernel, int nwarps, int E, size_t* bytes) {
  *bytes = group_smem_bytes(nwarps, E);
  if (E > kMaxGroupExperts || *bytes > kMaxGroupSmem) return B200MOE_ERR_TOO_LARGE;
  if (*bytes > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(kMaxGroupSmem)) != cudaSuccess)
    return B200MOE_ERR_CUDA;
  return B200MOE_OK;
}

}  // namespace

int align_capacity(int n_slots, int n_experts, int block) {
  long long cap = static_cast<long long>(n_slots) + static_cast<long long>(n_experts) * (block - 1);
  if (n_slots < n_experts) {
    long long alt = static_cast<long long>(n_slots) * block;
    if (alt < cap) cap = alt;
  }
  if (cap > 0x7fffffffLL) return -1;
  return static_cast<int>(cap);
}

int routing_max_tiles(int n_slots, int n_experts) {
  if (n_slots <= n_experts) return n_slots;
  // floor division of a negative numerator, as the dependency's Python does
  int num = n_experts - n_slots - 1;  // negative
  int fl = -((-num + 15) / 16);
  return n_experts - 1 - fl;
}

int launch_align_block(const void* ids, int is64, const int* map, int map_len, const float* weights, int P, int E,
                       int block, int cap, int* sorted_ids, int* expert_ids, int* num_post_pad,
                       float* row_gamma, int* blk_off, int* meta, cudaStream_t stream, bool pdl, const FlagWait* wait, bool one_cta,
                       int* slot_row) {
  if (P < 0 || E <= 0 || block <= 0 || cap < 0) return B200MOE_ERR_BAD_ARG;
  const int nw = pick_warps(E);
  size_t smem;
  if (const int rc = group_smem_for(align_block_kernel, nw, E, &smem)) return rc;
  note_launch("align_block_kernel");
  FlagWait fw = {};
  if (wait != nullptr) fw = *wait;
  const int ctas = one_cta ? 1 : pick_ctas(P);
  cudaError_t err = launch_kernel_cluster(align_block_kernel, dim3(ctas), ctas, dim3(kAlignThreads), smem, stream, pdl, ids,
                                          is64, map, map_len, weights, P, E, block, cap, nw, sorted_ids, expert_ids,
                                          num_post_pad, row_gamma, blk_off, meta, slot_row, fw);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

int launch_align_from_routing(const int* hist, const int* topk_indx, const float* gate_scal, int P,
                              int E, int block, int cap, int* sorted_ids, float* row_gamma,
                              int* blk_off, int* meta, cudaStream_t stream, bool pdl) {
  if (P < 0 || E <= 0 || block <= 0) return B200MOE_ERR_BAD_ARG;
  size_t smem = (2 * static_cast<size_t>(E + 1) + 40) * sizeof(int);
  if (smem > 48 * 1024) return B200MOE_ERR_TOO_LARGE;
  note_launch("align_from_routing_kernel");
  int ctas = (cap + kAlignThreads - 1) / kAlignThreads;
  if (ctas > 32) ctas = 32;
  if (ctas < 1) ctas = 1;
  cudaError_t err = launch_kernel(align_from_routing_kernel, dim3(ctas), dim3(kAlignThreads), smem, stream, pdl, hist, topk_indx,
                                  gate_scal, P, E, block, cap, sorted_ids, row_gamma, blk_off, meta);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

int launch_routing_from_topk(const float* weights, const void* ids, int is64, int M, int k, int E,
                             int* expt_indx, int* topk_indx, int* gate_indx, float* gate_scal,
                             int* hist, int* token_offs_raw, int* token_offs_pad, int* block_pid_map,
                             cudaStream_t stream, bool pdl) {
  if (M < 0 || k <= 0 || E <= 0) return B200MOE_ERR_BAD_ARG;
  const int nw = pick_warps(E);
  size_t smem;
  if (const int rc = group_smem_for(routing_from_topk_kernel, nw, E, &smem)) return rc;
  const int mt = routing_max_tiles(M * k, E);
  note_launch("routing_from_topk_kernel");
  const int ctas = pick_ctas(M * k);
  cudaError_t err = launch_kernel_cluster(routing_from_topk_kernel, dim3(ctas), ctas, dim3(kAlignThreads), smem, stream, pdl,
                                          weights, ids, is64, M, k, E, mt, nw, expt_indx, topk_indx, gate_indx, gate_scal,
                                          hist, token_offs_raw, token_offs_pad, block_pid_map);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

}  // namespace b200moe
