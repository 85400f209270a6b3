// Decode-sized calls: the grouped GEMMs sort the (token, choice) slots by expert themselves.
//
// Every CTA counts the slots of each expert in its own shared memory, straight from the routing input (count_slots); with the
// experts' starts the tiles are known and the weights of the first ones are under way.  Which slots a tile holds is looked up by
// the warps that need it, one scan over the slots' experts per tile (block_slots).  No alignment is launched, and the
// 16-bit gate/up projection fetches the token rows where they lie.  The later kernels of a call do the same while the one before
// them drains, and have their ring full of weights before they may read what it wrote.
#pragma once
#include "gemm.cuh"

namespace b200moe {

constexpr unsigned kNoSlot = 0xffffu;

struct RowTables {
  int* blk;         // [E+1] first block of each expert
  int* raw;         // [E+1] slots before each expert
  int* scan;        // [32]
  uint16_t* ids;    // local expert of slot i at ids_at(i), kNoSlot: none
};
// 256 slots are 32 vectors of eight, lane l of a warp with slots l, l + 32, ...: a warp compares them with one load.
__host__ __device__ __forceinline__ int ids_at(int i) { return (i & ~255) + ((i & 31) << 3) + ((i >> 5) & 7); }
__host__ __device__ __forceinline__ size_t route_table_bytes(int E, int P) {
  return 2 * static_cast<size_t>(E + 1) * 4 + 128 + 16 + ((static_cast<size_t>(P) + 255) & ~static_cast<size_t>(255)) * 2;
}
__device__ __forceinline__ RowTables row_tables(void* smem, int E) {
  RowTables t;
  t.blk = reinterpret_cast<int*>(smem);
  t.raw = t.blk + (E + 1);
  t.scan = t.raw + (E + 1);
  t.ids = reinterpret_cast<uint16_t*>((reinterpret_cast<uintptr_t>(t.scan + 32) + 15) & ~static_cast<uintptr_t>(15));
  return t;
}

// The experts of a thread's next kAhead slots, fetched together (i0, i0 + blockDim.x, ...); -1 past the end or outside [0, bound).
// Reads bypass L1: a dependent launch may get here before griddep_wait(), when an earlier kernel's lines could still be cached.
constexpr int kAhead = 4;
template <typename I>
__device__ __forceinline__ void fetch_experts(const I* ids, int i0, int P, int bound, int (&ev)[kAhead]) {
  I v[kAhead];
#pragma unroll
  for (int q = 0; q < kAhead; ++q) {
    const int i = i0 + q * blockDim.x;
    v[q] = i < P ? __ldcg(ids + i) : static_cast<I>(-1);
  }
#pragma unroll
  for (int q = 0; q < kAhead; ++q) ev[q] = (v[q] >= 0 && v[q] < bound) ? static_cast<int>(v[q]) : -1;
}

// All threads of the CTA: starts of the experts in slots and in blocks.  Ends with a barrier.
__device__ __forceinline__ void count_slots(const RouteSource& r, int P, int E, int BT, const RowTables& t) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool triple = r.hist != nullptr;
  if (!triple) {
    const int bound = r.map != nullptr ? r.map_len : E;
    int ev[kAhead];
    auto fetch = [&](int i0) {
      if (r.is64) fetch_experts(reinterpret_cast<const long long*>(r.ids), i0, P, bound, ev);
      else fetch_experts(reinterpret_cast<const int*>(r.ids), i0, P, bound, ev);
      if (r.map != nullptr) {
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
          if (ev[q] >= 0) {
            const int e = __ldcg(r.map + ev[q]);
            ev[q] = e < E ? e : -1;
          }
      }
    };
    fetch(threadIdx.x);
    for (int i = P + threadIdx.x; i < ((P + 255) & ~255); i += blockDim.x) t.ids[ids_at(i)] = kNoSlot;
    for (int e = threadIdx.x; e < E; e += blockDim.x) t.raw[e] = 0;
    __syncthreads();
    for (int i0 = threadIdx.x; i0 < P; i0 += kAhead * blockDim.x) {
      if (i0 != static_cast<int>(threadIdx.x)) fetch(i0);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int i = i0 + q * blockDim.x;
        if (i >= P) break;
        t.ids[ids_at(i)] = static_cast<uint16_t>(ev[q] >= 0 ? ev[q] : kNoSlot);
        if (ev[q] >= 0) atomicAdd(&t.raw[ev[q]], 1);
      }
    }
    __syncthreads();
  }
  // Exclusive scan over the experts of (slots, blocks), packed two to a word: both stay below 2^16.  A thread has
  // consecutive experts.
  const int per = (E + blockDim.x - 1) / blockDim.x;
  const int e0 = min(E, static_cast<int>(threadIdx.x) * per), e1 = min(E, e0 + per);
  auto packed = [&](int n) { return static_cast<unsigned>(n) | (static_cast<unsigned>((n + BT - 1) / BT) << 16); };
  unsigned mine = 0;
  for (int e = e0; e < e1; ++e) {
    if (triple) t.raw[e] = max(0, min(P, __ldcg(r.hist + e)));
    mine += packed(t.raw[e]);
  }
  unsigned inc = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += v;
  }
  if (lane == 31) t.scan[warp] = static_cast<int>(inc);
  __syncthreads();
  unsigned base = inc - mine;
  for (int w = 0; w < warp; ++w) base += static_cast<unsigned>(t.scan[w]);
  for (int e = e0; e < e1; ++e) {
    const int n = t.raw[e];
    t.raw[e] = static_cast<int>(base & 0xffffu);
    t.blk[e] = static_cast<int>(base >> 16);
    base += packed(n);
  }
  if (threadIdx.x == blockDim.x - 1) {      // the last thread ends at E
    t.raw[E] = static_cast<int>(base & 0xffffu);
    t.blk[E] = static_cast<int>(base >> 16);
  }
  __syncthreads();
}

// Which of the eight experts at t.ids[at] are the one in both halves of `both`.
__device__ __forceinline__ unsigned ids_equal(const RowTables& t, int at, unsigned both) {
  const uint4 v = *reinterpret_cast<const uint4*>(t.ids + at);
  const unsigned w[4] = {v.x ^ both, v.y ^ both, v.z ^ both, v.w ^ both};
  unsigned hit = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) hit |= ((w[q] & 0xffffu) == 0 ? 1u << (2 * q) : 0u) | (w[q] < 0x10000u ? 2u << (2 * q) : 0u);
  return hit;
}
// A warp: lane r gets the slot of row r of the block that starts at padded row row0 of expert e (r < rows <= 32), -1 for
// padding.  Slots of an expert stand in ascending order (triple: in the order given).
__device__ __forceinline__ int block_slots(const RouteSource& r, const RowTables& t, int P, int BT, int e, int row0, int rows) {
  const int lane = threadIdx.x & 31;
  const int first = row0 - t.blk[e] * BT;
  if (r.hist != nullptr) {
    const int q = t.raw[e] + first + lane;
    int slot = (lane < rows && q < t.raw[e + 1] && q < P) ? __ldcg(r.topk_indx + q) : -1;
    return slot < P ? slot : -1;
  }
  // Everything below is uniform over the warp but the last select: with a divergent search of the set bits a scan over 256
  // slots took 1060 cycles.
  int mine = -1, seen = 0;
  const unsigned both = static_cast<unsigned>(e) * 0x10001u;
  for (int i0 = 0; i0 < P && seen < first + rows; i0 += 256) {
    const unsigned hit = ids_equal(t, i0 + lane * 8, both);      // bit q: slot i0 + 32 q + lane
    // A later block of the expert: pass over 256 slots at once.  (By rounds of 32, with the slots behind the block looked at too, a
    // zipf-skewed call of 208 tokens on 128 experts of 2048 x 768 took 181 us against 152, of 400 tokens 266 against 207.)
    if (seen < first) {
      const int n = __reduce_add_sync(0xffffffffu, __popc(hit));
      if (seen + n <= first) {
        seen += n;
        continue;
      }
    }
    for (unsigned rounds = __reduce_or_sync(0xffffffffu, hit); rounds != 0 && seen < first + rows; rounds &= rounds - 1) {
      const int q = __ffs(rounds) - 1;
      unsigned bits = __ballot_sync(0xffffffffu, (hit >> q) & 1u);
      const int n = __popc(bits);
      if (seen + n <= first) {
        seen += n;
        continue;
      }
      for (; bits != 0; bits &= bits - 1, ++seen)
        if (lane == seen - first) mine = i0 + 32 * q + __ffs(bits) - 1;
    }
  }
  return lane < rows ? mine : -1;
}
// Slot (lane r: of row r, see block_slots) and routing weight of a block's rows: from this CTA's tables, or from those of an
// alignment launch.  Whole warp.
__device__ __forceinline__ int rows_slot(const GemmArgs& a, const RowTables& t, int BT, int e, int row0, int rows) {
  if (a.route.own) return block_slots(a.route, t, a.P, BT, e, row0, rows);
  const int lane = threadIdx.x & 31;
  const int slot = lane < rows ? a.sorted_ids[row0 + lane] : -1;
  return slot >= 0 && slot < a.P ? slot : -1;
}
__device__ __forceinline__ float rows_weight(const GemmArgs& a, const RowTables& t, int BT, int e, int row0, int slot) {
  const int lane = threadIdx.x & 31;
  if (slot < 0) return 0.f;
  if (!a.route.own) return a.row_gamma[row0 + lane];
  if (a.route.hist == nullptr) return __ldcg(a.route.weights + slot);
  return __ldcg(a.route.gate_scal + t.raw[e] + row0 - t.blk[e] * BT + lane);
}
// A warp: number of slots before `slot` that name the same expert e.
__device__ __forceinline__ int slot_rank(const RowTables& t, int slot, unsigned e) {
  const int lane = threadIdx.x & 31;
  const unsigned both = e * 0x10001u;
  int n = 0;
#pragma unroll 1
  for (int i0 = 0; i0 < slot; i0 += 256) {
    const int rounds = (max(0, min(256, slot - i0 - lane)) + 31) >> 5;      // of this lane's slots i0 + 32 q + lane
    n += __popc(ids_equal(t, i0 + lane * 8, both) & ((1u << rounds) - 1));
  }
  return __reduce_add_sync(0xffffffffu, n);
}

// One warp copies the token rows of a block of BT rows into swizzled operand tiles, 128 bytes of every row at a time, and hands
// them to the MMA thread: plain copies become visible to the tensor core with a proxy fence of the thread that waited
// for them.  kLag stages are in flight.
template <int BT, int kLag>
struct RowCopier {
  const uint8_t* src[BT / 4];     // this lane's 16 bytes of row 4 i + lane / 8
  int lane, n;                    // stages issued
  uint32_t bars[kLag];            // barriers of the stages in flight

  __device__ __forceinline__ RowCopier() : lane(threadIdx.x & 31), n(0) {}
  // Padding rows repeat the block's first token: what is computed for them is never stored where it is read.
  __device__ __forceinline__ void block(const GemmArgs& a, const RowTables& t, int e, int row0, size_t row_bytes) {
    const int mine = block_slots(a.route, t, a.P, BT, e, row0, BT);
    const int first = max(0, __shfl_sync(0xffffffffu, mine, 0));
#pragma unroll
    for (int i = 0; i < BT / 4; ++i) {
      int slot = __shfl_sync(0xffffffffu, mine, 4 * i + (lane >> 3));
      if (slot < 0) slot = first;
      src[i] = reinterpret_cast<const uint8_t*>(a.rows) + static_cast<size_t>(slot / a.topk) * row_bytes + (lane & 7) * 16;
    }
  }
  // 128 bytes from byte `at` of every row into the tile at `tile`; bytes past the row are zero
  __device__ __forceinline__ void copy(uint32_t tile, size_t at, size_t row_bytes) const {
    const uint32_t bytes = at + (lane & 7) * 16 < row_bytes ? 16u : 0u;
#pragma unroll
    for (int i = 0; i < BT / 4; ++i) {
      const int row = 4 * i + (lane >> 3);
      const uint32_t d = tile + static_cast<uint32_t>(row * 128 + (((lane & 7) ^ (row & 7)) << 4));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(bytes ? src[i] + at : src[i]), "r"(bytes)
                   : "memory");
    }
  }
  __device__ __forceinline__ void hand_over(uint32_t bar) const {
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  }
  // the copies of a stage have been issued; the oldest stage in flight is handed over
  __device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (n >= kLag) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kLag) : "memory");
      hand_over(bars[0]);
    }
#pragma unroll
    for (int i = 0; i + 1 < kLag; ++i) bars[i] = bars[i + 1];
    bars[kLag - 1] = bar;
    ++n;
  }
  // everything has landed (also on the way out after a time-out); hands over what is left
  __device__ __forceinline__ void drain() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    fence_proxy_async_smem();
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kLag; ++i)
      if (lane == 0 && n >= kLag - i) mbar_arrive(bars[i]);
  }
};

// The combine buffer is cleared by the kernel before the one that adds to it: `threads` threads of each CTA.
__device__ __forceinline__ void clear_combine_buffer(const GemmArgs& a, int tid, int threads) {
  uint4* z = reinterpret_cast<uint4*>(a.zero);
  const long long step = static_cast<long long>(gridDim.x) * threads;
  for (long long i = static_cast<long long>(blockIdx.x) * threads + tid; i < a.zero_chunks; i += step)
    z[i] = make_uint4(0, 0, 0, 0);
}

}  // namespace b200moe
