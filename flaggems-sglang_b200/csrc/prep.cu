// Row movers around the grouped GEMMs: gather token rows into expert-sorted,
// block-padded order (optionally quantising them to FP8 per 1x128 group),
// and turn the fp32 combine buffer into the 16-bit output.
#include "gemm_route.cuh"
#include "prep.cuh"

namespace b200moe {

namespace {

// A warp copies 2 KiB of a row at a time: one row id, then four 16-byte loads per lane, then the stores.  What bounds it is
// the write to HBM at prefill sizes and two memory latencies at decode (a row id and a 64-bit division per 16-byte chunk
// bound it by its instructions: 32768 rows of 7168 bytes 118 us, 80 like this; a decode graph of the 128-expert layer
// 182.0 and 179.4).  Padding rows are left alone, whatever they hold: every GEMM keeps a row's results to itself and none
// of a padding row's is ever stored where it is read.  (Quantising and zeroing them, three quarters of the rows of a
// 64-token call on 256 experts, cost 8 us of 439.)
// The same launch clears the fp32 combine buffer (`zero`, `zero_chunks`).
// With sc_src: the rows are already quantised (one byte per element) and each has G group scales
// [tokens][G]; they are re-laid group-major for the GEMMs, sc_dst [G][ld].
constexpr int kGatherSeg = 128;      // 16-byte chunks per warp and step

__global__ void __launch_bounds__(256)
gather_rows_kernel(const uint4* __restrict__ x, uint4* __restrict__ xs, const int* __restrict__ sorted_ids,
                   const int* __restrict__ meta, int P, int topk, int chunks_per_row, int cap,
                   uint4* __restrict__ zero, long long zero_chunks, const float* __restrict__ sc_src,
                   float* __restrict__ sc_dst, int G, int ld, const FlagWait fw) {
  griddep_wait();
  griddep_launch_dependents();
  wait_for_peers(fw);     // expert parallelism: the rows come from the peers
  const int rows = min(meta[1], cap);
  const int threads = gridDim.x * blockDim.x;
  const int thread = blockIdx.x * blockDim.x + threadIdx.x;
  if (sc_src != nullptr) {
    // lanes along the rows: a group's scales of 32 rows are one store
    const int blocks = (rows + 31) >> 5;
    for (int u = thread >> 5; u < blocks * G; u += threads >> 5) {
      const int g = u / blocks;
      const int r = ((u - g * blocks) << 5) + (thread & 31);
      if (r >= rows) continue;
      const int slot = sorted_ids[r];
      if (slot >= 0 && slot < P)
        sc_dst[static_cast<size_t>(g) * ld + r] = __ldg(sc_src + static_cast<size_t>(slot / topk) * G + g);
    }
  }
  const int lane = thread & 31;
  const int segs = (chunks_per_row + kGatherSeg - 1) / kGatherSeg;
  const int units = rows * segs;       // (2 KiB each, or a shorter row of at most 2^25: far below 2^31)
  for (int u = thread >> 5; u < units; u += threads >> 5) {
    const int r = u / segs;
    const int slot = sorted_ids[r];
    if (slot < 0 || slot >= P) continue;
    const int c0 = (u - r * segs) * kGatherSeg + lane;
    const uint4* src = x + static_cast<size_t>(slot / topk) * chunks_per_row;
    uint4* dst = xs + static_cast<size_t>(r) * chunks_per_row;
    uint4 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c0 + 32 * q < chunks_per_row) v[q] = __ldg(src + c0 + 32 * q);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c0 + 32 * q < chunks_per_row) dst[c0 + 32 * q] = v[q];
  }
  for (long long i = thread; i < zero_chunks; i += threads) zero[i] = make_uint4(0, 0, 0, 0);
}

// The same for a call whose GEMMs sort the slots themselves (gemm_route.cuh): a warp takes 2 KiB of a slot's row and puts it where
// the GEMMs look for it.
// Padded row of slot i (triple: of the i-th sorted row); -1: no expert here.  Whole warp.
__device__ __forceinline__ int routed_row(const RouteSource& route, const RowTables& t, int P, int E, int BT, int i) {
  if (route.hist == nullptr) {
    const unsigned e = t.ids[ids_at(i)];
    return e == kNoSlot ? -1 : t.blk[e] * BT + slot_rank(t, i, e);
  }
  const int slot = __ldcg(route.topk_indx + i);
  if (i >= t.raw[E] || slot < 0 || slot >= P) return -1;
  int lo = 0, hi = E;         // last expert that starts at or before row i
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (t.raw[mid] <= i) lo = mid; else hi = mid;
  }
  return t.blk[lo] * BT + i - t.raw[lo];
}

__global__ void __launch_bounds__(256)
gather_routed_kernel(const uint4* __restrict__ x, uint4* __restrict__ xs, const RouteSource route, int P, int E, int BT, int topk,
                     int chunks_per_row, uint4* __restrict__ zero, long long zero_chunks) {
  extern __shared__ __align__(16) uint8_t route_smem[];
  const RowTables t = row_tables(route_smem, E);
  griddep_wait();
  griddep_launch_dependents();
  const int threads = gridDim.x * blockDim.x;
  const int thread = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = thread & 31;
  const int segs = (chunks_per_row + kGatherSeg - 1) / kGatherSeg;
  // The first unit's row is on its way while the slots are counted: the next kernel's weights fill the memory's queues by then,
  // and a second trip through them costs 4 us.
  uint4 v[4];
  auto fetch = [&](int u) {
    const int i = u / segs, c0 = (u - i * segs) * kGatherSeg + lane;
    int slot = route.hist == nullptr ? i : __ldcg(route.topk_indx + i);
    if (slot < 0 || slot >= P) slot = 0;
    const uint4* src = x + static_cast<size_t>(slot / topk) * chunks_per_row;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c0 + 32 * q < chunks_per_row) v[q] = __ldg(src + c0 + 32 * q);
  };
  const int units = P * segs;
  int u = thread >> 5;
  if (u < units) fetch(u);
  for (long long i = thread; i < zero_chunks; i += threads) zero[i] = make_uint4(0, 0, 0, 0);
  count_slots(route, P, E, BT, t);
  for (bool first = true; u < units; u += threads >> 5, first = false) {
    if (!first) fetch(u);
    const int i = u / segs;
    const int r = routed_row(route, t, P, E, BT, i);
    if (r < 0) continue;
    const int c0 = (u - i * segs) * kGatherSeg + lane;
    uint4* dst = xs + static_cast<size_t>(r) * chunks_per_row;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c0 + 32 * q < chunks_per_row) dst[c0 + 32 * q] = v[q];
  }
}

template <typename T>
__device__ __forceinline__ void load4(const T* p, float (&v)[4]);
template <>
__device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[4]) {
  uint2 raw = *reinterpret_cast<const uint2*>(p);
  __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&raw.x);
  __nv_bfloat162 b = *reinterpret_cast<__nv_bfloat162*>(&raw.y);
  v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(b); v[3] = __high2float(b);
}
template <>
__device__ __forceinline__ void load4<__half>(const __half* p, float (&v)[4]) {
  uint2 raw = *reinterpret_cast<const uint2*>(p);
  __half2 a = *reinterpret_cast<__half2*>(&raw.x);
  __half2 b = *reinterpret_cast<__half2*>(&raw.y);
  v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(b); v[3] = __high2float(b);
}

// One 128-wide group over a warp: four e4m3 values of this lane; lane u receives the group's scale in `mine`.
// scale = max(amax, eps)/448, q = rne_satfinite(x / scale) with an IEEE divide so that the bits match a CPU restatement.
__device__ __forceinline__ uint32_t quantise_group(const float (&v)[4], int lane, int u, float& mine) {
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
  // non-negative floats order like their bit patterns: one redux instead of five shuffles
  amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
  const float s = __fdiv_rn(fmaxf(amax, 1e-10f), 448.0f);
  if (lane == u) mine = s;
  uint32_t packed = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    packed |= static_cast<uint32_t>(__nv_cvt_float_to_fp8(__fdiv_rn(v[i], s), __NV_SATFINITE, __NV_E4M3)) << (8 * i);
  return packed;
}

// One warp per (row, run of up to eight 128-wide groups): the loads of the run are issued
// together (one 8-byte load per lane and group in flight is too little to cover the memory
// latency), then quantise_group per group.
// sorted_ids == nullptr: rows map to themselves.
// scale_t != 0: scales stored [K/128][ld_scale] (group-major) instead of [rows][K/128].
template <typename T>
__global__ void __launch_bounds__(256)
group_quant_fp8_kernel(const T* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scales,
                       const int* __restrict__ sorted_ids, const int* __restrict__ meta, int P, int topk,
                       int n_rows_static, int K, int scale_t, int ld_scale, uint4* __restrict__ zero,
                       long long zero_chunks) {
  griddep_wait();
  griddep_launch_dependents();
  // clear the fp32 combine buffer alongside (grid-stride, 16 bytes per thread)
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < zero_chunks;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    zero[i] = make_uint4(0, 0, 0, 0);
  constexpr int RUN = 8;
  const int groups = K >> 7;
  const int runs = (groups + RUN - 1) / RUN;
  const int lane = threadIdx.x & 31;
  const int rows = (meta != nullptr) ? min(meta[1], n_rows_static) : n_rows_static;
  const long long total = static_cast<long long>(rows) * runs;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (long long w = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; w < total;
       w += warps) {
    const int r = static_cast<int>(w / runs);
    const int g0 = static_cast<int>(w - static_cast<long long>(r) * runs) * RUN;
    int src_row = r;
    if (sorted_ids != nullptr) {
      const int slot = sorted_ids[r];
      if (slot < 0 || slot >= P) continue;     // padding rows are left alone (see gather_rows_kernel)
      src_row = slot / topk;
    }
    float v[RUN][4];
#pragma unroll
    for (int u = 0; u < RUN; ++u) {
      v[u][0] = v[u][1] = v[u][2] = v[u][3] = 0.f;
      if (g0 + u < groups) load4<T>(x + static_cast<size_t>(src_row) * K + (g0 + u) * 128 + lane * 4, v[u]);
    }
#pragma unroll
    for (int u = 0; u < RUN; ++u) {
      const int g = g0 + u;
      if (g >= groups) break;
      float s = 0.f;
      *reinterpret_cast<uint32_t*>(q + static_cast<size_t>(r) * K + g * 128 + lane * 4) = quantise_group(v[u], lane, 0, s);
      if (lane == 0) {
        if (scale_t) scales[static_cast<size_t>(g) * ld_scale + r] = s;
        else scales[static_cast<size_t>(r) * groups + g] = s;
      }
    }
  }
}

// The quantisation by token: a warp quantises a run of groups once and stores it for each of the token's slots, in the row that
// the alignment gave it (slot_row) or, where the GEMMs sort the slots themselves (gemm_route.cuh), in the one they
// look for.  (Quantising the tokens and gathering the bytes: 4096 tokens of 56 groups, top-8, 38 + 67 us.)  At decode the
// kernel is a few microseconds long, so its loops stay rolled: straight-line code for eight groups and eight slots spent more time being
// fetched than executed (64 tokens of 56 groups, top-8: 18.5 us; an alignment and one warp per slot: 20).
constexpr int kQuantRun = 8;      // groups of a run at most; few tokens are dealt out in shorter ones
template <typename T>
__global__ void __launch_bounds__(256)
group_quant_slots_kernel(const T* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scales, const RouteSource route,
                         const int* __restrict__ slot_row, int P, int E, int BT, int topk, int M, int K, int run, int ld_scale,
                         uint4* __restrict__ zero, long long zero_chunks) {
  extern __shared__ __align__(16) uint8_t route_smem[];
  __shared__ __align__(16) uint2 s_x[8][kQuantRun][32];
  const RowTables t = row_tables(route_smem, E);
  griddep_wait();
  griddep_launch_dependents();
  const int threads = gridDim.x * blockDim.x;
  const int thread = blockIdx.x * blockDim.x + threadIdx.x;
  const int groups = K >> 7, runs = (groups + run - 1) / run, lane = thread & 31;
  uint2(*mine)[32] = s_x[threadIdx.x >> 5];
  auto fetch = [&](int w) {
    const int tok = w / runs, g0 = (w - tok * runs) * run, n = min(run, groups - g0);
    const T* src = x + static_cast<size_t>(tok) * K + g0 * 128 + lane * 4;
#pragma unroll 1
    for (int u = 0; u < n; ++u)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(&mine[u][lane])), "l"(src + u * 128) : "memory");
  };
  // the first run is on its way while the slots are counted: by then the next kernel's weights fill the memory's queues
  int w = thread >> 5;
  if (w < M * runs) fetch(w);
  for (long long i = thread; i < zero_chunks; i += threads) zero[i] = make_uint4(0, 0, 0, 0);
  if (slot_row == nullptr) count_slots(route, P, E, BT, t);
  for (bool first_run = true; w < M * runs; w += threads >> 5, first_run = false) {
    if (!first_run) fetch(w);
    const int tok = w / runs, g0 = (w - tok * runs) * run, n = min(run, groups - g0);
    asm volatile("cp.async.wait_all;" ::: "memory");        // (a lane reads only what it copied)
    for (int j0 = 0; j0 < topk; j0 += 32) {
      const int nj = min(32, topk - j0);
      int row = -1;             // lane j: padded row of the token's slot j0 + j
      if (slot_row != nullptr && lane < nj) row = slot_row[tok * topk + j0 + lane];
#pragma unroll 1
      for (int j = 0; slot_row == nullptr && j < nj; ++j) {
        const int slot = tok * topk + j0 + j;
        const unsigned e = t.ids[ids_at(slot)];
        const int rank = e == kNoSlot ? -1 : slot_rank(t, slot, e);
        if (lane == j && rank >= 0) row = t.blk[e] * BT + rank;
      }
#pragma unroll 1
      for (int u = 0; u < n; ++u) {
        float v[4];
        load4<T>(reinterpret_cast<const T*>(&mine[u][lane]), v);
        float scale = 0.f;
        const uint32_t packed = quantise_group(v, 0, 0, scale);      // (every lane has the scale)
#pragma unroll 1
        for (int j = 0; j < nj; ++j) {
          const int r = __shfl_sync(0xffffffffu, row, j);
          if (r >= 0) *reinterpret_cast<uint32_t*>(q + static_cast<size_t>(r) * K + (g0 + u) * 128 + lane * 4) = packed;
        }
        if (row >= 0) scales[static_cast<size_t>(g0 + u) * ld_scale + row] = scale;
      }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
finalize_kernel(const float4* __restrict__ acc, T* __restrict__ out, size_t n4, float scale, const FlagWait fw) {
  griddep_wait();
  griddep_launch_dependents();
  wait_for_peers(fw);
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    float4 v = acc[i];
    T o[4] = {from_f32<T>(v.x * scale), from_f32<T>(v.y * scale), from_f32<T>(v.z * scale),
              from_f32<T>(v.w * scale)};
    *reinterpret_cast<uint2*>(out + i * 4) = *reinterpret_cast<uint2*>(o);
  }
}

// One thread per (token, run of 8 columns): fp32 sum of the token's valid pair rows.
template <typename T>
__global__ void __launch_bounds__(256)
finalize_pairs_kernel(const uint4* __restrict__ pairs, const uint8_t* __restrict__ pair_valid, uint4* __restrict__ out,
                      int M, int topk, int chunks_per_row, float scale, const FlagWait fw) {
  griddep_wait();
  griddep_launch_dependents();
  wait_for_peers(fw);
  const long long total = static_cast<long long>(M) * chunks_per_row;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(i / chunks_per_row);
    const int c = static_cast<int>(i - static_cast<long long>(t) * chunks_per_row);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // four pairs at a time: the validity bytes first, then the row chunks, so that the loads of a
    // batch are in flight together
    for (int j0 = 0; j0 < topk; j0 += 4) {
      uint4 v[4];
      bool ok[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const size_t slot = static_cast<size_t>(t) * topk + j0 + u;
        ok[u] = (j0 + u < topk) && pair_valid[slot] != 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const size_t slot = static_cast<size_t>(t) * topk + j0 + u;
        v[u] = ok[u] ? __ldg(pairs + slot * chunks_per_row + c) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const T* e = reinterpret_cast<const T*>(&v[u]);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] += to_f32<T>(e[k]);   // zeros for pairs that are not there
      }
    }
    T o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = from_f32<T>(acc[k] * scale);
    out[i] = *reinterpret_cast<uint4*>(o);
  }
}

}  // namespace

int launch_finalize_pairs(const void* pairs, const uint8_t* pair_valid, void* out, int dtype, int M, int topk,
                          int H, float scale, int num_sms, cudaStream_t stream, bool pdl, const FlagWait* wait) {
  FlagWait fw = {};
  if (wait != nullptr) fw = *wait;
  if (H % 8 != 0) return B200MOE_ERR_UNSUPPORTED;
  const long long total = static_cast<long long>(M) * (H / 8);
  long long ctas = (total + 255) / 256;
  if (ctas > static_cast<long long>(num_sms) * 16) ctas = static_cast<long long>(num_sms) * 16;
  if (ctas < 1) ctas = 1;
  cudaError_t err;
  note_launch("finalize_pairs_kernel");
  if (dtype == B200MOE_DTYPE_BF16)
    err = launch_kernel(finalize_pairs_kernel<__nv_bfloat16>, dim3(static_cast<unsigned>(ctas)), dim3(256), 0, stream,
                        pdl, reinterpret_cast<const uint4*>(pairs), pair_valid, reinterpret_cast<uint4*>(out), M, topk,
                        H / 8, scale, fw);
  else
    err = launch_kernel(finalize_pairs_kernel<__half>, dim3(static_cast<unsigned>(ctas)), dim3(256), 0, stream, pdl,
                        reinterpret_cast<const uint4*>(pairs), pair_valid, reinterpret_cast<uint4*>(out), M, topk, H / 8,
                        scale, fw);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

int launch_gather_rows(const void* x, void* xs, const int* sorted_ids, const int* meta, int P, int topk,
                       int row_bytes, int cap, void* zero, size_t zero_bytes, int num_sms,
                       cudaStream_t stream, bool pdl, const float* sc_src, float* sc_dst, int G, int ld,
                       const FlagWait* wait) {
  FlagWait fw = {};
  if (wait != nullptr) fw = *wait;
  if (row_bytes % 16 != 0 || zero_bytes % 16 != 0) return B200MOE_ERR_UNSUPPORTED;
  const int segs = (row_bytes / 16 + kGatherSeg - 1) / kGatherSeg;
  const long long copy_warps = static_cast<long long>(cap) * segs, zero_threads = static_cast<long long>(zero_bytes / 16);
  long long ctas = (copy_warps * 32 > zero_threads ? copy_warps * 32 + 255 : zero_threads + 255) / 256;
  if (ctas > static_cast<long long>(num_sms) * 8) ctas = static_cast<long long>(num_sms) * 8;
  if (ctas < 1) ctas = 1;
  note_launch("gather_rows_kernel");
  cudaError_t err = launch_kernel(gather_rows_kernel, dim3(static_cast<unsigned>(ctas)), dim3(256), 0, stream, pdl,
                                  reinterpret_cast<const uint4*>(x), reinterpret_cast<uint4*>(xs), sorted_ids, meta,
                                  P, topk, row_bytes / 16, cap, reinterpret_cast<uint4*>(zero),
                                  static_cast<long long>(zero_bytes / 16), sc_src, sc_dst, G, ld, fw);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

int launch_gather_routed(const void* x, void* xs, const RouteSource& route, int P, int E, int BT, int topk, int row_bytes, void* zero,
                         size_t zero_bytes, int num_sms, cudaStream_t stream, bool pdl) {
  if (row_bytes % 16 != 0 || zero_bytes % 16 != 0) return B200MOE_ERR_UNSUPPORTED;
  const size_t smem = route_table_bytes(E, P);
  if (smem > 48 * 1024) return B200MOE_ERR_TOO_LARGE;
  const int segs = (row_bytes / 16 + kGatherSeg - 1) / kGatherSeg;
  int ctas = (P * segs + 7) / 8;
  if (ctas > 2 * num_sms) ctas = 2 * num_sms;
  if (ctas < 1) ctas = 1;
  note_launch("gather_routed_kernel");
  cudaError_t err = launch_kernel(gather_routed_kernel, dim3(ctas), dim3(256), smem, stream, pdl, reinterpret_cast<const uint4*>(x),
                                  reinterpret_cast<uint4*>(xs), route, P, E, BT, topk, row_bytes / 16,
                                  reinterpret_cast<uint4*>(zero), static_cast<long long>(zero_bytes / 16));
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

int launch_group_quant_fp8(const void* x, int dtype, void* q, float* scales, const int* sorted_ids,
                           const int* meta, int P, int topk, int rows, int K, int scale_t, int ld_scale,
                           void* zero, size_t zero_bytes, int num_sms, cudaStream_t stream, bool pdl) {
  if (K % 128 != 0 || zero_bytes % 16 != 0) return B200MOE_ERR_UNSUPPORTED;
  long long warps = static_cast<long long>(rows) * ((K / 128 + 7) / 8);
  long long ctas = (warps + 7) / 8;
  if (ctas > num_sms * 16) ctas = num_sms * 16;
  if (ctas < 1) ctas = 1;
  cudaError_t err;
  const long long zc = static_cast<long long>(zero_bytes / 16);
  note_launch("group_quant_fp8_kernel");
  if (dtype == B200MOE_DTYPE_BF16)
    err = launch_kernel(group_quant_fp8_kernel<__nv_bfloat16>, dim3(static_cast<unsigned>(ctas)), dim3(256), 0, stream,
                        pdl, reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<uint8_t*>(q), scales,
                        sorted_ids, meta, P, topk, rows, K, scale_t, ld_scale, reinterpret_cast<uint4*>(zero), zc);
  else
    err = launch_kernel(group_quant_fp8_kernel<__half>, dim3(static_cast<unsigned>(ctas)), dim3(256), 0, stream, pdl,
                        reinterpret_cast<const __half*>(x), reinterpret_cast<uint8_t*>(q), scales, sorted_ids, meta, P,
                        topk, rows, K, scale_t, ld_scale, reinterpret_cast<uint4*>(zero), zc);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

int launch_group_quant_slots(const void* x, int dtype, void* q, float* scales, const RouteSource& route, const int* slot_row, int P,
                             int E, int BT, int topk, int M, int K, int ld_scale, void* zero, size_t zero_bytes, int num_sms,
                             cudaStream_t stream, bool pdl) {
  const size_t smem = slot_row != nullptr ? 16 : route_table_bytes(E, P);
  if (K % 128 != 0 || zero_bytes % 16 != 0 || route.hist != nullptr) return B200MOE_ERR_UNSUPPORTED;
  if (smem > 30 * 1024) return B200MOE_ERR_TOO_LARGE;
  const int groups = K / 128;
  int run = (M * groups + 16 * num_sms - 1) / (16 * num_sms);
  if (run > kQuantRun) run = kQuantRun;
  int ctas = (M * ((groups + run - 1) / run) + 7) / 8;
  const int most = (slot_row != nullptr ? 8 : 2) * num_sms;      // (few where each CTA counts the slots first)
  if (ctas > most) ctas = most;
  if (ctas < 1) ctas = 1;
  const long long zc = static_cast<long long>(zero_bytes / 16);
  note_launch("group_quant_slots_kernel");
  cudaError_t err;
  if (dtype == B200MOE_DTYPE_BF16)
    err = launch_kernel(group_quant_slots_kernel<__nv_bfloat16>, dim3(ctas), dim3(256), smem, stream, pdl,
                        reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<uint8_t*>(q), scales, route, slot_row, P, E,
                        BT, topk, M, K, run, ld_scale, reinterpret_cast<uint4*>(zero), zc);
  else
    err = launch_kernel(group_quant_slots_kernel<__half>, dim3(ctas), dim3(256), smem, stream, pdl,
                        reinterpret_cast<const __half*>(x), reinterpret_cast<uint8_t*>(q), scales, route, slot_row, P, E, BT,
                        topk, M, K, run, ld_scale, reinterpret_cast<uint4*>(zero), zc);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

int launch_finalize(const float* acc, void* out, int dtype, size_t n, float scale, int num_sms,
                    cudaStream_t stream, bool pdl, const FlagWait* wait) {
  FlagWait fw = {};
  if (wait != nullptr) fw = *wait;
  if (n % 4 != 0) return B200MOE_ERR_UNSUPPORTED;
  size_t n4 = n / 4;
  size_t ctas = (n4 + 255) / 256;
  if (ctas > static_cast<size_t>(num_sms) * 8) ctas = static_cast<size_t>(num_sms) * 8;
  if (ctas < 1) ctas = 1;
  cudaError_t err;
  note_launch("finalize_kernel");
  if (dtype == B200MOE_DTYPE_BF16)
    err = launch_kernel(finalize_kernel<__nv_bfloat16>, dim3(static_cast<unsigned>(ctas)), dim3(256), 0, stream, pdl,
                        reinterpret_cast<const float4*>(acc), reinterpret_cast<__nv_bfloat16*>(out), n4, scale, fw);
  else
    err = launch_kernel(finalize_kernel<__half>, dim3(static_cast<unsigned>(ctas)), dim3(256), 0, stream, pdl,
                        reinterpret_cast<const float4*>(acc), reinterpret_cast<__half*>(out), n4, scale, fw);
  return err == cudaSuccess ? B200MOE_OK : B200MOE_ERR_CUDA;
}

}  // namespace b200moe
