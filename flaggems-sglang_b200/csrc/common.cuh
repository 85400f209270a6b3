// Shared device helpers: mbarrier, TMA and tcgen05 wrappers for sm_100a.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/b200moe.h"

namespace b200moe {

// Device-side status codes written to the caller's status word.
enum DevStatus : int {
  DEV_OK = 0,
  DEV_TIMEOUT_PRODUCER = 101,
  DEV_TIMEOUT_MMA = 102,
  DEV_TIMEOUT_EPILOGUE = 103,
  DEV_TIMEOUT_PEER = 104,      // a flag another rank raises (expert parallelism) did not arrive
  DEV_TIMEOUT_SELFTEST = 105,  // the wait the self-test lets run out on purpose
};

// A wait gives up after this many nanoseconds of wall clock.
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31; }

// Index of the thread's warp as a value the compiler knows to be the same for the whole warp.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0); }
// True in exactly one lane of a converged warp.  The role threads that issue TMA loads and MMAs are
// picked with it rather than with `lane == 0`: a branch on elect.sync is one the compiler knows to
// hold a single thread, and it then issues the operands of a tcgen05.mma without a loop over the
// active lanes.  Four dependent MMAs with a commit and a wait per stage: 137 cycles per MMA behind
// `lane == 0`, 99 behind elect.sync (128 x 128 x 16; the tensor core itself needs 64).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_inval(uint32_t bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: returns false when the CTA-wide abort flag is raised or `limit_ns` of wall clock
// ran out (it then raises the flag itself).
__device__ __forceinline__ bool mbar_wait_limit(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code,
                                                unsigned long long limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  unsigned long long t0 = 0;
#pragma unroll 1
  for (uint32_t spin = 1;; ++spin) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spin & 0xff) == 0) {
      if (*abort_flag) return false;
      unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > limit_ns) {
        *abort_flag = code;
        return false;
      }
    }
  }
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int code) {
  return mbar_wait_limit(bar, parity, abort_flag, code, kWaitLimitNs);
}

// Wait with optional stall accounting (development builds with -DB200MOE_STALL_STATS): the
// cycles spent in the wait are added to `acc`.
__device__ __forceinline__ bool mbar_wait_t(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code,
                                            unsigned long long& acc) {
#ifdef B200MOE_STALL_STATS
  const long long t0 = clock64();
  const bool ok = mbar_wait(bar, parity, abort_flag, code);
  acc += static_cast<unsigned long long>(clock64() - t0);
  return ok;
#else
  (void)acc;
  return mbar_wait(bar, parity, abort_flag, code);
#endif
}

// Meeting point of several warps with a bounded wait, in place of a named bar.sync (which would
// hang the CTA if one of the warps had given up on a time-out): `bar` is an mbarrier initialised to
// the number of warps, lane 0 of each arrives, `phase` is the caller's running parity.
__device__ __forceinline__ bool warps_meet(uint32_t bar, uint32_t& phase, int lane, volatile int* abort_flag,
                                           int code) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
  const bool ok = mbar_wait(bar, phase, abort_flag, code);
  phase ^= 1u;
  return ok;
}

// Short bounded wait used on the abort path to let copies in flight land.
__device__ __forceinline__ void mbar_wait_brief(uint32_t bar, uint32_t parity) {
#pragma unroll 1
  for (int spin = 0; spin < 4096; ++spin) {
    if (mbar_try_wait(bar, parity)) return;
  }
}

// ---------------------------------------------------------------- TMA (tiled bulk tensor loads)
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0,
                                            int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
      "[%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0,
                                            int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, "
      "%5}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2,
                                            int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// Untiled bulk copy global -> shared (both addresses 16-byte aligned, size a multiple of 16),
// completing on an mbarrier like the tiled loads.
__device__ __forceinline__ void bulk_copy_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
      : "memory");
}

// ---------------------------------------------------------------- tcgen05 / tensor memory
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Arrive on an mbarrier once every MMA issued so far by this thread has finished.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]; 16-bit inputs, fp32 accumulate.
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                           uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Same with the A operand read from tensor memory (lane = row, 32-bit columns hold two
// consecutive k) instead of shared memory.
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[smem] * B[smem] for 8-bit float inputs (e4m3 / e5m2).
__device__ __forceinline__ void tc_mma_f8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Each thread of the warp reads 16 consecutive fp32 columns of its own TMEM lane.  The load
// and the wait for it sit in one asm statement so that no use of the registers can be
// scheduled in between.
#define B200MOE_R16(r, o)                                                                            \
  "=r"(r[o + 0]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]),   \
      "=r"(r[o + 6]), "=r"(r[o + 7]), "=r"(r[o + 8]), "=r"(r[o + 9]), "=r"(r[o + 10]),              \
      "=r"(r[o + 11]), "=r"(r[o + 12]), "=r"(r[o + 13]), "=r"(r[o + 14]), "=r"(r[o + 15])

__device__ __forceinline__ void tmem_ld16_wait(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
      "%13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : B200MOE_R16(r, 0)
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Two loads (e.g. gate and up accumulators) in flight before the single wait.
__device__ __forceinline__ void tmem_ld16x2_wait(uint32_t taddr0, uint32_t taddr1, float (&v0)[16],
                                                 float (&v1)[16]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
      "%13, %14, %15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, "
      "%27, %28, %29, %30, %31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : B200MOE_R16(r, 0), B200MOE_R16(r, 16)
      : "r"(taddr0), "r"(taddr1)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v0[i] = __uint_as_float(r[i]);
    v1[i] = __uint_as_float(r[16 + i]);
  }
}

// Raw 32-bit words of a 16-column read (for packed f32x2 arithmetic on register pairs).
__device__ __forceinline__ void tmem_ld16_wait_u32(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
      "%13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : B200MOE_R16(r, 0)
      : "r"(taddr)
      : "memory");
}

#define B200MOE_R32(r, o) B200MOE_R16(r, o), B200MOE_R16(r, o + 16)
// Two 32-column loads in flight before the single wait.
__device__ __forceinline__ void tmem_ld32x2_wait(uint32_t taddr0, uint32_t taddr1, float (&v0)[32],
                                                 float (&v1)[32]) {
  uint32_t r[64];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%64];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, "
      "%44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, "
      "[%65];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : B200MOE_R32(r, 0), B200MOE_R32(r, 32)
      : "r"(taddr0), "r"(taddr1)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    v0[i] = __uint_as_float(r[i]);
    v1[i] = __uint_as_float(r[32 + i]);
  }
}

// Shared-memory matrix descriptor: rows of 128 bytes (reduction dim contiguous),
// 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_k_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFF) >> 4);  // start address, 16-byte units
  d |= static_cast<uint64_t>(1) << 16;                 // leading byte offset (unused for swizzled K-major)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;         // stride byte offset between 8-row groups
  d |= static_cast<uint64_t>(1) << 46;                 // descriptor version for sm_100
  d |= static_cast<uint64_t>(2) << 61;                 // 128-byte swizzle
  return d;
}

// Instruction descriptor: fp32 accumulate, A and B both with the reduction dim
// contiguous, M x N tile.  fmt: 0 = fp16, 1 = bf16 (kind::f16); 0 = e4m3 (kind::f8f6f4).
__host__ __device__ __forceinline__ uint32_t make_idesc(uint32_t fmt, uint32_t m, uint32_t n) {
  uint32_t d = 0;
  d |= 1u << 4;           // accumulator format fp32
  d |= (fmt & 7u) << 7;   // A format
  d |= (fmt & 7u) << 10;  // B format
  d |= (n >> 3) << 17;
  d |= (m >> 4) << 24;
  return d;
}

// Two fp32 fused multiply-adds in one instruction (packed f32x2, sm_100) on accumulators that stay
// packed, two fp32 to a 64-bit register, across a whole reduction loop, so that no pack / unpack
// moves surround the instruction: c += {a0, a1} * s2.
__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void ffma2_packed(unsigned long long& c, uint32_t a0, uint32_t a1, unsigned long long s2) {
  asm("{\n\t.reg .b64 ra;\n\t"
      "mov.b64 ra, {%1, %2};\n\t"
      "fma.rn.f32x2 %0, ra, %3, %0;\n\t}"
      : "+l"(c)
      : "r"(a0), "r"(a1), "l"(s2));
}

// Programmatic dependent launch: a kernel launched with the stream-serialisation attribute may
// start while its predecessor still runs; everything it does before griddep_wait() must not
// touch global memory the predecessor writes.  Without the attribute both are no-ops.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// ---------------------------------------------------------------- flags raised by other ranks
// Expert parallelism: a kernel that consumes what the peers wrote first waits until every peer's
// epoch flag (in THIS rank's memory, written by the peers with release stores) has reached this
// rank's own epoch.  world == 0: nothing to wait for.  The wait is bounded; when it runs out the
// status word receives DEV_TIMEOUT_PEER and the kernel goes on (its output is then meaningless,
// the context stays usable).
struct FlagWait {
  const unsigned long long* flags;   // [world]
  const unsigned long long* epoch;   // this rank's epoch counter
  int world;
  unsigned long long limit_ns;
  int* status;
};
__device__ __forceinline__ unsigned long long ld_acquire_sys_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// Called by every thread of a CTA (after griddep_wait); contains a __syncthreads.
__device__ __forceinline__ void wait_for_peers(const FlagWait& w) {
  if (w.world <= 0) return;
  // a wait that already ran out in this call (another CTA, an earlier kernel) is not repeated
  if (static_cast<int>(threadIdx.x) < w.world && *reinterpret_cast<const volatile int*>(w.status) == 0) {
    const unsigned long long want = *reinterpret_cast<const volatile unsigned long long*>(w.epoch);
    const unsigned long long* f = w.flags + threadIdx.x;
    unsigned long long t0 = 0;
#pragma unroll 1
    for (unsigned int spin = 0;; ++spin) {
      if (ld_acquire_sys_u64(f) >= want) break;
      if ((spin & 0x3f) == 0x3f) {
        const unsigned long long now = globaltimer_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 > w.limit_ns) {
          atomicCAS(w.status, 0, static_cast<int>(DEV_TIMEOUT_PEER));
          break;
        }
      }
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------- host: launch accounting
// Every launcher names the kernel it starts; the C ABI reports the total and the kernels of the
// most recent forward call (b200moe_launch_stats), so that benchmarks count launches instead of
// mirroring the launch logic.
void note_launch(const char* name);

// ---------------------------------------------------------------- host: launch with / without PDL
// cluster > 1: CTAs per cluster along x
template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel_cluster(void (*kernel)(KArgs...), dim3 grid, int cluster, dim3 block, size_t smem,
                                         cudaStream_t stream, bool pdl, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                 bool pdl, Args&&... args) {
  return launch_kernel_cluster(kernel, grid, 1, block, smem, stream, pdl, static_cast<Args&&>(args)...);
}

// ---------------------------------------------------------------- small math helpers
template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) {
  return __bfloat162float(v);
}
template <>
__device__ __forceinline__ float to_f32<__half>(__half v) {
  return __half2float(v);
}
template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}
template <>
__device__ __forceinline__ __half from_f32<__half>(float v) {
  return __float2half_rn(v);
}

__device__ __forceinline__ float gelu_f32(float g) {
  return 0.5f * g * (1.0f + erff(g * 0.70710678118654752f));
}

}  // namespace b200moe
