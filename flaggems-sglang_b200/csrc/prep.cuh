// Host-callable launchers of the row movers around the grouped GEMMs.
#pragma once
#include "gemm.cuh"

namespace b200moe {

// xs[r] = x[sorted_ids[r] / topk] for r < meta[1]; padding rows are left alone.  Also clears
// `zero_bytes` bytes at `zero` (the fp32 combine buffer) in the same launch.  With sc_src
// ([tokens][G] group scales of already quantised rows) the scales follow their rows into the
// group-major table sc_dst [G][ld].  `wait` (expert parallelism): every CTA first waits for the
// peers' flags (common.cuh: FlagWait).
int launch_gather_rows(const void* x, void* xs, const int* sorted_ids, const int* meta, int P, int topk,
                       int row_bytes, int cap, void* zero, size_t zero_bytes, int num_sms,
                       cudaStream_t stream, bool pdl, const float* sc_src = nullptr, float* sc_dst = nullptr,
                       int G = 0, int ld = 0, const FlagWait* wait = nullptr);

// The same from the routing input, for calls whose GEMMs sort the slots themselves (gemm_route.cuh).
int launch_gather_routed(const void* x, void* xs, const RouteSource& route, int P, int E, int BT, int topk, int row_bytes, void* zero,
                         size_t zero_bytes, int num_sms, cudaStream_t stream, bool pdl);

// The quantisation by token (FP8 weights): rows as above, or slot_row[slot] where that is given (-1: none).
int launch_group_quant_slots(const void* x, int dtype, void* q, float* scales, const RouteSource& route, const int* slot_row, int P,
                             int E, int BT, int topk, int M, int K, int ld_scale, void* zero, size_t zero_bytes, int num_sms,
                             cudaStream_t stream, bool pdl);

// Per-token-group (1x128) FP8 quantisation, optionally gathering rows through
// sorted_ids like launch_gather_rows.  scale_t: store scales group-major.
int launch_group_quant_fp8(const void* x, int dtype, void* q, float* scales, const int* sorted_ids,
                           const int* meta, int P, int topk, int rows, int K, int scale_t, int ld_scale,
                           void* zero, size_t zero_bytes, int num_sms, cudaStream_t stream, bool pdl);

// out[i] = cast(acc[i] * scale)
// `wait` (expert parallelism): every CTA first waits for the peers' flags (common.cuh: FlagWait).
int launch_finalize(const float* acc, void* out, int dtype, size_t n, float scale, int num_sms,
                    cudaStream_t stream, bool pdl, const FlagWait* wait = nullptr);

// out[t][c] = cast(scale * sum_j pairs[t * topk + j][c]) over the pairs marked valid.
int launch_finalize_pairs(const void* pairs, const uint8_t* pair_valid, void* out, int dtype, int M, int topk,
                          int H, float scale, int num_sms, cudaStream_t stream, bool pdl,
                          const FlagWait* wait = nullptr);

// Provokes a device-side time-out on purpose (see selftest.cu): observed[0] = 0 when the short wait
// ran out, observed[1] = 0 when the sibling wait was released by the abort flag, observed[2] = the
// microseconds the sibling waited; the status word receives DEV_TIMEOUT_SELFTEST.
int launch_selftest_timeout(unsigned long long limit_ns, int* status, int* observed, cudaStream_t stream);

}  // namespace b200moe
