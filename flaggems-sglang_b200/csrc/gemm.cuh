// Grouped expert GEMMs: argument block and launchers.
#pragma once
#include "common.cuh"

namespace b200moe {

// Orientation: the expert weight tile sits on the 128-row side of the tensor-core
// instruction and the (block of) tokens on its N side, so a decode-sized token
// block of 16 wastes nothing and a prefill block of 256 fills the widest shape.
constexpr int kMaxPeers = 8;   // ranks of one NVSwitch domain that an expert-parallel call may span

// Routing input of a call whose GEMMs sort the slots by expert themselves (gemm_route.cuh).
struct RouteSource {
  int own;                   // 1: they do; 0: the tables come from an alignment launch, the rows lie in expert order
  int early;                 // own: a kernel of this call lies between the routing input and this one (see griddep_wait below)
  const void* ids;           // [P] expert of each slot, with an optional global -> local map
  int is64;
  const int* map;
  int map_len;
  const float* weights;      // [P]
  const int* hist;           // or the routing triple: slots per expert, slots by expert, their weights
  const int* topk_indx;
  const float* gate_scal;
};

struct GemmArgs {
  int mode;        // 0: gate/up projection + activation; 1: down projection + weighted scatter-add
  int dtype;       // B200MOE_DTYPE_* of activations / 16-bit weights
  int wmode;       // B200MOE_W_*
  int E;           // local experts
  int K;           // reduction length (H for mode 0, I for mode 1)
  int N;           // output rows per expert covered by tiles of 128 (I for mode 0, H for mode 1)
  int up_row_off;  // mode 0: row of the first "up" weight inside an expert (= I)
  int orient;      // 0: weight rows on the MMA's M side (decode); 1: tokens on the M side (BT = 128); 2: CTA pairs
  int BT;          // tokens per block (16..256, multiple of 16); CTA pairs, w4_var: upper bound of the tokens per tile
  int w4_var;      // int4: 1 = tiles of a variable number of tokens (16..192), 0 = decode blocks of BT (16 or 32) tokens
  int stages;      // shared-memory ring depth
  int table_off;   // FP8 blocks of 128: where the block tables stand in shared memory
  int stages_cold; // FP8 blocks of 128: the same of the CTAs that take the blocks of at most 16 tokens
  int acc_stages;  // accumulator buffers in tensor memory (1 or 2)
  int tmem_cols;   // allocated tensor-memory columns (power of two >= 32)
  int num_nt;      // ceil(N / 128)
  int kblocks;     // ceil(K / kblock elements)
  int topk;
  int P;           // M * topk
  int flags;       // B200MOE_FLAG_*
  int activation;  // B200MOE_ACT_*
  int max_split;   // mode 1: upper bound for the reduction split
  int pdl;         // launch with programmatic stream serialisation
  const int* meta;        // [0] = token blocks, [1] = padded rows
  const int* blk_off;     // [E+1] first block of each expert
  const int* sorted_ids;  // [cap] slot of each padded row (>= P: padding)
  const float* row_gamma; // [cap] routing weight of each padded row
  void* out;              // mode 0: activations [cap, N]; mode 1: fp32 combine buffer [M, N]
  long long ld_out;       // row stride of out in elements
  int* status;            // device status word
  // FP8 block-scaled mode
  const float* w_scale;   // [E, ceil(rows/128), ceil(K/128)] (rows = 2I for mode 0)
  const float* x_scale;   // [K/128][ld_xscale] group-major activation scales
  int ld_xscale;
  int w_scale_rows;       // scale rows per expert
  const float* bias;      // optional per-expert bias of this GEMM's output rows: [E, rows] fp32 (mode 0: gate rows then up rows)
  float act_alpha;        // B200MOE_ACT_SWIGLU_OAI: s = g * sigmoid(alpha * g)
  float act_limit;        // B200MOE_ACT_SWIGLU_OAI: clamp gate to <= limit and linear to [-limit, limit]; <= 0: none
  uint8_t* out_q;         // mode 0 FP8: quantised activations [cap, N]
  float* out_scale;       // mode 0 FP8: [N/128][ld_xscale]
  // mode 1, optional: instead of adding into the fp32 combine buffer, store each (token, choice)
  // pair's weighted row in the 16-bit type at out_pairs[slot][N] and mark pair_valid[slot]; the
  // output conversion then sums a token's rows.  Plain 16-byte stores instead of fp32 atomics,
  // which bound the tail once M * topk * N is large.  Requires an unsplit reduction.
  void* out_pairs;
  uint8_t* pair_valid;
  // mode 1 under expert parallelism (FP8 kernels): the output row of a token (fp32 combine buffer)
  // or of a pair (16-bit pair rows) lives on the rank that owns the token.  Output row index r
  // (token, or pair slot, numbered rank-major over all ranks) -> rank r / rows_per_peer, row
  // r % rows_per_peer of that rank's buffer, reached through its peer mapping.  n_peers <= 1:
  // everything stays in `out` / `out_pairs` of this GPU.
  int n_peers;
  int rows_per_peer;
  void* peer_out[kMaxPeers];          // out (fp32) or out_pairs (16-bit) of every rank
  uint8_t* peer_valid[kMaxPeers];     // pair_valid of every rank (pair rows only)
  RouteSource route;
  const void* rows;       // mode 0, route.own: the token rows
  void* zero;             // mode 0, route.own: the combine buffer, cleared here
  long long zero_chunks;  // of 16 bytes
};

// Base address of output row `orow` (row_bytes bytes per row): local, or on the owning rank.
__device__ __forceinline__ uint8_t* out_row_base(const GemmArgs& a, void* local, int orow, size_t row_bytes) {
  if (a.n_peers <= 1) return reinterpret_cast<uint8_t*>(local) + static_cast<size_t>(orow) * row_bytes;
  const int peer = orow / a.rows_per_peer;
  return reinterpret_cast<uint8_t*>(a.peer_out[peer]) + static_cast<size_t>(orow - peer * a.rows_per_peer) * row_bytes;
}
__device__ __forceinline__ void mark_pair_valid(const GemmArgs& a, int slot) {
  if (a.n_peers <= 1) {
    a.pair_valid[slot] = 1;
  } else {
    const int peer = slot / a.rows_per_peer;
    a.peer_valid[peer][slot - peer * a.rows_per_peer] = 1;
  }
}

size_t gemm_smem_bytes(const GemmArgs& a);
void gemm_plan(GemmArgs* a);  // fills stages / acc_stages / tmem_cols / num_nt / kblocks from the rest

int launch_gemm_tc(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const GemmArgs& a, int num_sms,
                   cudaStream_t stream);
void gemm_plan_fp8(GemmArgs* a);
// tm_xc (blocks of 128): boxes of 16 rows for blocks that hold no more
int launch_gemm_fp8(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const CUtensorMap& tm_xc, const GemmArgs& a, int num_sms,
                    cudaStream_t stream);
// int4 AWQ: see gemm_w4.cu.  Token maps: boxes of 16 (i + 1) rows x the 64-k halves of a group;
// decode blocks use m[0] (their rows, two groups).
struct W4TokenMaps {
  CUtensorMap m[12];
};
bool gemm_w4_ok(int E);
bool gemm_w4_own_ok(int E, int P, int BT);
void gemm_plan_w4(GemmArgs* a);
// tm_w: packed rows, mode 0 [E][I][2][K/2] in boxes of 64 rows of both halves, mode 1 [E][rows][K/2] in boxes of 128
// rows; tm_sz: their scale / zero words [E * K/128][2][I] in boxes of 64 of both halves, or [E * K/128][1][rows] in boxes of 128
int launch_gemm_w4(const CUtensorMap& tm_w, const CUtensorMap& tm_sz, const W4TokenMaps& tm_x, const GemmArgs& a,
                   int num_sms, cudaStream_t stream);
// 16-bit, more than 25 tokens per expert, on CTA pairs (tcgen05.mma.cta_group::2): see gemm_tc2.cu
bool gemm_tc2_ok(int E, int num_sms);
int gemm_tc2_resident_pairs();   // CTA pairs the device kept resident for the last such launch (0: none yet)
void gemm_plan_tc2(GemmArgs* a);
// Token maps of a pair launch: m[i] has boxes of 16 (i + 1) rows, half of a tile of 32 (i + 1) tokens.
struct PairTokenMaps {
  CUtensorMap m[8];
};
// tm_w: mode 0 [E][2][I][K] in boxes of 64 rows of both halves, mode 1 [E][rows][K] in boxes of 128 rows
int launch_gemm_tc2(const CUtensorMap& tm_w, const PairTokenMaps& tm_x, const GemmArgs& a, int num_sms,
                    cudaStream_t stream);
int launch_gemm_simt(const void* w, const void* x, const GemmArgs& a, cudaStream_t stream, int cap);

}  // namespace b200moe
