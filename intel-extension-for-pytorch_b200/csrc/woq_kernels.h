// Internal interface between the C ABI (woq_capi.cu) and the kernel translation units.
#pragma once
#include <cuda.h>

#include "woq_common.cuh"

namespace woq {

// ---- tensor-parallel exchange fused into the decode kernel's epilogue ---------------------
// Every rank of one node owns a "symmetric" buffer with the same layout and maps all peers'
// buffers (CUDA IPC).  Layout of one buffer:
//   [0, 4096)               control words: epoch (u32 @0), finished CTAs of the running grid (u32 @4)
//   [4096, +slot_n*2048)    exchange words {2 x bf16, stamp}, 8 bytes each:
//                           [epoch & 3][source rank][tile][token][lane]
//   [gather_off, ..)        gather area (the caller places gathered tensors here)
// A launch with a comm mode is one "epoch" (the same number on every rank, because all ranks
// issue the same sequence of launches); its stamp is epoch + 1.  The warp that finishes a
// tile stores each lane's two results and the stamp as one 8-byte word into every other
// rank's slot (data and mark arrive together, no fence).
//   all-reduce: the same warp then reads its own slots for the other ranks' words of the same
//     tile (all ranks' loads in flight together) and adds them in rank order;
//   all-gather: nobody waits.  The NEXT launch on the comm (or comm_fence) copies the words of
//     the other ranks into this rank's gathered tensor with its otherwise idle epilogue warps,
//     while its own weights stream: the gathered tensor is complete when that launch ends.
// Four slot sets, indexed by epoch & 3: finishing the launch of epoch X takes every peer's
// words of epoch X - 1 at least, so a rank that writes set E & 3 knows every peer has finished
// the launches up to E - 3, and with them the reading of epoch E - 4.
constexpr int kCommMaxRanks = 8;
constexpr int kCommMaxTiles = 1024;
constexpr int kCommCtlBytes = 4096;
constexpr int kCommSets = 4;
enum CommMode { kCommNone = 0, kCommAllReduce = 1, kCommAllGather = 2 };

// The all-gather of the previous launch on the comm, still to be received on this rank.
struct CommPending {
  __nv_bfloat16* dst;  // this rank's gathered tensor [m][world * n_out]; null: nothing pending
  int m, n, n_out, tiles, gate_up, pair;  // of the launch that sent it (pair: two values per word)
};

struct CommParams {
  uint8_t* peer[kCommMaxRanks];  // base of every rank's buffer as mapped here (peer[rank]: own)
  int mode, world, rank;
  int64_t ar_n;        // 64 x the tiles a slot set holds
  CommPending pend;
};

// ---- INT4 decode (M <= 16) -----------------------------------------------------------
struct DecodeParams {
  const uint8_t* wq;       // tiled nibbles [tiles][kb_per_tile][2048]
  const uint32_t* sz;      // [tiles][groups][64] {bf16 scale, bf16 128+zp}
  const float* bias;       // [n] or null
  const __nv_bfloat16* x;  // [m][ldx]
  __nv_bfloat16* y;        // [m][ldy]  (scatter: [*][ldy])
  const __nv_bfloat16* other0;
  const __nv_bfloat16* other1;
  const int32_t* row_idx;       // scatter epilogue
  const __nv_bfloat16* row_w;   // scatter epilogue
  float* partials;         // [2 * grid][16][64]
  uint32_t* counters;      // [tiles], zero between calls
  int* status;             // 0, or the code of the wait that gave up
  int64_t ldx, ldy;
  int64_t ldo;  // row length of other0 / other1
  int m, n, n_out, k;
  int tiles, kb_per_tile, kbpg_shift, groups, gps;  // gps = groups a full stage can touch
  int fusion, gate_up, stages;
  int exact;  // 0: scale after the sum; 1, 2: per-weight bf16 rounding (2: shift-free high nibbles)
  int unit;   // CTA shares are multiples of this many k-blocks
  int x_rows, red_tok;  // shared-memory rows for x per stage / tokens in the reduction buffer
#ifdef WOQ_B200_TIMELINE
  unsigned long long* stamps;  // measuring build only: [8 launches][1024 CTAs][8] global-timer stamps
  int launch_seq;
#endif
  CommParams comm;
};

// How a launch cuts the weight: `cluster` == 0 is the stream-K grid (equal contiguous shares of
// the k-block sequence, split tiles reduced through the workspace); `cluster` == C >= 1 is
// tiles x C CTAs in thread-block clusters of C that reduce through distributed shared memory.
struct DecodePlan {
  int grid, cluster, kpw, unit, smem_budget;
};

template <class P>
__device__ __forceinline__ int decode_row_to_n(const P& p, int tile, int row) {
  if (p.gate_up) return row < 32 ? tile * 32 + row : p.n / 2 + tile * 32 + (row - 32);
  return tile * kTileN + row;
}

// 0 per-layer choice, 1 always stream-K, 2 cluster grid whenever the tiles fit (see DecodePlan)
void decode_int4_set_split(int mode);
DecodePlan decode_int4_plan(int m, int tiles, int kb_per_tile, int kb_per_group, int num_sms);
size_t decode_int4_partial_bytes(int grid);
cudaError_t launch_decode_int4(DecodeParams p, const DecodePlan& plan, cudaStream_t stream);
// Receives a pending all-gather without running a linear (status: the workspace-style status word).
cudaError_t launch_comm_fence(const CommParams& c, int* status, int num_sms, cudaStream_t stream);

// ---- INT4 tensor-core path, one CTA per tile (M <= 16; above: the CTA-pair path below) -----
// Row layout: tiles of 128 output rows x 64 k, 4096 bytes each, [tile][k-block][half][row][16 B].
// Word j' = 4 * half + j of a row holds k = 8 j' + 2 s in nibble s (bits 4s..4s+3) and
// k = 8 j' + 2 s + 1 in nibble s + 4, so (w >> 4s) & 0x000f000f is the bf16x2 pair (k, k+1).
// Scales: [tile][group][128] words, same {bf16 scale, bf16 128 + zp} format.
constexpr int kTcTileN = 128;
constexpr int kTcBlockBytes = kTcTileN * kBlockK / 2;  // 4096

struct TcParams {
  const uint8_t* wq;
  const uint32_t* sz;
  const float* bias;
  __nv_bfloat16* y;
  const __nv_bfloat16* other0;
  const __nv_bfloat16* other1;
  const int32_t* row_idx;
  const __nv_bfloat16* row_w;
  float* partials;     // [2 * grid][n_tok][128]
  uint32_t* counters;  // [tiles]
  int* status;
  int64_t ldy;
  int m, n, n_out, k;
  int n_tok;           // token columns of the MMA: 16 (the pipeline shapes go up to 256)
  int tiles, kb_per_tile, kbpg_shift, groups;
  int kbs, stages;     // k-blocks per stage; slots of the A-group / activation ring
  int w_ring, a_col0;  // slots of the packed-weight ring (a multiple of four); first TMEM column of the A groups
  int fusion, gate_up;
};

// The decode kernel, the CTA-pair kernels, the K-block tcgen05 kernel and the per-token quantiser opt into
// programmatic dependent launch unless WOQ_B200_PDL=0 was set before first use (all other kernels launch plainly).
bool dependent_launch_enabled();
// Lets `kern` (no static shared memory) be launched with all the shared memory a block can have.  Always the same
// limit, set before each launch: with the launch's own size, two host threads with different token counts could
// interleave so that one launches above the limit the other has just set.
constexpr int kMaxSmemBytes = 227 * 1024;
template <class K>
inline cudaError_t allow_max_smem(K* kern) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmemBytes);
}
int tc_pick_grid(int tiles, int kb_per_tile, int num_sms);
size_t tc_partial_bytes(int grid, int n_tok);
size_t tc_plan(TcParams& p);  // fills a_col0, kbs, stages, w_ring from n_tok; returns the dynamic shared memory (0: none)
cudaError_t launch_int4_tc(TcParams p, const CUtensorMap& xmap, int grid, cudaStream_t stream);

// ---- tensor-core path on CTA pairs (INT4: more than 16 tokens; INT8 / NF4 with bf16 compute: any) ----
// Row layouts of a 128-row x 64-k block: INT4 as above; NF4 the same words (codes are table indices);
// INT8 8192 bytes [quarter][row][16 B], codes biased by 128 (u8), a word holds k, k + 2, k + 1, k + 3
// from its low byte up, so w & 0x00ff00ff and (w >> 8) & 0x00ff00ff are pairs of neighbouring k.
// Scale words: INT4 {bf16 scale, bf16 128 + zp}; INT8 {bf16 scale, 128 + zp as an integer}; NF4 {bf16 scale, 0}.
enum WeightKind { kWeightInt4InPlace = 0, kWeightInt4, kWeightInt8InPlace, kWeightInt8, kWeightNf4 };
__host__ __device__ constexpr int pair_block_bytes(int kind) {
  return kind == kWeightInt8InPlace || kind == kWeightInt8 ? 2 * kTcBlockBytes : kTcBlockBytes;
}
// A launch runs one linear, or several of one shape on consecutive row ranges of x (the experts of a
// mixture): `groups` of them, their items one after the other.
constexpr int kMaxPairGroups = 32;
struct PairGroup {
  const uint8_t* wq;   // row layout
  const uint32_t* sz;
  const float* bias;
  __nv_bfloat16* y;    // result of the group's first token
  int row0, m;         // first row of x, tokens
  int tok_tiles;       // tiles of tokens
  int item0;           // number of the group's first (256-row tile, token tile) item
};
struct PairParams {
  PairGroup group[kMaxPairGroups];
  int n_groups, items;
  float nf4[16];       // NF4: the table
  const __nv_bfloat16* other0;  // extra operands: one group only
  const __nv_bfloat16* other1;
  const int32_t* row_idx;
  const __nv_bfloat16* row_w;
  float* partials;     // [CTAs][2][part_tok][128]
  uint32_t* counters;  // [CTAs], zero between calls
  int* status;
  int64_t ldy;
  int n, n_out;
  int n_tok;                    // token columns of a tile (a multiple of 32, <= 256)
  int tiles, w_tiles;           // 128-row tiles; pairs of them (rounded up)
  int kb_per_tile, kbpg_shift, groups;
  int kbs, kpw, stages, w_ring; // k-blocks per stage, and of them per warpgroup; slots of the two rings
  int whole, split;             // pairs take whole tiles; pairs of a cluster that share a tile (0, 1: none)
  int unit;                     // shares are multiples of this many k-blocks
  int fusion, gate_up;
  int kind;      // WeightKind
  int part_tok;  // tokens of a partial tile: min(most tokens of a group, n_tok)
  int vec;  // y and the extra operands can be accessed 16 bytes at a time
};
// How a launch is cut: token columns, tiles of tokens, and whether pairs take whole tiles (or equal shares of
// the k sequence).  `kind`: a WeightKind, or kPairCutInt8 for the INT8 compute kernel (k steps of 128, not 64).
constexpr int kPairCutInt8 = -1;
struct PairCut {
  int n_tok, tok_tiles, whole, split;  // split > 1: so many pairs, a cluster, share each tile
};
PairCut pair_cut(int64_t m, int w_tiles, int k_steps, int pairs, int kind);
int pair_group_columns(const int64_t* rows, int groups, int kind);
size_t pair_plan(PairParams& p, int num_sms);  // fills kbs, stages, w_ring, unit; dynamic shared memory (0: none)
size_t pair_partial_bytes(int num_sms, int part_tok);
cudaError_t launch_pair(PairParams p, const CUtensorMap& xmap, int num_sms, cudaStream_t stream);

__host__ __device__ inline int tc_tile_row_to_n(int n_total, int gate_up, int tile, int row) {
  if (gate_up) return row < 64 ? tile * 64 + row : n_total / 2 + tile * 64 + (row - 64);
  return tile * kTcTileN + row;
}

// ---- INT8 compute path ----------------------------------------------------------------------
struct I8PairParams {
  const float* sw;      // per-channel weight scales [n_pad]
  const float* sa;      // per-token activation scales [m]
  const int32_t* zpa;   // per-token activation zero points [m] (asymmetric codes are u8), or null
  const int32_t* comp;  // with zpa: per-row sums of the weight codes [n_pad]
  const float* bias;
  __nv_bfloat16* y;     // may be null when only the accumulators are wanted
  const __nv_bfloat16* other0;
  const __nv_bfloat16* other1;
  int* acc_out;         // optional [m][n] int32 accumulators
  int* partials;        // [CTAs][2][part_tok][128]
  uint32_t* counters;   // [CTAs], zero between calls
  int* status;
  int64_t ldy;
  int m, n, n_out;
  int n_tok, tok_tiles, unit;  // as pair_cut; shares are multiples of `unit` k-chunks
  int tiles, w_tiles;    // 128-row tiles; pairs of them (rounded up)
  int kc_per_tile, part_tok, stages, fusion, gate_up;
  int split;  // pairs of a cluster that share a tile (0, 1: none)
  int vec;  // y and the extra operands can be accessed 16 bytes at a time
};
size_t i8_pair_partial_bytes(int num_sms, int part_tok);
cudaError_t launch_i8_pair(I8PairParams p, const CUtensorMap& wmap, const CUtensorMap& qamap, int num_sms,
                           cudaStream_t stream);
cudaError_t launch_pack_int8(const int8_t* plain, int8_t* tiled, int n, int k, int tiles64,
                             int gate_up, cudaStream_t stream);
cudaError_t launch_unpack_int8(const int8_t* tiled, int8_t* plain, int n, int k, int gate_up,
                               cudaStream_t stream);
cudaError_t launch_pad_scale(const void* src, float* dst, int n, int n_pad, int dtype,
                             cudaStream_t stream);
cudaError_t launch_quant_act(const __nv_bfloat16* x, int64_t ldx, int m, int k, int asym, int per_tensor,
                             int8_t* qa, float* sa, int32_t* zpa, float* range, cudaStream_t stream);
cudaError_t launch_rmsnorm_quant(const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* gamma, float eps, int m,
                                 int k, int asym, __nv_bfloat16* y, int64_t ldy, int8_t* qa, float* sa, int32_t* zpa,
                                 cudaStream_t stream);
cudaError_t launch_weight_row_sum(const int8_t* plain, int n, int k, int32_t* comp, cudaStream_t stream);

// ---- INT8 compute with K-block scaling (woq_int8_block.cu) --------------------------------
struct I8BlockParams {
  const uint8_t* w;      // plain [n][k/2] nibbles (w4) or [n][k] s8
  const float* sw;       // [n][groups] weight scales
  const float* zpw;      // [n][groups] weight zero points or null (default_zp)
  const uint32_t* zw;    // not null: w, sw and zw in the layout of I8BlockTcParams, natural code order, m <= 16
  const int32_t* comp;   // [n][kc] sums of (qw - zp_w) per K block (asymmetric activations)
  const uint8_t* qa;     // [m][k] activation codes (w4: even / odd interleaved inside every 8)
  const float* sa;       // [m][kc]
  const int32_t* zpa;    // [m][kc]
  const int32_t* sumqa;  // [m][kc] sums of the activation codes per K block
  const float* bias;
  __nv_bfloat16* y;      // may be null when only the accumulators are wanted
  const __nv_bfloat16* other0;
  const __nv_bfloat16* other1;
  int32_t* acc_out;      // optional [kc][m][n] block accumulators after the compensation
  int64_t ldy;
  int m, n, k, kb, kc, group, groups, fusion, w4, asym;
  float default_zp;
};
cudaError_t launch_act_block_quant(const __nv_bfloat16* x, int64_t ldx, int m, int k, int kb, int act_mode,
                                   int interleave, uint8_t* qa, float* sa, int32_t* zpa, int32_t* sumqa,
                                   float* range, float* folded, cudaStream_t stream);
cudaError_t launch_weight_block_sum(const uint8_t* w, const float* zpw, int n, int k, int kb, int group, int groups,
                                    float default_zp, int w4, int32_t* comp, cudaStream_t stream);
cudaError_t launch_i8_block(const I8BlockParams& p, cudaStream_t stream);

// ---- the same for INT4 weights, symmetric activations and K blocks of 128 on tcgen05 (woq_i8_block_tc.cu) ----
struct I8BlockTcParams {
  const uint8_t* w;      // [tiles][kc][8192] nibbles, see btc_pack_kernel
  const uint32_t* zw;    // [tiles][groups][128] zero point in every byte
  const float* sw;       // [tiles][groups][128] weight scales
  const float* sat;      // [tok_tiles][kc][n_tok] activation scales
  const float* bias;
  __nv_bfloat16* y;      // may be null when only the accumulators are wanted
  const __nv_bfloat16* other0;
  const __nv_bfloat16* other1;
  int32_t* acc_out;      // optional [kc][m][n] block accumulators
  float* partials;       // [CTAs][2][part_tok][128]
  uint32_t* counters;    // [CTAs], zero between calls
  int* status;
  int64_t ldy;
  int m, n, kc, groups, bpg;  // bpg: K blocks per weight group (a large number: one group)
  int n_tok, tok_tiles, tiles, part_tok;
  int w_ring, unit;           // slots of the packed-weight ring; shares are multiples of `unit` K blocks (kc: whole tiles)
  int cut;                    // 0: by estimate, 1: shares, 2: whole tiles
  int fusion;
};
int i8_block_tc_columns(int64_t m);
size_t i8_block_tc_partial_bytes(int num_sms, int part_tok);
cudaError_t launch_i8_block_tc(I8BlockTcParams p, const CUtensorMap& qamap, int num_sms, cudaStream_t stream);
cudaError_t launch_act_block128_quant(const __nv_bfloat16* x, int64_t ldx, int m, int kc, uint8_t* qa, float* sa,
                                      int32_t* zpa, int32_t* sumqa, float* sat, int n_tok, cudaStream_t stream);
// whether a call of m tokens on n x (kc * 128) weights runs on woq_i8_block_kernel instead
bool i8_block_tc_few_tokens(int64_t m, int64_t n, int kc);
cudaError_t launch_transpose_scales(const float* sa, int m, int kc, float* sat, int n_tok, cudaStream_t stream);
cudaError_t launch_btc_pack(const uint8_t* plain, uint8_t* packed, int n, int k, cudaStream_t stream);
cudaError_t launch_btc_unpack(const uint8_t* packed, uint8_t* plain, int n, int k, cudaStream_t stream);
cudaError_t launch_btc_pack_scales(const float* scales, const float* zps, float* sw, uint32_t* zw, int n, int groups,
                                   int* flag, cudaStream_t stream);

// ---- general route: any weight dtype, fp32 / fp16 / bf16 compute, plain layout -----------
struct GenericParams {
  const uint8_t* w;     // plain [n][row_bytes]: nibbles (even k low) or bytes; kb_per_tile > 0: row layout
  const float* scales;  // [n][groups] fp32 as given (rounded to the compute dtype in the kernel)
  const float* zps;     // [n][groups] or null (then default_zp)
  const float* bias;    // [n] or null
  const void* x;        // [m][ldx] of io_dtype
  void* y;              // [m][ldy] of io_dtype
  const void* other0;
  const void* other1;
  int64_t ldx, ldy;
  int m, n, k, group, groups, row_bytes;
  int kb_per_tile;      // K / 64 when w is in the row layout of INT8 / NF4 (see WeightKind), else 0
  int weight_dtype, compute_dtype, io_dtype, fusion;  // WOQ_B200_DTYPE_* / WOQ_B200_T_*
  float default_zp;
};
cudaError_t launch_generic(const GenericParams& p, cudaStream_t stream);
cudaError_t launch_dump_generic(const GenericParams& p, float* out, cudaStream_t stream);
// Row layout of plain INT8 (`int8`) or NF4 weights and of their scales, and the weights back.  `flag`
// (zeroed): bit 0 a zero point is not an integer in -128..127 or a scale not finite or above 2^100 (the
// layout cannot be used), bit 1 a scale is outside the in-place range.
cudaError_t launch_pack_rows(const uint8_t* plain, uint8_t* rows, int n, int k, int int8, cudaStream_t stream);
cudaError_t launch_unpack_rows(const uint8_t* rows, uint8_t* plain, int n, int k, int int8, cudaStream_t stream);
cudaError_t launch_pack_row_scales(const float* scales, const float* zps, uint32_t* sz, int n, int groups, int* flag,
                                   cudaStream_t stream);

// ---- pack / unpack / dump ------------------------------------------------------------
struct PackInt4Args {
  const uint8_t* plain;  // [n][ceil(k/2)]
  uint8_t* tiled;
  int n, k, tiles, kb_per_tile, gate_up;
  int tc;  // 0: 64-row fragment layout, 1: 128-row row layout
};
cudaError_t launch_pack_int4(const PackInt4Args& a, cudaStream_t stream);
cudaError_t launch_unpack_int4(const uint8_t* tiled, uint8_t* plain, int n, int k, int tiles,
                               int kb_per_tile, int gate_up, cudaStream_t stream);

struct PackScaleArgs {
  const void* scales;  // [n][groups] (or transposed [groups][n])
  const void* zps;     // same shape or null
  uint32_t* sz;        // [tiles][groups][64]
  int* bad_zp;         // bit 0: a zero point is not an integer in 0..127; bit 1: see pack_scales_kernel
  int n, tiles, groups, gate_up;
  int transposed;     // scales are [groups][n]
  int zp_transposed;  // zero points are [groups][n]
  int scale_dtype, zp_dtype, default_zp;
  int tc;  // 0: [tiles64][groups][64] fragment order, 1: [tiles128][groups][128] row order
};
cudaError_t launch_pack_scales(const PackScaleArgs& a, cudaStream_t stream);

cudaError_t launch_dump_dequant_int4(const uint8_t* tiled, const uint32_t* sz, __nv_bfloat16* w,
                                     int n, int k, int tiles, int kb_per_tile, int kb_per_group,
                                     int groups, int gate_up, cudaStream_t stream);
cudaError_t launch_dump_dequant_int4_tc(const uint8_t* tiled, const uint32_t* sz, __nv_bfloat16* w,
                                        int n, int k, int tiles, int kb_per_tile, int kbpg_shift,
                                        int groups, int gate_up, cudaStream_t stream);

cudaError_t launch_gather_rows(const __nv_bfloat16* x, int64_t ldx, const int32_t* idx,
                               __nv_bfloat16* out, int64_t rows, int k, cudaStream_t stream);

// ---- mixture of experts: routing, activation and combination around the experts' linears (woq_moe.cu) ----
cudaError_t launch_moe_route(const int64_t* ids, int64_t pairs, int top_k, int experts, int32_t* counts,
                             int32_t* token_of, int32_t* pos_of, cudaStream_t stream);
cudaError_t launch_silu_mul(const __nv_bfloat16* gate, const __nv_bfloat16* up, __nv_bfloat16* out, int64_t count,
                            cudaStream_t stream);
cudaError_t launch_moe_combine(const __nv_bfloat16* rows, const int64_t* ids, const int32_t* pos_of,
                               const __nv_bfloat16* w, int64_t tokens, int top_k, int hidden, __nv_bfloat16* out,
                               cudaStream_t stream);

// AWQ / GPTQ int32 checkpoints -> plain nibble layout [n][k/2]
cudaError_t launch_awq_to_plain(const int32_t* qweight_kn8, uint8_t* plain, int n, int k,
                                cudaStream_t stream);
cudaError_t launch_gptq_to_plain(const int32_t* qweight_k8n, uint8_t* plain, int n, int k,
                                 cudaStream_t stream);
// packed int32 zero points [groups][n/8] -> u8 [n][groups]; gptq_plus_one adds 1 (GPTQ v1)
cudaError_t launch_unpack_qzeros(const int32_t* qzeros, uint8_t* zps, int n, int groups, int awq,
                                 int plus_one, cudaStream_t stream);

__host__ __device__ inline int tile_row_to_n(int n_total, int gate_up, int tile, int row) {
  if (gate_up) return row < 32 ? tile * 32 + row : n_total / 2 + tile * 32 + (row - 32);
  return tile * kTileN + row;
}

void count_launch();

}  // namespace woq
