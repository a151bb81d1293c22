// Weight-only-quantised GEMM on CTA pairs (tcgen05 cta_group::2 + TMEM) for more than 16 tokens.
//
// A pair of CTAs on neighbouring SMs owns 256 output rows x up to 256 tokens: each CTA dequantises
// its own 128 weight rows into its tensor memory (the A operand), each loads half of the
// activation tile into its shared memory (the B operand), and the leader's MMAs (M = 256) read both
// halves.  Against one CTA per tile that halves the activation bytes an SM takes from L2 and writes
// to shared memory per FLOP: 20 KB per 128 rows x 256 tokens x 64 k instead of 36 KB.
//
//   warp 0      producer: bulk copies of packed weights + group scales of this CTA's rows
//   warp 1      producer: TMA loads of this CTA's half of the activation tile; both CTAs' loads
//               complete on the leader's barrier
//   warp 2      (leader) issues the MMAs, one commit per stage frees the stage in both CTAs
//   warp 3      tensor-memory allocation
//   warps 4-11  epilogue: accumulators -> bias -> bf16 tile in shared memory -> fused post-op -> y.
//               The accumulators are free again once the bf16 tile is written; the copy to global
//               memory runs beside the next tile's MMAs.
//   warps 12-27 dequantise: thread = output row, one k-block of a stage per warpgroup
//
// Work split: the sequence of (linear, 256-row tile, token tile, k-block), token tiles innermost but
// for k, is cut into equal contiguous shares, one per pair ("stream-K").  A tile that several
// pairs share is summed in k order: whoever arrives last adds the others' fp32 partial tiles from
// the workspace (the pair that holds the beginning of the tile reaches it at the end of its own
// share, when the others are normally done, and then adds its accumulators straight from TMEM).
// Nobody waits for an arrival, and the order of the sum does not depend on timing.
//
// SPLIT: few tiles (p.split = S = 2 .. 4 pairs each).  The S pairs of a tile form one cluster and take a
// contiguous part of k each; they leave their fp32 accumulators in shared memory, and after a cluster barrier
// each CTA adds 1 / S of the tokens over distributed shared memory, in k order.  With shares of the k sequence
// the same tiles pay three trips through L2 and one CTA per tile reads all the parts: 4096 x 4096, 128 tokens
// took 26 us for 4 us of MMAs.
//
// What bounds it.  At 256 token columns: the tensor cores under the power limit (57344 x 8192, 512 tokens: 333 us,
// 1440 TFLOP/s; one CTA per tile and 256 tokens per launch took 501).  At 32 columns: the dequantiser's issue
// slots and the hand-overs between roles (57344 x 8192, 32 tokens: 72 us, 3.4 TB/s of weights; 91 us with one
// k-block per visit and polling idle warps, 125 us with one CTA per tile).  A lone thread beside sixteen
// dequantising warps gets an instruction issued every ten cycles or so, so the roles' work per stage is what has
// to be small: one activation copy per stage, several k-blocks per stage, no wait or fence that is not needed.
//
// Weights: INT4, INT8 and NF4 in the row layout of their kind (WeightKind); only the dequantiser and
// the bytes of a k-block differ.
#include "woq_kernels.h"
#include <atomic>

#include "woq_nf4.cuh"
#include "woq_pair_epilogue.cuh"

namespace woq {

namespace {

constexpr int kRoleWarps = 4, kDeqGroups = 4;
constexpr int kDeqWarp0 = kRoleWarps + kEpiWarps;
constexpr int kPairThreads = (kDeqWarp0 + 4 * kDeqGroups) * 32;
constexpr int kPairTmemCols = 512;
constexpr int kMaxXRing = 8, kMaxPairWRing = 24;
constexpr int kPairHeaderBytes = 1024;
constexpr int kEpiBar = 1;

struct PairHeader {
  uint64_t w_full[kMaxPairWRing];  // packed weights + scales of the slot have landed
  uint64_t w_free[kMaxPairWRing];  // the dequantising warps have read the slot
  uint64_t full[kMaxXRing];        // leader: the A halves of both CTAs written, both x halves landed
  uint64_t free_[kMaxXRing];       // the stage's MMAs have completed
  uint64_t d_full, d_empty;        // accumulators complete / (leader) read by all epilogue warps of the pair
  uint32_t tmem_base;
  int abort_flag;
  int decision;
};
constexpr int kNf4LutBytes = 16 * 32 * 4;  // the NF4 table, one copy per lane (no bank conflicts)
static_assert(sizeof(PairHeader) <= kPairHeaderBytes, "header too large");

__device__ __forceinline__ int pair_owner_of(int64_t b, int64_t total, int64_t pairs) {
  return static_cast<int>(((b + 1) * pairs - 1) / total);
}

// group of an item, and the item's place in it
__device__ __forceinline__ int pair_group_of(const PairParams& p, int item) {
  int g = 0;
  while (g + 1 < p.n_groups && item >= p.group[g + 1].item0) ++g;
  return g;
}

// A k-block's 64 weights of one row -> 32 bf16x2 registers (k order).  `ws` + 16 * row is the row's first
// 16 bytes, the next ones are kTcTileN * 16 further on.  All variants give bf16((code - zp) * bf16(scale)),
// rounded once, bit for bit the general kernel's values.
//
// INT4 in place: every scale is normal and below 0.5 and every zero point below 16, so nibbles at bits 4..7
// of a half-word can be used where they are: masked, the half-word read as bf16 is 16 q 2^-133 exactly
// (the encoding is linear below 2^-125); subtract 16 zp 2^-133, multiply by scale * 2^129.  13 instead
// of 15 instructions per eight weights.
template <bool IN_PLACE>
__device__ __forceinline__ void pair_dequant_int4(const uint8_t* ws, int row, uint32_t szw, uint32_t (&r)[32]) {
  const uint4* wp = reinterpret_cast<const uint4*>(ws) + row;
  const uint4 v0 = wp[0], v1 = wp[kTcTileN];
  const uint32_t z0 = __byte_perm(szw, 0, 0x1010), s0 = __byte_perm(szw, 0, 0x3232);
  const uint32_t z1 = IN_PLACE ? (szw & 0xfu) * 0x00100010u : z0;
  const uint32_t s1 = IN_PLACE ? s0 + 0x40804080u : s0;
  const uint32_t words[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t w = words[j], u = w >> 8;
    r[j * 4] = bf16x2_mul(bf16x2_sub(lop3_and_or(w, 0x000f000fu, kBf16Magic), z0), s0);
    r[j * 4 + 2] = bf16x2_mul(bf16x2_sub(lop3_and_or(u, 0x000f000fu, kBf16Magic), z0), s0);
    if (IN_PLACE) {
      r[j * 4 + 1] = bf16x2_mul(bf16x2_sub(w & 0x00f000f0u, z1), s1);
      r[j * 4 + 3] = bf16x2_mul(bf16x2_sub(u & 0x00f000f0u, z1), s1);
    } else {
      r[j * 4 + 1] = bf16x2_mul(bf16x2_sub(lop3_and_or(w >> 4, 0x000f000fu, kBf16Magic), z0), s0);
      r[j * 4 + 3] = bf16x2_mul(bf16x2_sub(lop3_and_or(u >> 4, 0x000f000fu, kBf16Magic), z0), s0);
    }
  }
}

// INT8: codes biased by 128; a byte in a half-word read as bf16 is q 2^-133 exactly (0..255: the subnormals
// and the first binade), so the difference to the zero point's byte is exact too and one multiplication by
// scale * 2^133 finishes (IN_PLACE: every scale normal and below 2^-5); otherwise 2^120 first, exact, then
// scale * 2^13 with the same single rounding.
template <bool IN_PLACE>
__device__ __forceinline__ void pair_dequant_int8(const uint8_t* ws, int row, uint32_t szw, uint32_t (&r)[32]) {
  const uint4* wp = reinterpret_cast<const uint4*>(ws) + row;
  const uint32_t z = (szw & 0xffu) * 0x00010001u, s = __byte_perm(szw, 0, 0x3232);
  const uint32_t s1 = IN_PLACE ? s + 0x42804280u : bf16x2_mul(s, 0x46004600u);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 v = wp[q * kTcTileN];
    const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t lo = bf16x2_sub(words[j] & 0x00ff00ffu, z), hi = bf16x2_sub(__byte_perm(words[j], 0, 0x4341), z);
      r[q * 8 + j * 2] = bf16x2_mul(IN_PLACE ? lo : bf16x2_mul(lo, 0x7b807b80u), s1);
      r[q * 8 + j * 2 + 1] = bf16x2_mul(IN_PLACE ? hi : bf16x2_mul(hi, 0x7b807b80u), s1);
    }
  }
}

// NF4: fp32 table values (24 bits) times the bf16 scale, rounded to fp32 and then to bf16 as the general
// kernel does, so a table of bf16 values would not do.  One conflict-free shared load per weight: lane l
// reads its own copy at 128 * code + 4 l.
__device__ __forceinline__ void pair_dequant_nf4(const uint8_t* ws, int row, uint32_t szw, const uint8_t* lut_lane,
                                                 uint32_t (&r)[32]) {
  const uint4* wp = reinterpret_cast<const uint4*>(ws) + row;
  const float s = __uint_as_float(szw & 0xffff0000u);
  auto value = [&](uint32_t code128) { return *reinterpret_cast<const float*>(lut_lane + (code128 & 0x780u)) * s; };
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint4 v = wp[h * kTcTileN];
    const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t w = words[j];
      r[h * 16 + j * 4] = bf_pack(value(w << 7), value(w >> 9));
      r[h * 16 + j * 4 + 1] = bf_pack(value(w << 3), value(w >> 13));
      r[h * 16 + j * 4 + 2] = bf_pack(value(w >> 1), value(w >> 17));
      r[h * 16 + j * 4 + 3] = bf_pack(value(w >> 5), value(w >> 21));
    }
  }
}

template <int KIND>
__device__ __forceinline__ void pair_dequant(const uint8_t* ws, int row, uint32_t szw, const uint8_t* lut_lane,
                                             uint32_t (&r)[32]) {
  if (KIND == kWeightInt4InPlace) pair_dequant_int4<true>(ws, row, szw, r);
  if (KIND == kWeightInt4) pair_dequant_int4<false>(ws, row, szw, r);
  if (KIND == kWeightInt8InPlace) pair_dequant_int8<true>(ws, row, szw, r);
  if (KIND == kWeightInt8) pair_dequant_int8<false>(ws, row, szw, r);
  if (KIND == kWeightNf4) pair_dequant_nf4(ws, row, szw, lut_lane, r);
}

template <int KIND, int KPW, bool SPLIT>
__global__ void __launch_bounds__(kPairThreads, 1)
    woq_pair_kernel(const __grid_constant__ PairParams p, const __grid_constant__ CUtensorMap xmap) {
  extern __shared__ __align__(1024) uint8_t smem[];
  PairHeader* hdr = reinterpret_cast<PairHeader*>(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (smem_u32(smem) & 1023u) {  // swizzled tiles need a 1024-byte aligned base (the same in both CTAs)
    if (tid == 0) atomicCAS(p.status, 0, 99);
    return;
  }
  const int half_tok = p.n_tok >> 1;
  const int x_blk = half_tok * 128;
  const int x_stage_bytes = p.kbs * x_blk;
  constexpr int kBlock = pair_block_bytes(KIND);
  const int w_stage_bytes = p.kbs * (kBlock + 512);
  uint8_t* x_stages = smem + kPairHeaderBytes;
  uint8_t* w_stages = x_stages + static_cast<size_t>(p.stages) * x_stage_bytes;
  uint8_t* out_tile = w_stages + static_cast<size_t>(p.w_ring) * w_stage_bytes;
  uint8_t* lut = out_tile + p.n_tok * kOutPitch;  // NF4 only
  if (KIND == kWeightNf4 && tid < 512) reinterpret_cast<float*>(lut)[tid] = p.nf4[tid >> 5];

  const uint32_t crank = pair_cta_rank(), rank = crank & 1, leader = crank - rank;  // rank in cluster / pair
  const uint16_t pair_mask = static_cast<uint16_t>(3u << leader);
  const int pair = blockIdx.x >> 1;
  const int64_t pairs = gridDim.x >> 1;
  const int kbpt = p.kb_per_tile, kbs = p.kbs, n_stages = p.stages, n_wring = p.w_ring;
  // shares are dealt in units of p.unit k-blocks
  const int64_t units = static_cast<int64_t>(p.items) * kbpt / p.unit;
  int item0, kb00, rem0;  // item0 - group.item0 = weight tile * tok_tiles + token tile
  if (SPLIT) {
    const int sub = crank >> 1, n_st = (kbpt + kbs - 1) / kbs;  // whole stages, at least one each
    item0 = pair / p.split;
    kb00 = sub * n_st / p.split * kbs;
    const int kb_end = (sub + 1) * n_st / p.split * kbs;
    rem0 = (kb_end < kbpt ? kb_end : kbpt) - kb00;
  } else {
    const int64_t b_begin = pair * units / pairs * p.unit, b_end = (pair + 1) * units / pairs * p.unit;
    item0 = static_cast<int>(b_begin / kbpt);
    kb00 = static_cast<int>(b_begin % kbpt);
    rem0 = static_cast<int>(b_end - b_begin);
  }

  if (tid == 0) {
    for (int s = 0; s < n_stages; ++s) {
      mbar_init(&hdr->full[s], 8 * kbs / KPW + 1);  // the dequantising warps of both CTAs, the leader's x producer
      mbar_init(&hdr->free_[s], 1);
    }
    for (int s = 0; s < n_wring; ++s) {
      mbar_init(&hdr->w_full[s], 1);
      mbar_init(&hdr->w_free[s], 4 * kbs / KPW);
    }
    mbar_init(&hdr->d_full, 1);
    mbar_init(&hdr->d_empty, 2 * kEpiWarps);
    hdr->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 3) {
    pair_tmem_alloc(&hdr->tmem_base, kPairTmemCols);
    pair_tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  pair_sync();
  tc_fence_after_sync();
  grid_launch_dependents();
  const uint32_t tmem_base = hdr->tmem_base;
  volatile int* abort_flag = &hdr->abort_flag;

  if (warp == 0) {
    // ---- packed weights and their group scales (never written by an earlier launch) ----
    if (lane == 0) {
      int item = item0, kb0 = kb00, rem = rem0, wslot = 0, g = pair_group_of(p, item0);
      uint32_t wphase = 0;
      while (rem > 0) {
        if (g + 1 < p.n_groups && item >= p.group[g + 1].item0) ++g;
        int tile = (item - p.group[g].item0) / p.group[g].tok_tiles * 2 + static_cast<int>(rank);
        if (tile >= p.tiles) tile = p.tiles - 1;  // odd tile count: the last pair's second half repeats it
        const uint8_t* wsrc = p.group[g].wq + (static_cast<size_t>(tile) * kbpt + kb0) * kBlock;
        const uint32_t* ssrc = p.group[g].sz + static_cast<size_t>(tile) * p.groups * kTcTileN;
        int seg = kbpt - kb0 < rem ? kbpt - kb0 : rem;
        rem -= seg;
        while (seg > 0) {
          const int nkb = seg < kbs ? seg : kbs;
          uint8_t* ws = w_stages + static_cast<size_t>(wslot) * w_stage_bytes;
          const int g0 = kb0 >> p.kbpg_shift;
          const int ng = ((kb0 + nkb - 1) >> p.kbpg_shift) - g0 + 1;
          mbar_wait<true>(&hdr->w_free[wslot], wphase ^ 1, abort_flag, p.status, 31);
          mbar_arrive_expect_tx(&hdr->w_full[wslot], nkb * kBlock + ng * 512);
          bulk_g2s(ws, wsrc, nkb * kBlock, &hdr->w_full[wslot]);
          bulk_g2s(ws + kbs * kBlock, ssrc + static_cast<size_t>(g0) * kTcTileN, ng * 512, &hdr->w_full[wslot]);
          wsrc += nkb * kBlock;
          kb0 += nkb;
          seg -= nkb;
          if (++wslot == n_wring) {
            wslot = 0;
            wphase ^= 1;
          }
        }
        if (kb0 == kbpt) {
          kb0 = 0;
          ++item;
        }
      }
    }
  } else if (warp == 1) {
    // ---- this CTA's half of the activation tile, one copy per stage (a stage cut short by the end of
    // ---- the share still loads whole: its last k-blocks are not used) ----
    if (lane == 0) {
      grid_dependency_wait();
      int item = item0, kb0 = kb00, rem = rem0, slot = 0, g = pair_group_of(p, item0);
      uint32_t phase = 0;
      const uint32_t full0 = pair_map(&hdr->full[0], leader);
      while (rem > 0) {
        if (g + 1 < p.n_groups && item >= p.group[g + 1].item0) ++g;
        // (rows past the group's last belong to another group or to nobody: their columns are not used)
        const int row = p.group[g].row0 + (item - p.group[g].item0) % p.group[g].tok_tiles * p.n_tok +
                        static_cast<int>(rank) * half_tok;
        int seg = kbpt - kb0 < rem ? kbpt - kb0 : rem;
        rem -= seg;
        for (; seg > 0; seg -= kbs) {
          mbar_wait<true>(&hdr->free_[slot], phase ^ 1, abort_flag, p.status, 32);
          if (rank == 0) mbar_arrive_expect_tx(&hdr->full[slot], 2 * x_stage_bytes);
          pair_tma_load_3d(x_stages + slot * x_stage_bytes, &xmap, 0, row, kb0, full0 + slot * 8);
          kb0 += kbs;
          if (++slot == n_stages) {
            slot = 0;
            phase ^= 1;
          }
        }
        kb0 = 0;
        ++item;
      }
    }
  } else if (warp == 2) {
    if (rank == 0) {
      // ---- the whole warp walks the stages, one elected lane issues ----
      const uint32_t idesc = pair_idesc(p.n_tok, /*bf16*/ 1, /*bf16*/ 1, /*f32*/ 1);
      const uint64_t desc0 = umma_desc_k128(smem_u32(x_stages));
      const uint32_t a_base = tmem_base + p.n_tok;
      const uint32_t x_blk16 = static_cast<uint32_t>(x_blk >> 4);
      int kb0 = kb00, rem = rem0, slot = 0;
      uint32_t phase = 0, seg_no = 0;
      while (rem > 0) {
        int seg = kbpt - kb0 < rem ? kbpt - kb0 : rem;
        rem -= seg;
        kb0 = 0;
        uint32_t accumulate = 0;
        mbar_wait(&hdr->d_empty, (seg_no & 1) ^ 1, abort_flag, p.status, 33);
        for (; seg > 0; seg -= kbs) {
          mbar_wait(&hdr->full[slot], phase, abort_flag, p.status, 34);
          tc_fence_after_sync();
          if (elect_one()) {
            const int nkb = seg < kbs ? seg : kbs;
            uint32_t a = a_base + slot * (kbs * 32);
            uint64_t b = desc0 + static_cast<uint32_t>(slot * kbs) * x_blk16;
            for (int j = 0; j < nkb; ++j) {
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) {
                pair_mma_f16_ts(tmem_base, a + ks * 8, b + ks * 2, idesc, accumulate);
                accumulate = 1;
              }
              a += 32;
              b += x_blk16;
            }
            pair_commit(&hdr->free_[slot], pair_mask);
            if (seg <= kbs) pair_commit(&hdr->d_full, pair_mask);
          }
          __syncwarp();
          accumulate = 1;
          if (++slot == n_stages) {
            slot = 0;
            phase ^= 1;
          }
        }
        ++seg_no;
      }
    }
  } else if (warp >= kDeqWarp0) {
    // ---- dequantise: KPW neighbouring k-blocks of a stage per warpgroup, so kbs / KPW warpgroups share a
    // ---- stage and each takes every step-th one ----
    const int wg = (warp - kDeqWarp0) >> 2, q = warp & 3;
    const int row = q * 32 + lane;
    const int wgs = kbs / KPW, step = kDeqGroups / wgs;
    const int j0 = wg % wgs * KPW;  // first k-block within the stage
    const uint32_t a_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + p.n_tok + j0 * 32;
    const uint32_t full0 = pair_map(&hdr->full[0], leader);
    int kb_seg = kb00, rem = rem0;
    int own = wg / wgs, slot = own, wslot = own;  // `own`: this warpgroup's next stage, counted over all segments
    int st = 0;
    uint32_t phase = 0, wphase = 0;
    while (rem > 0) {
      const int seg_len = kbpt - kb_seg < rem ? kbpt - kb_seg : rem;
      const int ns = (seg_len + kbs - 1) / kbs;
      for (; own < st + ns; own += step) {
        const int in_seg = (own - st) * kbs;   // k-blocks of the segment before this stage
        const int kb0 = kb_seg + in_seg;
        const int nj = seg_len - in_seg - j0;  // below KPW where the stage was cut short
        const uint8_t* ws = w_stages + wslot * w_stage_bytes;
        const uint32_t a_slot = a_lane + slot * (kbs * 32);
        mbar_wait(&hdr->w_full[wslot], wphase, abort_flag, p.status, 35);
        const int g0 = kb0 >> p.kbpg_shift;
#pragma unroll
        for (int j = 0; j < KPW; ++j) {
          uint32_t r[32];
          if (j < nj) {
            const int gl = ((kb0 + j0 + j) >> p.kbpg_shift) - g0;
            const uint32_t szw = reinterpret_cast<const uint32_t*>(ws + kbs * kBlock)[gl * kTcTileN + row];
            pair_dequant<KIND>(ws + (j0 + j) * kBlock, row, szw, lut + lane * 4, r);
          }
          if (j == KPW - 1) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&hdr->w_free[wslot]);
          }
          if (j == 0) {
            mbar_wait(&hdr->free_[slot], phase ^ 1, abort_flag, p.status, 36);
            tc_fence_after_sync();
            __syncwarp();  // the TMEM store is a warp-wide instruction
          }
          if (j < nj) tmem_st_x32(a_slot + j * 32, r);
        }
        if (nj > 0) tc_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) pair_arrive(full0 + slot * 8);
        slot += step;
        if (slot >= n_stages) {
          slot -= n_stages;
          phase ^= 1;
        }
        wslot += step;
        if (wslot >= n_wring) {
          wslot -= n_wring;
          wphase ^= 1;
        }
      }
      st += ns;
      rem -= seg_len;
      kb_seg = 0;
    }
  } else if (warp >= kRoleWarps) {
    // ---- epilogue: two warpgroups, 16 tokens at a time in turn ----
    const int q = warp & 3, eg = (warp - kRoleWarps) >> 2, et = tid - kRoleWarps * 32;
    const int row = q * 32 + lane;
    const uint32_t d_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t d_empty0 = pair_map(&hdr->d_empty, leader);
    grid_dependency_wait();  // y, the fused operands and the workspace belong to this grid now
    int item = item0, kb0 = kb00, rem = rem0, g = pair_group_of(p, item0);
    uint32_t seg_no = 0;
    auto to_tile = [&](int c0, const float (&v)[16], float bias) {  // 16 tokens of this row, as bf16
      uint8_t* dst = out_tile + c0 * kOutPitch + row * 2;
#pragma unroll
      for (int e = 0; e < 16; ++e) *reinterpret_cast<__nv_bfloat16*>(dst + e * kOutPitch) = __float2bfloat16_rn(v[e] + bias);
    };
    auto accumulators_read = [&]() {
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) pair_arrive(d_empty0);
    };
    while (rem > 0) {
      const int seg_len = kbpt - kb0 < rem ? kbpt - kb0 : rem;
      const bool whole = seg_len == kbpt;
      if (g + 1 < p.n_groups && item >= p.group[g + 1].item0) ++g;
      const PairGroup& grp = p.group[g];
      const int in_group = item - grp.item0;
      const int tile = in_group / grp.tok_tiles * 2 + static_cast<int>(rank);
      const int tok0 = in_group % grp.tok_tiles * p.n_tok;
      const int mv = grp.m - tok0 < p.n_tok ? grp.m - tok0 : p.n_tok;
      const bool real = tile < p.tiles;
      float bias = 0.f;
      if (grp.bias && real) {
        const int n = tc_tile_row_to_n(p.n, p.gate_up, tile, row);
        if (n < p.n) bias = grp.bias[n];
      }
      // the bf16 tile of the previous segment has been copied out by everybody
      named_bar_sync(kEpiBar, kEpiThreads);
      mbar_wait<true>(&hdr->d_full, seg_no & 1, abort_flag, p.status, 37);
      tc_fence_after_sync();
      __syncwarp();
      if (SPLIT) {  // this pair's part of the tile, for the CTAs that add it up
        float* part = reinterpret_cast<float*>(x_stages) + row;
        for (int c0 = eg * 16; c0 < mv; c0 += 32) {
          uint32_t t[16];
          tmem_ld_x16(d_lane + c0, t);
          tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) part[(c0 + e) * kTcTileN] = __uint_as_float(t[e]);
        }
        break;
      }
      bool finish = whole && real;
      if (whole || !real) {
        if (real)
          for (int c0 = eg * 16; c0 < mv; c0 += 32) {
            uint32_t t[16];
            tmem_ld_x16(d_lane + c0, t);
            tc_wait_ld();
            float v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(t[e]);
            to_tile(c0, v, bias);
          }
        accumulators_read();
      } else {
        // part of a tile
        const int64_t tb0 = static_cast<int64_t>(item) * kbpt / p.unit;  // the tile's first unit
        const int c_first = pair_owner_of(tb0, units, pairs), c_last = pair_owner_of(tb0 + kbpt / p.unit - 1, units, pairs);
        const unsigned others = static_cast<unsigned>(c_last - c_first);
        uint32_t* counter = p.counters + c_first * 2 + rank;
        auto slot_of = [&](int c) {  // partial tile of pair c, this CTA's rows
          const int s = (c == c_first && c * units / pairs < tb0) ? 1 : 0;
          return p.partials + static_cast<size_t>((c * 2 + static_cast<int>(rank)) * 2 + s) * p.part_tok * kTcTileN + row;
        };
        bool from_tmem = false;
        if (kb0 == 0) {
          // the beginning of the tile, the last segment of this pair: have all others arrived?
          if (et == 0) {
            uint32_t seen;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
            if (seen == others) *counter = 0;
            hdr->decision = seen == others;
          }
          named_bar_sync(kEpiBar, kEpiThreads);
          from_tmem = hdr->decision != 0;
          finish = from_tmem;
        }
        if (!from_tmem) {
          float* dst = slot_of(pair);
          for (int c0 = eg * 16; c0 < mv; c0 += 32) {
            uint32_t t[16];
            tmem_ld_x16(d_lane + c0, t);
            tc_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (c0 + e < mv) __stcg(dst + static_cast<size_t>(c0 + e) * kTcTileN, __uint_as_float(t[e]));
          }
          accumulators_read();
          __threadfence();
          named_bar_sync(kEpiBar, kEpiThreads);
          if (et == 0) {
            const unsigned old = atomicAdd(counter, 1u);
            if (old == others) *counter = 0;
            hdr->decision = old == others;
          }
          named_bar_sync(kEpiBar, kEpiThreads);
          finish = hdr->decision != 0;
        }
        if (finish) {
          __threadfence();
          for (int c0 = eg * 16; c0 < mv; c0 += 32) {
            float v[16];
            int c = c_first;
            if (from_tmem) {
              uint32_t t[16];
              tmem_ld_x16(d_lane + c0, t);
              tc_wait_ld();
#pragma unroll
              for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(t[e]);
              ++c;
            } else {
#pragma unroll
              for (int e = 0; e < 16; ++e) v[e] = 0.f;
            }
            // two parts in flight together: a round trip to L2 per part was most of a shared tile's cost
            for (; c <= c_last; c += 2) {
              const bool two = c < c_last;
              const float* src = slot_of(c) + static_cast<size_t>(c0) * kTcTileN;
              const float* src2 = slot_of(two ? c + 1 : c) + static_cast<size_t>(c0) * kTcTileN;
              float t[16], t2[16];
#pragma unroll
              for (int e = 0; e < 16; ++e) t[e] = c0 + e < mv ? __ldcg(src + e * kTcTileN) : 0.f;
#pragma unroll
              for (int e = 0; e < 16; ++e) t2[e] = two && c0 + e < mv ? __ldcg(src2 + e * kTcTileN) : 0.f;
#pragma unroll
              for (int e = 0; e < 16; ++e) v[e] = two ? v[e] + t[e] + t2[e] : v[e] + t[e];
            }
            to_tile(c0, v, bias);
          }
          if (from_tmem) accumulators_read();
        }
      }
      named_bar_sync(kEpiBar, kEpiThreads);
      if (finish) pair_copy_out<true>(p, grp.y, out_tile, tile, tok0, mv, et);
      rem -= seg_len;
      kb0 = 0;
      ++item;
      ++seg_no;
    }
  }

  if (SPLIT) {
    __syncwarp();
    pair_sync();  // every pair's part is in its shared memory
    const PairGroup& grp = p.group[0];
    const int tile = item0 / grp.tok_tiles * 2 + static_cast<int>(rank), tok0 = item0 % grp.tok_tiles * p.n_tok;
    const int mv = grp.m - tok0 < p.n_tok ? grp.m - tok0 : p.n_tok;
    const int slice = (mv + p.split - 1) / p.split, t0 = static_cast<int>(crank >> 1) * slice;
    const int nt = mv - t0 < slice ? mv - t0 : slice;  // this CTA's tokens t0 .. t0 + nt (none: <= 0)
    if (tile < p.tiles) {
      // a warp: 32 rows of a token; four tokens' reads in flight together
      constexpr int kWarps = kPairThreads / 32, kBatch = 4;
      const int row = (warp & 3) * 32 + lane, n = tc_tile_row_to_n(p.n, p.gate_up, tile, row);
      const float bias = grp.bias && n < p.n ? grp.bias[n] : 0.f;
      const uint32_t part0 = pair_map(reinterpret_cast<const float*>(x_stages) + row, rank);
      const uint32_t part_step = pair_map(x_stages, 2) - pair_map(x_stages, 0);  // to the next pair's part
      for (int t = warp >> 2; t < nt; t += kWarps / 4 * kBatch) {
        float v[kBatch][4];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int tok = t + u * (kWarps / 4);
#pragma unroll
          for (int s = 0; s < 4; ++s)
            v[u][s] = tok < nt && s < p.split ? pair_ld_f32(part0 + s * part_step + (t0 + tok) * (kTcTileN * 4)) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int tok = t + u * (kWarps / 4);
          if (tok < nt)
            *reinterpret_cast<__nv_bfloat16*>(out_tile + tok * kOutPitch + row * 2) =
                __float2bfloat16_rn(((v[u][0] + v[u][1]) + v[u][2]) + v[u][3] + bias);
        }
      }
    }
    __syncthreads();
    if (tile < p.tiles && nt > 0 && warp >= kRoleWarps && warp < kDeqWarp0)
      pair_copy_out<true>(p, grp.y, out_tile, tile, tok0 + t0, nt, tid - kRoleWarps * 32);
  }

  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  pair_sync();
  if (warp == 3) {
    tc_fence_after_sync();
    pair_tmem_dealloc(tmem_base, kPairTmemCols);
  }
}

}  // namespace

// What a k step costs a tile of n columns, in us: the larger of its dequantisation and hand-overs (or, for INT8
// compute, its L2 traffic) and its MMAs.  Fitted to 57344 x 8192 INT4 (72 / 77 / 89 / 101 / 176 / 333 us at
// 32 / 64 / 96 / 128 / 256 / 512 tokens), 57344 x 4096 INT8 with bf16 compute (44 / 52 / 68 us at 8 / 64 / 128) and
// INT8 compute on 28672 x 4096 (121 / 220 us at 1024 / 2048).
static double pair_step_us(int kind, int n) {
  const double mma = (kind == kPairCutInt8 ? 0.0011 : 0.0017) * n;
  const double step = kind == kPairCutInt8                                    ? 0.26 + 0.001 * n
                      : kind == kWeightInt4 || kind == kWeightInt4InPlace     ? 0.165 + 0.00075 * n
                      : kind == kWeightNf4                                    ? 0.25 + 0.001 * n
                                                                              : 0.19 + 0.00125 * n;
  return step < mma ? mma : step;
}

// Token tiles of a call, and how its tiles are dealt, by estimated time.  Whole tiles take as many rounds as the
// fullest pair has tiles.  Equal shares of the k sequence
// keep every pair busy to the end, but then the parts of shared tiles go through the workspace, one after
// another and behind the last MMA: 4096 x 4096, 1000 tokens took 46 us with shares for 25 us of MMAs.  With few
// tiles, clusters of pairs split k (see SPLIT).
static int pair_cluster_capacity(int ctas);
PairCut pair_cut(int64_t m, int w_tiles, int k_steps, int pairs, int kind) {
  PairCut best{};
  double best_cost = -1;
  const int t0 = static_cast<int>(m > 256 ? (m + 255) / 256 : 1);
  for (int t = t0; t <= 2 * t0 + 1; ++t) {
    int n = static_cast<int>(((m + t - 1) / t + 31) / 32 * 32);
    if (n < 32) n = 32;
    if ((m + n - 1) / n != t) continue;  // fewer tiles of this width do
    const double step = pair_step_us(kind, n);
    const int64_t items = static_cast<int64_t>(w_tiles) * t;
    const double shares = step * k_steps * items / pairs + 4 + 0.04 * n + 2.0 * pairs / items;
    const double rounds = step * k_steps * static_cast<double>((items + pairs - 1) / pairs);
    auto consider = [&](double cost, int whole, int split) {
      if (best_cost >= 0 && cost >= best_cost) return;
      best_cost = cost;
      best = PairCut{n, t, whole, split};
    };
    consider(shares, 0, 1);
    consider(rounds, 1, 1);
    // (a part has at least one stage of four k-blocks)
    for (int s = 2; s <= 4; ++s)
      if (k_steps >= 4 * s && items <= pair_cluster_capacity(2 * s))
        consider(step * ((k_steps + s - 1) / s) + 2 + 0.01 * n, 0, s);
  }
  return best;
}

// Token columns for several linears in one launch, by the number of tokens each has: the width with the least
// sum over their tiles.
int pair_group_columns(const int64_t* rows, int groups, int kind) {
  int best = 256;
  double best_cost = -1;
  for (int n = 256; n >= 32; n -= 32) {
    int64_t tiles = 0;
    for (int g = 0; g < groups; ++g) tiles += (rows[g] + n - 1) / n;
    const double cost = static_cast<double>(tiles) * pair_step_us(kind, n);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = n;
    }
  }
  return best;
}

// Pipeline shape for p.n_tok token columns; returns the dynamic shared memory in bytes.
//   k-blocks per stage: four up to 128 columns, two above.  Every stage costs each single-thread role
//     300-400 cycles of waiting, issuing and bookkeeping beside the busy dequantising warps, whatever
//     the stage holds; a k-block's MMAs take at least 64 cycles, 4 x n_tok / 2 when that is more.
//   k-blocks per warpgroup and visit: two up to 128 columns, because the two waits, the store's completion and
//     the arrival (600 of 1490 cycles, most of it latency) then come once per two k-blocks (57344 x 8192 INT4, 32 /
//     64 / 128 tokens: 72 / 77 / 101 us, with one 80 / 83 / 105).  One at 128 columns of 8-bit weights: only three
//     weight slots fit, too few for two warpgroups to hold one each and a third to land (73 us with two, 68 with one).
//   Rings: a parity wait cannot tell a barrier that is one completion short from one that is three
//     short, so whoever waits for use u of a slot must know that use u - 1 has completed.  A warpgroup sees
//     every step-th stage (step = 4 kpw / kbs: 1 or 2).  A weight ring that is a multiple of step gives each
//     slot to the same warpgroups every time; on the A / activation ring the wait for stage s - step (the
//     MMAs of stage s - step - stages, which complete in order) covers stage s - 2 * stages when there are
//     at least step stages.
size_t pair_plan(PairParams& p, int num_sms) {
  const int lut = p.kind == kWeightNf4 ? kNf4LutBytes : 0;
  const int budget = kMaxSmemBytes - kPairHeaderBytes - lut - p.n_tok * kOutPitch;
  p.kbs = p.n_tok <= 128 ? 4 : 2;
  p.kpw = p.kbs == 4 && (p.n_tok < 128 || pair_block_bytes(p.kind) == kTcBlockBytes) ? 2 : 1;
  const int step = kDeqGroups * p.kpw / p.kbs;
  const int x_stage = p.kbs * (p.n_tok / 2) * 128;
  const int w_stage = p.kbs * (pair_block_bytes(p.kind) + 512);
  int stages = (kPairTmemCols - p.n_tok) / 32 / p.kbs;
  if (stages > kMaxXRing) stages = kMaxXRing;
  // (two slots of 17 KB are enough for the 8-bit weights of a 256-column tile: the A ring buffers as well)
  const int min_ring = p.kbs == 2 && w_stage > 16 * 1024 ? 2 : 3;
  while (stages > 2 && budget - stages * x_stage < min_ring * w_stage) --stages;
  int ring = (budget - stages * x_stage) / w_stage;
  if (ring > kMaxPairWRing) ring = kMaxPairWRing;
  ring -= ring % step;
  if (stages < 2 || ring < 2) return 0;
  p.stages = stages;
  p.w_ring = ring;
  // shares in whole stages where they are long enough for the rounding not to matter
  const int64_t total = static_cast<int64_t>(p.items) * p.kb_per_tile;
  p.unit = p.whole ? p.kb_per_tile : p.kb_per_tile % p.kbs == 0 && total >= static_cast<int64_t>(num_sms / 2) * 8 * p.kbs ? p.kbs : 1;
  return kPairHeaderBytes + static_cast<size_t>(stages) * x_stage + static_cast<size_t>(ring) * w_stage +
         static_cast<size_t>(p.n_tok) * kOutPitch + lut;
}

// Pairs of a launch: all SMs, or one per unit of work when there are fewer.
int pair_grid(const PairParams& p, int num_sms) {
  const int64_t total = static_cast<int64_t>(p.items) * p.kb_per_tile / p.unit;
  int64_t pairs = num_sms / 2;
  if (pairs > total) pairs = total;
  return static_cast<int>(pairs < 1 ? 1 : pairs) * 2;
}

// Clusters of that many CTAs of this kernel's size that the current device runs at a time: a split whose
// clusters need a second round takes twice as long (16 clusters of 8: 27 us for a 4096 x 14336 layer that 20 us
// of shares do).  Asked once per device and size; an error counts as none.
static int pair_cluster_capacity(int ctas) {
  static std::atomic<int> known[64][9];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 0;
  int n = known[dev][ctas].load(std::memory_order_relaxed);
  if (n) return n - 1;
  auto* kern = woq_pair_kernel<kWeightInt4, 1, true>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas * 32));
  cfg.blockDim = dim3(kPairThreads);
  cfg.dynamicSmemBytes = kMaxSmemBytes;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = ctas;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (allow_max_smem(kern) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    clusters = 0;
  }
  known[dev][ctas].store(clusters + 1, std::memory_order_relaxed);
  return clusters;
}

size_t pair_partial_bytes(int num_sms, int part_tok) {
  return static_cast<size_t>(num_sms) * 2 * part_tok * kTcTileN * sizeof(float);
}

template <int KIND>
static void (*pick_pair_kernel(const PairParams& p))(const PairParams, const CUtensorMap) {
  if (p.split > 1) return p.kpw == 2 ? woq_pair_kernel<KIND, 2, true> : woq_pair_kernel<KIND, 1, true>;
  return p.kpw == 2 ? woq_pair_kernel<KIND, 2, false> : woq_pair_kernel<KIND, 1, false>;
}

cudaError_t launch_pair(PairParams p, const CUtensorMap& xmap, int num_sms, cudaStream_t stream) {
  const size_t smem = pair_plan(p, num_sms);
  if (smem == 0) return cudaErrorInvalidConfiguration;
  if (p.kind == kWeightNf4) {
    static constexpr float values[16] = WOQ_NF4_VALUES;
    for (int i = 0; i < 16; ++i) p.nf4[i] = values[i];
  }
  void (*kern)(const PairParams, const CUtensorMap) = nullptr;
  switch (p.kind) {
    case kWeightInt4InPlace: kern = pick_pair_kernel<kWeightInt4InPlace>(p); break;
    case kWeightInt4: kern = pick_pair_kernel<kWeightInt4>(p); break;
    case kWeightInt8InPlace: kern = pick_pair_kernel<kWeightInt8InPlace>(p); break;
    case kWeightInt8: kern = pick_pair_kernel<kWeightInt8>(p); break;
    case kWeightNf4: kern = pick_pair_kernel<kWeightNf4>(p); break;
    default: return cudaErrorInvalidValue;
  }
  cudaError_t e = allow_max_smem(kern);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  if (p.split > 1 && (p.n_groups != 1 || (p.kb_per_tile + p.kbs - 1) / p.kbs < p.split ||
                      static_cast<size_t>(p.n_tok) * kTcTileN * 4 >
                          smem - kPairHeaderBytes - static_cast<size_t>(p.n_tok) * kOutPitch - kNf4LutBytes))
    return cudaErrorInvalidValue;  // (pair_cut does not ask for these)
  cfg.gridDim = dim3(p.split > 1 ? p.items * p.split * 2 : pair_grid(p, num_sms));
  cfg.blockDim = dim3(kPairThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.split > 1 ? 2 * p.split : 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (dependent_launch_enabled()) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  return cudaLaunchKernelEx(&cfg, kern, p, xmap);
}

}  // namespace woq
