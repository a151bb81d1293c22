// INT4 weights with INT8 compute and symmetric activation codes, K blocks of 128, on the tensor cores:
// C[m,n] += (float(sum_k qa[m,k] * (qw[n,k] - zp[n,g])) * scale_a[m,block]) * scale_w[n,g] per K block
// (csrc/cpu/aten/utils/woq.h:962-1126), the sum as int32 by tcgen05.mma kind::i8, exact.
//
// A CTA owns 128 output rows x up to 128 tokens of a share of the (row tile, token tile, K block) sequence
// (equal contiguous shares, or whole tiles where that is quicker; tiles that several CTAs share are summed in k order through the workspace by
// whoever arrives last, so nobody waits and the order does not depend on timing).
//
//   warp 0       producer: packed weights + zero points, two K blocks per stage
//   warp 1       producer: activation codes (TMA), their scales, the weight scales
//   warp 2       MMAs: one accumulator buffer per K block
//   warp 3       tensor-memory allocation
//   warps 4-19   drain: int32 accumulators of a K block -> fp32 -> scaled -> running sums in registers;
//                at the end of a tile bias, bf16, post-op, y
//   warps 20-27  unpack: thread = output row; nibbles -> s8 codes minus zero point -> tensor memory (the A
//                operand), one K block of the stage per warpgroup
//
// What bounds it: the drain.  Every K block's 128 x columns accumulators pass through the CUDA cores once,
// 2.5 issue slots per value (an integer add that makes the accumulator a float, then pairs: subtract,
// multiply, multiply-add); the unpacking adds 7 per eight weights.  The kernels of mma.sync fragments
// (woq_int8_block.cu) spend the same on the drain and the MMAs' operand traffic on top, and read the weights
// once per 64 tokens.
#include "woq_kernels.h"
#include "woq_pair_common.cuh"

namespace woq {

namespace {

constexpr int kDrainWarps = 16, kUnpackWarps = 8;
constexpr int kDrainWarp0 = 4, kUnpackWarp0 = kDrainWarp0 + kDrainWarps;
constexpr int kBtcThreads = (kUnpackWarp0 + kUnpackWarps) * 32;
constexpr int kDrainThreads = kDrainWarps * 32;
constexpr int kBtcStages = 4, kBtcSRing = 6, kBtcMaxWRing = 8, kBtcMaxBufs = 4;
constexpr int kBtcHeaderBytes = 1024;
constexpr int kWBlock = 8192;           // 128 rows x 128 k nibbles
constexpr int kWStage = 2 * (kWBlock + 512);
constexpr int kACol0 = 256;             // first tensor-memory column of the A slots

struct BtcHeader {
  uint64_t w_full[kBtcMaxWRing], w_free[kBtcMaxWRing];
  uint64_t full[kBtcStages], free_[kBtcStages];
  uint64_t s_full[kBtcSRing], s_free[kBtcSRing];
  uint64_t d_full[kBtcMaxBufs], d_empty[kBtcMaxBufs];
  uint32_t tmem_base;
  int abort_flag;
  int decision;
};
static_assert(sizeof(BtcHeader) <= kBtcHeaderBytes, "header too large");

__device__ __forceinline__ int btc_owner_of(int64_t u, int64_t units, int64_t ctas) {
  return static_cast<int>(((u + 1) * ctas - 1) / units);
}

// D[tmem] (+)= A[tmem] * B[smem descriptor], 8-bit operands, M = 128, K = 32
__device__ __forceinline__ void umma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      :
      : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst_smem, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst_smem)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ uint64_t f32x2(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
// c += ((float(acc) * sa) * sw) for two neighbouring tokens.  |acc| < 2^22, so acc + the bits of 1.5 * 2^23 is
// the float 1.5 * 2^23 + acc.
__device__ __forceinline__ void drain2(uint64_t& c, uint32_t a0, uint32_t a1, uint64_t sa, uint64_t sw) {
  uint64_t v = f32x2(__uint_as_float(a0 + 0x4b400000u), __uint_as_float(a1 + 0x4b400000u));
  const uint64_t m = f32x2(-12582912.f, -12582912.f);
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(m));
  asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(sa));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(v), "l"(sw));
}

__device__ __forceinline__ void btc_store(const I8BlockTcParams& p, int n, int tok, float v) {
  if (p.bias) v = p.bias[n] + v;
  float r = bf16_round(v);
  const size_t o = static_cast<size_t>(tok) * p.ldy + n;
  if (p.fusion == FUSE_ADD || p.fusion == FUSE_ADD_ADD) {
    r = bf16_round(r + __bfloat162float(p.other0[o]));
    if (p.fusion == FUSE_ADD_ADD) r = bf16_round(r + __bfloat162float(p.other1[o]));
  } else if (p.fusion == FUSE_MUL) {
    r = bf16_round(r * __bfloat162float(p.other0[o]));
  } else {
    r = unary_post_op(r, p.fusion);
  }
  p.y[o] = __float2bfloat16_rn(r);
}

// NCH: groups of eight token columns per drain warpgroup (n_tok = 32 * NCH)
template <int NCH>
__global__ void __launch_bounds__(kBtcThreads, 1)
    woq_i8_block_tc_kernel(const __grid_constant__ I8BlockTcParams p, const __grid_constant__ CUtensorMap qamap) {
  extern __shared__ __align__(1024) uint8_t smem[];
  BtcHeader* hdr = reinterpret_cast<BtcHeader*>(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (smem_u32(smem) & 1023u) {
    if (tid == 0) atomicCAS(p.status, 0, 99);
    return;
  }
  constexpr int n_tok = 32 * NCH, cw = 8 * NCH;
  constexpr int x_blk = n_tok * 128, x_stage = 2 * x_blk, s_stage = 2 * (512 + n_tok * 4);
  constexpr int n_bufs = NCH == 4 ? 2 : 4;
  uint8_t* x_stages = smem + kBtcHeaderBytes;
  uint8_t* s_stages = x_stages + kBtcStages * x_stage;
  uint8_t* w_stages = s_stages + kBtcSRing * s_stage;

  const int kc = p.kc, n_wring = p.w_ring;
  const int64_t ctas = gridDim.x, units = static_cast<int64_t>(p.tiles) * p.tok_tiles * kc / p.unit;
  const int64_t b_begin = blockIdx.x * units / ctas * p.unit, b_end = (blockIdx.x + 1) * units / ctas * p.unit;
  const int item0 = static_cast<int>(b_begin / kc);  // item = row tile * tok_tiles + token tile
  const int kb00 = static_cast<int>(b_begin % kc);
  const int rem0 = static_cast<int>(b_end - b_begin);

  if (tid == 0) {
    for (int s = 0; s < kBtcStages; ++s) {
      mbar_init(&hdr->full[s], kUnpackWarps + 1);
      mbar_init(&hdr->free_[s], 1);
    }
    for (int s = 0; s < kBtcSRing; ++s) {
      mbar_init(&hdr->s_full[s], 1);
      mbar_init(&hdr->s_free[s], kDrainWarps);
    }
    for (int s = 0; s < n_wring; ++s) {
      mbar_init(&hdr->w_full[s], 1);
      mbar_init(&hdr->w_free[s], kUnpackWarps);
    }
    for (int s = 0; s < n_bufs; ++s) {
      mbar_init(&hdr->d_full[s], 1);
      mbar_init(&hdr->d_empty[s], kDrainWarps);
    }
    hdr->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 3) {
    tmem_alloc(&hdr->tmem_base, 512);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  grid_launch_dependents();
  const uint32_t tmem_base = hdr->tmem_base;
  volatile int* abort_flag = &hdr->abort_flag;

  // Every role walks the same segments (runs of K blocks of one item) and in them the same stages of two K
  // blocks (one, where the segment ends).
  if (warp == 0) {
    if (lane == 0) {
      int item = item0, kb0 = kb00, rem = rem0, slot = 0;
      uint32_t phase = 0;
      while (rem > 0) {
        const int tile = item / p.tok_tiles;
        int seg = kc - kb0 < rem ? kc - kb0 : rem;
        rem -= seg;
        for (; seg > 0; seg -= 2, kb0 += 2) {
          const int nkb = seg < 2 ? 1 : 2;
          uint8_t* ws = w_stages + slot * kWStage;
          const int g0 = kb0 / p.bpg, ng = (kb0 + nkb - 1) / p.bpg - g0 + 1;
          mbar_wait(&hdr->w_free[slot], phase ^ 1, abort_flag, p.status, 41);
          mbar_arrive_expect_tx(&hdr->w_full[slot], nkb * kWBlock + ng * 512);
          bulk_g2s(ws, p.w + (static_cast<size_t>(tile) * kc + kb0) * kWBlock, nkb * kWBlock, &hdr->w_full[slot]);
          bulk_g2s(ws + 2 * kWBlock, p.zw + (static_cast<size_t>(tile) * p.groups + g0) * kTcTileN, ng * 512,
                   &hdr->w_full[slot]);
          if (++slot == n_wring) {
            slot = 0;
            phase ^= 1;
          }
        }
        kb0 = 0;
        ++item;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      grid_dependency_wait();  // the quantiser's codes and scales
      int item = item0, kb0 = kb00, rem = rem0, slot = 0, sslot = 0;
      uint32_t phase = 0, sphase = 0;
      while (rem > 0) {
        const int tile = item / p.tok_tiles, tt = item % p.tok_tiles;
        int seg = kc - kb0 < rem ? kc - kb0 : rem;
        rem -= seg;
        for (; seg > 0; seg -= 2, kb0 += 2) {
          const int nkb = seg < 2 ? 1 : 2;
          mbar_wait(&hdr->free_[slot], phase ^ 1, abort_flag, p.status, 42);
          mbar_arrive_expect_tx(&hdr->full[slot], x_stage);  // (whole even where the second block is not used)
          tma_load_3d(x_stages + slot * x_stage, &qamap, 0, tt * n_tok, kb0, &hdr->full[slot]);
          const int g0 = kb0 / p.bpg, ng = (kb0 + nkb - 1) / p.bpg - g0 + 1;
          uint8_t* ss = s_stages + sslot * s_stage;
          mbar_wait(&hdr->s_free[sslot], sphase ^ 1, abort_flag, p.status, 43);
          mbar_arrive_expect_tx(&hdr->s_full[sslot], ng * 512 + nkb * n_tok * 4);
          bulk_g2s(ss, p.sw + (static_cast<size_t>(tile) * p.groups + g0) * kTcTileN, ng * 512, &hdr->s_full[sslot]);
          bulk_g2s(ss + 1024, p.sat + (static_cast<size_t>(tt) * kc + kb0) * n_tok, nkb * n_tok * 4, &hdr->s_full[sslot]);
          if (++slot == kBtcStages) {
            slot = 0;
            phase ^= 1;
          }
          if (++sslot == kBtcSRing) {
            sslot = 0;
            sphase ^= 1;
          }
        }
        kb0 = 0;
        ++item;
      }
    }
  } else if (warp == 2) {
    // the whole warp walks the stages, one elected lane issues
    const uint32_t idesc = umma_idesc(n_tok, /*s8*/ 1, /*s8*/ 1, /*s32*/ 2);
    const uint64_t desc0 = umma_desc_k128(smem_u32(x_stages));
    int kb0 = kb00, rem = rem0, slot = 0, buf = 0;
    uint32_t phase = 0, bphase = 0;
    while (rem > 0) {
      int seg = kc - kb0 < rem ? kc - kb0 : rem;
      rem -= seg;
      kb0 = 0;
      for (; seg > 0; seg -= 2) {
        const int nkb = seg < 2 ? 1 : 2;
        mbar_wait(&hdr->full[slot], phase, abort_flag, p.status, 44);
        for (int j = 0; j < nkb; ++j) {
          mbar_wait(&hdr->d_empty[buf], bphase ^ 1, abort_flag, p.status, 45);
          tc_fence_after_sync();
          if (elect_one()) {
            const uint32_t a = tmem_base + kACol0 + (slot * 2 + j) * 32;
            const uint64_t b = desc0 + static_cast<uint32_t>((slot * 2 + j) * (x_blk >> 4));
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_i8_ts(tmem_base + buf * n_tok, a + ks * 8, b + ks * 2, idesc, ks > 0 ? 1u : 0u);
            tc_commit(&hdr->d_full[buf]);
            if (j + 1 == nkb) tc_commit(&hdr->free_[slot]);
          }
          __syncwarp();
          if (++buf == n_bufs) {
            buf = 0;
            bphase ^= 1;
          }
        }
        if (++slot == kBtcStages) {
          slot = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp >= kUnpackWarp0) {
    const int j = (warp - kUnpackWarp0) >> 2, q = warp & 3, row = q * 32 + lane;
    const uint32_t a_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + kACol0 + j * 32;
    int kb0 = kb00, rem = rem0, slot = 0, wslot = 0;
    uint32_t phase = 0, wphase = 0;
    while (rem > 0) {
      int seg = kc - kb0 < rem ? kc - kb0 : rem;
      rem -= seg;
      for (; seg > 0; seg -= 2, kb0 += 2) {
        const bool some = j < seg;
        const uint8_t* ws = w_stages + wslot * kWStage;
        mbar_wait(&hdr->w_full[wslot], wphase, abort_flag, p.status, 46);
        uint32_t r[32];
        if (some) {
          const int gl = (kb0 + j) / p.bpg - kb0 / p.bpg;
          const uint32_t z = reinterpret_cast<const uint32_t*>(ws + 2 * kWBlock)[gl * kTcTileN + row];
          const uint4* wp = reinterpret_cast<const uint4*>(ws + j * kWBlock) + row;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 v = wp[i * kTcTileN];
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              // per byte 128 + q - zp in 1..143 (no borrow), its top bit flipped: q - zp as s8
              r[i * 8 + e * 2] = (lop3_and_or(w[e], 0x0f0f0f0fu, 0x80808080u) - z) ^ 0x80808080u;
              r[i * 8 + e * 2 + 1] = (lop3_and_or(w[e] >> 4, 0x0f0f0f0fu, 0x80808080u) - z) ^ 0x80808080u;
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&hdr->w_free[wslot]);
        mbar_wait(&hdr->free_[slot], phase ^ 1, abort_flag, p.status, 47);
        tc_fence_after_sync();
        __syncwarp();
        if (some) {
          tmem_st_x32(a_lane + slot * 64, r);
          tc_wait_st();
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&hdr->full[slot]);
        if (++slot == kBtcStages) {
          slot = 0;
          phase ^= 1;
        }
        if (++wslot == n_wring) {
          wslot = 0;
          wphase ^= 1;
        }
      }
      kb0 = 0;
    }
  } else if (warp >= kDrainWarp0) {
    const int q = warp & 3, eg = (warp - kDrainWarp0) >> 2, et = tid - kDrainWarp0 * 32;
    const int row = q * 32 + lane, col0 = eg * cw;
    const uint32_t d_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + col0;
    grid_dependency_wait();  // y, the fused operands and the workspace belong to this grid now
    int item = item0, kb0 = kb00, rem = rem0, sslot = 0, buf = 0;
    uint32_t sphase = 0, bphase = 0;
    while (rem > 0) {
      const int seg_len = kc - kb0 < rem ? kc - kb0 : rem;
      const int tile = item / p.tok_tiles, tok0 = item % p.tok_tiles * n_tok;
      const int mv = p.m - tok0 < n_tok ? p.m - tok0 : n_tok;
      const int n = tile * kTcTileN + row;
      uint64_t c[cw / 2];
#pragma unroll
      for (int e = 0; e < cw / 2; ++e) c[e] = 0ull;
      for (int kb = kb0; kb < kb0 + seg_len; kb += 2) {
        const int nkb = kb0 + seg_len - kb < 2 ? 1 : 2;
        const uint8_t* ss = s_stages + sslot * s_stage;
        mbar_wait(&hdr->s_full[sslot], sphase, abort_flag, p.status, 48);
        for (int j = 0; j < nkb; ++j) {
          const int gl = (kb + j) / p.bpg - kb / p.bpg;
          const float s1 = reinterpret_cast<const float*>(ss)[gl * kTcTileN + row];
          const uint64_t sw = f32x2(s1, s1);
          const float4* sa = reinterpret_cast<const float4*>(ss + 1024 + (j * n_tok + col0) * 4);
          mbar_wait(&hdr->d_full[buf], bphase, abort_flag, p.status, 49);
          tc_fence_after_sync();
          __syncwarp();
#pragma unroll
          for (int h = 0; h < NCH; ++h) {
            uint32_t t[8];
            tmem_ld_x8(d_lane + buf * n_tok + h * 8, t);
            tc_wait_ld();
            if (h == NCH - 1) {
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&hdr->d_empty[buf]);
            }
            if (p.acc_out && n < p.n) {
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (col0 + h * 8 + e < mv)
                  p.acc_out[(static_cast<size_t>(kb + j) * p.m + tok0 + col0 + h * 8 + e) * p.n + n] = static_cast<int>(t[e]);
            }
            const float4 sa0 = sa[h * 2], sa1 = sa[h * 2 + 1];
            drain2(c[h * 4], t[0], t[1], f32x2(sa0.x, sa0.y), sw);
            drain2(c[h * 4 + 1], t[2], t[3], f32x2(sa0.z, sa0.w), sw);
            drain2(c[h * 4 + 2], t[4], t[5], f32x2(sa1.x, sa1.y), sw);
            drain2(c[h * 4 + 3], t[6], t[7], f32x2(sa1.z, sa1.w), sw);
          }
          if (++buf == n_bufs) {
            buf = 0;
            bphase ^= 1;
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&hdr->s_free[sslot]);
        if (++sslot == kBtcSRing) {
          sslot = 0;
          sphase ^= 1;
        }
      }
      auto value = [&](int e) {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(c[e >> 1]));
        return (e & 1) ? hi : lo;
      };
      if (p.y) {
        if (seg_len == kc) {
          if (n < p.n)
#pragma unroll
            for (int e = 0; e < cw; ++e)
              if (col0 + e < mv) btc_store(p, n, tok0 + col0 + e, value(e));
        } else {
          // part of a tile: whoever comes last adds the parts in k order
          const int64_t tb0 = static_cast<int64_t>(item) * kc / p.unit;  // the tile's first unit
          const int c_first = btc_owner_of(tb0, units, ctas), c_last = btc_owner_of(tb0 + kc / p.unit - 1, units, ctas);
          auto slot_of = [&](int cc) {
            const int s = (cc == c_first && cc * units / ctas < tb0) ? 1 : 0;
            return p.partials + static_cast<size_t>(cc * 2 + s) * p.part_tok * kTcTileN + row;
          };
          float* dst = slot_of(blockIdx.x);
#pragma unroll
          for (int e = 0; e < cw; ++e)
            if (col0 + e < mv) __stcg(dst + static_cast<size_t>(col0 + e) * kTcTileN, value(e));
          __threadfence();
          named_bar_sync(1, kDrainThreads);
          if (et == 0) {
            uint32_t* counter = p.counters + c_first;
            const unsigned old = atomicAdd(counter, 1u), others = static_cast<unsigned>(c_last - c_first);
            if (old == others) *counter = 0;
            hdr->decision = old == others;
          }
          named_bar_sync(1, kDrainThreads);
          if (hdr->decision) {
            __threadfence();
#pragma unroll
            for (int h = 0; h < NCH; ++h) {
              float v[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) v[e] = 0.f;
              for (int cc = c_first; cc <= c_last; ++cc) {
                const float* src = slot_of(cc) + static_cast<size_t>(col0 + h * 8) * kTcTileN;
                float t[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) t[e] = col0 + h * 8 + e < mv ? __ldcg(src + e * kTcTileN) : 0.f;
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] += t[e];
              }
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (n < p.n && col0 + h * 8 + e < mv) btc_store(p, n, tok0 + col0 + h * 8 + e, v[e]);
            }
          }
          named_bar_sync(1, kDrainThreads);  // `decision` has been read
        }
      }
      rem -= seg_len;
      kb0 = 0;
      ++item;
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 3) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// Per-token, per-block symmetric codes (the qconfig factory's default mode): one warp per (token, 128-wide
// block) holds its 128 elements in registers, so range and codes are one pass and one launch instead of two.
__global__ void __launch_bounds__(256) act_block128_quant_kernel(const __nv_bfloat16* x, int64_t ldx, int m, int kc,
                                                                 uint8_t* qa, float* sa, int32_t* zpa, int32_t* sumqa,
                                                                 float* sat, int n_tok) {
  grid_launch_dependents();  // the GEMM's weight loads need nothing from here
  const int item = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= m * kc) return;
  const int tok = item / kc, c = item - tok * kc;
  const uint2 v = *reinterpret_cast<const uint2*>(x + static_cast<int64_t>(tok) * ldx + c * 128 + lane * 4);
  const float f[4] = {__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                      __uint_as_float(v.y & 0xffff0000u)};
  float lo = fminf(fminf(f[0], f[1]), fminf(f[2], f[3])), hi = fmaxf(fmaxf(f[0], f[1]), fmaxf(f[2], f[3]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  const float scale = __fdiv_rn(fmaxf(fabsf(hi), fabsf(lo)), 127.0f);
  uint32_t word = 0;
  int sum = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float q = 0.f;
    if (scale > 0.f) q = fminf(fmaxf(rintf(__fdiv_rn(f[e], scale)), -128.f), 127.f);
    sum += static_cast<int>(q);
    word |= (static_cast<uint32_t>(static_cast<int>(q)) & 0xffu) << (8 * e);
  }
  reinterpret_cast<uint32_t*>(qa + static_cast<size_t>(tok) * kc * 128 + c * 128)[lane] = word;
  if (sumqa) {  // (for the kernel of few tokens)
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) sumqa[item] = sum;
  }
  if (lane == 0) {
    sa[item] = scale;
    zpa[item] = 0;
    sat[(static_cast<size_t>(tok / n_tok) * kc + c) * n_tok + tok % n_tok] = scale;
  }
}

__global__ void transpose_scales_kernel(const float* sa, int m, int kc, float* sat, int n_tok) {
  const int item = blockIdx.x * 256 + threadIdx.x;
  if (item >= m * kc) return;
  const int tok = item / kc, c = item - tok * kc;
  sat[(static_cast<size_t>(tok / n_tok) * kc + c) * n_tok + tok % n_tok] = sa[item];
}

// plain [n][k/2] nibbles (even k low) <-> [tile][block][part][row][16 B]: word 4 part + j of a row holds
// k = 8 i .. 8 i + 3 in the low nibbles of its bytes and k = 8 i + 4 .. + 7 in the high ones
__device__ __forceinline__ uint32_t btc_word_from_plain(uint32_t v) {
  uint32_t w = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) w |= ((v >> (4 * i)) & 15u) << (8 * (i & 3) + 4 * (i >> 2));
  return w;
}
__device__ __forceinline__ uint32_t btc_word_to_plain(uint32_t w) {
  uint32_t v = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) v |= ((w >> (8 * (i & 3) + 4 * (i >> 2))) & 15u) << (4 * i);
  return v;
}
__global__ void btc_pack_kernel(const uint8_t* plain, uint32_t* out, int n, int k, int64_t words) {
  const int64_t wi = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (wi >= words) return;
  const int64_t blk = wi >> 11;
  const int in = static_cast<int>(wi & 2047), j = in & 3, row = (in >> 2) & 127, part = in >> 9, kc = k / 128;
  const int64_t nn = blk / kc * kTcTileN + row;
  const int k0 = static_cast<int>(blk % kc) * 128 + (part * 4 + j) * 8;
  out[wi] = nn < n ? btc_word_from_plain(*reinterpret_cast<const uint32_t*>(plain + (nn * k + k0) / 2)) : 0u;
}
__global__ void btc_unpack_kernel(const uint32_t* packed, uint8_t* plain, int n, int k, int64_t words) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;  // 32-bit word of the plain weight
  if (i >= words) return;
  const int nn = static_cast<int>(i / (k / 8)), k0 = static_cast<int>(i % (k / 8)) * 8, wr = (k0 & 127) / 8;
  const int64_t blk = static_cast<int64_t>(nn / kTcTileN) * (k / 128) + k0 / 128;
  const uint32_t v = btc_word_to_plain(packed[blk * 2048 + ((wr >> 2) * kTcTileN + nn % kTcTileN) * 4 + (wr & 3)]);
#pragma unroll
  for (int b = 0; b < 4; ++b) plain[i * 4 + b] = static_cast<uint8_t>(v >> (8 * b));  // maybe unaligned
}
__global__ void btc_pack_scales_kernel(const float* scales, const float* zps, float* sw, uint32_t* zw, int n, int groups,
                                       int64_t words, int* flag) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= words) return;
  const int row = static_cast<int>(i % kTcTileN), g = static_cast<int>(i / kTcTileN % groups);
  const int64_t nn = i / (static_cast<int64_t>(kTcTileN) * groups) * kTcTileN + row;
  float s = 0.f;
  int z = 0;
  if (nn < n) {
    s = scales[nn * groups + g];
    const float zf = zps ? zps[nn * groups + g] : 8.f;
    if (zf > -1.f && zf < 128.f) z = static_cast<int>(zf);  // the truncation of the other kernels
    else atomicOr(flag, 1);
  }
  sw[i] = s;
  zw[i] = static_cast<uint32_t>(z) * 0x01010101u;
}

}  // namespace

// Token columns of a tile: the width whose tiles cost least, a K block costing a tile about 60 + columns (in
// units of a column's drain) whatever its tokens.
int i8_block_tc_columns(int64_t m) {
  int best = 128;
  int64_t best_cost = -1;
  for (int n = 128; n >= 32; n >>= 1) {
    const int64_t cost = (m + n - 1) / n * (60 + n);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = n;
    }
  }
  return best;
}

// Up to 8 tokens the kernel of 16 rows x 8 tokens per CTA (mma.sync, woq_int8_block.cu) is quicker: nothing waits for a
// tile's other parts and nothing is drained through tensor memory.  9 to 16 tokens are two CTAs that read the weights
// twice: quicker where the second time comes from L2, so up to half of its 126 MB.  That kernel / this one, us: one
// token, 1024 x 2048 5.1 / 12.7, 4096 x 4096 7.4 / 16.1, 4096 x 14336 17.2 / 27.2, 28672 x 4096 16.7 / 41.3, 57344 x 8192
// 71.5 / 131, 512 x 16384 18.8 / 21.4; 16 tokens, 4096 x 4096 9.5 / 18.2, 28672 x 4096 (59 MB) 34.9 / 44.8, but
// 8192 x 28672 (117 MB) 92.4 / 74.8, 57344 x 8192 (235 MB) 141 / 137.
bool i8_block_tc_few_tokens(int64_t m, int64_t n, int kc) {
  return m <= 8 || (m <= 16 && n * kc * 64 <= (64ll << 20));
}

size_t i8_block_tc_partial_bytes(int num_sms, int part_tok) {
  return static_cast<size_t>(num_sms) * 2 * part_tok * kTcTileN * sizeof(float);
}

cudaError_t launch_i8_block_tc(I8BlockTcParams p, const CUtensorMap& qamap, int num_sms, cudaStream_t stream) {
  const int fixed = kBtcHeaderBytes + kBtcStages * 2 * p.n_tok * 128 + kBtcSRing * 2 * (512 + p.n_tok * 4);
  p.w_ring = (226 * 1024 - fixed) / kWStage;
  if (p.w_ring > kBtcMaxWRing) p.w_ring = kBtcMaxWRing;
  if (p.w_ring < 2) return cudaErrorInvalidConfiguration;
  const size_t smem = fixed + static_cast<size_t>(p.w_ring) * kWStage;
  const int64_t total = static_cast<int64_t>(p.tiles) * p.tok_tiles * p.kc;
  // Shares in whole stages where they are long enough for the rounding not to matter, or whole tiles: the parts of a
  // shared tile are added one after another and behind its last K block.  In us, for c = columns / 32: a K block 0.54 +
  // 0.085 c, a tile's end 3 c, a shared tile's 5.2 c + 0.31 c for each part (fitted to 512 x 512 .. 4096 x 4096).
  // Shared / whole: 512 x 512, 128 tokens 29.2 / 18.7, 1024 x 2048, 128 tokens 46.0 / 28.8, 4096 x 4096, 512 tokens
  // 56.3 / 47.5, but 1024 x 4096, 33 tokens 26.4 / 30.4.
  const int64_t items = static_cast<int64_t>(p.tiles) * p.tok_tiles, ctas = total < num_sms ? total : num_sms;
  const int64_t parts = items >= ctas ? 2 : ceil_div(ctas, items) + 1;
  const double c = p.n_tok / 32, step = 0.54 + 0.085 * c;
  const double shares = step * ceil_div(total, ctas) + c * (5.2 + 0.31 * (parts < p.kc ? parts : p.kc));
  const double whole = step * p.kc * ceil_div(items, num_sms) + 3 * c;
  p.unit = (p.cut ? p.cut == 2 : whole <= shares) ? p.kc : p.kc % 2 == 0 && total >= static_cast<int64_t>(num_sms) * 16 ? 2 : 1;
  void (*kern)(const I8BlockTcParams, const CUtensorMap) = nullptr;
  switch (p.n_tok) {
    case 32: kern = woq_i8_block_tc_kernel<1>; break;
    case 64: kern = woq_i8_block_tc_kernel<2>; break;
    case 128: kern = woq_i8_block_tc_kernel<4>; break;
    default: return cudaErrorInvalidValue;
  }
  cudaError_t e = allow_max_smem(kern);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  const int64_t units = total / p.unit;
  cfg.gridDim = dim3(static_cast<unsigned>(units < num_sms ? units : num_sms));
  cfg.blockDim = dim3(kBtcThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  cfg.attrs = attr;
  if (dependent_launch_enabled()) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 1;
  }
  return cudaLaunchKernelEx(&cfg, kern, p, qamap);
}

cudaError_t launch_act_block128_quant(const __nv_bfloat16* x, int64_t ldx, int m, int kc, uint8_t* qa, float* sa,
                                      int32_t* zpa, int32_t* sumqa, float* sat, int n_tok, cudaStream_t stream) {
  const unsigned blocks = static_cast<unsigned>(ceil_div(static_cast<int64_t>(m) * kc, 8));
  act_block128_quant_kernel<<<blocks, 256, 0, stream>>>(x, ldx, m, kc, qa, sa, zpa, sumqa, sat, n_tok);
  return cudaGetLastError();
}

cudaError_t launch_transpose_scales(const float* sa, int m, int kc, float* sat, int n_tok, cudaStream_t stream) {
  const unsigned blocks = static_cast<unsigned>(ceil_div(static_cast<int64_t>(m) * kc, 256));
  transpose_scales_kernel<<<blocks, 256, 0, stream>>>(sa, m, kc, sat, n_tok);
  return cudaGetLastError();
}

cudaError_t launch_btc_pack(const uint8_t* plain, uint8_t* packed, int n, int k, cudaStream_t stream) {
  const int64_t words = ceil_div(n, kTcTileN) * (k / 128) * 2048;
  btc_pack_kernel<<<static_cast<unsigned>(ceil_div(words, 256)), 256, 0, stream>>>(
      plain, reinterpret_cast<uint32_t*>(packed), n, k, words);
  return cudaGetLastError();
}

cudaError_t launch_btc_unpack(const uint8_t* packed, uint8_t* plain, int n, int k, cudaStream_t stream) {
  const int64_t words = static_cast<int64_t>(n) * k / 8;
  btc_unpack_kernel<<<static_cast<unsigned>(ceil_div(words, 256)), 256, 0, stream>>>(
      reinterpret_cast<const uint32_t*>(packed), plain, n, k, words);
  return cudaGetLastError();
}

cudaError_t launch_btc_pack_scales(const float* scales, const float* zps, float* sw, uint32_t* zw, int n, int groups,
                                   int* flag, cudaStream_t stream) {
  const int64_t words = ceil_div(n, kTcTileN) * groups * kTcTileN;
  btc_pack_scales_kernel<<<static_cast<unsigned>(ceil_div(words, 256)), 256, 0, stream>>>(scales, zps, sw, zw, n, groups,
                                                                                          words, flag);
  return cudaGetLastError();
}

}  // namespace woq
