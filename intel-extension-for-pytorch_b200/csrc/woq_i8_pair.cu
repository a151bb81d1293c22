// INT8 weights with INT8 compute and one activation range per token (or tensor) on CTA pairs: tcgen05.mma
// kind::i8, cta_group::2, exact int32 accumulators.
//
// A pair of CTAs on neighbouring SMs owns 256 output rows x up to 256 tokens; each loads its own 128 weight rows
// (operand images, ready for the tensor core) and half of the activation codes, and the leader's MMAs read both
// halves.  Work split, reduction of shared tiles and roles are those of woq_pair_tc.cu (equal contiguous shares of
// (256-row tile, token tile, k-chunk); whoever arrives last adds the parts):
//
//   warp 0      producer: weights (they are in flight before the launch may read what the quantiser writes)
//   warp 1      producer: this CTA's half of the activation codes; all four loads of a stage complete on the
//               leader's barrier
//   warp 2      (leader) MMAs
//   warp 3      tensor-memory allocation
//   warps 4-11  epilogue: int32 -> scales, bias -> bf16 tile of 64 tokens in shared memory -> post-op -> y.  Two
//               accumulator buffers, so the next tile's MMAs run meanwhile.
//
// SPLIT: few tiles; the p.split pairs of a tile form a cluster, take a part of k each and add their int32
// accumulators over distributed shared memory (as in woq_pair_tc.cu).
//
// What bounds it: with 256 columns the tensor cores (16 KB weights + 16 KB codes per SM and 512 cycles of MMAs;
// one CTA per tile and launch of 256 tokens moved 48 KB); with few columns the weights' HBM traffic.
#include "woq_pair_epilogue.cuh"

namespace woq {

namespace {

constexpr int kIpThreads = (4 + kEpiWarps) * 32;
constexpr int kIpMaxStages = 12;
constexpr int kIpHeaderBytes = 3072;      // barriers, then scales and zero points of the tile's tokens
constexpr int kIpPassTok = 64;            // tokens of the bf16 tile
constexpr int kIpOutBytes = kIpPassTok * kOutPitch;
constexpr int kIpABytes = 16384;          // 128 rows x 128 k

struct IpHeader {
  uint64_t full[kIpMaxStages];   // leader: both CTAs' weights and codes have landed
  uint64_t free_[kIpMaxStages];  // the stage's MMAs have completed
  uint64_t d_full[2], d_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  int decision;
};
static_assert(sizeof(IpHeader) <= 1024, "header too large");

__device__ __forceinline__ int ip_owner_of(int64_t b, int64_t total, int64_t pairs) {
  return static_cast<int>(((b + 1) * pairs - 1) / total);
}

__device__ __forceinline__ void pair_mma_i8_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// bias + (float(acc - compensation * zp) * scale_a) * scale_w, the integer part exact
// (csrc/cpu/aten/utils/woq.h:2310-2321)
__device__ __forceinline__ __nv_bfloat16 ip_result(int acc, int comp, int zp, float sa, float sw, const float* bias, float b) {
  float f = (static_cast<float>(acc - comp * zp) * sa) * sw;
  if (bias) f = b + f;
  return __float2bfloat16_rn(f);
}

template <bool SPLIT>
__global__ void __launch_bounds__(kIpThreads, 1)
    woq_i8_pair_kernel(const __grid_constant__ I8PairParams p, const __grid_constant__ CUtensorMap wmap,
                       const __grid_constant__ CUtensorMap qamap) {
  extern __shared__ __align__(1024) uint8_t smem[];
  IpHeader* hdr = reinterpret_cast<IpHeader*>(smem);
  float* s_sa = reinterpret_cast<float*>(smem + 1024);
  int* s_zp = reinterpret_cast<int*>(smem + 2048);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (smem_u32(smem) & 1023u) {  // (the same in both CTAs)
    if (tid == 0) atomicCAS(p.status, 0, 99);
    return;
  }
  const int half_tok = p.n_tok >> 1, b_bytes = half_tok * 128, n_stages = p.stages;
  uint8_t* a_stages = smem + kIpHeaderBytes;
  uint8_t* b_stages = a_stages + n_stages * kIpABytes;
  uint8_t* out_tile = b_stages + n_stages * b_bytes;

  const uint32_t crank = pair_cta_rank(), rank = crank & 1, leader = crank - rank;  // rank in cluster / pair
  const uint16_t pair_mask = static_cast<uint16_t>(3u << leader);
  const int pair = blockIdx.x >> 1, kcpt = p.kc_per_tile;
  // shares are dealt in units of p.unit chunks
  const int64_t pairs = gridDim.x >> 1, total = static_cast<int64_t>(p.w_tiles) * p.tok_tiles * kcpt / p.unit;
  int item0, kc00, rem0;  // item = weight tile * tok_tiles + token tile
  if (SPLIT) {
    const int sub = crank >> 1;
    item0 = pair / p.split;
    kc00 = sub * kcpt / p.split;
    rem0 = (sub + 1) * kcpt / p.split - kc00;
  } else {
    const int64_t b_begin = pair * total / pairs * p.unit, b_end = (pair + 1) * total / pairs * p.unit;
    item0 = static_cast<int>(b_begin / kcpt);
    kc00 = static_cast<int>(b_begin % kcpt);
    rem0 = static_cast<int>(b_end - b_begin);
  }

  if (tid == 0) {
    for (int s = 0; s < n_stages; ++s) {
      mbar_init(&hdr->full[s], 1);
      mbar_init(&hdr->free_[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&hdr->d_full[s], 1);
      mbar_init(&hdr->d_empty[s], 2 * kEpiWarps);
    }
    hdr->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 3) {
    pair_tmem_alloc(&hdr->tmem_base, 512);
    pair_tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  pair_sync();
  tc_fence_after_sync();
  grid_launch_dependents();
  const uint32_t tmem_base = hdr->tmem_base;
  volatile int* abort_flag = &hdr->abort_flag;

  if (warp < 2) {
    if (lane == 0) {
      if (warp == 1) grid_dependency_wait();  // the quantiser's codes
      int item = item0, kc = kc00, rem = rem0, slot = 0;
      uint32_t phase = 0;
      const uint32_t full0 = pair_map(&hdr->full[0], leader);
      while (rem > 0) {
        int tile = item / p.tok_tiles * 2 + static_cast<int>(rank);
        if (tile >= p.tiles) tile = p.tiles - 1;  // odd tile count: the last pair's second half repeats it
        const int row = item % p.tok_tiles * p.n_tok + static_cast<int>(rank) * half_tok;
        const int seg = kcpt - kc < rem ? kcpt - kc : rem;
        rem -= seg;
        for (const int end = kc + seg; kc < end; ++kc) {
          mbar_wait(&hdr->free_[slot], phase ^ 1, abort_flag, p.status, 51 + warp);
          if (warp == 0) {
            pair_tma_load_3d(a_stages + slot * kIpABytes, &wmap, 0, kc * 64, tile * 2, full0 + slot * 8);
          } else {
            if (rank == 0) mbar_arrive_expect_tx(&hdr->full[slot], 2 * (kIpABytes + b_bytes));
            pair_tma_load_3d(b_stages + slot * b_bytes, &qamap, 0, row, kc, full0 + slot * 8);
          }
          if (++slot == n_stages) {
            slot = 0;
            phase ^= 1;
          }
        }
        kc = 0;
        ++item;
      }
    }
  } else if (warp == 2) {
    if (rank == 0) {
      // the whole warp walks the stages, one elected lane issues
      // A = weights (s8), B = activations (s8, or u8 when quantised asymmetrically)
      const uint32_t idesc = pair_idesc(p.n_tok, /*s8*/ 1, p.zpa ? /*u8*/ 0 : /*s8*/ 1, /*s32*/ 2);
      const uint64_t a0 = umma_desc_k128(smem_u32(a_stages)), b0 = umma_desc_k128(smem_u32(b_stages));
      int kc = kc00, rem = rem0, slot = 0;
      uint32_t phase = 0, seg_no = 0;
      while (rem > 0) {
        int seg = kcpt - kc < rem ? kcpt - kc : rem;
        rem -= seg;
        kc = 0;
        uint32_t accumulate = 0;
        const uint32_t buf = seg_no & 1;
        mbar_wait(&hdr->d_empty[buf], ((seg_no >> 1) & 1) ^ 1, abort_flag, p.status, 53);
        for (; seg > 0; --seg) {
          mbar_wait(&hdr->full[slot], phase, abort_flag, p.status, 54);
          tc_fence_after_sync();
          if (elect_one()) {
            const uint64_t a = a0 + static_cast<uint32_t>(slot * (kIpABytes >> 4));
            const uint64_t b = b0 + static_cast<uint32_t>(slot * (b_bytes >> 4));
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              pair_mma_i8_ss(tmem_base + buf * p.n_tok, a + ks * 2, b + ks * 2, idesc, accumulate);
              accumulate = 1;
            }
            pair_commit(&hdr->free_[slot], pair_mask);
            if (seg == 1) pair_commit(&hdr->d_full[buf], pair_mask);
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
  } else if (warp >= 4) {
    const int q = warp & 3, eg = (warp - 4) >> 2, et = tid - 4 * 32;
    const int row = q * 32 + lane;
    grid_dependency_wait();  // scales, y, the fused operands and the workspace belong to this grid now
    int item = item0, kc = kc00, rem = rem0;
    uint32_t seg_no = 0;
    while (rem > 0) {
      const int seg_len = kcpt - kc < rem ? kcpt - kc : rem;
      const bool whole = seg_len == kcpt;
      const uint32_t buf = seg_no & 1;
      const uint32_t d_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * p.n_tok;
      const uint32_t d_empty0 = pair_map(&hdr->d_empty[buf], leader);
      const int tile = item / p.tok_tiles * 2 + static_cast<int>(rank);
      const int tok0 = item % p.tok_tiles * p.n_tok;
      const int mv = p.m - tok0 < p.n_tok ? p.m - tok0 : p.n_tok;
      const bool real = tile < p.tiles;
      const int n = tc_tile_row_to_n(p.n, p.gate_up, real ? tile : 0, row);
      const bool row_ok = real && n < p.n;
      const float sw = row_ok ? p.sw[n] : 0.f, bias = row_ok && p.bias ? p.bias[n] : 0.f;
      const int comp = row_ok && p.zpa ? p.comp[n] : 0;
      if (et < mv) {
        s_sa[et] = p.sa[tok0 + et];
        s_zp[et] = p.zpa ? p.zpa[tok0 + et] : 0;
      }
      named_bar_sync(1, kEpiThreads);
      mbar_wait(&hdr->d_full[buf], (seg_no >> 1) & 1, abort_flag, p.status, 55);
      tc_fence_after_sync();
      __syncwarp();
      if (SPLIT) {  // this pair's part of the tile, for the CTAs that add it up
        int* part = reinterpret_cast<int*>(a_stages) + row;
        for (int c0 = eg * 16; c0 < mv; c0 += 32) {
          uint32_t t[16];
          tmem_ld_x16(d_lane + c0, t);
          tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) part[(c0 + e) * kTcTileN] = static_cast<int>(t[e]);
        }
        break;
      }
      auto accumulators_read = [&]() {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) pair_arrive(d_empty0);
      };
      bool finish = whole && real, from_tmem = finish;
      int c_first = pair, c_last = pair;
      const int64_t tb0 = static_cast<int64_t>(item) * kcpt;  // the tile's first chunk (units of one where tiles are shared)
      auto slot_of = [&](int c) {  // partial tile of pair c, this CTA's rows
        const int s = (c == c_first && c * total / pairs < tb0) ? 1 : 0;
        return p.partials + static_cast<size_t>((c * 2 + static_cast<int>(rank)) * 2 + s) * p.part_tok * kTcTileN + row;
      };
      if (!real) {
        accumulators_read();
      } else if (!whole) {
        c_first = ip_owner_of(tb0, total, pairs);
        c_last = ip_owner_of(tb0 + kcpt - 1, total, pairs);
        const unsigned others = static_cast<unsigned>(c_last - c_first);
        uint32_t* counter = p.counters + c_first * 2 + rank;
        if (kc == 0) {
          // the beginning of the tile, the last segment of this pair: have all others arrived?
          if (et == 0) {
            uint32_t seen;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
            if (seen == others) *counter = 0;
            hdr->decision = seen == others;
          }
          named_bar_sync(1, kEpiThreads);
          from_tmem = finish = hdr->decision != 0;
        }
        if (!from_tmem) {
          int* dst = slot_of(pair);
          for (int c0 = eg * 16; c0 < mv; c0 += 32) {
            uint32_t t[16];
            tmem_ld_x16(d_lane + c0, t);
            tc_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (c0 + e < mv) __stcg(dst + static_cast<size_t>(c0 + e) * kTcTileN, static_cast<int>(t[e]));
          }
          accumulators_read();
          __threadfence();
          named_bar_sync(1, kEpiThreads);
          if (et == 0) {
            const unsigned old = atomicAdd(counter, 1u);
            if (old == others) *counter = 0;
            hdr->decision = old == others;
          }
          named_bar_sync(1, kEpiThreads);
          finish = hdr->decision != 0;
        }
        if (finish) __threadfence();
      }
      if (finish) {
        for (int t0 = 0; t0 < mv; t0 += kIpPassTok) {
          const int t1 = t0 + kIpPassTok < mv ? t0 + kIpPassTok : mv;
          for (int c0 = t0 + eg * 16; c0 < t1; c0 += 32) {
            int v[16];
            int c = c_first;
            if (from_tmem) {
              uint32_t t[16];
              tmem_ld_x16(d_lane + c0, t);
              tc_wait_ld();
#pragma unroll
              for (int e = 0; e < 16; ++e) v[e] = static_cast<int>(t[e]);
              ++c;
            } else {
#pragma unroll
              for (int e = 0; e < 16; ++e) v[e] = 0;
            }
            // three parts in flight together: a round trip to L2 per part was most of a shared tile's cost
            if (!whole)
              for (; c <= c_last; c += 3) {
                int t[3][16];
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                  const bool some = c + u <= c_last;
                  const int* src = slot_of(some ? c + u : c) + static_cast<size_t>(c0) * kTcTileN;
#pragma unroll
                  for (int e = 0; e < 16; ++e) t[u][e] = some && c0 + e < mv ? __ldcg(src + e * kTcTileN) : 0;
                }
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] += t[0][e] + t[1][e] + t[2][e];
              }
            if (p.acc_out && row_ok) {
#pragma unroll
              for (int e = 0; e < 16; ++e)
                if (c0 + e < mv) p.acc_out[static_cast<size_t>(tok0 + c0 + e) * p.n + n] = v[e];
            }
            // (columns past the last token hold anything)
            uint8_t* dst = out_tile + (c0 - t0) * kOutPitch + row * 2;
#pragma unroll
            for (int e = 0; e < 16; ++e)
              *reinterpret_cast<__nv_bfloat16*>(dst + e * kOutPitch) =
                  ip_result(v[e], comp, s_zp[c0 + e], s_sa[c0 + e], sw, p.bias, bias);
          }
          if (from_tmem && t1 == mv) accumulators_read();
          named_bar_sync(1, kEpiThreads);
          if (p.y) pair_copy_out<false>(p, p.y, out_tile, tile, tok0 + t0, t1 - t0, et);
          named_bar_sync(1, kEpiThreads);
        }
      }
      rem -= seg_len;
      kc = 0;
      ++item;
      ++seg_no;
      named_bar_sync(1, kEpiThreads);  // scales and `decision` have been read
    }
  }

  if (SPLIT) {
    __syncwarp();
    pair_sync();  // every pair's part is in its shared memory
    const int tile = item0 / p.tok_tiles * 2 + static_cast<int>(rank), tok0 = item0 % p.tok_tiles * p.n_tok;
    const int mv = p.m - tok0 < p.n_tok ? p.m - tok0 : p.n_tok;
    const int slice = (mv + p.split - 1) / p.split, t0 = static_cast<int>(crank >> 1) * slice;
    const int nt = tile >= p.tiles ? 0 : mv - t0 < slice ? mv - t0 : slice;  // this CTA's tokens t0 .. t0 + nt
    const int row = (warp & 3) * 32 + lane, n = tc_tile_row_to_n(p.n, p.gate_up, tile < p.tiles ? tile : 0, row);
    const bool row_ok = n < p.n;
    const float sw = row_ok ? p.sw[n] : 0.f, bias = row_ok && p.bias ? p.bias[n] : 0.f;
    const int comp = row_ok && p.zpa ? p.comp[n] : 0;
    const uint32_t part0 = pair_map(reinterpret_cast<const int*>(a_stages) + row, rank);
    const uint32_t part_step = pair_map(a_stages, 2) - pair_map(a_stages, 0);  // to the next pair's part
    for (int s0 = 0; s0 < nt; s0 += kIpPassTok) {
      const int ns = nt - s0 < kIpPassTok ? nt - s0 : kIpPassTok;
      // a warp: 32 rows of a token; four tokens' reads in flight together
      constexpr int kGroups = kIpThreads / 128, kBatch = 4;
      for (int t = warp >> 2; t < ns; t += kGroups * kBatch) {
        int v[kBatch][4];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int tok = t + u * kGroups;
#pragma unroll
          for (int s = 0; s < 4; ++s)
            v[u][s] = tok < ns && s < p.split
                          ? __float_as_int(pair_ld_f32(part0 + s * part_step + (t0 + s0 + tok) * (kTcTileN * 4)))
                          : 0;
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int tok = t + u * kGroups, col = t0 + s0 + tok, acc = v[u][0] + v[u][1] + v[u][2] + v[u][3];
          if (tok >= ns) break;
          if (p.acc_out && row_ok) p.acc_out[static_cast<size_t>(tok0 + col) * p.n + n] = acc;
          *reinterpret_cast<__nv_bfloat16*>(out_tile + tok * kOutPitch + row * 2) =
              ip_result(acc, comp, s_zp[col], s_sa[col], sw, p.bias, bias);
        }
      }
      __syncthreads();
      if (p.y && warp >= 4) pair_copy_out<false>(p, p.y, out_tile, tile, tok0 + t0 + s0, ns, tid - 4 * 32);
      __syncthreads();
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  pair_sync();
  if (warp == 3) {
    tc_fence_after_sync();
    pair_tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

size_t i8_pair_partial_bytes(int num_sms, int part_tok) {
  return static_cast<size_t>(num_sms) * 2 * part_tok * kTcTileN * sizeof(int);
}

cudaError_t launch_i8_pair(I8PairParams p, const CUtensorMap& wmap, const CUtensorMap& qamap, int num_sms,
                           cudaStream_t stream) {
  const int stage = kIpABytes + p.n_tok / 2 * 128;
  p.stages = (kMaxSmemBytes - kIpHeaderBytes - kIpOutBytes) / stage;
  if (p.stages > kIpMaxStages) p.stages = kIpMaxStages;
  const size_t smem = kIpHeaderBytes + static_cast<size_t>(p.stages) * stage + kIpOutBytes;
  const int64_t total = static_cast<int64_t>(p.w_tiles) * p.tok_tiles * p.kc_per_tile / p.unit;
  if (p.split > 1 && (p.kc_per_tile < p.split || static_cast<size_t>(p.n_tok) * kTcTileN * 4 >
                                                     static_cast<size_t>(p.stages) * stage))
    return cudaErrorInvalidValue;  // (pair_cut does not ask for these)
  const int64_t pairs = p.split > 1 ? static_cast<int64_t>(p.w_tiles) * p.tok_tiles * p.split
                        : total < num_sms / 2 ? total : num_sms / 2;
  auto* kern = p.split > 1 ? woq_i8_pair_kernel<true> : woq_i8_pair_kernel<false>;
  cudaError_t e = allow_max_smem(kern);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(pairs * 2));
  cfg.blockDim = dim3(kIpThreads);
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
  return cudaLaunchKernelEx(&cfg, kern, p, wmap, qamap);
}

}  // namespace woq
