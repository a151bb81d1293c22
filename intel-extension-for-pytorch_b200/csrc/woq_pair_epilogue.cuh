// The end of a tile of the CTA-pair kernels: the finished bf16 tile in shared memory -> fused post-op -> y.
#pragma once
#include "woq_kernels.h"
#include "woq_pair_common.cuh"

namespace woq {

constexpr int kEpiWarps = 8;
constexpr int kEpiThreads = kEpiWarps * 32;
constexpr int kOutPitch = kTcTileN * 2 + 16;  // bytes of one token's row of the bf16 tile (+16: bank spread)

__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ uint32_t bf_pack(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = bf_lo(w[i]);
    f[2 * i + 1] = bf_hi(w[i]);
  }
}

// Eight neighbouring columns from column n of row `o` (element offset) that may be unaligned or run
// past the limit.
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p, size_t o, int valid, bool vec) {
  if (vec && valid >= 8) return *reinterpret_cast<const uint4*>(p + o);
  const unsigned short* s = reinterpret_cast<const unsigned short*>(p) + o;
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    w[i] = 0u;
    if (2 * i < valid) w[i] = s[2 * i];
    if (2 * i + 1 < valid) w[i] |= static_cast<uint32_t>(s[2 * i + 1]) << 16;
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, size_t o, const float (&f)[8], int valid, bool vec) {
  const uint4 v = make_uint4(bf_pack(f[0], f[1]), bf_pack(f[2], f[3]), bf_pack(f[4], f[5]), bf_pack(f[6], f[7]));
  if (vec && valid >= 8) {
    *reinterpret_cast<uint4*>(p + o) = v;
    return;
  }
  unsigned short* s = reinterpret_cast<unsigned short*>(p) + o;
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i < valid) s[i] = static_cast<unsigned short>(w[i >> 1] >> (16 * (i & 1)));
}

// The finished bf16 tile S[token][128 rows] -> fused post-op -> y, by the epilogue warps.  A thread
// takes eight neighbouring columns of a token at a time, two such pieces together, so that the
// operand loads of both are in flight before the first is used.
template <bool SCATTER, class P>
__device__ __forceinline__ void pair_copy_out(const P& p, __nv_bfloat16* y, const uint8_t* S, int tile, int tok0, int mv, int tid) {
  constexpr int kBatch = 2;
  const bool silu_mul = p.fusion == FUSE_SILU_MUL;
  const int sh = silu_mul ? 3 : 4;  // pieces per token: 8 or 16
  const int items = mv << sh;
  const bool vec = p.vec != 0;
  const int fusion = p.fusion;
  for (int base = tid; base < items; base += kBatch * kEpiThreads) {
    uint4 f0[kBatch], f1[kBatch];
    size_t off[kBatch];
    int valid[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int idx = base + u * kEpiThreads;
      valid[u] = 0;
      if (idx >= items) continue;
      const int tok = idx >> sh, c = idx & ((1 << sh) - 1);
      int n0, limit;
      if (silu_mul) {
        n0 = tile * 64 + c * 8;
        limit = p.n_out;
      } else if (p.gate_up) {
        n0 = (c < 8 ? 0 : p.n / 2 - 64) + tile * 64 + c * 8;
        limit = c < 8 ? p.n / 2 : p.n;
      } else {
        n0 = tile * kTcTileN + c * 8;
        limit = p.n;
      }
      valid[u] = limit - n0 < 8 ? limit - n0 : 8;
      int64_t row = tok0 + tok;
      if constexpr (SCATTER)
        if (fusion == FUSE_SCALED_SCATTER_ADD) row = p.row_idx[tok0 + tok];
      off[u] = static_cast<size_t>(row) * p.ldy + n0;
      if (valid[u] > 0) {
        if (fusion == FUSE_ADD || fusion == FUSE_ADD_ADD || fusion == FUSE_MUL) f0[u] = load8(p.other0, off[u], valid[u], vec);
        if (fusion == FUSE_ADD_ADD) f1[u] = load8(p.other1, off[u], valid[u], vec);
        if (SCATTER && fusion == FUSE_SCALED_SCATTER_ADD) f0[u] = load8(y, off[u], valid[u], vec);
      }
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (valid[u] <= 0) continue;
      const int idx = base + u * kEpiThreads;
      const int tok = idx >> sh, c = idx & ((1 << sh) - 1);
      const uint8_t* src = S + tok * kOutPitch + c * 16;
      float r[8];
      unpack8(*reinterpret_cast<const uint4*>(src), r);
      if (silu_mul) {
        float up[8];
        unpack8(*reinterpret_cast<const uint4*>(src + 128), up);
#pragma unroll
        for (int e = 0; e < 8; ++e) r[e] = up[e] * silu_bf16(r[e]);
      } else if (fusion == FUSE_ADD || fusion == FUSE_ADD_ADD) {
        float a[8];
        unpack8(f0[u], a);
#pragma unroll
        for (int e = 0; e < 8; ++e) r[e] += a[e];
        if (fusion == FUSE_ADD_ADD) {
          unpack8(f1[u], a);
#pragma unroll
          for (int e = 0; e < 8; ++e) r[e] = bf16_round(r[e]) + a[e];
        }
      } else if (fusion == FUSE_MUL) {
        float a[8];
        unpack8(f0[u], a);
#pragma unroll
        for (int e = 0; e < 8; ++e) r[e] *= a[e];
      } else if (SCATTER && fusion == FUSE_SCALED_SCATTER_ADD) {
        if constexpr (SCATTER) {
          float a[8];
          unpack8(f0[u], a);
          const float w = __bfloat162float(p.row_w[tok0 + tok]);
#pragma unroll
          for (int e = 0; e < 8; ++e) r[e] = a[e] + r[e] * w;
        }
      } else if (fusion != FUSE_NONE) {
#pragma unroll
        for (int e = 0; e < 8; ++e) r[e] = unary_post_op(r[e], fusion);
      }
      store8(y, off[u], r, valid[u], vec);
    }
  }
}

}  // namespace woq
