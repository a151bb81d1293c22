// What surrounds the experts' linears of a mixture-of-experts layer: the (token, slot) pairs sorted by expert,
// silu(gate) * up, and the weighted sum of the experts' results.
#include "woq_kernels.h"

namespace woq {

namespace {

// Block e places the pairs of expert e, in pair order, behind those of the experts before it (a stable sort
// by expert): it counts the smaller ids first, then walks the ids again and ranks its own with ballots.  All
// blocks read all ids (64 KB for 4096 tokens and two slots, from L2): bound by the latency of a few dozen
// dependent steps, where a radix sort needs several launches.  counts[experts] is set when an id is outside
// 0 .. experts - 1 (such a pair gets position 0 and is never used).
__global__ void __launch_bounds__(1024) moe_route_kernel(const int64_t* ids, int pairs, int top_k, int experts,
                                                         int32_t* counts, int32_t* token_of, int32_t* pos_of) {
  __shared__ int warp_sum[32], warp_bad[32];
  const int e = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int below = 0, bad = 0;
  for (int i = tid; i < pairs; i += 1024) {
    const int64_t id = ids[i];
    below += id >= 0 && id < e;
    if (id < 0 || id >= experts) {
      bad = 1;
      if (e == 0) pos_of[i] = 0;
    }
  }
  below = __reduce_add_sync(0xffffffffu, below);
  bad = __reduce_or_sync(0xffffffffu, bad);
  if (lane == 0) {
    warp_sum[warp] = below;
    warp_bad[warp] = bad;
  }
  __syncthreads();
  int base = 0, any_bad = 0;
  for (int w = 0; w < 32; ++w) {
    base += warp_sum[w];
    any_bad |= warp_bad[w];
  }
  const int first = base;
  for (int i0 = 0; i0 < pairs; i0 += 1024) {
    const int i = i0 + tid;
    const bool mine = i < pairs && ids[i] == e;
    const unsigned vote = __ballot_sync(0xffffffffu, mine);
    __syncthreads();  // everyone has read the previous step's sums
    if (lane == 0) warp_sum[warp] = __popc(vote);
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) before += warp_sum[w];
      all += warp_sum[w];
    }
    if (mine) {
      const int pos = base + before + __popc(vote & ((1u << lane) - 1u));
      token_of[pos] = i / top_k;
      pos_of[i] = pos;
    }
    base += all;
  }
  if (tid == 0) {
    counts[e] = base - first;
    if (e == 0) counts[experts] = any_bad;
  }
}

// bf16(up * silu(gate)), the sigmoid and its product rounded as the linears' fused form does; memory bound.
__global__ void __launch_bounds__(256) silu_mul_kernel(const uint4* gate, const uint4* up, uint4* out, int64_t chunks) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= chunks) return;
  const uint4 a = gate[i], b = up[i];
  const uint32_t g[4] = {a.x, a.y, a.z, a.w}, u[4] = {b.x, b.y, b.z, b.w};
  uint32_t r[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float lo = __uint_as_float(u[j] << 16) * silu_bf16(__uint_as_float(g[j] << 16));
    const float hi = __uint_as_float(u[j] & 0xffff0000u) * silu_bf16(__uint_as_float(g[j] & 0xffff0000u));
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    r[j] = *reinterpret_cast<const uint32_t*>(&v);
  }
  out[i] = make_uint4(r[0], r[1], r[2], r[3]);
}

// out[t] = the experts' results of token t times their routing weights, added in expert order with one bf16
// rounding per addition (what scattering expert after expert into a zeroed tensor gives).
constexpr int kMaxTopK = 64;
__global__ void __launch_bounds__(256) moe_combine_kernel(const __nv_bfloat16* rows, const int64_t* ids,
                                                          const int32_t* pos_of, const __nv_bfloat16* w, int top_k,
                                                          int hidden, __nv_bfloat16* out) {
  __shared__ int pos[kMaxTopK];
  __shared__ float weight[kMaxTopK];
  const int64_t t = blockIdx.x;
  if (threadIdx.x < top_k) {
    // rank of this slot among the token's slots, by expert and then by slot
    const int s = threadIdx.x;
    const int64_t mine = ids[t * top_k + s];
    int rank = 0;
    for (int o = 0; o < top_k; ++o) {
      const int64_t other = ids[t * top_k + o];
      rank += other < mine || (other == mine && o < s);
    }
    pos[rank] = pos_of[t * top_k + s];
    weight[rank] = __bfloat162float(w[t * top_k + s]);
  }
  __syncthreads();
  for (int c = threadIdx.x * 8; c < hidden; c += 256 * 8) {
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    for (int s = 0; s < top_k; ++s) {
      const uint4 v = *reinterpret_cast<const uint4*>(rows + static_cast<int64_t>(pos[s]) * hidden + c);
      const uint32_t r[4] = {v.x, v.y, v.z, v.w};
      const float f = weight[s];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[2 * e] = bf16_round(acc[2 * e] + __uint_as_float(r[e] << 16) * f);
        acc[2 * e + 1] = bf16_round(acc[2 * e + 1] + __uint_as_float(r[e] & 0xffff0000u) * f);
      }
    }
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      o[e] = (__float_as_uint(acc[2 * e]) >> 16) | (__float_as_uint(acc[2 * e + 1]) & 0xffff0000u);
    *reinterpret_cast<uint4*>(out + t * hidden + c) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace

cudaError_t launch_moe_route(const int64_t* ids, int64_t pairs, int top_k, int experts, int32_t* counts,
                             int32_t* token_of, int32_t* pos_of, cudaStream_t stream) {
  moe_route_kernel<<<experts, 1024, 0, stream>>>(ids, static_cast<int>(pairs), top_k, experts, counts, token_of, pos_of);
  return cudaGetLastError();
}

cudaError_t launch_silu_mul(const __nv_bfloat16* gate, const __nv_bfloat16* up, __nv_bfloat16* out, int64_t count,
                            cudaStream_t stream) {
  const int64_t chunks = count / 8;
  silu_mul_kernel<<<static_cast<unsigned>(ceil_div(chunks, 256)), 256, 0, stream>>>(
      reinterpret_cast<const uint4*>(gate), reinterpret_cast<const uint4*>(up), reinterpret_cast<uint4*>(out), chunks);
  return cudaGetLastError();
}

cudaError_t launch_moe_combine(const __nv_bfloat16* rows, const int64_t* ids, const int32_t* pos_of,
                               const __nv_bfloat16* w, int64_t tokens, int top_k, int hidden, __nv_bfloat16* out,
                               cudaStream_t stream) {
  moe_combine_kernel<<<static_cast<unsigned>(tokens), 256, 0, stream>>>(rows, ids, pos_of, w, top_k, hidden, out);
  return cudaGetLastError();
}

}  // namespace woq
