// INT8-compute path (WoqLowpMode.INT8 with INT8 symmetric per-channel weights):
//   * prepack of the plain [N, K] int8 weight into "operand images": tiles of 64 rows x 128 k,
//     8 KB each, stored exactly as the tensor core wants a K-major 128-byte-swizzled operand
//     (row r of an 8-row group at r*128 bytes, its 16-byte chunk c at position c ^ r), so a
//     bulk copy of two consecutive images is a ready 128-row A operand - no tensor map needed;
//   * dynamic per-token symmetric quantisation of the bf16 activations (true division, round
//     half to even): the reference's dynamic_quantize_per_block for QUANT_A_PER_M_SYM;
// The GEMM is woq_i8_pair.cu.
#include <cuda_fp16.h>

#include "woq_kernels.h"

namespace woq {

namespace {

// ---- operand image layout -------------------------------------------------------------
__host__ __device__ inline int image_offset(int r /*0..63*/, int kbyte /*0..127*/) {
  return (r >> 3) * 1024 + (r & 7) * 128 + ((((kbyte >> 4) ^ (r & 7))) << 4) + (kbyte & 15);
}

__global__ void pack_int8_kernel(const int8_t* plain, int8_t* tiled, int n, int k, int tiles64,
                                 int kc_per_tile, int gate_up) {
  // one thread per 16 bytes of the image
  const int64_t total = static_cast<int64_t>(tiles64) * kc_per_tile * 512;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int chunk = i & 7, r = (i >> 3) & 63;
  const int64_t blk = i >> 9;
  const int kc = static_cast<int>(blk % kc_per_tile), t64 = static_cast<int>(blk / kc_per_tile);
  const int row128 = (t64 & 1) * 64 + r;
  const int nn = tc_tile_row_to_n(n, gate_up, t64 >> 1, row128);
  uint4 v = make_uint4(0, 0, 0, 0);
  if (nn < n) v = *reinterpret_cast<const uint4*>(plain + static_cast<int64_t>(nn) * k + kc * 128 + chunk * 16);
  *reinterpret_cast<uint4*>(tiled + blk * 8192 + image_offset(r, chunk * 16)) = v;
}

__global__ void unpack_int8_kernel(const int8_t* tiled, int8_t* plain, int n, int k, int kc_per_tile,
                                   int gate_up) {
  const int64_t chunks_per_row = k / 16;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<int64_t>(n) * chunks_per_row) return;
  const int nn = static_cast<int>(i / chunks_per_row), ch = static_cast<int>(i % chunks_per_row);
  int tile128, row128;
  if (gate_up) {
    const int half = n / 2, idx = nn < half ? nn : nn - half;
    tile128 = idx / 64;
    row128 = (idx % 64) + (nn < half ? 0 : 64);
  } else {
    tile128 = nn / 128;
    row128 = nn % 128;
  }
  const int t64 = tile128 * 2 + (row128 >> 6), r = row128 & 63;
  const int kc = ch / 8, chunk = ch % 8;
  const int64_t blk = static_cast<int64_t>(t64) * kc_per_tile + kc;
  *reinterpret_cast<uint4*>(plain + static_cast<int64_t>(nn) * k + ch * 16) =
      *reinterpret_cast<const uint4*>(tiled + blk * 8192 + image_offset(r, chunk * 16));
}

__global__ void pad_scale_kernel(const void* src, float* dst, int n, int n_pad, int dtype) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pad) return;
  float v = 0.f;
  if (i < n) {
    if (dtype == 1) v = reinterpret_cast<const float*>(src)[i];
    else if (dtype == 2) v = __half2float(reinterpret_cast<const __half*>(src)[i]);
    else v = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(src)[i]);
  }
  dst[i] = v;
}

// ---- dynamic activation quantisation ------------------------------------------------------
// Follows dynamic_quantize_per_block (csrc/cpu/aten/utils/woq_dynamic_quant.h:1526-1750).
// Symmetric: scale = max(|max|, |min|) / 127, q = clamp(nearbyint(x / scale), -128, 127) as s8.
// Asymmetric: scale = (max - min) / 255, zp = -nearbyint(min / scale),
// q = clamp(nearbyint(x / scale + zp), 0, 255) as u8.  True division, round-half-even; no
// clamping of the range to zero and no epsilon; a constant row of zeros gets codes 0.
// Per token: one range per row.  Per tensor: one range over all rows (act_row_range_kernel
// first, then every CTA folds the row ranges).  One CTA per token row.
__device__ __forceinline__ void block_min_max(float& lo, float& hi, float* red) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((tid & 31) == 0) {
    red[tid >> 5] = lo;
    red[8 + (tid >> 5)] = hi;
  }
  __syncthreads();
  lo = red[0];
  hi = red[8];
#pragma unroll
  for (int i = 1; i < 8; ++i) {
    lo = fminf(lo, red[i]);
    hi = fmaxf(hi, red[8 + i]);
  }
  __syncthreads();
}

__device__ __forceinline__ void row_min_max(const __nv_bfloat16* xr, int k, float& lo, float& hi) {
  lo = INFINITY;
  hi = -INFINITY;
  for (int i = threadIdx.x * 8; i < k; i += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(xr + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = __uint_as_float(w[j] << 16), b = __uint_as_float(w[j] & 0xffff0000u);
      lo = fminf(lo, fminf(a, b));
      hi = fmaxf(hi, fmaxf(a, b));
    }
  }
}

__global__ void __launch_bounds__(256) act_row_range_kernel(const __nv_bfloat16* x, int64_t ldx, int k,
                                                            float* range) {
  __shared__ float red[16];
  float lo, hi;
  row_min_max(x + static_cast<int64_t>(blockIdx.x) * ldx, k, lo, hi);
  block_min_max(lo, hi, red);
  if (threadIdx.x == 0) {
    range[2 * blockIdx.x] = lo;
    range[2 * blockIdx.x + 1] = hi;
  }
}

// range: null (per token) or the [m_total][2] row ranges of the whole tensor (per tensor)
template <bool ASYM>
__global__ void __launch_bounds__(256) quant_act_kernel(const __nv_bfloat16* x, int64_t ldx, int k,
                                                        int8_t* qa, float* sa, int32_t* zpa,
                                                        const float* range, int m_total) {
  __shared__ float red[16];
  const int m = blockIdx.x, tid = threadIdx.x;
  const __nv_bfloat16* xr = x + static_cast<int64_t>(m) * ldx;
  float lo, hi;
  if (range) {
    lo = INFINITY;
    hi = -INFINITY;
    for (int i = tid; i < m_total; i += 256) {
      lo = fminf(lo, range[2 * i]);
      hi = fmaxf(hi, range[2 * i + 1]);
    }
  } else {
    row_min_max(xr, k, lo, hi);
  }
  block_min_max(lo, hi, red);
  float scale, zp = 0.f;
  if (ASYM) {
    scale = __fdiv_rn(hi - lo, 255.0f);
    const float z = -rintf(__fdiv_rn(lo, scale));
    zp = z;
    if (tid == 0) zpa[m] = scale > 0.f ? static_cast<int32_t>(z) : 0;
  } else {
    scale = __fdiv_rn(fmaxf(fabsf(hi), fabsf(lo)), 127.0f);
  }
  if (tid == 0) sa[m] = scale;
  const float q_lo = ASYM ? 0.f : -128.f, q_hi = ASYM ? 255.f : 127.f;
  int8_t* qr = qa + static_cast<int64_t>(m) * k;
  for (int i = tid * 8; i < k; i += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(xr + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t out[2] = {0u, 0u};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = __uint_as_float(w[j] << 16), b = __uint_as_float(w[j] & 0xffff0000u);
      float ql = 0.f, qh = 0.f;
      if (scale > 0.f) {
        ql = fminf(fmaxf(rintf(__fdiv_rn(a, scale) + zp), q_lo), q_hi);
        qh = fminf(fmaxf(rintf(__fdiv_rn(b, scale) + zp), q_lo), q_hi);
      }
      const uint32_t c = (static_cast<uint32_t>(static_cast<int>(ql)) & 0xffu) |
                         ((static_cast<uint32_t>(static_cast<int>(qh)) & 0xffu) << 8);
      out[j >> 1] |= c << ((j & 1) * 16);
    }
    *reinterpret_cast<uint2*>(qr + i) = make_uint2(out[0], out[1]);
  }
}

// Per-token ranges (the usual modes): a row is read once, into registers (a thread holds up to eight pieces of
// eight elements), by a cluster of CL CTAs that exchange their ranges through distributed shared memory.  Bound
// by latency: 8 tokens x 14336 on one CTA per row took 5.3 us, the divisions alone keep an SM busy for 1.5 us.
// The launch after this one may start at once (its weight loads need nothing from here), and this one starts
// before the kernel that makes x has ended.
__device__ __forceinline__ float cluster_ld(const float* p, uint32_t rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
constexpr int kQuantPieces = 8;

template <bool ASYM, int CL>
__global__ void __launch_bounds__(256) quant_act_row_kernel(const __nv_bfloat16* x, int64_t ldx, int k, int8_t* qa,
                                                            float* sa, int32_t* zpa) {
  __shared__ float red[16], mine[2];
  const int m = blockIdx.x / CL, slice = blockIdx.x % CL, tid = threadIdx.x;
  const int per = (k / 8 + CL - 1) / CL, p0 = slice * per, p1 = min(k / 8, p0 + per);  // pieces of this CTA
  grid_launch_dependents();
  grid_dependency_wait();
  const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<int64_t>(m) * ldx);
  uint4 v[kQuantPieces];
  float lo = INFINITY, hi = -INFINITY;
#pragma unroll
  for (int i = 0; i < kQuantPieces; ++i)
    if (p0 + tid + i * 256 < p1) v[i] = xr[p0 + tid + i * 256];
#pragma unroll
  for (int i = 0; i < kQuantPieces; ++i) {
    if (p0 + tid + i * 256 >= p1) break;
    const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = __uint_as_float(w[j] << 16), b = __uint_as_float(w[j] & 0xffff0000u);
      lo = fminf(lo, fminf(a, b));
      hi = fmaxf(hi, fmaxf(a, b));
    }
  }
  block_min_max(lo, hi, red);
  if (CL > 1) {
    if (tid == 0) {
      mine[0] = lo;
      mine[1] = hi;
    }
    cluster_sync_all();
#pragma unroll
    for (int r = 0; r < CL; ++r) {
      lo = fminf(lo, cluster_ld(&mine[0], r));
      hi = fmaxf(hi, cluster_ld(&mine[1], r));
    }
    cluster_sync_all();  // nobody leaves while another CTA may still read its range
  }
  float scale, zp = 0.f;
  if (ASYM) {
    scale = __fdiv_rn(hi - lo, 255.0f);
    zp = -rintf(__fdiv_rn(lo, scale));
    if (tid == 0 && slice == 0) zpa[m] = scale > 0.f ? static_cast<int32_t>(zp) : 0;
  } else {
    scale = __fdiv_rn(fmaxf(fabsf(hi), fabsf(lo)), 127.0f);
  }
  if (tid == 0 && slice == 0) sa[m] = scale;
  const float q_lo = ASYM ? 0.f : -128.f, q_hi = ASYM ? 255.f : 127.f;
  uint2* qr = reinterpret_cast<uint2*>(qa + static_cast<int64_t>(m) * k);
#pragma unroll
  for (int i = 0; i < kQuantPieces; ++i) {
    if (p0 + tid + i * 256 >= p1) break;
    const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
    uint32_t out[2] = {0u, 0u};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = __uint_as_float(w[j] << 16), b = __uint_as_float(w[j] & 0xffff0000u);
      float ql = 0.f, qh = 0.f;
      if (scale > 0.f) {
        ql = fminf(fmaxf(rintf(__fdiv_rn(a, scale) + zp), q_lo), q_hi);
        qh = fminf(fmaxf(rintf(__fdiv_rn(b, scale) + zp), q_lo), q_hi);
      }
      const uint32_t c = (static_cast<uint32_t>(static_cast<int>(ql)) & 0xffu) |
                         ((static_cast<uint32_t>(static_cast<int>(qh)) & 0xffu) << 8);
      out[j >> 1] |= c << ((j & 1) * 16);
    }
    qr[p0 + tid + i * 256] = make_uint2(out[0], out[1]);
  }
}

// RMSNorm fused with the per-token quantiser: one CTA per token row.
//   y = bf16(x * rsqrt(mean(x^2) + eps) * gamma)   (fp32 arithmetic, one rounding)
// and then exactly what quant_act_kernel does on y, without y making a round trip through
// memory (it is written only when the caller wants it).  Three passes over the row, which
// stays in L1 after the first.
template <bool ASYM>
__global__ void __launch_bounds__(256) rmsnorm_quant_kernel(const __nv_bfloat16* x, int64_t ldx,
                                                            const __nv_bfloat16* gamma, float eps, int k,
                                                            __nv_bfloat16* y, int64_t ldy, int8_t* qa, float* sa,
                                                            int32_t* zpa) {
  __shared__ float red[16];
  const int m = blockIdx.x, tid = threadIdx.x;
  const __nv_bfloat16* xr = x + static_cast<int64_t>(m) * ldx;
  // pass 1: sum of squares
  float ss = 0.f;
  for (int i = tid * 8; i < k; i += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(xr + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = __uint_as_float(w[j] << 16), b = __uint_as_float(w[j] & 0xffff0000u);
      ss = fmaf(a, a, ss);
      ss = fmaf(b, b, ss);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  ss = red[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) ss += red[i];
  __syncthreads();
  const float inv = rsqrtf(__fdiv_rn(ss, static_cast<float>(k)) + eps);
  auto normed = [&](uint32_t xw, uint32_t gw, float& a, float& b) {
    a = bf16_round(__uint_as_float(xw << 16) * inv * __uint_as_float(gw << 16));
    b = bf16_round(__uint_as_float(xw & 0xffff0000u) * inv * __uint_as_float(gw & 0xffff0000u));
  };
  // pass 2: range of the normalised row (and y itself, if wanted)
  float lo = INFINITY, hi = -INFINITY;
  for (int i = tid * 8; i < k; i += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(xr + i);
    const uint4 g = *reinterpret_cast<const uint4*>(gamma + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w}, gw[4] = {g.x, g.y, g.z, g.w};
    uint32_t out[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float a, b;
      normed(w[j], gw[j], a, b);
      lo = fminf(lo, fminf(a, b));
      hi = fmaxf(hi, fmaxf(a, b));
      out[j] = (__float_as_uint(a) >> 16) | (__float_as_uint(b) & 0xffff0000u);
    }
    if (y) *reinterpret_cast<uint4*>(y + static_cast<int64_t>(m) * ldy + i) = make_uint4(out[0], out[1], out[2], out[3]);
  }
  block_min_max(lo, hi, red);
  float scale, zp = 0.f;
  if (ASYM) {
    scale = __fdiv_rn(hi - lo, 255.0f);
    const float z = -rintf(__fdiv_rn(lo, scale));
    zp = z;
    if (tid == 0) zpa[m] = scale > 0.f ? static_cast<int32_t>(z) : 0;
  } else {
    scale = __fdiv_rn(fmaxf(fabsf(hi), fabsf(lo)), 127.0f);
  }
  if (tid == 0) sa[m] = scale;
  const float q_lo = ASYM ? 0.f : -128.f, q_hi = ASYM ? 255.f : 127.f;
  int8_t* qr = qa + static_cast<int64_t>(m) * k;
  // pass 3: codes
  for (int i = tid * 8; i < k; i += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(xr + i);
    const uint4 g = *reinterpret_cast<const uint4*>(gamma + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w}, gw[4] = {g.x, g.y, g.z, g.w};
    uint32_t out[2] = {0u, 0u};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float a, b;
      normed(w[j], gw[j], a, b);
      float ql = 0.f, qh = 0.f;
      if (scale > 0.f) {
        ql = fminf(fmaxf(rintf(__fdiv_rn(a, scale) + zp), q_lo), q_hi);
        qh = fminf(fmaxf(rintf(__fdiv_rn(b, scale) + zp), q_lo), q_hi);
      }
      const uint32_t c = (static_cast<uint32_t>(static_cast<int>(ql)) & 0xffu) |
                         ((static_cast<uint32_t>(static_cast<int>(qh)) & 0xffu) << 8);
      out[j >> 1] |= c << ((j & 1) * 16);
    }
    *reinterpret_cast<uint2*>(qr + i) = make_uint2(out[0], out[1]);
  }
}

// compensation[n] = sum over k of the weight codes of row n (plain [n][k] int8): what an
// activation zero point contributes to every accumulator of that row.  One warp per row.
__global__ void __launch_bounds__(256) weight_row_sum_kernel(const int8_t* w, int n, int k, int32_t* comp) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= n) return;
  const int8_t* wr = w + static_cast<int64_t>(row) * k;
  int sum = 0;
  for (int i = lane * 16; i < k; i += 32 * 16) {
    const uint4 v = *reinterpret_cast<const uint4*>(wr + i);
    const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) sum = __dp4a(static_cast<int>(q[j]), 0x01010101, sum);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) comp[row] = sum;
}

inline unsigned blocks_for(int64_t n, int threads) {
  return static_cast<unsigned>((n + threads - 1) / threads);
}

}  // namespace

cudaError_t launch_pack_int8(const int8_t* plain, int8_t* tiled, int n, int k, int tiles64,
                             int gate_up, cudaStream_t stream) {
  const int64_t total = static_cast<int64_t>(tiles64) * (k / 128) * 512;
  pack_int8_kernel<<<blocks_for(total, 256), 256, 0, stream>>>(plain, tiled, n, k, tiles64, k / 128,
                                                               gate_up);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_unpack_int8(const int8_t* tiled, int8_t* plain, int n, int k, int gate_up,
                               cudaStream_t stream) {
  const int64_t total = static_cast<int64_t>(n) * (k / 16);
  unpack_int8_kernel<<<blocks_for(total, 256), 256, 0, stream>>>(tiled, plain, n, k, k / 128, gate_up);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_pad_scale(const void* src, float* dst, int n, int n_pad, int dtype,
                             cudaStream_t stream) {
  pad_scale_kernel<<<blocks_for(n_pad, 256), 256, 0, stream>>>(src, dst, n, n_pad, dtype);
  count_launch();
  return cudaGetLastError();
}

template <bool ASYM, int CL>
static cudaError_t launch_quant_rows(const __nv_bfloat16* x, int64_t ldx, int m, int k, int8_t* qa, float* sa,
                                     int32_t* zpa, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(m) * CL);
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (CL > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = CL;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  if (dependent_launch_enabled()) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  return cudaLaunchKernelEx(&cfg, quant_act_row_kernel<ASYM, CL>, x, ldx, k, qa, sa, zpa);
}

cudaError_t launch_quant_act(const __nv_bfloat16* x, int64_t ldx, int m, int k, int asym, int per_tensor,
                             int8_t* qa, float* sa, int32_t* zpa, float* range, cudaStream_t stream) {
  constexpr int kRowMax = kQuantPieces * 8 * 256;  // elements of a row that one CTA holds in registers
  count_launch();
  // few rows: four CTAs each, so that 8 rows x 14336 use 32 SMs
  const bool split = m <= 128 && k >= 2048 && k <= 4 * kRowMax;
  if (!per_tensor && (split || k <= kRowMax)) {
    if (split)
      return asym ? launch_quant_rows<true, 4>(x, ldx, m, k, qa, sa, zpa, stream)
                  : launch_quant_rows<false, 4>(x, ldx, m, k, qa, sa, zpa, stream);
    return asym ? launch_quant_rows<true, 1>(x, ldx, m, k, qa, sa, zpa, stream)
                : launch_quant_rows<false, 1>(x, ldx, m, k, qa, sa, zpa, stream);
  }
  if (per_tensor) {
    act_row_range_kernel<<<m, 256, 0, stream>>>(x, ldx, k, range);
    count_launch();
  }
  const float* r = per_tensor ? range : nullptr;
  if (asym)
    quant_act_kernel<true><<<m, 256, 0, stream>>>(x, ldx, k, qa, sa, zpa, r, m);
  else
    quant_act_kernel<false><<<m, 256, 0, stream>>>(x, ldx, k, qa, sa, zpa, r, m);
  return cudaGetLastError();
}

cudaError_t launch_rmsnorm_quant(const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* gamma, float eps, int m,
                                 int k, int asym, __nv_bfloat16* y, int64_t ldy, int8_t* qa, float* sa, int32_t* zpa,
                                 cudaStream_t stream) {
  if (asym)
    rmsnorm_quant_kernel<true><<<m, 256, 0, stream>>>(x, ldx, gamma, eps, k, y, ldy, qa, sa, zpa);
  else
    rmsnorm_quant_kernel<false><<<m, 256, 0, stream>>>(x, ldx, gamma, eps, k, y, ldy, qa, sa, zpa);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_weight_row_sum(const int8_t* plain, int n, int k, int32_t* comp, cudaStream_t stream) {
  weight_row_sum_kernel<<<(n + 7) / 8, 256, 0, stream>>>(plain, n, k, comp);
  count_launch();
  return cudaGetLastError();
}

}  // namespace woq
