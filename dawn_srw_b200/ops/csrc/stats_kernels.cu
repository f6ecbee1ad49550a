// Per-token score statistics of the SRW pool op without a pass over the scores.
//
// With s_u = <h, e_u> over a pool of U units,
//   mean_U s   = <h, sum_u e_u> / U               (esum, [r])
//   mean_U s^2 = h (E^T E) h^T / U                (Gram matrix G, [r, r])
// so mu, sigma, the threshold tau = mu + tau_off * sigma and 1 / sigma of every
// token follow from hg = h . G (a [N, r] x [r, r] GEMM on the tensor engine, G
// split into two bf16 terms so that the product is fp32-accurate) and one row
// kernel.  The reference sweeps all [T, U] scores for the same numbers
// (models/dawn_spatial_v41_exp.py:433-464).  The kernels here are the row parts,
// forward and backward; the column sums of h (the per-unit mean score used by the
// load-balance and dead-unit terms is emb . mean_t h) ride along.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common/ptx.cuh"
#include "dsb_api_ops.h"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

constexpr float kVarFloor = 1e-12f;   // variance floor under the square root
constexpr float kSdEps = 1e-8f;       // sigma = sqrt(var) + eps, as in the reference
constexpr int kMaxR = 512;            // d_route of every supported model is <= 384

// One warp per row, grid-stride; a block adds its column sums of h into hsum
// once at the end (shared-memory partials first).
// KR: values of a row per lane (r <= 32 KR); with room for 512 columns at every r, a row of 128 spent
// three quarters of its instructions on predicated-off ones (see score_route_bwd_kernel).
// hg = g1 + g2 (row stride ldg): the products with the two bf16 terms of G, side by side in one
// GEMM's output; g2 may be null.  Row n is token n % T of route n / T, off has strides (o_st, o_sr).
template <int KR>
__global__ void score_stats_fwd_kernel(const float* __restrict__ g1, const float* __restrict__ g2,
                                       long long ldg, const __nv_bfloat16* __restrict__ h,
                                       long long ldh, const float* __restrict__ esum,
                                       const float* __restrict__ off, long long o_st, long long o_sr,
                                       int T, float inv_u, int N, int r,
                                       float* __restrict__ tau, float* __restrict__ isd,
                                       float* __restrict__ mu_out, float* __restrict__ sd_out,
                                       float* __restrict__ hsum) {
  __shared__ float s_sum[kMaxR];
  for (int j = threadIdx.x; j < r; j += blockDim.x) s_sum[j] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  float csum[KR];
#pragma unroll
  for (int k = 0; k < KR; ++k) csum[k] = 0.f;
  for (int row = blockIdx.x * warps + (threadIdx.x >> 5); row < N; row += gridDim.x * warps) {
    const float* g = g1 + static_cast<size_t>(row) * ldg;
    const float* gl = g2 != nullptr ? g2 + static_cast<size_t>(row) * ldg : nullptr;
    const __nv_bfloat16* hr = h + static_cast<size_t>(row) * ldh;
    float m2 = 0.f, m1 = 0.f;
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      const int j = lane + 32 * k;
      if (j < r) {
        const float hv = __bfloat162float(hr[j]);
        m2 = fmaf(gl != nullptr ? g[j] + gl[j] : g[j], hv, m2);
        m1 = fmaf(esum[j], hv, m1);
        csum[k] += hv;
      }
    }
    m2 = warp_sum(m2) * inv_u;
    const float mu = warp_sum(m1) * inv_u;
    if (lane == 0) {
      const float sd = sqrtf(fmaxf(m2 - mu * mu, kVarFloor)) + kSdEps;
      tau[row] = fmaf(off[(row % T) * o_st + (row / T) * o_sr], sd, mu);
      isd[row] = 1.f / sd;
      mu_out[row] = mu;
      sd_out[row] = sd;
    }
  }
  if (hsum != nullptr) {
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      const int j = lane + 32 * k;
      if (j < r) atomicAdd(&s_sum[j], csum[k]);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < r; j += blockDim.x) atomicAdd(hsum + j, s_sum[j]);
  }
}

// Backward of the row part.  Given the cotangents of tau, 1/sigma and of the
// column sums of h:
//   d_sd = d_tau * off - d_isd / sd^2,   d_off = d_tau * sd
//   d_var = d_sd / (2 sqrt(var))  (0 where the variance floor is active)
//   d_mu  = d_tau - 2 mu d_var
//   dh    = (2 d_var / U) hg + (d_mu / U) esum + d_hsum + d_hb   (d_hb: cotangent that
//           reached the bf16 copy of h from the gate kernels)
//   w     = bf16(d_var * h)      operand of  dG = w^T h / U  (engine GEMM)
//   d_esum += (d_mu / U) h       (shared-memory partials, one atomic per column and block)
__global__ void score_stats_bwd_kernel(const float* __restrict__ d_tau, const float* __restrict__ d_isd,
                                       const float* __restrict__ d_hsum,
                                       const __nv_bfloat16* __restrict__ d_hb,
                                       const float* __restrict__ off,
                                       const float* __restrict__ mu_in, const float* __restrict__ sd_in,
                                       const float* __restrict__ hg, const __nv_bfloat16* __restrict__ h,
                                       long long ldh, const float* __restrict__ esum, float inv_u, int N,
                                       int r, float* __restrict__ dh, __nv_bfloat16* __restrict__ w,
                                       long long ldw, float* __restrict__ d_off,
                                       float* __restrict__ d_esum) {
  __shared__ float s_sum[kMaxR];
  for (int j = threadIdx.x; j < r; j += blockDim.x) s_sum[j] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  float csum[kMaxR / 32];
#pragma unroll
  for (int k = 0; k < kMaxR / 32; ++k) csum[k] = 0.f;
  for (int row = blockIdx.x * warps + (threadIdx.x >> 5); row < N; row += gridDim.x * warps) {
    const float sd = sd_in[row], mu = mu_in[row];
    const float dt = d_tau != nullptr ? d_tau[row] : 0.f;
    const float di = d_isd != nullptr ? d_isd[row] : 0.f;
    const float d_sd = dt * off[row] - di / (sd * sd);
    const float sq = sd - kSdEps;
    const float d_var = sq > 1.5e-6f ? d_sd / (2.f * sq) : 0.f;   // sqrt(floor) = 1e-6
    const float d_mu = dt - 2.f * mu * d_var;
    if (lane == 0) d_off[row] = dt * sd;
    const float a = 2.f * d_var * inv_u, b = d_mu * inv_u;
    const float* g = hg + static_cast<size_t>(row) * r;
    const __nv_bfloat16* hr = h + static_cast<size_t>(row) * ldh;
    float* dr = dh + static_cast<size_t>(row) * r;
    __nv_bfloat16* wr = w + static_cast<size_t>(row) * ldw;
#pragma unroll
    for (int k = 0; k < kMaxR / 32; ++k) {
      const int j = lane + 32 * k;
      if (j < r) {
        const float hv = __bfloat162float(hr[j]);
        float acc = fmaf(a, g[j], fmaf(b, esum[j], d_hsum != nullptr ? d_hsum[j] : 0.f));
        if (d_hb != nullptr) acc += __bfloat162float(d_hb[static_cast<size_t>(row) * r + j]);
        dr[j] = acc;
        wr[j] = __float2bfloat16(d_var * hv);
        csum[k] = fmaf(b, hv, csum[k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kMaxR / 32; ++k) {
    const int j = lane + 32 * k;
    if (j < r) atomicAdd(&s_sum[j], csum[k]);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < r; j += blockDim.x) atomicAdd(d_esum + j, s_sum[j]);
}

// The routes of one pool call, packed for the tensor engine: h fp32 [T, R, r] (strides h_st, h_sr)
// -> bf16 [R * T, r], route-major, so that a route's rows are one operand.  The buffers that
// the kernels after it add into (denominators, column sums) are cleared on the way.
template <bool kVec>
__global__ void __launch_bounds__(256) score_pack_kernel(const float* __restrict__ h, long long h_st,
                                                         long long h_sr, int T, int R, int r,
                                                         __nv_bfloat16* __restrict__ hb,
                                                         float* __restrict__ z1, int n1,
                                                         float* __restrict__ z2, int n2) {
  const long long stride = static_cast<long long>(gridDim.x) * 256;
  const long long first = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  for (long long i = first; i < n1; i += stride) z1[i] = 0.f;
  for (long long i = first; i < n2; i += stride) z2[i] = 0.f;
  const int per = r >> 3;                              // r % 8 == 0
  const long long total = static_cast<long long>(T) * R * per;
  for (long long i = first; i < total; i += stride) {
    const int n = static_cast<int>(i / per), c = static_cast<int>(i - static_cast<long long>(n) * per);
    const float* src = h + (n % T) * h_st + (n / T) * h_sr + 8 * c;
    float v[8];
    if constexpr (kVec) {
      const float4 a = reinterpret_cast<const float4*>(src)[0], b = reinterpret_cast<const float4*>(src)[1];
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = src[j];
    }
    uint4 q;
    uint32_t* w = reinterpret_cast<uint32_t*>(&q);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 p2 = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
      w[j] = *reinterpret_cast<const uint32_t*>(&p2);
    }
    *reinterpret_cast<uint4*>(hb + static_cast<size_t>(n) * r + 8 * c) = q;
  }
}

// Everything of a call's backward pass that is a matter of token rows, one warp per row n
// (route-major): the sigma path of the gate, the statistics, and the sum of what reaches h.
//   dsz = (1/sigma) (<h, dh32> + tau dtau),  d_isd = dsz sigma^2      (gates that use sigma)
//   then the row part above with d_tau = dtau; dh = ... + d_hsum + dh32.
// dh32 (fp32 [N, r]) is ds . emb straight from its GEMM.  dh is [T, R, r], d_off [T, R].  16 x 512 tokens on
// the 40M model: 24.7 us a call with KR = 16, 13.8 with the KR of their r = 128.
template <int KR>
__global__ void __launch_bounds__(256) score_route_bwd_kernel(
    const float* __restrict__ dtau, const float* __restrict__ dh32, const float* __restrict__ d_hsum,
    const float* __restrict__ off, long long o_st, long long o_sr, const float* __restrict__ tau,
    const float* __restrict__ isd, const float* __restrict__ mu_in, const float* __restrict__ sd_in,
    const float* __restrict__ g1, const float* __restrict__ g2, long long ldg,
    const __nv_bfloat16* __restrict__ h, const float* __restrict__ esum, float inv_u, int sigma_path,
    int T, int R, int r, float* __restrict__ dh, __nv_bfloat16* __restrict__ w,
    float* __restrict__ d_off, float* __restrict__ d_esum) {
  __shared__ float s_sum[kMaxR];
  for (int j = threadIdx.x; j < r; j += blockDim.x) s_sum[j] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5, N = T * R;
  float csum[KR];
#pragma unroll
  for (int k = 0; k < KR; ++k) csum[k] = 0.f;
  for (int row = blockIdx.x * warps + (threadIdx.x >> 5); row < N; row += gridDim.x * warps) {
    const int t = row % T, ri = row / T;
    const float sd = sd_in[row], mu = mu_in[row], dt = dtau[row];
    const __nv_bfloat16* hr = h + static_cast<size_t>(row) * r;
    const float* dr32 = dh32 + static_cast<size_t>(row) * r;
    float hv[KR], dv[KR];
    float dot = 0.f;
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      const int j = lane + 32 * k;
      hv[k] = j < r ? __bfloat162float(hr[j]) : 0.f;
      dv[k] = j < r ? dr32[j] : 0.f;
      dot = fmaf(hv[k], dv[k], dot);
    }
    float di = 0.f;
    if (sigma_path) {
      const float is = isd[row];
      di = is * (warp_sum(dot) + tau[row] * dt) / (is * is);
    }
    const float d_sd = dt * off[t * o_st + ri * o_sr] - di / (sd * sd);
    const float sq = sd - kSdEps;
    const float d_var = sq > 1.5e-6f ? d_sd / (2.f * sq) : 0.f;   // sqrt(floor) = 1e-6
    const float d_mu = dt - 2.f * mu * d_var;
    if (lane == 0) d_off[static_cast<size_t>(t) * R + ri] = dt * sd;
    const float a = 2.f * d_var * inv_u, b = d_mu * inv_u;
    const float* gr1 = g1 + static_cast<size_t>(row) * ldg;
    const float* gr2 = g2 + static_cast<size_t>(row) * ldg;
    float* dr = dh + (static_cast<size_t>(t) * R + ri) * r;
    __nv_bfloat16* wr = w + static_cast<size_t>(row) * r;
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      const int j = lane + 32 * k;
      if (j < r) {
        const float acc = fmaf(a, gr1[j] + gr2[j], fmaf(b, esum[j], d_hsum != nullptr ? d_hsum[j] : 0.f));
        dr[j] = acc + dv[k];
        wr[j] = __float2bfloat16(d_var * hv[k]);
        csum[k] = fmaf(b, hv[k], csum[k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    const int j = lane + 32 * k;
    if (j < r) atomicAdd(&s_sum[j], csum[k]);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < r; j += blockDim.x) atomicAdd(d_esum + j, s_sum[j]);
}

// A handful of rows (decoding): the whole statistic in one launch, fp32 throughout.
// Row n is token t = n % T of route ri = n / T (route-major output rows, the order in which
// the routes of one pool are stacked into one gate-kernel call).  h G h^T is a sum over the rows of
// G, so a cluster of eight CTAs shares them and only scalars meet in the first CTA; thread j owns
// column j of the symmetric G (consecutive addresses), sixteen loads in flight.  One block per row
// pulled all of G through one SM: 7.2 us at r = 256 (256 KB) and 15 us at r = 384, a tenth of a
// decoded token (400M, one sequence: 3.03 ms a token, 2.80 with this; 1B, six: 9.25 and 8.58).  `zero` is scratch of the launch that follows (partial sums, counters).
constexpr int kRowCtas = 8, kRowThreads = 256;
__global__ void __cluster_dims__(kRowCtas, 1, 1) __launch_bounds__(kRowThreads)
score_stats_rows_kernel(const float* __restrict__ h, long long h_st, long long h_sr,
                        const float* __restrict__ off, long long o_st, long long o_sr,
                        const float* __restrict__ gram, const float* __restrict__ esum, float inv_u,
                        int T, int r, float* __restrict__ tau, float* __restrict__ isd,
                        __nv_bfloat16* __restrict__ hb, float* __restrict__ zero, long long n_zero) {
  __shared__ float s_h[kMaxR];
  __shared__ float s_red[2][kRowThreads / 32];
  __shared__ float s_m2;
  const int cta = blockIdx.x, n = blockIdx.y, t = n % T, ri = n / T, tid = threadIdx.x;
  const float* hr = h + t * h_st + ri * h_sr;
  for (long long i = (static_cast<long long>(n) * kRowCtas + cta) * kRowThreads + tid; i < n_zero;
       i += static_cast<long long>(gridDim.y) * kRowCtas * kRowThreads)
    zero[i] = 0.f;
  for (int j = tid; j < r; j += kRowThreads) {
    const __nv_bfloat16 q = __float2bfloat16(hr[j]);     // the gate kernels see bf16(h)
    if (cta == 0) hb[static_cast<size_t>(n) * r + j] = q;
    s_h[j] = __bfloat162float(q);
  }
  __syncthreads();
  const int per = (r + kRowCtas - 1) / kRowCtas;
  const int i0 = cta * per, i1 = min(r, i0 + per);
  float m2 = 0.f, m1 = 0.f;
  for (int j = tid; j < r; j += kRowThreads) {
    float a[4] = {0.f, 0.f, 0.f, 0.f};
    const float* col = gram + j;
    int i = i0;
    for (; i + 16 <= i1; i += 16) {
      float v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = col[static_cast<size_t>(i + k) * r];
#pragma unroll
      for (int k = 0; k < 16; ++k) a[k & 3] = fmaf(v[k], s_h[i + k], a[k & 3]);
    }
    for (; i < i1; ++i) a[0] = fmaf(col[static_cast<size_t>(i) * r], s_h[i], a[0]);
    m2 = fmaf((a[0] + a[1]) + (a[2] + a[3]), s_h[j], m2);
    if (cta == 0) m1 = fmaf(esum[j], s_h[j], m1);
  }
  m2 = warp_sum(m2);
  m1 = warp_sum(m1);
  if ((tid & 31) == 0) { s_red[0][tid >> 5] = m2; s_red[1][tid >> 5] = m1; }
  __syncthreads();
  m2 = m1 = 0.f;
#pragma unroll
  for (int w = 0; w < kRowThreads / 32; ++w) { m2 += s_red[0][w]; m1 += s_red[1][w]; }
  if (tid == 0) s_m2 = m2;
  dsb::cluster_sync_all();
  if (cta == 0 && tid == 0) {
    m2 = 0.f;
#pragma unroll
    for (int k = 0; k < kRowCtas; ++k) m2 += dsb::ld_cluster_f32(dsb::mapa_shared(dsb::smem_u32(&s_m2), k));
    const float mu = m1 * inv_u;
    const float sd = sqrtf(fmaxf(m2 * inv_u - mu * mu, kVarFloor)) + kSdEps;
    tau[n] = fmaf(off[t * o_st + ri * o_sr], sd, mu);
    isd[n] = 1.f / sd;
  }
  dsb::cluster_sync_all();   // nobody leaves while its shared memory may still be read
}

// ------------------------------------------------------------ load balance
// m_u = <e_u, hbar>, hbar = hsum * inv_n (mean score of unit u over the tokens), and from it
//   lb = var / (mean^2 + var + 0.01),   mean = sum_u m_u / U,   var = sum_u m_u^2 / U - mean^2.
// The op reads the pool's bf16 embedding rows once (51 MB for 100 000 units of 256) and is bound
// by those bytes at that size, by its launches below a few MB; so it is one pass that also takes
// the sums (per-block partials, fixed order), and one block that finishes the scalar.  As a chain
// of tensor ops on an fp32 copy of the rows it was 14 launches forward and about 35 backward.
// A unit belongs to `lpu` lanes (a power of two), each with every lpu-th 16-byte chunk of the row.
constexpr int kLbThreads = 256, kLbUnroll = 4;
constexpr float kLbEps = 1e-2f;

__device__ __forceinline__ void unpack_bf16x8(const uint4& q, float (&f)[8]) {
  const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __bfloat1622float2(h2[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}

// KC: chunks per lane (r <= 8 * lpu * KC).
template <int KC>
__global__ void __launch_bounds__(kLbThreads) lb_fwd_kernel(const __nv_bfloat16* __restrict__ emb,
                                                            long long lde, const float* __restrict__ hsum,
                                                            float inv_n, int U, int r, int lpu,
                                                            float* __restrict__ m_u,
                                                            float* __restrict__ part) {
  __shared__ float s_red[2][kLbThreads / 32];
  const int lane = threadIdx.x & 31, sub = lane & (lpu - 1), chunks = r >> 3;
  const int per_warp = 32 / lpu;
  float hb[KC][8];
#pragma unroll
  for (int k = 0; k < KC; ++k) {
    const int c = sub + lpu * k;
#pragma unroll
    for (int j = 0; j < 8; ++j) hb[k][j] = c < chunks ? hsum[8 * c + j] * inv_n : 0.f;
  }
  const int stride = gridDim.x * (kLbThreads / 32) * per_warp;
  const int first = (blockIdx.x * (kLbThreads / 32) + (threadIdx.x >> 5)) * per_warp;   // of the warp
  float s1 = 0.f, s2 = 0.f;
  for (int u0 = first; u0 < U; u0 += kLbUnroll * stride) {                // warp-uniform trip count
    uint4 q[kLbUnroll][KC];
#pragma unroll
    for (int i = 0; i < kLbUnroll; ++i) {
      const int u = u0 + i * stride + lane / lpu;
#pragma unroll
      for (int k = 0; k < KC; ++k) {
        const int c = sub + lpu * k;
        q[i][k] = u < U && c < chunks
                      ? *reinterpret_cast<const uint4*>(emb + static_cast<size_t>(u) * lde + 8 * c)
                      : make_uint4(0u, 0u, 0u, 0u);
      }
    }
#pragma unroll
    for (int i = 0; i < kLbUnroll; ++i) {
      const int u = u0 + i * stride + lane / lpu;
      float a = 0.f;
#pragma unroll
      for (int k = 0; k < KC; ++k) {
        float e[8];
        unpack_bf16x8(q[i][k], e);
#pragma unroll
        for (int j = 0; j < 8; ++j) a = fmaf(e[j], hb[k][j], a);
      }
      for (int o = lpu >> 1; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if (sub == 0 && u < U) {
        m_u[u] = a;
        s1 += a;
        s2 = fmaf(a, a, s2);
      }
    }
  }
  s1 = warp_sum(s1);
  s2 = warp_sum(s2);
  if (lane == 0) { s_red[0][threadIdx.x >> 5] = s1; s_red[1][threadIdx.x >> 5] = s2; }
  __syncthreads();
  if (threadIdx.x < 2) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kLbThreads / 32; ++w) t += s_red[threadIdx.x][w];
    part[2 * blockIdx.x + threadIdx.x] = t;
  }
}

// lb[0] and stat = (mean, mean^2 + var + eps) from the blocks' partial sums.
__global__ void __launch_bounds__(256) lb_finish_kernel(const float* __restrict__ part, int blocks,
                                                        float units, float* __restrict__ lb,
                                                        float* __restrict__ stat) {
  __shared__ float s_red[2][8];
  float s1 = 0.f, s2 = 0.f;
  for (int b = threadIdx.x; b < blocks; b += 256) { s1 += part[2 * b]; s2 += part[2 * b + 1]; }
  s1 = warp_sum(s1);
  s2 = warp_sum(s2);
  if ((threadIdx.x & 31) == 0) { s_red[0][threadIdx.x >> 5] = s1; s_red[1][threadIdx.x >> 5] = s2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    s1 = s2 = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) { s1 += s_red[0][w]; s2 += s_red[1][w]; }
    const float mean = s1 / units, var = s2 / units - mean * mean;
    const float q = mean * mean + var + kLbEps;
    lb[0] = var / q;
    stat[0] = mean;
    stat[1] = q;
  }
}

// With q = mean^2 + var + eps:  d mean = -2 mean / q,  d (sum m^2 / U) = (mean^2 + eps) / q^2, so
//   dm_u = g / U * (d mean + 2 m_u d(sum m^2 / U)),   dmn[u] = dm_u * inv_n,
//   d_hsum = sum_u dmn[u] e_u: a slab of shared memory per warp, a row of part per block, and a launch
// that adds the rows up in order, so that it repeats bit by bit.  The embedding gradient dmn[u] * hsum is left to
// rank1_add_kernel, which takes the calls of all layers in one pass over the gradient buffer.
template <int KC>
__global__ void __launch_bounds__(kLbThreads) lb_bwd_kernel(const __nv_bfloat16* __restrict__ emb,
                                                            long long lde, const float* __restrict__ m_u,
                                                            const float* __restrict__ stat,
                                                            const float* __restrict__ g_lb, float units,
                                                            float inv_n, int U, int r, int lpu,
                                                            float* __restrict__ dmn,
                                                            float* __restrict__ part) {
  __shared__ float s_sum[kLbThreads / 32][kMaxR];
  const int lane = threadIdx.x & 31, sub = lane & (lpu - 1), chunks = r >> 3;
  const int per_warp = 32 / lpu;
  const float mean = stat[0], q = stat[1], g = g_lb[0] * inv_n / units;
  const float c0 = -2.f * mean / q * g, c1 = 2.f * (fmaf(mean, mean, kLbEps) / q) / q * g;
  float acc[KC][8];
#pragma unroll
  for (int k = 0; k < KC; ++k)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[k][j] = 0.f;
  const int stride = gridDim.x * (kLbThreads / 32) * per_warp;
  const int first = (blockIdx.x * (kLbThreads / 32) + (threadIdx.x >> 5)) * per_warp;
  for (int u0 = first; u0 < U; u0 += kLbUnroll * stride) {
    uint4 e4[kLbUnroll][KC];
    float d[kLbUnroll];
#pragma unroll
    for (int i = 0; i < kLbUnroll; ++i) {
      const int u = u0 + i * stride + lane / lpu;
      d[i] = u < U ? fmaf(c1, m_u[u], c0) : 0.f;
#pragma unroll
      for (int k = 0; k < KC; ++k) {
        const int c = sub + lpu * k;
        e4[i][k] = u < U && c < chunks
                       ? *reinterpret_cast<const uint4*>(emb + static_cast<size_t>(u) * lde + 8 * c)
                       : make_uint4(0u, 0u, 0u, 0u);
      }
    }
#pragma unroll
    for (int i = 0; i < kLbUnroll; ++i) {
      const int u = u0 + i * stride + lane / lpu;
      if (sub == 0 && u < U) dmn[u] = d[i];
#pragma unroll
      for (int k = 0; k < KC; ++k) {
        float e[8];
        unpack_bf16x8(e4[i][k], e);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[k][j] = fmaf(d[i], e[j], acc[k][j]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < KC; ++k) {
    const int c = sub + lpu * k;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      for (int o = lpu; o < 32; o <<= 1) acc[k][j] += __shfl_xor_sync(0xffffffffu, acc[k][j], o);
      if (lane < lpu && c < chunks) s_sum[threadIdx.x >> 5][8 * c + j] = acc[k][j];
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < r; j += kLbThreads) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kLbThreads / 32; ++w) t += s_sum[w][j];
    part[static_cast<size_t>(blockIdx.x) * r + j] = t;
  }
}

// g[u, :] += sum_l dm[l, u] * hs[l, :] (fp32 [U, r], row stride ldg): one read and write of the
// gradient rows for up to kRank1Max layers instead of one per layer.
constexpr int kRank1Max = 24;
__global__ void __launch_bounds__(256) rank1_add_kernel(float* __restrict__ g, long long ldg,
                                                        const float* __restrict__ dm,
                                                        const float* __restrict__ hs, int L, int U,
                                                        int r) {
  extern __shared__ __align__(16) float s_hs[];                  // [L][r]
  for (int i = threadIdx.x; i < L * r; i += 256) s_hs[i] = hs[i];
  __syncthreads();
  const int c4 = r >> 2;
  const long long total = static_cast<long long>(U) * c4;
  for (long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * 256) {
    const int u = static_cast<int>(i / c4), c = static_cast<int>(i - static_cast<long long>(u) * c4);
    float4* dst = reinterpret_cast<float4*>(g + static_cast<size_t>(u) * ldg) + c;
    float4 a = *dst;
#pragma unroll 4
    for (int l = 0; l < L; ++l) {
      const float d = dm[static_cast<size_t>(l) * U + u];
      const float4 h = *reinterpret_cast<const float4*>(s_hs + l * r + 4 * c);
      a.x = fmaf(d, h.x, a.x); a.y = fmaf(d, h.y, a.y);
      a.z = fmaf(d, h.z, a.z); a.w = fmaf(d, h.w, a.w);
    }
    *dst = a;
  }
}

int lb_lanes(int r) {
  int lpu = 1;
  while (lpu < 32 && 8 * lpu < r) lpu *= 2;
  return lpu;
}

int stats_grid(int N) {
  const int blocks = (N + 7) / 8;
  return blocks < 148 * 4 ? (blocks < 1 ? 1 : blocks) : 148 * 4;
}

}  // namespace

extern "C" int dsb_score_stats_fwd(const float* hg, const float* hg2, long long ldg, const void* h_bf16,
                                   long long ldh, const float* esum, const float* off, long long o_st,
                                   long long o_sr, int T, float inv_u, int N, int r,
                                   float* tau, float* isd, float* mu, float* sd, float* hsum,
                                   cudaStream_t stream) {
  if (N <= 0) return 0;
  if (r <= 0 || r > kMaxR) return 801;
  auto kern = r <= 128 ? score_stats_fwd_kernel<4> : r <= 256 ? score_stats_fwd_kernel<8> : score_stats_fwd_kernel<16>;
  kern<<<stats_grid(N), 256, 0, stream>>>(
      hg, hg2, ldg, static_cast<const __nv_bfloat16*>(h_bf16), ldh, esum, off, o_st, o_sr, T, inv_u, N, r,
      tau, isd, mu, sd, hsum);
  return cudaGetLastError() == cudaSuccess ? 0 : 802;
}

extern "C" int dsb_score_pack(const float* h, long long h_st, long long h_sr, int T, int R, int r,
                              void* hb_bf16, float* z1, int n1, float* z2, int n2,
                              cudaStream_t stream) {
  if (T <= 0 || R <= 0) return 0;
  if (r <= 0 || r % 8 != 0 || r > kMaxR) return 801;
  const long long n = static_cast<long long>(T) * R * (r >> 3);
  const int blocks = static_cast<int>(n / 256 + 1 < 148 * 8 ? n / 256 + 1 : 148 * 8);
  __nv_bfloat16* hb = static_cast<__nv_bfloat16*>(hb_bf16);
  if (((reinterpret_cast<uintptr_t>(h) & 15) | (h_st & 3) | (h_sr & 3)) == 0)
    score_pack_kernel<true><<<blocks, 256, 0, stream>>>(h, h_st, h_sr, T, R, r, hb, z1, n1, z2, n2);
  else
    score_pack_kernel<false><<<blocks, 256, 0, stream>>>(h, h_st, h_sr, T, R, r, hb, z1, n1, z2, n2);
  return cudaGetLastError() == cudaSuccess ? 0 : 802;
}

extern "C" int dsb_score_route_bwd(const float* dtau, const float* dh32, const float* d_hsum,
                                   const float* off, long long o_st, long long o_sr, const float* tau,
                                   const float* isd, const float* mu, const float* sd, const float* hg,
                                   const float* hg2, long long ldg, const void* h_bf16,
                                   const float* esum, float inv_u, int sigma_path, int T, int R, int r,
                                   float* dh, void* w_bf16, float* d_off, float* d_esum,
                                   cudaStream_t stream) {
  if (T <= 0 || R <= 0) return 0;
  if (r <= 0 || r > kMaxR) return 801;
  auto kern = r <= 128 ? score_route_bwd_kernel<4> : r <= 256 ? score_route_bwd_kernel<8> : score_route_bwd_kernel<16>;
  kern<<<stats_grid(T * R), 256, 0, stream>>>(
      dtau, dh32, d_hsum, off, o_st, o_sr, tau, isd, mu, sd, hg, hg2, ldg,
      static_cast<const __nv_bfloat16*>(h_bf16), esum, inv_u, sigma_path, T, R, r, dh,
      static_cast<__nv_bfloat16*>(w_bf16), d_off, d_esum);
  return cudaGetLastError() == cudaSuccess ? 0 : 802;
}

extern "C" int dsb_score_stats_bwd(const float* d_tau, const float* d_isd, const float* d_hsum,
                                   const void* d_hb_bf16, const float* off, const float* mu,
                                   const float* sd,
                                   const float* hg, const void* h_bf16, long long ldh,
                                   const float* esum, float inv_u, int N, int r, float* dh,
                                   void* w_bf16, long long ldw, float* d_off, float* d_esum,
                                   cudaStream_t stream) {
  if (N <= 0) return 0;
  if (r <= 0 || r > kMaxR) return 801;
  score_stats_bwd_kernel<<<stats_grid(N), 256, 0, stream>>>(
      d_tau, d_isd, d_hsum, static_cast<const __nv_bfloat16*>(d_hb_bf16), off, mu, sd, hg,
      static_cast<const __nv_bfloat16*>(h_bf16), ldh, esum,
      inv_u, N, r, dh, static_cast<__nv_bfloat16*>(w_bf16), ldw, d_off, d_esum);
  return cudaGetLastError() == cudaSuccess ? 0 : 802;
}

extern "C" int dsb_score_stats_rows(const float* h, long long h_st, long long h_sr, const float* off,
                                    long long o_st, long long o_sr, const float* gram,
                                    const float* esum, float inv_u, int T, int R, int r, float* tau,
                                    float* isd, void* hb_bf16, float* zero, long long n_zero,
                                    cudaStream_t stream) {
  if (T <= 0 || R <= 0) return 0;
  if (r <= 0 || r > kMaxR) return 801;
  if (static_cast<long long>(T) * R > 65535) return 804;
  score_stats_rows_kernel<<<dim3(kRowCtas, T * R), kRowThreads, 0, stream>>>(
      h, h_st, h_sr, off, o_st, o_sr, gram, esum, inv_u, T, r, tau, isd,
      static_cast<__nv_bfloat16*>(hb_bf16), zero, n_zero);
  return cudaGetLastError() == cudaSuccess ? 0 : 802;
}

extern "C" int dsb_load_balance_blocks(int U, int r) {
  const int warps_units = (kLbThreads / 32) * (32 / lb_lanes(r));      // units of a block per pass
  const int b = (U + warps_units - 1) / warps_units;
  return b < 148 * 4 ? (b < 1 ? 1 : b) : 148 * 4;
}

extern "C" int dsb_load_balance_fwd(const void* emb_bf16, long long lde, const float* hsum, float inv_n,
                                    float units, int U, int r, float* m_u, float* part, float* lb,
                                    float* stat, cudaStream_t stream) {
  if (U <= 0 || r <= 0 || r > kMaxR || r % 8 != 0 || lde % 8 != 0) return 803;
  const int lpu = lb_lanes(r), blocks = dsb_load_balance_blocks(U, r);
  const __nv_bfloat16* e = static_cast<const __nv_bfloat16*>(emb_bf16);
  if (r <= 8 * lpu) lb_fwd_kernel<1><<<blocks, kLbThreads, 0, stream>>>(e, lde, hsum, inv_n, U, r, lpu, m_u, part);
  else lb_fwd_kernel<2><<<blocks, kLbThreads, 0, stream>>>(e, lde, hsum, inv_n, U, r, lpu, m_u, part);
  lb_finish_kernel<<<1, 256, 0, stream>>>(part, blocks, units, lb, stat);
  return cudaGetLastError() == cudaSuccess ? 0 : 802;
}

extern "C" int dsb_load_balance_bwd(const void* emb_bf16, long long lde, const float* m_u,
                                    const float* stat, const float* g_lb, float inv_n, float units,
                                    int U, int r, float* dmn, float* d_hsum, float* part,
                                    cudaStream_t stream) {
  if (U <= 0 || r <= 0 || r > kMaxR || r % 8 != 0 || lde % 8 != 0) return 803;
  const int lpu = lb_lanes(r), blocks = dsb_load_balance_blocks(U, r);
  const __nv_bfloat16* e = static_cast<const __nv_bfloat16*>(emb_bf16);
  if (r <= 8 * lpu)
    lb_bwd_kernel<1><<<blocks, kLbThreads, 0, stream>>>(e, lde, m_u, stat, g_lb, units, inv_n, U, r, lpu, dmn, part);
  else
    lb_bwd_kernel<2><<<blocks, kLbThreads, 0, stream>>>(e, lde, m_u, stat, g_lb, units, inv_n, U, r, lpu, dmn, part);
  if (cudaGetLastError() != cudaSuccess) return 802;
  return dsb_column_sum(part, blocks, r, d_hsum, stream);
}

extern "C" int dsb_rank1_add(float* g, long long ldg, const float* dm, const float* hs, int L, int U,
                             int r, cudaStream_t stream) {
  if (L <= 0 || U <= 0) return 0;
  if (r <= 0 || r > kMaxR || r % 4 != 0 || ldg % 4 != 0) return 803;
  const long long n = static_cast<long long>(U) * (r >> 2);
  const int blocks = static_cast<int>(n / 256 + 1 < 148 * 8 ? n / 256 + 1 : 148 * 8);
  for (int l0 = 0; l0 < L; l0 += kRank1Max) {
    const int cnt = L - l0 < kRank1Max ? L - l0 : kRank1Max;      // 24 x 512 floats = 48 KB
    rank1_add_kernel<<<blocks, 256, static_cast<size_t>(cnt) * r * sizeof(float), stream>>>(
        g, ldg, dm + static_cast<size_t>(l0) * U, hs + static_cast<size_t>(l0) * r, cnt, U, r);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 802;
}
