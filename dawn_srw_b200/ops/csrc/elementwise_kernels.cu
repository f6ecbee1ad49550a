// Memory-bound kernels around the GEMMs: LayerNorm forward/backward (bf16 out),
// row-wise softmax cross-entropy statistics and gradient for the chunked tied
// LM head, and the AdamW update with the clip factor read from device memory.
// Reference math: LayerNorm eps 1e-6, population variance
// (models/dawn_spatial_v41_exp.py:321-324); CE on shifted labels (:1642-1668);
// optimizer chain (scripts/train_jax.py:2083-2089).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "dsb_api_ops.h"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One warp per row.  x fp32 [T, D]; y bf16 [T, D]; mean/rstd fp32 [T].
// kRegs > 0: the row (D <= 32 * kRegs) is read once and kept in registers, all
// loads in flight together; kRegs == 0: three passes over the row for any D.
template <int kRegs>
__global__ void ln_fwd_kernel(const float* __restrict__ x, const float* __restrict__ w,
                              const float* __restrict__ b, __nv_bfloat16* __restrict__ y,
                              float* __restrict__ mean, float* __restrict__ rstd, int T, int D,
                              float eps) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= T) return;
  const float* xr = x + static_cast<size_t>(row) * D;
  __nv_bfloat16* yr = y + static_cast<size_t>(row) * D;
  if constexpr (kRegs > 0) {
    float v[kRegs];
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kRegs; ++k) {
      const int i = lane + 32 * k;
      v[k] = i < D ? xr[i] : 0.f;
      s += v[k];
    }
    const float mu = warp_sum(s) / D;
    float q = 0.f;
#pragma unroll
    for (int k = 0; k < kRegs; ++k) {
      const float d = lane + 32 * k < D ? v[k] - mu : 0.f;
      q += d * d;
    }
    const float rs = rsqrtf(warp_sum(q) / D + eps);
#pragma unroll
    for (int k = 0; k < kRegs; ++k) {
      const int i = lane + 32 * k;
      if (i < D) yr[i] = __float2bfloat16((v[k] - mu) * rs * w[i] + b[i]);
    }
    if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
  } else {
    float s = 0.f;
    for (int i = lane; i < D; i += 32) s += xr[i];
    const float mu = warp_sum(s) / D;
    float q = 0.f;
    for (int i = lane; i < D; i += 32) { const float d = xr[i] - mu; q += d * d; }
    const float rs = rsqrtf(warp_sum(q) / D + eps);
    for (int i = lane; i < D; i += 32) yr[i] = __float2bfloat16((xr[i] - mu) * rs * w[i] + b[i]);
    if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
  }
}

__device__ __forceinline__ float4 bf16x4(const uint2& u) {
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

// The same for rows that can be read as float4 (D % 4 == 0, D <= 128 * NV, 16-byte aligned): one
// warp per row, the row in registers after NV loads in flight.  Bound by its bytes (6 per element) for
// many rows, by one round trip to memory for few: 4.4 us for 512 x 1280 and 5.1 us for 8192 x 384
// (3.7 TB/s); with scalar loads 14.5 and 8.2 us.
template <int NV>
__global__ void __launch_bounds__(128) ln_fwd_vec_kernel(const float* __restrict__ x,
                                                         const float* __restrict__ w,
                                                         const float* __restrict__ b,
                                                         __nv_bfloat16* __restrict__ y,
                                                         float* __restrict__ mean, float* __restrict__ rstd,
                                                         int T, int D, float eps) {
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= T) return;
  const int d4 = D >> 2;
  const float4* xr = reinterpret_cast<const float4*>(x + static_cast<size_t>(row) * D);
  float4 v[NV];
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = lane + 32 * k;
    v[k] = i < d4 ? xr[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) s += (v[k].x + v[k].y) + (v[k].z + v[k].w);
  const float mu = warp_sum(s) / D;
  float q = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    if (lane + 32 * k < d4) {
      const float a = v[k].x - mu, c = v[k].y - mu, d = v[k].z - mu, e = v[k].w - mu;
      q += (a * a + c * c) + (d * d + e * e);
    }
  }
  const float rs = rsqrtf(warp_sum(q) / D + eps);
  uint2* yr = reinterpret_cast<uint2*>(y + static_cast<size_t>(row) * D);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = lane + 32 * k;
    if (i < d4) {
      const float4 g = reinterpret_cast<const float4*>(w)[i], c = reinterpret_cast<const float4*>(b)[i];
      const __nv_bfloat162 lo = __floats2bfloat162_rn((v[k].x - mu) * rs * g.x + c.x, (v[k].y - mu) * rs * g.y + c.y);
      const __nv_bfloat162 hi = __floats2bfloat162_rn((v[k].z - mu) * rs * g.z + c.z, (v[k].w - mu) * rs * g.w + c.w);
      yr[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  }
  if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
}

// dx of the backward pass under the same conditions: dy and x are read once (7.2 us for 8192 x 384, 8.6
// with a second read).  Narrow rows take fewer steps per lane: 65 536 x 8 took 23.2 us with NV = 4,
// 10.6 with 1.
template <int NV>
__global__ void __launch_bounds__(128) ln_bwd_dx_vec_kernel(const __nv_bfloat16* __restrict__ dy,
                                                            const float* __restrict__ x,
                                                            const float* __restrict__ w,
                                                            const float* __restrict__ mean,
                                                            const float* __restrict__ rstd,
                                                            float* __restrict__ dx, int T, int D) {
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= T) return;
  const int d4 = D >> 2;
  const float mu = mean[row], rs = rstd[row];
  const float4* xr = reinterpret_cast<const float4*>(x + static_cast<size_t>(row) * D);
  const uint2* dyr = reinterpret_cast<const uint2*>(dy + static_cast<size_t>(row) * D);
  float4 v[NV];
  uint2 g2[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = lane + 32 * k;
    v[k] = i < d4 ? xr[i] : make_float4(mu, mu, mu, mu);
    g2[k] = i < d4 ? dyr[i] : make_uint2(0u, 0u);
  }
  float s1 = 0.f, s2 = 0.f;
  auto scaled = [&](int k) {                       // dy * w of this lane's four columns
    const int i = lane + 32 * k;
    const float4 d = bf16x4(g2[k]);
    const float4 c = i < d4 ? reinterpret_cast<const float4*>(w)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(d.x * c.x, d.y * c.y, d.z * c.z, d.w * c.w);
  };
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const float4 g = scaled(k);
    s1 += (g.x + g.y) + (g.z + g.w);
    s2 += (g.x * ((v[k].x - mu) * rs) + g.y * ((v[k].y - mu) * rs)) +
          (g.z * ((v[k].z - mu) * rs) + g.w * ((v[k].w - mu) * rs));
  }
  s1 = warp_sum(s1) / D;
  s2 = warp_sum(s2) / D;
  float4* dxr = reinterpret_cast<float4*>(dx + static_cast<size_t>(row) * D);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = lane + 32 * k;
    if (i < d4) {
      const float4 g = scaled(k);
      dxr[i] = make_float4(rs * (g.x - s1 - (v[k].x - mu) * rs * s2), rs * (g.y - s1 - (v[k].y - mu) * rs * s2),
                           rs * (g.z - s1 - (v[k].z - mu) * rs * s2), rs * (g.w - s1 - (v[k].w - mu) * rs * s2));
    }
  }
}

// dw, db under the same conditions: a block covers 128 columns (four per thread) of 64 rows (4.3 us for
// 8192 x 384, 8.9 with 32 columns of 256 rows and scalar loads), or of more where that would be more than 256
// blocks that add to the same columns: 65 536 x 64 took 12.2 us in 1024 blocks, 8.0 in 256, x 384 32.7 and 29.9.
int ln_rows_per_block(int T) { return T <= 64 * 256 ? 64 : (T / 256 / 8 + 1) * 8; }
__global__ void __launch_bounds__(256) ln_bwd_dwdb_vec_kernel(const __nv_bfloat16* __restrict__ dy,
                                                              const float* __restrict__ x,
                                                              const float* __restrict__ mean,
                                                              const float* __restrict__ rstd,
                                                              float* __restrict__ dw, float* __restrict__ db,
                                                              int T, int D, int rows) {
  __shared__ float s_w[8][128], s_b[8][128];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5, c = blockIdx.x * 128 + 4 * cx;
  const int lo = blockIdx.y * rows, hi = T - lo < rows ? T : lo + rows;
  float aw[4] = {0.f, 0.f, 0.f, 0.f}, ab[4] = {0.f, 0.f, 0.f, 0.f};
  if (c < D) {
#pragma unroll 4
    for (int row = lo + ry; row < hi; row += 8) {
      const float4 d = bf16x4(*reinterpret_cast<const uint2*>(dy + static_cast<size_t>(row) * D + c));
      const float4 v = *reinterpret_cast<const float4*>(x + static_cast<size_t>(row) * D + c);
      const float mu = mean[row], rs = rstd[row];
      aw[0] += d.x * ((v.x - mu) * rs); aw[1] += d.y * ((v.y - mu) * rs);
      aw[2] += d.z * ((v.z - mu) * rs); aw[3] += d.w * ((v.w - mu) * rs);
      ab[0] += d.x; ab[1] += d.y; ab[2] += d.z; ab[3] += d.w;
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) { s_w[ry][4 * cx + j] = aw[j]; s_b[ry][4 * cx + j] = ab[j]; }
  __syncthreads();
  const int col = threadIdx.x & 127, out = blockIdx.x * 128 + col;
  if (out < D) {
    const float (*src)[128] = threadIdx.x < 128 ? s_w : s_b;
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += src[k][col];
    atomicAdd((threadIdx.x < 128 ? dw : db) + out, t);
  }
}

bool aligned16(const void* a, const void* b, const void* c, const void* d) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
           reinterpret_cast<uintptr_t>(d)) & 15) == 0;
}

// A few rows only (decoding): one block of 256 threads per row, the row in
// registers (D <= 256 * 8), two block reductions.
__global__ void __launch_bounds__(256) ln_fwd_block_kernel(
    const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b,
    __nv_bfloat16* __restrict__ y, float* __restrict__ mean, float* __restrict__ rstd, int D,
    float eps) {
  __shared__ float s_red[2][8];
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* xr = x + static_cast<size_t>(row) * D;
  float v[8];
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int i = tid + 256 * k;
    v[k] = i < D ? xr[i] : 0.f;
    s += v[k];
  }
  s = warp_sum(s);
  if (lane == 0) s_red[0][warp] = s;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) tot += s_red[0][k];
  const float mu = tot / D;
  float q = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float d = tid + 256 * k < D ? v[k] - mu : 0.f;
    q += d * d;
  }
  q = warp_sum(q);
  if (lane == 0) s_red[1][warp] = q;
  __syncthreads();
  tot = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) tot += s_red[1][k];
  const float rs = rsqrtf(tot / D + eps);
  __nv_bfloat16* yr = y + static_cast<size_t>(row) * D;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int i = tid + 256 * k;
    if (i < D) yr[i] = __float2bfloat16((v[k] - mu) * rs * w[i] + b[i]);
  }
  if (tid == 0) { mean[row] = mu; rstd[row] = rs; }
}

// LayerNorm backward in two kernels.  (1) dx: one warp per row, two passes over
// the row (row sums, then dx).  (2) dw, db: a block covers 32 columns x 256
// rows (a warp reads 32 consecutive columns of one row, so loads are
// coalesced), reduces over its rows in shared memory and adds one partial per
// column to dw / db.
__global__ void ln_bwd_dx_kernel(const __nv_bfloat16* __restrict__ dy, const float* __restrict__ x,
                                 const float* __restrict__ w, const float* __restrict__ mean,
                                 const float* __restrict__ rstd, float* __restrict__ dx, int T,
                                 int D) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= T) return;
  const float mu = mean[row], rs = rstd[row];
  const float* xr = x + static_cast<size_t>(row) * D;
  const __nv_bfloat16* dyr = dy + static_cast<size_t>(row) * D;
  float s1 = 0.f, s2 = 0.f;
  for (int i = lane; i < D; i += 32) {
    const float g = __bfloat162float(dyr[i]) * w[i];
    s1 += g;
    s2 += g * (xr[i] - mu) * rs;
  }
  s1 = warp_sum(s1) / D;
  s2 = warp_sum(s2) / D;
  float* dxr = dx + static_cast<size_t>(row) * D;
  for (int i = lane; i < D; i += 32) {
    const float xh = (xr[i] - mu) * rs;
    dxr[i] = rs * (__bfloat162float(dyr[i]) * w[i] - s1 - xh * s2);
  }
}

constexpr int kLnRowsPerBlock = 256;
__global__ void ln_bwd_dwdb_kernel(const __nv_bfloat16* __restrict__ dy, const float* __restrict__ x,
                                   const float* __restrict__ mean, const float* __restrict__ rstd,
                                   float* __restrict__ dw, float* __restrict__ db, int T, int D) {
  __shared__ float sw[8][33], sb[8][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;      // 32 columns x 8 row lanes
  const int col = blockIdx.x * 32 + cx;
  const int row_lo = blockIdx.y * kLnRowsPerBlock;
  const int row_hi = min(T, row_lo + kLnRowsPerBlock);
  float aw = 0.f, ab = 0.f;
  if (col < D) {
    for (int row = row_lo + ry; row < row_hi; row += 8) {
      const float d = __bfloat162float(dy[static_cast<size_t>(row) * D + col]);
      const float xh = (x[static_cast<size_t>(row) * D + col] - mean[row]) * rstd[row];
      aw += d * xh;
      ab += d;
    }
  }
  sw[ry][cx] = aw;
  sb[ry][cx] = ab;
  __syncthreads();
  if (ry == 0 && col < D) {
    float tw = 0.f, tb = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) { tw += sw[k][cx]; tb += sb[k][cx]; }
    atomicAdd(dw + col, tw);
    atomicAdd(db + col, tb);
  }
}

// One block per row of logits [R, ld] (fp32, V valid columns).
__global__ void ce_fwd_kernel(const float* __restrict__ logits, long long ld,
                              const long long* __restrict__ labels, int V, float* __restrict__ lse,
                              float* __restrict__ label_logit, long long* __restrict__ argmax) {
  const int row = blockIdx.x;
  const float* lr = logits + row * ld;
  float m = -FLT_MAX;
  int mi = 0;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    const float v = lr[i];
    if (v > m) { m = v; mi = i; }
  }
  __shared__ float sm[32];
  __shared__ int si[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, m, o);
    const int oi = __shfl_xor_sync(0xffffffffu, mi, o);
    if (om > m || (om == m && oi < mi)) { m = om; mi = oi; }
  }
  if (lane == 0) { sm[warp] = m; si[warp] = mi; }
  __syncthreads();
  if (warp == 0) {
    m = lane < nwarp ? sm[lane] : -FLT_MAX;
    mi = lane < nwarp ? si[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float om = __shfl_xor_sync(0xffffffffu, m, o);
      const int oi = __shfl_xor_sync(0xffffffffu, mi, o);
      if (om > m || (om == m && oi < mi)) { m = om; mi = oi; }
    }
    if (lane == 0) { sm[0] = m; si[0] = mi; }
  }
  __syncthreads();
  m = sm[0];
  float s = 0.f;
  for (int i = threadIdx.x; i < V; i += blockDim.x) s += __expf(lr[i] - m);
  s = warp_sum(s);
  __shared__ float ss[32];
  if (lane == 0) ss[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int k = 0; k < nwarp; ++k) t += ss[k];
    lse[row] = m + logf(t);
    long long lab = labels[row];
    if (lab < 0) lab = 0;
    label_logit[row] = lr[lab];
    argmax[row] = si[0];
  }
}

// dl[row, i] = scale[row] * (softmax(logits[row])[i] - [i == label]) as bf16 [R, ldo].
__global__ void ce_bwd_kernel(const float* __restrict__ logits, long long ld,
                              const long long* __restrict__ labels, const float* __restrict__ lse,
                              const float* __restrict__ scale, int V, __nv_bfloat16* __restrict__ dl,
                              long long ldo) {
  const int row = blockIdx.x;
  const float* lr = logits + row * ld;
  __nv_bfloat16* dr = dl + row * ldo;
  const float l = lse[row], sc = scale[row];
  long long lab = labels[row];
  if (lab < 0) lab = 0;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    float v = __expf(lr[i] - l);
    if (i == lab) v -= 1.f;
    dr[i] = __float2bfloat16(v * sc);
  }
  for (long long i = V + threadIdx.x; i < ldo; i += blockDim.x) dr[i] = __float2bfloat16(0.f);
}

__global__ void adamw_kernel(float* __restrict__ p, const float* __restrict__ g,
                             float* __restrict__ m, float* __restrict__ v, long long n,
                             const float* __restrict__ clip_scale, float lr, float b1, float b2,
                             float eps, float wd, float bc1, float bc2) {
  const float cs = *clip_scale;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += stride) {
    const float gi = g[i] * cs;
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i];
    const float upd = (mi / bc1) / (sqrtf(vi / bc2) + eps) + wd * pi;
    p[i] = pi - lr * upd;
  }
}

// out[0] += sum(g^2)
__global__ void sqnorm_kernel(const float* __restrict__ g, long long n, float* __restrict__ out) {
  float s = 0.f;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += stride) {
    const float v = g[i];
    s += v * v;
  }
  s = warp_sum(s);
  __shared__ float sh[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) sh[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int k = 0; k < (blockDim.x >> 5); ++k) t += sh[k];
    atomicAdd(out, t);
  }
}


// ---------------------------------------------------------------------------
// Token + position embedding.  out[t, :] = tok[ids[t], :] + pos[t % S, :]
// (models/dawn_spatial_v41_exp.py:1504-1507).  One warp per token, float4 lanes.
__global__ void embed_fwd_kernel(const long long* __restrict__ ids, const float* __restrict__ tok,
                                 const float* __restrict__ pos, float* __restrict__ out, int T,
                                 int S, int D, int V) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  long long id = ids[t];
  id = id < 0 ? 0 : (id >= V ? V - 1 : id);
  const float4* a = reinterpret_cast<const float4*>(tok + static_cast<size_t>(id) * D);
  const float4* b = reinterpret_cast<const float4*>(pos + static_cast<size_t>(t % S) * D);
  float4* o = reinterpret_cast<float4*>(out + static_cast<size_t>(t) * D);
  for (int i = lane; i < (D >> 2); i += 32) {
    const float4 x = a[i], y = b[i];
    o[i] = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
  }
}

// dtok[ids[t], :] += dy[t, :] (atomic: a token may repeat), one warp per token.
__global__ void embed_bwd_tok_kernel(const long long* __restrict__ ids, const float* __restrict__ dy,
                                     float* __restrict__ dtok, int T, int D, int V) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  long long id = ids[t];
  id = id < 0 ? 0 : (id >= V ? V - 1 : id);
  const float* g = dy + static_cast<size_t>(t) * D;
  float* d = dtok + static_cast<size_t>(id) * D;
  for (int i = lane; i < D; i += 32) atomicAdd(d + i, g[i]);
}

// dpos[s, :] = sum_b dy[b*S + s, :]; one thread per (s, column), fixed order.
__global__ void embed_bwd_pos_kernel(const float* __restrict__ dy, float* __restrict__ dpos, int B,
                                     int S, int D) {
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<long long>(S) * D) return;
  float acc = 0.f;
  for (int b = 0; b < B; ++b) acc += dy[static_cast<size_t>(b) * S * D + idx];
  dpos[idx] = acc;
}

// ---------------------------------------------------------------------------
// Off-diagonal |cos| statistics of a similarity matrix sim [m, m] (fp32, row
// stride ld): total[0] += sum_{i != j} |sim_ij|, and sgn[i, j] = sign(sim_ij)
// (0 on the diagonal) as bf16 for the backward GEMM.
__global__ void offdiag_abs_kernel(const float* __restrict__ sim, long long ld, int m,
                                   __nv_bfloat16* __restrict__ sgn, long long ld_s,
                                   float* __restrict__ total) {
  float acc = 0.f;
  const long long n = static_cast<long long>(m) * m;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long k = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; k < n;
       k += stride) {
    const int i = static_cast<int>(k / m), j = static_cast<int>(k % m);
    const float v = sim[i * ld + j];
    float sg = 0.f;
    if (i != j) {
      acc += fabsf(v);
      sg = v > 0.f ? 1.f : (v < 0.f ? -1.f : 0.f);
    }
    sgn[i * ld_s + j] = __float2bfloat16(sg);
  }
  acc = warp_sum(acc);
  __shared__ float sh[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) sh[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int k = 0; k < (blockDim.x >> 5); ++k) t += sh[k];
    atomicAdd(total, t);
  }
}

// ---------------------------------------------------------------------------
// Backward prologue of a scaled, sum-normalised SRW route y = s * raw / den:
//   dy_bf[t, :] = bf16(dy[t, :] * row_scale[t])        (row_scale = s / max(den, 1))
//   rowdot[t]   = sum_d dy[t, d] * y[t, d]             (feeds d_den and d_s)
// One warp per row; dy and y fp32.
__global__ void route_bwd_prologue_kernel(const float* __restrict__ dy, const float* __restrict__ y,
                                          const float* __restrict__ row_scale,
                                          __nv_bfloat16* __restrict__ dy_bf,
                                          float* __restrict__ rowdot, int T, int D) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  const float rs = row_scale[t];
  const float4* g = reinterpret_cast<const float4*>(dy + static_cast<size_t>(t) * D);
  const float4* yy = reinterpret_cast<const float4*>(y + static_cast<size_t>(t) * D);
  uint2* o = reinterpret_cast<uint2*>(dy_bf + static_cast<size_t>(t) * D);
  float acc = 0.f;
  for (int i = lane; i < (D >> 2); i += 32) {
    const float4 a = g[i], b = yy[i];
    acc += a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w;
    __nv_bfloat162 lo = __floats2bfloat162_rn(a.x * rs, a.y * rs);
    __nv_bfloat162 hi = __floats2bfloat162_rn(a.z * rs, a.w * rs);
    uint2 w;
    w.x = *reinterpret_cast<uint32_t*>(&lo);
    w.y = *reinterpret_cast<uint32_t*>(&hi);
    o[i] = w;
  }
  acc = warp_sum(acc);
  if (lane == 0) rowdot[t] = acc;
}

// The same for a route whose denominator and scale are still separate, with all that follows per
// row: row_scale = s / max(den, 1);  d_den = -rowdot / den where den > 1 (+ ext_dden);
// dots[block] = its rows' sum of rowdot (scale_grad_kernel);  dtau = 0 (the gate kernel adds into it).  One pass over dy and y
// instead of that plus nine tensor ops on [T].
__global__ void __launch_bounds__(256) route_bwd_rows_kernel(
    const float* __restrict__ dy, const float* __restrict__ y, const float* __restrict__ den,
    const float* __restrict__ scale_ptr, float scale, const float* __restrict__ ext_dden,
    __nv_bfloat16* __restrict__ dy_bf, float* __restrict__ d_den, float* __restrict__ dtau,
    float* __restrict__ dots, int T, int D) {
  __shared__ float s_dot[8];
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  float acc = 0.f;
  const float sc = scale_ptr != nullptr ? scale_ptr[0] : scale;
  if (t < T) {
    const float dn = den[t];
    const float rs = sc / (dn < 1.f ? 1.f : dn);                 // a NaN stays one
    const float4* g = reinterpret_cast<const float4*>(dy + static_cast<size_t>(t) * D);
    const float4* yy = reinterpret_cast<const float4*>(y + static_cast<size_t>(t) * D);
    uint2* o = reinterpret_cast<uint2*>(dy_bf + static_cast<size_t>(t) * D);
#pragma unroll 4
    for (int i = lane; i < (D >> 2); i += 32) {
      const float4 a = g[i], b = yy[i];
      acc += a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w;
      const __nv_bfloat162 lo = __floats2bfloat162_rn(a.x * rs, a.y * rs);
      const __nv_bfloat162 hi = __floats2bfloat162_rn(a.z * rs, a.w * rs);
      uint2 w;
      w.x = *reinterpret_cast<const uint32_t*>(&lo);
      w.y = *reinterpret_cast<const uint32_t*>(&hi);
      o[i] = w;
    }
    acc = warp_sum(acc);
    if (lane == 0) {
      d_den[t] = (dn > 1.f ? -acc / dn : 0.f) + (ext_dden != nullptr ? ext_dden[t] : 0.f);
      dtau[t] = 0.f;
    }
  }
  if (dots != nullptr) {
    if (lane == 0) s_dot[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      float tot = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) tot += s_dot[k];
      dots[blockIdx.x] = tot;
    }
  }
}

// d_scale += (dots[0] + dots[1] + ...) / s, in a fixed order: the gradient of a scale repeats bit by bit.
__global__ void __launch_bounds__(256) scale_grad_kernel(const float* __restrict__ dots, int n,
                                                         const float* __restrict__ scale_ptr, float scale,
                                                         float* __restrict__ d_scale) {
  __shared__ float s_sum[8];
  float a = 0.f;
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += 256) a += dots[i];
  a = warp_sum(a);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    a = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) a += s_sum[k];
    d_scale[0] += a / (scale_ptr != nullptr ? scale_ptr[0] : scale);
  }
}

inline int grid_for(long long n, int block, int cap) {
  long long g = (n + block - 1) / block;
  return static_cast<int>(g < cap ? (g < 1 ? 1 : g) : cap);
}

}  // namespace

extern "C" int dsb_layernorm_fwd(const float* x, const float* w, const float* b, void* y_bf16,
                                 float* mean, float* rstd, int T, int D, float eps,
                                 cudaStream_t stream) {
  if (T <= 0) return 0;
  __nv_bfloat16* y = reinterpret_cast<__nv_bfloat16*>(y_bf16);
  if (T <= 296 && D <= 2048) {   // few rows: a block per row instead of a warp per row
    ln_fwd_block_kernel<<<T, 256, 0, stream>>>(x, w, b, y, mean, rstd, D, eps);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
  }
  if (D % 4 == 0 && D <= 2048 && aligned16(x, w, b, y)) {
    const int blocks = (T + 3) / 4;
    if (D <= 512) ln_fwd_vec_kernel<4><<<blocks, 128, 0, stream>>>(x, w, b, y, mean, rstd, T, D, eps);
    else if (D <= 1280) ln_fwd_vec_kernel<10><<<blocks, 128, 0, stream>>>(x, w, b, y, mean, rstd, T, D, eps);
    else ln_fwd_vec_kernel<16><<<blocks, 128, 0, stream>>>(x, w, b, y, mean, rstd, T, D, eps);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
  }
  // rows of other lengths or alignments
  const int warps = 8;
  const dim3 grid((T + warps - 1) / warps), block(warps * 32);
  if (D <= 32 * 16) ln_fwd_kernel<16><<<grid, block, 0, stream>>>(x, w, b, y, mean, rstd, T, D, eps);
  else if (D <= 32 * 40) ln_fwd_kernel<40><<<grid, block, 0, stream>>>(x, w, b, y, mean, rstd, T, D, eps);
  else if (D <= 32 * 64) ln_fwd_kernel<64><<<grid, block, 0, stream>>>(x, w, b, y, mean, rstd, T, D, eps);
  else ln_fwd_kernel<0><<<grid, block, 0, stream>>>(x, w, b, y, mean, rstd, T, D, eps);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_layernorm_bwd(const void* dy_bf16, const float* x, const float* w,
                                 const float* mean, const float* rstd, float* dx, float* dw,
                                 float* db, int T, int D, cudaStream_t stream) {
  if (T <= 0) return 0;
  const __nv_bfloat16* dy = reinterpret_cast<const __nv_bfloat16*>(dy_bf16);
  if (D % 4 == 0 && D <= 2048 && aligned16(x, w, dy, dx)) {
    const int blocks = (T + 3) / 4;
    if (D <= 128) ln_bwd_dx_vec_kernel<1><<<blocks, 128, 0, stream>>>(dy, x, w, mean, rstd, dx, T, D);
    else if (D <= 256) ln_bwd_dx_vec_kernel<2><<<blocks, 128, 0, stream>>>(dy, x, w, mean, rstd, dx, T, D);
    else if (D <= 512) ln_bwd_dx_vec_kernel<4><<<blocks, 128, 0, stream>>>(dy, x, w, mean, rstd, dx, T, D);
    else if (D <= 1280) ln_bwd_dx_vec_kernel<10><<<blocks, 128, 0, stream>>>(dy, x, w, mean, rstd, dx, T, D);
    else ln_bwd_dx_vec_kernel<16><<<blocks, 128, 0, stream>>>(dy, x, w, mean, rstd, dx, T, D);
    const int rows = ln_rows_per_block(T);
    ln_bwd_dwdb_vec_kernel<<<dim3((D + 127) / 128, T / rows + (T % rows != 0)), 256, 0, stream>>>(
        dy, x, mean, rstd, dw, db, T, D, rows);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
  }
  ln_bwd_dx_kernel<<<(T + 7) / 8, 256, 0, stream>>>(dy, x, w, mean, rstd, dx, T, D);
  const dim3 grid((D + 31) / 32, (T + kLnRowsPerBlock - 1) / kLnRowsPerBlock);
  ln_bwd_dwdb_kernel<<<grid, 256, 0, stream>>>(dy, x, mean, rstd, dw, db, T, D);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_ce_fwd(const float* logits, long long ld, const long long* labels, int R, int V,
                          float* lse, float* label_logit, long long* argmax, cudaStream_t stream) {
  if (R <= 0) return 0;
  ce_fwd_kernel<<<R, 256, 0, stream>>>(logits, ld, labels, V, lse, label_logit, argmax);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_ce_bwd(const float* logits, long long ld, const long long* labels,
                          const float* lse, const float* scale, int R, int V, void* dl_bf16,
                          long long ldo, cudaStream_t stream) {
  if (R <= 0) return 0;
  ce_bwd_kernel<<<R, 256, 0, stream>>>(logits, ld, labels, lse, scale, V,
                                       reinterpret_cast<__nv_bfloat16*>(dl_bf16), ldo);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_adamw(float* p, const float* g, float* m, float* v, long long n,
                         const float* clip_scale, float lr, float b1, float b2, float eps, float wd,
                         float bc1, float bc2, cudaStream_t stream) {
  if (n <= 0) return 0;
  adamw_kernel<<<grid_for(n, 256, 148 * 16), 256, 0, stream>>>(p, g, m, v, n, clip_scale, lr, b1,
                                                               b2, eps, wd, bc1, bc2);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_sqnorm_accumulate(const float* g, long long n, float* out,
                                     cudaStream_t stream) {
  if (n <= 0) return 0;
  sqnorm_kernel<<<grid_for(n, 256, 148 * 8), 256, 0, stream>>>(g, n, out);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_embed_fwd(const long long* ids, const float* tok, const float* pos, float* out,
                             int T, int S, int D, int V, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (D & 3) return 2;
  embed_fwd_kernel<<<(T + 7) / 8, 256, 0, stream>>>(ids, tok, pos, out, T, S, D, V);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_embed_bwd(const long long* ids, const float* dy, float* dtok, float* dpos, int B,
                             int S, int D, int V, cudaStream_t stream) {
  const int T = B * S;
  if (T <= 0) return 0;
  embed_bwd_tok_kernel<<<(T + 7) / 8, 256, 0, stream>>>(ids, dy, dtok, T, D, V);
  const long long n = static_cast<long long>(S) * D;
  embed_bwd_pos_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(dy, dpos, B, S, D);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_offdiag_abs(const float* sim, long long ld, int m, void* sgn_bf16,
                               long long ld_s, float* total, cudaStream_t stream) {
  if (m <= 0) return 0;
  const long long n = static_cast<long long>(m) * m;
  offdiag_abs_kernel<<<grid_for(n, 256, 148 * 8), 256, 0, stream>>>(
      sim, ld, m, reinterpret_cast<__nv_bfloat16*>(sgn_bf16), ld_s, total);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_route_bwd_prologue(const float* dy, const float* y, const float* row_scale,
                                      void* dy_bf16, float* rowdot, int T, int D,
                                      cudaStream_t stream) {
  if (T <= 0) return 0;
  if (D & 3) return 2;
  route_bwd_prologue_kernel<<<(T + 7) / 8, 256, 0, stream>>>(
      dy, y, row_scale, reinterpret_cast<__nv_bfloat16*>(dy_bf16), rowdot, T, D);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_route_bwd_rows(const float* dy, const float* y, const float* den,
                                  const float* scale_ptr, float scale, const float* ext_dden,
                                  void* dy_bf16, float* d_den, float* dtau, float* d_scale, float* dots,
                                  int T, int D, cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((D & 3) || (d_scale != nullptr && dots == nullptr)) return 2;
  route_bwd_rows_kernel<<<(T + 7) / 8, 256, 0, stream>>>(
      dy, y, den, scale_ptr, scale, ext_dden, reinterpret_cast<__nv_bfloat16*>(dy_bf16), d_den, dtau,
      d_scale != nullptr ? dots : nullptr, T, D);
  if (d_scale != nullptr)
    scale_grad_kernel<<<1, 256, 0, stream>>>(dots, (T + 7) / 8, scale_ptr, scale, d_scale);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

// ------------------------------------------------------------------ dropout
// Keep-mask dropout scaled by 1 / keep, optionally fused with the residual add
// that follows it (y = res + dropout(x)).  The mask is a counter-based hash of
// (seed, element index): nothing is stored, the backward kernel regenerates it.
// (The reference draws from the JAX key stream, models/dawn_spatial_v41_exp.py:
// 308-318; same distribution, different bits.)
namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// element 4*i4 + k of the tensor is kept iff its 32 hash bits are >= thresh
__device__ __forceinline__ void keep4(uint64_t seed, long long i4, uint32_t thresh, float scale,
                                      float (&m)[4]) {
  const uint64_t a = mix64(seed + static_cast<uint64_t>(2 * i4) * 0x9E3779B97F4A7C15ull);
  const uint64_t b = mix64(seed + static_cast<uint64_t>(2 * i4 + 1) * 0x9E3779B97F4A7C15ull);
  m[0] = static_cast<uint32_t>(a) >= thresh ? scale : 0.f;
  m[1] = static_cast<uint32_t>(a >> 32) >= thresh ? scale : 0.f;
  m[2] = static_cast<uint32_t>(b) >= thresh ? scale : 0.f;
  m[3] = static_cast<uint32_t>(b >> 32) >= thresh ? scale : 0.f;
}

__global__ void dropout_kernel(const float4* __restrict__ res, const float4* __restrict__ x,
                               float4* __restrict__ y, long long n4, uint64_t seed, uint32_t thresh,
                               float scale) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n4;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float m[4];
    keep4(seed, i, thresh, scale, m);
    const float4 v = x[i];
    float4 o = make_float4(v.x * m[0], v.y * m[1], v.z * m[2], v.w * m[3]);
    if (res != nullptr) {
      const float4 r = res[i];
      o.x += r.x; o.y += r.y; o.z += r.z; o.w += r.w;
    }
    y[i] = o;
  }
}

}  // namespace

extern "C" int dsb_dropout(const float* res, const float* x, float* y, long long n,
                           unsigned long long seed, float p, cudaStream_t stream) {
  if (n <= 0) return 0;
  if ((n & 3) || !(p >= 0.f && p < 1.f)) return 2;
  const long long n4 = n >> 2;
  const uint32_t thresh = static_cast<uint32_t>(static_cast<double>(p) * 4294967296.0);
  long long blocks = (n4 + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  dropout_kernel<<<static_cast<int>(blocks), 256, 0, stream>>>(
      reinterpret_cast<const float4*>(res), reinterpret_cast<const float4*>(x),
      reinterpret_cast<float4*>(y), n4, seed, thresh, 1.f / (1.f - p));
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

// ------------------------------------------------- operand of a linear layer's backward
// dst bf16 [T, n] = bf16(sum of the sources that cover a column), 0 where none does, and the column
// sums of the same values (the bias gradient) in one pass: a source is an fp32 [T, cols] block at
// column col0; the columns of the sum below n_drop are optionally under the keep mask of a
// [T, n_drop]-shaped dropout.  Bound by its bytes (6 per element): separate cast, sum, slice and pad ops
// read a gradient three times, and a column sum of 8192 x 384 alone took 18.6 us.  A thread owns four
// columns, a block 128 columns of 64 rows (more where the grid could not hold them); the blocks' sums
// are added up in their order by column_sum_kernel, so that a bias gradient repeats bit by bit.
namespace {

constexpr int kPackRows = 64, kMaxGridY = 65535;
int pack_rows(int T) { return T <= kPackRows * kMaxGridY ? kPackRows : (T / kMaxGridY / 8 + 1) * 8; }

// out[j] = part[0][j] + part[1][j] + ... in a fixed order (n % 4 == 0, part 16-byte aligned): a block takes 32
// columns, its 32 groups of eight threads every 32nd row.
__global__ void __launch_bounds__(256) column_sum_kernel(const float* __restrict__ part, int rows, int n,
                                                         float* __restrict__ out) {
  __shared__ __align__(16) float s_sum[32][36];
  const int q = threadIdx.x & 7, ry = threadIdx.x >> 3, c = blockIdx.x * 32 + 4 * q;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < n) {
#pragma unroll 4
    for (int y = ry; y < rows; y += 32) {
      const float4 v = *reinterpret_cast<const float4*>(part + static_cast<size_t>(y) * n + c);
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
  }
  *reinterpret_cast<float4*>(&s_sum[ry][4 * q]) = a;
  __syncthreads();
  const int j = blockIdx.x * 32 + threadIdx.x;
  if (threadIdx.x < 32 && j < n) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) t += s_sum[k][threadIdx.x];
    out[j] = t;
  }
}

template <int kSrc>
__global__ void __launch_bounds__(256) linear_pack_kernel(const DsbPackSrc s0, const DsbPackSrc s1,
                                                          const DsbPackSrc s2, const DsbPackSrc s3,
                                                          const DsbPackSrc s4, int T, int n, int rows,
                                                          __nv_bfloat16* __restrict__ dst,
                                                          float* __restrict__ part, uint64_t seed,
                                                          uint32_t thresh, float keep_scale, int n_drop) {
  __shared__ float s_sum[8][128];
  const DsbPackSrc src[5] = {s0, s1, s2, s3, s4};
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int c = blockIdx.x * 128 + 4 * cx;
  const int lo = blockIdx.y * rows, hi = T - lo < rows ? T : lo + rows;
  float sum[4] = {0.f, 0.f, 0.f, 0.f};
  if (c < n) {                                            // n % 8 == 0
#pragma unroll 2
    for (int t = lo + ry; t < hi; t += 8) {
      float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < kSrc; ++k) {
        const DsbPackSrc& s = src[k];
        const int j0 = c - s.col0;
        if (j0 <= -4 || j0 >= s.cols) continue;
        const float* row = s.ptr + static_cast<size_t>(t) * s.ld;
        float a[4];
        if (s.vec && j0 >= 0 && j0 + 4 <= s.cols) {
          const float4 q = *reinterpret_cast<const float4*>(row + j0);
          a[0] = q.x; a[1] = q.y; a[2] = q.z; a[3] = q.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) a[j] = j0 + j >= 0 && j0 + j < s.cols ? row[j0 + j] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] += a[j];
      }
      if (thresh != 0u && c < n_drop) {                    // n_drop % 4 == 0
        float m[4];
        keep4(seed, (static_cast<long long>(t) * n_drop + c) >> 2, thresh, keep_scale, m);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] *= m[j];
      }
      const __nv_bfloat162 a2 = __floats2bfloat162_rn(v[0], v[1]), b2 = __floats2bfloat162_rn(v[2], v[3]);
      uint2 w;
      w.x = *reinterpret_cast<const uint32_t*>(&a2);
      w.y = *reinterpret_cast<const uint32_t*>(&b2);
      *reinterpret_cast<uint2*>(dst + static_cast<size_t>(t) * n + c) = w;
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[j] += v[j];
    }
  }
  if (part == nullptr) return;
#pragma unroll
  for (int j = 0; j < 4; ++j) s_sum[ry][4 * cx + j] = sum[j];
  __syncthreads();
  if (threadIdx.x < 128 && blockIdx.x * 128 + threadIdx.x < n) {
    float a = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) a += s_sum[r][threadIdx.x];
    part[static_cast<size_t>(blockIdx.y) * n + blockIdx.x * 128 + threadIdx.x] = a;
  }
}

// dropout of a [T, n] block with row stride ldx into a contiguous one (same mask as dropout_kernel
// on the contiguous tensor)
__global__ void __launch_bounds__(256) dropout_rows_kernel(const float* __restrict__ x, long long ldx,
                                                           float4* __restrict__ y, int T, int n4,
                                                           uint64_t seed, uint32_t thresh, float scale) {
  const long long total = static_cast<long long>(T) * n4;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    const long long t = i / n4;
    const int c = static_cast<int>(i - t * n4);
    float m[4];
    keep4(seed, i, thresh, scale, m);
    const float4 v = *reinterpret_cast<const float4*>(x + t * ldx + 4 * c);
    y[i] = make_float4(v.x * m[0], v.y * m[1], v.z * m[2], v.w * m[3]);
  }
}
}  // namespace

extern "C" int dsb_column_sum(const float* part, int rows, int n, float* out, cudaStream_t stream) {
  if (rows < 0 || n < 0 || (n & 3) || (reinterpret_cast<uintptr_t>(part) & 15) != 0) return 2;
  if (n == 0) return 0;
  column_sum_kernel<<<(n + 31) / 32, 256, 0, stream>>>(part, rows, n, out);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_linear_pack_blocks(int T) {
  const int rows = pack_rows(T);
  return T / rows + (T % rows != 0);
}

extern "C" int dsb_linear_pack(const DsbPackSrc* src, int n_src, int T, int n, void* dst_bf16,
                               float* colsum, float* part, unsigned long long seed, float p, int n_drop,
                               cudaStream_t stream) {
  if (T <= 0 || n <= 0) return 0;
  if (colsum != nullptr && (part == nullptr || (reinterpret_cast<uintptr_t>(part) & 15) != 0)) return 2;
  if (n_src < 1 || n_src > 5 || (n & 7) || (n_drop & 3) || !(p >= 0.f && p < 1.f)) return 2;
  DsbPackSrc s[5];
  for (int i = 0; i < 5; ++i) {
    s[i] = src[i < n_src ? i : 0];
    s[i].vec = (reinterpret_cast<uintptr_t>(s[i].ptr) & 15) == 0 && (s[i].ld & 3) == 0 && (s[i].col0 & 3) == 0;
  }
  const uint32_t thresh = static_cast<uint32_t>(static_cast<double>(p) * 4294967296.0);
  const int rows = pack_rows(T), row_blocks = dsb_linear_pack_blocks(T);
  const dim3 grid((n + 127) / 128, row_blocks);
  float* sums = colsum == nullptr ? nullptr : row_blocks == 1 ? colsum : part;
  __nv_bfloat16* d = static_cast<__nv_bfloat16*>(dst_bf16);
  const float sc = 1.f / (1.f - p);
  if (n_src == 1)
    linear_pack_kernel<1><<<grid, 256, 0, stream>>>(s[0], s[1], s[2], s[3], s[4], T, n, rows, d, sums, seed, thresh, sc, n_drop);
  else if (n_src == 2)
    linear_pack_kernel<2><<<grid, 256, 0, stream>>>(s[0], s[1], s[2], s[3], s[4], T, n, rows, d, sums, seed, thresh, sc, n_drop);
  else {
    for (int i = n_src; i < 5; ++i) s[i].cols = 0;         // covers nothing
    linear_pack_kernel<5><<<grid, 256, 0, stream>>>(s[0], s[1], s[2], s[3], s[4], T, n, rows, d, sums, seed, thresh, sc, n_drop);
  }
  if (sums != colsum) column_sum_kernel<<<(n + 31) / 32, 256, 0, stream>>>(part, row_blocks, n, colsum);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

extern "C" int dsb_dropout_rows(const float* x, long long ldx, float* y, int T, int n,
                                unsigned long long seed, float p, cudaStream_t stream) {
  if (T <= 0 || n <= 0) return 0;
  if ((n & 3) || (ldx & 3) || (reinterpret_cast<uintptr_t>(x) & 15) || !(p >= 0.f && p < 1.f)) return 2;
  const uint32_t thresh = static_cast<uint32_t>(static_cast<double>(p) * 4294967296.0);
  dropout_rows_kernel<<<grid_for(static_cast<long long>(T) * (n >> 2), 256, 148 * 16), 256, 0, stream>>>(
      x, ldx, reinterpret_cast<float4*>(y), T, n >> 2, seed, thresh, 1.f / (1.f - p));
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

// ------------------------------------------------------- operand of a router GEMM
// w [n, D] bf16 = bf16 of w1's n1 rows, then w2's n2, then zeros; b [n] = b1, b2, zeros.  Bound by its
// bytes (6 per element: 5.1 us for the 1152 + 3 rows of 2048 of the largest model, 1.6 for 384 + 3 of 384): made anew in
// every call, so that a kept copy need not be told of every way to write to a parameter.
namespace {
template <bool kVec>
__global__ void __launch_bounds__(256) router_operand_kernel(const float* __restrict__ w1,
                                                             const float* __restrict__ b1,
                                                             const float* __restrict__ w2,
                                                             const float* __restrict__ b2, int n1, int n2,
                                                             int n, int D, __nv_bfloat16* __restrict__ w,
                                                             float* __restrict__ b) {
  const long long first = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  const long long stride = static_cast<long long>(gridDim.x) * 256;
  const long long l1 = static_cast<long long>(n1) * D, l2 = l1 + static_cast<long long>(n2) * D;
  const long long total = static_cast<long long>(n) * D;
  for (long long i = first; i < n; i += stride) b[i] = i < n1 ? b1[i] : i < n1 + n2 ? b2[i - n1] : 0.f;
  if constexpr (kVec) {                                  // D % 4 == 0: a chunk lies in one row
    for (long long i = 4 * first; i < total; i += 4 * stride) {
      const float4 v = i < l1   ? *reinterpret_cast<const float4*>(w1 + i)
                       : i < l2 ? *reinterpret_cast<const float4*>(w2 + (i - l1))
                                : make_float4(0.f, 0.f, 0.f, 0.f);
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
      *reinterpret_cast<uint2*>(w + i) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  } else {
    for (long long i = first; i < total; i += stride)
      w[i] = __float2bfloat16(i < l1 ? w1[i] : i < l2 ? w2[i - l1] : 0.f);
  }
}
}  // namespace

extern "C" int dsb_router_operand(const float* w1, const float* b1, const float* w2, const float* b2, int n1,
                                  int n2, int n, int D, void* w_bf16, float* b, cudaStream_t stream) {
  if (n1 < 0 || n2 < 0 || n < n1 + n2 || D < 0) return 2;
  if (n == 0) return 0;
  __nv_bfloat16* w = static_cast<__nv_bfloat16*>(w_bf16);
  const long long total = static_cast<long long>(n) * D;
  if ((D & 3) == 0 && aligned16(w1, w2, w_bf16, nullptr))
    router_operand_kernel<true><<<grid_for(total / 4 + n, 256, 148 * 8), 256, 0, stream>>>(w1, b1, w2, b2, n1, n2, n, D, w, b);
  else
    router_operand_kernel<false><<<grid_for(total + n, 256, 148 * 8), 256, 0, stream>>>(w1, b1, w2, b2, n1, n2, n, D, w, b);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

// Prompt of a cached generation: q, k, v fp32 [B * S, H * dh] -> bf16 operands of the attention kernel
// and, for k and v, their fp32 rows in the caches [B, H, s_max, dh] at positions 0..S-1.  Bound by its
// bytes (12 read, 14 written per position and column) from a few thousand positions on, by being one
// launch in place of five below.
namespace {
__global__ void __launch_bounds__(256) prompt_qkv_kernel(const float4* __restrict__ q,
                                                         const float4* __restrict__ k,
                                                         const float4* __restrict__ v,
                                                         uint2* __restrict__ qb, uint2* __restrict__ kb,
                                                         uint2* __restrict__ vb, float* __restrict__ ck,
                                                         float* __restrict__ cv, int S, int H, int dh4,
                                                         int s_max, long long n) {
  auto bf = [](const float4& a) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(a.z, a.w);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  };
  const int d4 = H * dh4;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL) {
    const float4 a = q[i], b = k[i], c = v[i];
    qb[i] = bf(a);
    kb[i] = bf(b);
    vb[i] = bf(c);
    const long long row = i / d4;
    const int col = static_cast<int>(i - row * d4), h = col / dh4, j = col - h * dh4;
    const long long bi = row / S, s = row - bi * S;
    const long long at = ((bi * H + h) * s_max + s) * dh4 + j;
    reinterpret_cast<float4*>(ck)[at] = b;
    reinterpret_cast<float4*>(cv)[at] = c;
  }
}
}  // namespace

extern "C" int dsb_prompt_qkv(const float* q, const float* k, const float* v, void* qb, void* kb, void* vb,
                              float* cache_k, float* cache_v, int B, int S, int H, int dh, int s_max,
                              cudaStream_t stream) {
  if (B <= 0 || S <= 0 || H <= 0) return 0;
  if (dh <= 0 || (dh & 3) || S > s_max) return 2;
  const long long n = static_cast<long long>(B) * S * H * (dh >> 2);
  prompt_qkv_kernel<<<grid_for(n, 256, 148 * 16), 256, 0, stream>>>(
      reinterpret_cast<const float4*>(q), reinterpret_cast<const float4*>(k), reinterpret_cast<const float4*>(v),
      static_cast<uint2*>(qb), static_cast<uint2*>(kb), static_cast<uint2*>(vb), cache_k, cache_v, S, H,
      dh >> 2, s_max, n);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

// ----------------------------------------------------- multi-tensor launches
// AdamW and the squared gradient norm over a whole list of tensors in one launch
// each: a block takes one 64 K-element chunk of one tensor; the chunk -> tensor
// map is a prefix table in the kernel parameters (binary search, 8 steps).
namespace {

constexpr int kMultiMax = 160;                 // tensors per launch
constexpr long long kMultiChunk = 1 << 16;     // elements per block

struct MultiTable {
  const float* g[kMultiMax];
  float* p[kMultiMax];
  float* m[kMultiMax];
  float* v[kMultiMax];
  long long n[kMultiMax];
  int first_chunk[kMultiMax + 1];
  int count;
};

__device__ __forceinline__ int chunk_owner(const MultiTable& t, int chunk) {
  int lo = 0, hi = t.count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.first_chunk[mid] <= chunk) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(256) adamw_multi_kernel(const __grid_constant__ MultiTable t,
                                                          const float* __restrict__ clip_scale,
                                                          float lr, float b1, float b2, float eps,
                                                          float wd, float bc1, float bc2) {
  const int ti = chunk_owner(t, blockIdx.x);
  const long long off = static_cast<long long>(blockIdx.x - t.first_chunk[ti]) * kMultiChunk;
  const long long n = min(kMultiChunk, t.n[ti] - off);
  float* __restrict__ p = t.p[ti] + off;
  const float* __restrict__ g = t.g[ti] + off;
  float* __restrict__ m = t.m[ti] + off;
  float* __restrict__ v = t.v[ti] + off;
  const float cs = *clip_scale;
  auto update = [&](float& pi, float gi, float& mi, float& vi) {
    gi *= cs;
    mi = b1 * mi + (1.f - b1) * gi;
    vi = b2 * vi + (1.f - b2) * gi * gi;
    const float upd = (mi / bc1) / (sqrtf(vi / bc2) + eps) + wd * pi;
    pi = pi - lr * upd;
  };
  // Seven fp32 streams and nothing else to wait for: float4, two in flight per stream.  A step of the
  // 40M model's parameters takes 0.19 ms (0.64 with one float at a time), of the 400M model's 1.80 (2.79).
  long long i0 = 0;
  if (((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) |
        reinterpret_cast<uintptr_t>(v)) & 15) == 0) {
    const long long n4 = n >> 2;
    float4* p4 = reinterpret_cast<float4*>(p);
    const float4* g4 = reinterpret_cast<const float4*>(g);
    float4* m4 = reinterpret_cast<float4*>(m);
    float4* v4 = reinterpret_cast<float4*>(v);
    for (long long i = threadIdx.x; i < n4; i += 512) {
      float4 pq[2], gq[2], mq[2], vq[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (i + 256 * k < n4) {
          pq[k] = p4[i + 256 * k];
          gq[k] = __ldcs(g4 + i + 256 * k);
          mq[k] = m4[i + 256 * k];
          vq[k] = v4[i + 256 * k];
        }
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (i + 256 * k < n4) {
          update(pq[k].x, gq[k].x, mq[k].x, vq[k].x);
          update(pq[k].y, gq[k].y, mq[k].y, vq[k].y);
          update(pq[k].z, gq[k].z, mq[k].z, vq[k].z);
          update(pq[k].w, gq[k].w, mq[k].w, vq[k].w);
          p4[i + 256 * k] = pq[k];
          m4[i + 256 * k] = mq[k];
          v4[i + 256 * k] = vq[k];
        }
      }
    }
    i0 = n4 << 2;
  }
  for (long long i = i0 + threadIdx.x; i < n; i += blockDim.x) update(p[i], g[i], m[i], v[i]);
}

__global__ void __launch_bounds__(256) sqnorm_multi_kernel(const __grid_constant__ MultiTable t,
                                                           float* __restrict__ out) {
  const int ti = chunk_owner(t, blockIdx.x);
  const long long off = static_cast<long long>(blockIdx.x - t.first_chunk[ti]) * kMultiChunk;
  const long long n = min(kMultiChunk, t.n[ti] - off);
  const float* __restrict__ g = t.g[ti] + off;
  float s = 0.f;
  long long i0 = 0;
  if ((reinterpret_cast<uintptr_t>(g) & 15) == 0) {
    const long long n4 = n >> 2;
    const float4* g4 = reinterpret_cast<const float4*>(g);
#pragma unroll 4
    for (long long i = threadIdx.x; i < n4; i += 256) {
      const float4 x = g4[i];
      s = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, s))));
    }
    i0 = n4 << 2;
  }
  for (long long i = i0 + threadIdx.x; i < n; i += blockDim.x) {
    const float x = g[i];
    s = fmaf(x, x, s);
  }
  s = warp_sum(s);
  __shared__ float sh[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) sh[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int k = 0; k < 8; ++k) tot += sh[k];
    atomicAdd(out, tot);
  }
}

// Fills `t` with tensors [i0, i0 + cnt) of the lists; returns the number of chunks.
int fill_table(MultiTable& t, const float* const* g, float* const* p, float* const* m, float* const* v,
               const long long* n, int i0, int cnt) {
  int chunks = 0, k = 0;
  for (int i = i0; i < i0 + cnt; ++i) {
    if (n[i] <= 0) continue;
    t.g[k] = g[i];
    t.p[k] = p != nullptr ? p[i] : nullptr;
    t.m[k] = m != nullptr ? m[i] : nullptr;
    t.v[k] = v != nullptr ? v[i] : nullptr;
    t.n[k] = n[i];
    t.first_chunk[k] = chunks;
    chunks += static_cast<int>((n[i] + kMultiChunk - 1) / kMultiChunk);
    ++k;
  }
  t.first_chunk[k] = chunks;
  t.count = k;
  return chunks;
}

}  // namespace

extern "C" int dsb_adamw_multi(float* const* p, const float* const* g, float* const* m, float* const* v,
                               const long long* n, int count, const float* clip_scale, float lr,
                               float b1, float b2, float eps, float wd, float bc1, float bc2,
                               cudaStream_t stream) {
  for (int i0 = 0; i0 < count; i0 += kMultiMax) {
    MultiTable t;
    const int cnt = count - i0 < kMultiMax ? count - i0 : kMultiMax;
    const int chunks = fill_table(t, g, p, m, v, n, i0, cnt);
    if (chunks == 0) continue;
    adamw_multi_kernel<<<chunks, 256, 0, stream>>>(t, clip_scale, lr, b1, b2, eps, wd, bc1, bc2);
    if (cudaGetLastError() != cudaSuccess) return 1;
  }
  return 0;
}

extern "C" int dsb_sqnorm_multi(const float* const* g, const long long* n, int count, float* out,
                                cudaStream_t stream) {
  for (int i0 = 0; i0 < count; i0 += kMultiMax) {
    MultiTable t;
    const int cnt = count - i0 < kMultiMax ? count - i0 : kMultiMax;
    const int chunks = fill_table(t, g, nullptr, nullptr, nullptr, n, i0, cnt);
    if (chunks == 0) continue;
    sqnorm_multi_kernel<<<chunks, 256, 0, stream>>>(t, out);
    if (cudaGetLastError() != cudaSuccess) return 1;
  }
  return 0;
}
