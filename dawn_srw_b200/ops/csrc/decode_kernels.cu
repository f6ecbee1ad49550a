// SRW pool op for up to four stacked token rows (routes times sequences: V and Know of up to four
// sequences, Q and K of up to two; half of that above d_model 1280).
//
// With one to four rows the op is a stream over the pool: per unit u it needs
// e_u (r values), and r_u and w_u (d_model values each) where some row's gate is not
// zero (the relu-type gates of v3.9.4 / v4.0.1 are exactly zero below the threshold),
//   s_t  = <h_t, e_u>,   g_t = gate(s_t; tau_t, 1/sigma_t),   den_t += den_term
//   acc_t += bf16(g_t * <x_t, r_u>) * w_u
// and a few hundred FMAs.  A tensor-core tile would spend a 128-row MMA on those rows, so
// this path is plain SIMT and bound by HBM - if enough loads are in flight.  A block
// therefore takes its units in two phases: all scores first, four embedding rows in flight
// per group of lanes (eight with one token row and r <= 256), the units with a gate going on a list in shared memory; then the
// listed units, dealt evenly to the warps, with the next unit's read row and this unit's
// write row in flight.  (A warp that took a unit from score to write waited out the latency of
// HBM twice for every active one.)  Every sum has a fixed order: lists are compacted in unit order,
// blocks write partial outputs, and a second kernel adds those and applies scale / max(sum den, 1);
// adding them up with global reductions would save that launch, but a decoded token would no longer
// repeat bit by bit.  One row, 28 % of the units
// active: 100 000 units of 256 + 2 x 1280 and 10 400 of them in 31.2 us on average (39.2 for a warp per
// unit), 25 200 and 2 600 units of 128 + 2 x 384 in 8.8 (11.6); about half of the issue slots are used,
// a third of them for the loads' latency.
// The reference runs the generic chunked kernels for decoding
// (models/dawn_spatial_v41_exp.py:1713-1739, 1913-1957).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common/gate_math.cuh"
#include "common/ptx.cuh"
#include "dsb_api.h"
#include "dsb_api_ops.h"

namespace dsb {
namespace {

constexpr int kRowWarps = 8;        // warps per block
constexpr int kMaxRouteDim = 512;   // d_route <= 384 in every supported model

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// 8 bf16 -> 8 floats
__device__ __forceinline__ void unpack8(const uint4& q, float* f) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __bfloat1622float2(p[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}

__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

struct RowsParams {
  const __nv_bfloat16* h;       // [N, r]   contiguous
  const __nv_bfloat16* x;       // [N / x_rep, D] contiguous: row n of h goes with row n % (N / x_rep)
  const float* tau;             // [N]
  const float* isd;             // [N]
  const __nv_bfloat16* emb;     // [U, lde]
  const __nv_bfloat16* read;    // [U, ldr]
  const __nv_bfloat16* write;   // [U, ldw]
  const float* unit_mask;       // [U] or null
  long long lde, ldr, ldw;
  int N, x_rows, U, r, D;
  int lpu;                      // lanes that share a unit's embedding row (power of two)
  float* part;                  // [blocks, N, D] partial outputs
  float* den_part;              // [blocks, N]
  GateConsts gc;
};

constexpr int kListUnits = 512;     // units of a block between two list phases

// NR: rows handled (N <= NR); KC: 16-byte chunks of a d_model row per lane; EC: of an embedding row.
template <int KIND, int NR, int KC, int EC>
__global__ void __launch_bounds__(kRowWarps * 32, (NR == 1 && KC == 5) ? 2 : 1) srw_rows_kernel(const RowsParams p) {
  // registers allow the next read row to be in flight beside the accumulators
  constexpr bool kAhead = NR * KC <= 10;
  constexpr int kScoreUnroll = NR * EC == 1 ? 8 : 4;
  // One x row is kept in fp32 (used once per active unit, 31.2 us for 33.1); of several, reading twice the
  // shared memory costs more than unpacking: 100 000 units of 1280, all active, 2 rows 174 us in bf16, 196
  // in fp32; 4 rows 229 and 263; 28 % active 112 and 124, 186 and 217.
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* s_acc = reinterpret_cast<float*>(smem_raw);                                // [warps][NR][D]
  float* s_x = s_acc + kRowWarps * NR * p.D;                                        // [NR][D], fp32 or bf16
  __nv_bfloat16* s_h = reinterpret_cast<__nv_bfloat16*>(s_x + NR * p.D);                                            // [NR][r]
  float* s_g = reinterpret_cast<float*>(s_h + NR * p.r);                            // [kListUnits][NR]
  int* s_u = reinterpret_cast<int*>(s_g + kListUnits * NR);                         // [kListUnits] active units
  __shared__ float s_den[kRowWarps][NR];
  __shared__ int s_cnt[kRowWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int d_chunks = p.D >> 3, r_chunks = p.r >> 3;
  const uint4 none = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    const uint4* xs = reinterpret_cast<const uint4*>(p.x) + static_cast<size_t>(t % p.x_rows) * d_chunks;
    const uint4* hs = reinterpret_cast<const uint4*>(p.h) + static_cast<size_t>(t) * r_chunks;
    for (int c = tid; c < d_chunks; c += kRowWarps * 32) {
      if constexpr (NR >= 2) {
        reinterpret_cast<uint4*>(s_x)[t * d_chunks + c] = t < p.N ? xs[c] : none;
      } else {
        float f[8];
        unpack8(t < p.N ? xs[c] : none, f);
        float4* dst = reinterpret_cast<float4*>(s_x + t * p.D + 8 * c);
        dst[0] = make_float4(f[0], f[1], f[2], f[3]);
        dst[1] = make_float4(f[4], f[5], f[6], f[7]);
      }
    }
    for (int c = tid; c < r_chunks; c += kRowWarps * 32)
      reinterpret_cast<uint4*>(s_h)[t * r_chunks + c] = t < p.N ? hs[c] : none;
  }
  __syncthreads();
  RowGate rg[NR];
#pragma unroll
  for (int t = 0; t < NR; ++t)
    rg[t] = row_gate<KIND>(p.gc, t < p.N ? p.tau[t] : 0.f, t < p.N ? p.isd[t] : 1.f);

  const int lpu = p.lpu, sub = lane & (lpu - 1), groups = kRowWarps * 32 / lpu, grp = tid / lpu;
  float acc[NR][KC * 8];
  float den[NR];
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    den[t] = 0.f;
#pragma unroll
    for (int j = 0; j < KC * 8; ++j) acc[t][j] = 0.f;
  }
  const int per = (p.U + gridDim.x - 1) / gridDim.x;
  const int u_lo = blockIdx.x * per, u_hi = min(p.U, u_lo + per);
  for (int base = u_lo; base < u_hi; base += kListUnits) {
    const int end = min(u_hi, base + kListUnits);
    // ---- scores and gates of units [base, end)
    for (int u0 = base; u0 < end; u0 += kScoreUnroll * groups) {          // block-uniform trip count
      uint4 eq[kScoreUnroll][EC];
#pragma unroll
      for (int i = 0; i < kScoreUnroll; ++i) {
        const int u = u0 + i * groups + grp;
#pragma unroll
        for (int k = 0; k < EC; ++k) {
          const int c = sub + lpu * k;
          eq[i][k] = u < end && c < r_chunks ? ldg_stream(p.emb + static_cast<size_t>(u) * p.lde + 8 * c)
                                             : make_uint4(0u, 0u, 0u, 0u);
        }
      }
      float s[kScoreUnroll][NR];
#pragma unroll
      for (int i = 0; i < kScoreUnroll; ++i)
#pragma unroll
        for (int t = 0; t < NR; ++t) s[i][t] = 0.f;
#pragma unroll
      for (int k = 0; k < EC; ++k) {
        const int c = sub + lpu * k;
        if (c < r_chunks) {
#pragma unroll
          for (int t = 0; t < NR; ++t) {
            float hv[8];
            unpack8(*reinterpret_cast<const uint4*>(s_h + t * p.r + 8 * c), hv);
#pragma unroll
            for (int i = 0; i < kScoreUnroll; ++i) {
              float e[8];
              unpack8(eq[i][k], e);
#pragma unroll
              for (int j = 0; j < 8; ++j) s[i][t] = fmaf(e[j], hv[j], s[i][t]);
            }
          }
        }
      }
#pragma unroll
      for (int i = 0; i < kScoreUnroll; ++i)
#pragma unroll
        for (int t = 0; t < NR; ++t)
          for (int o = lpu >> 1; o > 0; o >>= 1) s[i][t] += __shfl_xor_sync(0xffffffffu, s[i][t], o);
      // every lane of a group holds the group's sums: lane `sub` evaluates the gate of unit `sub`
      // (of units sub, sub + lpu, .. in groups of fewer lanes), not the first lane that of all
      for (int i0 = 0; i0 < kScoreUnroll; i0 += lpu) {
        const int i = i0 + sub, u = u0 + i * groups + grp;
        float st[NR];
#pragma unroll
        for (int t = 0; t < NR; ++t) {
          st[t] = s[0][t];
#pragma unroll
          for (int k = 1; k < kScoreUnroll; ++k) st[t] = i == k ? s[k][t] : st[t];
        }
        if (i < kScoreUnroll && u < end) {
          const float um = p.unit_mask != nullptr ? p.unit_mask[u] : 1.f;
#pragma unroll
          for (int t = 0; t < NR; ++t) {
            float g, dt;
            gate_fwd_shifted<KIND>(p.gc, fmaf(st[t], rg[t].a, rg[t].b), g, dt);
            if (t < p.N) den[t] = fmaf(dt, um, den[t]);
            s_g[(u - base) * NR + t] = t < p.N ? g * um : 0.f;
          }
        }
      }
    }
    __syncthreads();
    // ---- the active units, in unit order: a warp compacts kListUnits / kRowWarps of them
    constexpr int kRounds = kListUnits / kRowWarps / 32;
    unsigned act[kRounds];
    int cnt = 0;
#pragma unroll
    for (int k = 0; k < kRounds; ++k) {
      const int l = (warp * kRounds + k) * 32 + lane;
      bool any = false;
      if (l < end - base) {
#pragma unroll
        for (int t = 0; t < NR; ++t) any = any || s_g[l * NR + t] != 0.f;
      }
      act[k] = __ballot_sync(0xffffffffu, any);
      cnt += __popc(act[k]);
    }
    if (lane == 0) s_cnt[warp] = cnt;
    __syncthreads();
    int n = 0, slot = 0;
#pragma unroll
    for (int w = 0; w < kRowWarps; ++w) {
      if (w == warp) slot = n;
      n += s_cnt[w];
    }
#pragma unroll
    for (int k = 0; k < kRounds; ++k) {
      if ((act[k] >> lane) & 1u)
        s_u[slot + __popc(act[k] & ((1u << lane) - 1u))] = (warp * kRounds + k) * 32 + lane;
      slot += __popc(act[k]);
    }
    __syncthreads();
    // ---- read scalars and gated writes of the listed units
    auto load_row = [&](const __nv_bfloat16* m, long long ld, int i, uint4 (&q)[KC]) {
      const __nv_bfloat16* row = m + static_cast<size_t>(i < n ? base + s_u[i] : 0) * ld;
#pragma unroll
      for (int k = 0; k < KC; ++k) {
        const int c = lane + 32 * k;
        q[k] = i < n && c < d_chunks ? ldg_stream(row + 8 * c) : make_uint4(0u, 0u, 0u, 0u);
      }
    };
    uint4 rq[KC], wq[KC];
    if (warp < n) {
      load_row(p.read, p.ldr, warp, rq);
      load_row(p.write, p.ldw, warp, wq);
    }
    for (int i = warp; i < n; i += kRowWarps) {
      uint4 rn[kAhead ? KC : 1];
      if constexpr (kAhead) load_row(p.read, p.ldr, i + kRowWarps, rn);
      float xr[NR];
#pragma unroll
      for (int t = 0; t < NR; ++t) xr[t] = 0.f;
#pragma unroll
      for (int k = 0; k < KC; ++k) {
        const int c = lane + 32 * k;
        if (c < d_chunks) {
          float rv[8];
          unpack8(rq[k], rv);
#pragma unroll
          for (int t = 0; t < NR; ++t) {
            float xv[8];
            if constexpr (NR >= 2) {
              unpack8(reinterpret_cast<const uint4*>(s_x)[t * d_chunks + c], xv);
            } else {
              const float4 a = *reinterpret_cast<const float4*>(s_x + t * p.D + 8 * c);
              const float4 b = *reinterpret_cast<const float4*>(s_x + t * p.D + 8 * c + 4);
              xv[0] = a.x; xv[1] = a.y; xv[2] = a.z; xv[3] = a.w;
              xv[4] = b.x; xv[5] = b.y; xv[6] = b.z; xv[7] = b.w;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) xr[t] = fmaf(rv[j], xv[j], xr[t]);
          }
        }
      }
      if constexpr (!kAhead) load_row(p.read, p.ldr, i + kRowWarps, rq);
      float pv[NR];
#pragma unroll
      for (int t = 0; t < NR; ++t)   // p is rounded to bf16, as the tile kernels store it
        pv[t] = __bfloat162float(__float2bfloat16(s_g[s_u[i] * NR + t] * warp_sum(xr[t])));
#pragma unroll
      for (int k = 0; k < KC; ++k) {
        float wv[8];
        unpack8(wq[k], wv);
#pragma unroll
        for (int t = 0; t < NR; ++t)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[t][8 * k + j] = fmaf(pv[t], wv[j], acc[t][8 * k + j]);
      }
      load_row(p.write, p.ldw, i + kRowWarps, wq);
      if constexpr (kAhead) {
#pragma unroll
        for (int k = 0; k < KC; ++k) rq[k] = rn[k];
      }
    }
    __syncthreads();               // the list has been read
  }
  // ---- the block's sums: a slab of shared memory per warp (floating-point atomics on shared memory
  // are compare-and-swap loops, and eight warps on the same words cost more than a small pool's
  // whole stream), summed on the way to global memory
  float* slab = s_acc + warp * NR * p.D;
#pragma unroll
  for (int t = 0; t < NR; ++t) {
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const int c = lane + 32 * k;
      if (c < d_chunks) {
        float4* dst = reinterpret_cast<float4*>(slab + t * p.D + 8 * c);
        const float* a = &acc[t][8 * k];
        dst[0] = make_float4(a[0], a[1], a[2], a[3]);
        dst[1] = make_float4(a[4], a[5], a[6], a[7]);
      }
    }
    const float d = warp_sum(den[t]);
    if (lane == 0) s_den[warp][t] = d;
  }
  __syncthreads();
  const int total = p.N * p.D;                                     // D % 8 == 0
  for (int i = 4 * tid; i < total; i += 4 * kRowWarps * 32) {
    float4 v = *reinterpret_cast<const float4*>(s_acc + i);
#pragma unroll
    for (int w = 1; w < kRowWarps; ++w) {
      const float4 o = *reinterpret_cast<const float4*>(s_acc + w * NR * p.D + i);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    *reinterpret_cast<float4*>(p.part + static_cast<size_t>(blockIdx.x) * total + i) = v;
  }
  if (tid < p.N) {
    float d = 0.f;
#pragma unroll
    for (int w = 0; w < kRowWarps; ++w) d += s_den[w][tid];
    p.den_part[blockIdx.x * p.N + tid] = d;
  }
}

// out[t, :] = (sum_b part[b, t, :]) * scale / max(sum_b den_part[b, t], 1).  A block covers 32
// columns of one row; sixteen warps share the blocks' partials (128-byte reads, eight in flight:
// with two in flight the launch was bound by their latency, 4.4 us for 1.5 MB).
constexpr int kFinishWarps = 16;
__global__ void __launch_bounds__(32 * kFinishWarps) srw_rows_finish_kernel(
    const float* __restrict__ part, const float* __restrict__ den_part, int blocks, int N, int D,
    float scale, const float* __restrict__ scale_ptr, float* __restrict__ out, float* __restrict__ den_out) {
  __shared__ float s_col[kFinishWarps][32];
  __shared__ float s_den[kFinishWarps];
  const int t = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int j = blockIdx.x * 32 + lane;
  float d = 0.f;
  for (int b = tid; b < blocks; b += 32 * kFinishWarps) d += den_part[b * N + t];
  d = warp_sum(d);
  if (lane == 0) s_den[warp] = d;
  float a = 0.f;
  if (j < D) {
    const float* col = part + static_cast<size_t>(t) * D + j;
    const size_t ld = static_cast<size_t>(N) * D;
    for (int b = warp; b < blocks; b += 8 * kFinishWarps) {
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = b + k * kFinishWarps < blocks ? col[(b + k * kFinishWarps) * ld] : 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) a += v[k];
    }
  }
  s_col[warp][lane] = a;
  __syncthreads();
  if (warp == 0) {
    float den = 0.f;
    a = 0.f;
#pragma unroll
    for (int g = 0; g < kFinishWarps; ++g) { den += s_den[g]; a += s_col[g][lane]; }
    const float sc = (scale_ptr != nullptr ? scale_ptr[0] : scale) / fmaxf(den, 1.f);
    if (j < D) out[static_cast<size_t>(t) * D + j] = a * sc;
    if (den_out != nullptr && blockIdx.x == 0 && lane == 0) den_out[t] = den;
  }
}

// ------------------------------------------------- attention over the KV cache
// One decoded token of one (batch, head): append k, v to the cache at position
// pos[0], then softmax(q . K[0..pos]^T / sqrt(dh)) . V[0..pos].  q, k, v, out are
// token-major fp32 [B, H * dh]; the caches are fp32 [B, H, S_max, dh].  The position
// is a device scalar so that the launch can sit in a captured graph.
//
// The op reads n * dh * 8 bytes per (batch, head) and is bound by how many of them are in
// flight, so the positions are split over the CTAs of a cluster, over warps and over
// eight groups of four lanes: a group takes a position, a lane every fourth 16-byte
// chunk of its K and V rows (64 contiguous bytes per group and load), all of them
// in flight together.  Every group keeps a running (max, sum, output), merged by shuffles,
// then in shared memory, then through the cluster's shared memory by its first CTA.
struct KvParams {
  const float *q, *k, *v;
  float *cache_k, *cache_v;
  const long long* pos;
  float* out;
  int H, dh, s_max;
  float scale;
};
constexpr int kKvThreads = 128, kKvGroups = kKvThreads / 4;
constexpr int kKvMaxDh = 128;
// Up to here the first CTA of a cluster takes all positions and the others leave: three rounds of its groups
// cost less than two cluster barriers.  6 x 16 heads of 128: 4.5 us for 9.7 at 3 positions, 7.2 for 9.9 at
// 96, 8.3 for 10.2 at 128; 6 heads of 64: 3.2 for 4.5, 4.4 for 4.7, and 5.0 for 4.8.  (A warp per position,
// the form for unaligned rows, takes 2.6 us at 3 positions and 16 to 20 at 96.)
constexpr int kSoloPositions = 96;

// A running maximum starts at the lowest finite value, not at -inf: a score of -inf then weighs
// nothing (exp(-inf - finite)) instead of turning into exp(-inf + inf), and a group without a
// position has nothing to weigh.
constexpr float kLowest = -3.402823466e38f;
__device__ __forceinline__ float merge_weight(float m, float m_all) { return __expf(m - m_all); }

// NV: 16-byte chunks of a head row per lane (dh <= 16 * NV, dh % 4 == 0).
template <int NV>
__global__ void __launch_bounds__(kKvThreads) kv_decode_split_kernel(const KvParams p) {
  __shared__ float s_m[kKvThreads / 32], s_l[kKvThreads / 32];
  __shared__ __align__(16) float s_o[kKvThreads / 32][kKvMaxDh];
  __shared__ float c_ml[2];
  __shared__ float c_o[kKvMaxDh];
  const int rank = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = lane & 3, grp = tid >> 2;
  const int nv4 = p.dh >> 2;
  long long pos = p.pos[0];
  pos = pos < 0 ? 0 : (pos >= p.s_max ? p.s_max - 1 : pos);
  const int n_old = static_cast<int>(pos);
  const int splits = n_old <= kSoloPositions ? 1 : gridDim.x;       // the same in every CTA of a cluster
  if (rank >= splits) return;
  const size_t row = (static_cast<size_t>(b) * p.H + h) * p.dh;
  float* ck = p.cache_k + row * p.s_max;
  float* cv = p.cache_v + row * p.s_max;
  const float4* q4 = reinterpret_cast<const float4*>(p.q + row);
  float4 qv[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = sub + 4 * i;
    qv[i] = c < nv4 ? q4[c] : make_float4(0.f, 0.f, 0.f, 0.f);
    qv[i].x *= p.scale; qv[i].y *= p.scale; qv[i].z *= p.scale; qv[i].w *= p.scale;
  }
  float m = kLowest, l = 0.f;
  float4 o[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  auto take = [&](const float* kr, const float* vr, bool valid) {
    float4 kq[NV], vq[NV];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = sub + 4 * i;
      const bool ok = valid && c < nv4;
      kq[i] = ok ? __ldcs(reinterpret_cast<const float4*>(kr) + c) : zero;
      vq[i] = ok ? __ldcs(reinterpret_cast<const float4*>(vr) + c) : zero;
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      s = fmaf(qv[i].x, kq[i].x, s);
      s = fmaf(qv[i].y, kq[i].y, s);
      s = fmaf(qv[i].z, kq[i].z, s);
      s = fmaf(qv[i].w, kq[i].w, s);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (!valid) return;
    const float mn = fmaxf(m, s);
    const float f = __expf(m - mn), e = __expf(s - mn);
    l = fmaf(l, f, e);
    m = mn;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      o[i].x = fmaf(o[i].x, f, e * vq[i].x);
      o[i].y = fmaf(o[i].y, f, e * vq[i].y);
      o[i].z = fmaf(o[i].z, f, e * vq[i].z);
      o[i].w = fmaf(o[i].w, f, e * vq[i].w);
    }
  };
  // cached positions 0..pos-1 of this CTA
  const int per = (n_old + splits - 1) / splits;
  const int j1 = min(n_old, (rank + 1) * per);
  for (int j0 = rank * per; j0 < j1; j0 += kKvGroups) {       // block-uniform trip count
    const int j = j0 + grp;
    take(ck + static_cast<size_t>(j) * p.dh, cv + static_cast<size_t>(j) * p.dh, j < j1);
  }
  // the new position comes from the inputs; the first warp of the first CTA appends it
  if (rank == 0 && warp == 0) {
    take(p.k + row, p.v + row, grp == 0);
    for (int c = lane; c < nv4; c += 32) {
      reinterpret_cast<float4*>(ck + pos * p.dh)[c] = reinterpret_cast<const float4*>(p.k + row)[c];
      reinterpret_cast<float4*>(cv + pos * p.dh)[c] = reinterpret_cast<const float4*>(p.v + row)[c];
    }
  }
  // ---- groups of a warp
  float mw = m;
#pragma unroll
  for (int x = 4; x < 32; x <<= 1) mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, x));
  const float fg = merge_weight(m, mw);
  l *= fg;
#pragma unroll
  for (int x = 4; x < 32; x <<= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float* e = reinterpret_cast<float*>(&o[i]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float t = e[k] * fg;
#pragma unroll
      for (int x = 4; x < 32; x <<= 1) t += __shfl_xor_sync(0xffffffffu, t, x);
      e[k] = t;
    }
    const int c = sub + 4 * i;
    if (lane < 4 && c < nv4) *reinterpret_cast<float4*>(&s_o[warp][4 * c]) = o[i];
  }
  if (lane == 0) { s_m[warp] = mw; s_l[warp] = l; }
  __syncthreads();
  // ---- warps of the CTA: thread t owns output column t
  float mc = s_m[0];
#pragma unroll
  for (int w = 1; w < kKvThreads / 32; ++w) mc = fmaxf(mc, s_m[w]);
  float lc = 0.f, oc = 0.f;
#pragma unroll
  for (int w = 0; w < kKvThreads / 32; ++w) {
    const float f = merge_weight(s_m[w], mc);
    lc = fmaf(f, s_l[w], lc);
    if (tid < p.dh) oc = fmaf(f, s_o[w][tid], oc);
  }
  if (splits == 1) {
    if (tid < p.dh) p.out[row + tid] = oc / lc;
    return;
  }
  // ---- CTAs of the cluster
  if (tid < p.dh) c_o[tid] = oc;
  if (tid == 0) { c_ml[0] = mc; c_ml[1] = lc; }
  cluster_sync_all();
  if (rank == 0) {
    float ms[8], ls[8], ma = kLowest;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < splits) {
        ms[r] = ld_cluster_f32(mapa_shared(smem_u32(&c_ml[0]), r));
        ls[r] = ld_cluster_f32(mapa_shared(smem_u32(&c_ml[1]), r));
        ma = fmaxf(ma, ms[r]);
      }
    }
    float lt = 0.f, ot = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < splits) {
        const float f = merge_weight(ms[r], ma);
        lt = fmaf(f, ls[r], lt);
        if (tid < p.dh) ot = fmaf(f, ld_cluster_f32(mapa_shared(smem_u32(&c_o[tid]), r)), ot);
      }
    }
    if (tid < p.dh) p.out[row + tid] = ot / lt;
  }
  cluster_sync_all();      // nobody leaves while its shared memory may still be read
}

// Any head dimension up to 128 and any alignment: a block per (batch, head), a warp per position.
__global__ void __launch_bounds__(128) kv_decode_attention_kernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
    float* __restrict__ cache_k, float* __restrict__ cache_v, const long long* __restrict__ pos_ptr,
    int H, int dh, int s_max, float inv_sqrt_dh, float* __restrict__ out) {
  extern __shared__ float s_p[];                 // [s_max] scores, then probabilities
  __shared__ float s_red[4];
  __shared__ float s_q[128];
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  long long pos = pos_ptr[0];
  if (pos < 0) pos = 0;
  if (pos >= s_max) pos = s_max - 1;
  const int n = static_cast<int>(pos) + 1;
  const size_t row = static_cast<size_t>(b) * H * dh + static_cast<size_t>(h) * dh;
  float* ck = cache_k + (static_cast<size_t>(b) * H + h) * s_max * dh;
  float* cv = cache_v + (static_cast<size_t>(b) * H + h) * s_max * dh;
  if (tid < dh) {
    ck[pos * dh + tid] = k[row + tid];
    cv[pos * dh + tid] = v[row + tid];
    s_q[tid] = q[row + tid] * inv_sqrt_dh;
  }
  __syncthreads();
  // scores: one warp per cache position
  float mx = -3.0e38f;
  for (int j = warp; j < n; j += 4) {
    float a = 0.f;
    for (int t = lane; t < dh; t += 32) a = fmaf(s_q[t], ck[static_cast<size_t>(j) * dh + t], a);
    a = warp_sum(a);
    if (lane == 0) s_p[j] = a;
    mx = fmaxf(mx, a);
  }
  if (lane == 0) s_red[warp] = mx;
  __syncthreads();
  mx = fmaxf(fmaxf(s_red[0], s_red[1]), fmaxf(s_red[2], s_red[3]));
  __syncthreads();
  float sum = 0.f;
  for (int j = tid; j < n; j += 128) {
    const float e = __expf(s_p[j] - mx);
    s_p[j] = e;
    sum += e;
  }
  sum = warp_sum(sum);
  if (lane == 0) s_red[warp] = sum;
  __syncthreads();
  const float inv = 1.f / (s_red[0] + s_red[1] + s_red[2] + s_red[3]);
  if (tid < dh) {
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
    int j = 0;
    for (; j + 4 <= n; j += 4) {
      a0 = fmaf(s_p[j], cv[static_cast<size_t>(j) * dh + tid], a0);
      a1 = fmaf(s_p[j + 1], cv[static_cast<size_t>(j + 1) * dh + tid], a1);
      a2 = fmaf(s_p[j + 2], cv[static_cast<size_t>(j + 2) * dh + tid], a2);
      a3 = fmaf(s_p[j + 3], cv[static_cast<size_t>(j + 3) * dh + tid], a3);
    }
    for (; j < n; ++j) a0 = fmaf(s_p[j], cv[static_cast<size_t>(j) * dh + tid], a0);
    out[row + tid] = ((a0 + a1) + (a2 + a3)) * inv;
  }
}

// y[t, n] = <x_t, W_n> + bias[n] for up to four rows x_t: one warp per output column, the
// weight matrix streamed once with 16-byte loads, x in shared memory.  x bf16 [N, K]
// contiguous, W bf16 [n_out, ldw], y fp32 [N, ldy]; K % 8 == 0.
template <int NR>
__global__ void __launch_bounds__(256) gemv_rows_kernel(const __nv_bfloat16* __restrict__ x,
                                                        const __nv_bfloat16* __restrict__ w, long long ldw,
                                                        const float* __restrict__ bias,
                                                        float* __restrict__ y, long long ldy, int N,
                                                        int n_out, int K) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __nv_bfloat16* s_x = reinterpret_cast<__nv_bfloat16*>(smem_raw);
  for (int i = threadIdx.x; i < NR * K; i += blockDim.x)
    s_x[i] = i / K < N ? x[i] : __float2bfloat16(0.f);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, chunks = K >> 3;
  for (int n = blockIdx.x * 8 + warp; n < n_out; n += gridDim.x * 8) {
    float acc[NR];
#pragma unroll
    for (int t = 0; t < NR; ++t) acc[t] = 0.f;
    const __nv_bfloat16* wr = w + static_cast<size_t>(n) * ldw;
    for (int c = lane; c < chunks; c += 32) {
      float wv[8];
      unpack8(ldg_stream(wr + 8 * c), wv);
#pragma unroll
      for (int t = 0; t < NR; ++t) {
        float xv[8];
        unpack8(*reinterpret_cast<const uint4*>(s_x + t * K + 8 * c), xv);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[t] = fmaf(wv[j], xv[j], acc[t]);
      }
    }
#pragma unroll
    for (int t = 0; t < NR; ++t) {
      const float a = warp_sum(acc[t]);
      if (lane == 0 && t < N) y[static_cast<size_t>(t) * ldy + n] = a + (bias != nullptr ? bias[n] : 0.f);
    }
  }
}

int device_sms() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 148;
}

template <int NV>
int launch_kv_nv(const KvParams& p, int splits, int B, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(splits, p.H, B);
  cfg.blockDim = dim3(kKvThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kv_decode_split_kernel<NV>, p) == cudaSuccess ? 0 : 913;
}

// The position is not known here, so the split follows from what the cache can hold: up to
// eight CTAs per (batch, head) until there are four CTAs per SM, none shorter than 32 positions.
int launch_kv(const KvParams& p, int B, cudaStream_t stream) {
  const int want = 4 * device_sms();
  int splits = 1;
  while (splits < 8 && B * p.H * splits < want && p.s_max / (2 * splits) >= kKvGroups) splits *= 2;
  if (p.dh <= 32) return launch_kv_nv<2>(p, splits, B, stream);
  if (p.dh <= 64) return launch_kv_nv<4>(p, splits, B, stream);
  if (p.dh <= 80) return launch_kv_nv<5>(p, splits, B, stream);
  return launch_kv_nv<8>(p, splits, B, stream);
}

template <int KIND, int NR, int KC, int EC>
int launch_rows(const RowsParams& p, int blocks, cudaStream_t stream) {
  const size_t smem = static_cast<size_t>(NR) * (p.D * 4 + p.r * 2) +
                      static_cast<size_t>(kRowWarps) * NR * p.D * 4 + static_cast<size_t>(kListUnits) * (NR + 1) * 4;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(srw_rows_kernel<KIND, NR, KC, EC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             200 * 1024) != cudaSuccess)
      return 902;
    attr_set = true;
  }
  if (smem > 200 * 1024) return 903;
  srw_rows_kernel<KIND, NR, KC, EC><<<blocks, kRowWarps * 32, smem, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : 904;
}

template <int KIND, int EC>
int dispatch_rows(const RowsParams& p, int NR, int KC, int blocks, cudaStream_t stream) {
  if (KC == 5) {
    if (NR == 1) return launch_rows<KIND, 1, 5, EC>(p, blocks, stream);
    if (NR == 2) return launch_rows<KIND, 2, 5, EC>(p, blocks, stream);
    return launch_rows<KIND, 4, 5, EC>(p, blocks, stream);
  }
  if (NR == 1) return launch_rows<KIND, 1, 8, EC>(p, blocks, stream);
  if (NR == 2) return launch_rows<KIND, 2, 8, EC>(p, blocks, stream);
  return 905;
}

template <int KIND>
int dispatch_rows(const RowsParams& p, int NR, int KC, int blocks, cudaStream_t stream) {
  return p.r <= 256 ? dispatch_rows<KIND, 1>(p, NR, KC, blocks, stream)
                    : dispatch_rows<KIND, 2>(p, NR, KC, blocks, stream);
}

}  // namespace
}  // namespace dsb

using namespace dsb;

extern "C" int dsb_srw_rows_max(int D) {
  if (D % 8 != 0 || D > 2048) return 0;
  return D <= 1280 ? 4 : 2;
}

extern "C" int dsb_srw_rows_blocks(int N, int D) {
  const int n = device_sms();
  return (N <= 1 && D <= 1280) ? 2 * n : n;   // one row needs 128 registers: two blocks per SM
}

extern "C" int dsb_srw_rows(const void* h, const void* x, int x_rows, const float* tau, const float* isd,
                            const void* emb, long long lde, const void* read, long long ldr,
                            const void* write, long long ldw, const float* unit_mask, int N, int U,
                            int r, int D, const DsbGate* gate, float scale, const float* scale_ptr,
                            float* part, float* out, float* den_out, cudaStream_t stream) {
  if (N <= 0 || U <= 0) return 0;
  if (x_rows <= 0 || (reinterpret_cast<uintptr_t>(part) & 15) != 0) return 907;
  const int max_rows = dsb_srw_rows_max(D);
  if (N > max_rows || r % 8 != 0 || r > kMaxRouteDim || lde % 8 != 0 || ldr % 8 != 0 || ldw % 8 != 0)
    return 901;
  const int NR = N <= 1 ? 1 : N <= 2 ? 2 : 4;
  const int KC = D <= 1280 ? 5 : 8;
  const int blocks = dsb_srw_rows_blocks(N, D);
  RowsParams p;
  p.h = static_cast<const __nv_bfloat16*>(h);
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.tau = tau;
  p.isd = isd;
  p.emb = static_cast<const __nv_bfloat16*>(emb);
  p.read = static_cast<const __nv_bfloat16*>(read);
  p.write = static_cast<const __nv_bfloat16*>(write);
  p.unit_mask = unit_mask;
  p.lde = lde; p.ldr = ldr; p.ldw = ldw;
  p.N = N; p.x_rows = x_rows; p.U = U; p.r = r; p.D = D;
  p.lpu = 1;
  while (p.lpu < 32 && 8 * p.lpu < r) p.lpu *= 2;
  p.part = part;
  p.den_part = part + static_cast<size_t>(blocks) * N * D;
  p.gc = {gate->kind, gate->sharpness, gate->act_threshold, gate->act_cutoff, gate->epsilon,
          gate->max_intensity, gate->clip_max, gate->dead_threshold};
  int rc;
  if (gate->kind == 0) rc = dispatch_rows<0>(p, NR, KC, blocks, stream);
  else if (gate->kind == 1) rc = dispatch_rows<1>(p, NR, KC, blocks, stream);
  else rc = dispatch_rows<2>(p, NR, KC, blocks, stream);
  if (rc) return rc;
  srw_rows_finish_kernel<<<dim3((D + 31) / 32, N), 32 * kFinishWarps, 0, stream>>>(
      part, p.den_part, blocks, N, D, scale, scale_ptr, out, den_out);
  return cudaGetLastError() == cudaSuccess ? 0 : 906;
}

extern "C" int dsb_kv_decode_attention(const float* q, const float* k, const float* v, float* cache_k,
                                       float* cache_v, const long long* pos, int B, int H, int dh,
                                       int s_max, float* out, cudaStream_t stream) {
  if (B <= 0 || H <= 0) return 0;
  if (dh <= 0 || dh > 128 || s_max <= 0 || s_max > 8192) return 911;
  const float scale = rsqrtf(static_cast<float>(dh));
  const uintptr_t bits = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
                         reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(cache_k) |
                         reinterpret_cast<uintptr_t>(cache_v);
  if (dh % 4 == 0 && (bits & 15) == 0) {
    const KvParams p = {q, k, v, cache_k, cache_v, pos, out, H, dh, s_max, scale};
    return launch_kv(p, B, stream);
  }
  const dim3 grid(H, B);
  kv_decode_attention_kernel<<<grid, 128, static_cast<size_t>(s_max) * sizeof(float), stream>>>(
      q, k, v, cache_k, cache_v, pos, H, dh, s_max, scale, out);
  return cudaGetLastError() == cudaSuccess ? 0 : 912;
}

extern "C" int dsb_gemv_rows(const void* x, const void* w, long long ldw, const float* bias, float* y,
                             long long ldy, int N, int n_out, int K, cudaStream_t stream) {
  if (N <= 0 || n_out <= 0) return 0;
  if (N > 4 || K % 8 != 0 || K > 8192 || ldw % 8 != 0) return 921;
  const int NR = N <= 1 ? 1 : N <= 2 ? 2 : 4;
  int blocks = (n_out + 7) / 8;
  const int cap = 8 * dsb_srw_rows_blocks(4, 2048);
  if (blocks > cap) blocks = cap;
  const size_t smem = static_cast<size_t>(NR) * K * 2;
  static bool attr_set = false;
  if (!attr_set) {
    cudaFuncSetAttribute(gemv_rows_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    cudaFuncSetAttribute(gemv_rows_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    cudaFuncSetAttribute(gemv_rows_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    attr_set = true;
  }
  const __nv_bfloat16* xb = static_cast<const __nv_bfloat16*>(x);
  const __nv_bfloat16* wb = static_cast<const __nv_bfloat16*>(w);
  if (NR == 1) gemv_rows_kernel<1><<<blocks, 256, smem, stream>>>(xb, wb, ldw, bias, y, ldy, N, n_out, K);
  else if (NR == 2) gemv_rows_kernel<2><<<blocks, 256, smem, stream>>>(xb, wb, ldw, bias, y, ldy, N, n_out, K);
  else gemv_rows_kernel<4><<<blocks, 256, smem, stream>>>(xb, wb, ldw, bias, y, ldy, N, n_out, K);
  return cudaGetLastError() == cudaSuccess ? 0 : 922;
}
