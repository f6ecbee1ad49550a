// C ABI of the memory-bound kernels (see elementwise_kernels.cu).  Device
// pointers; asynchronous on `stream`; return 0 on a successful launch.
#pragma once
#include <cuda_runtime.h>

#ifdef __cplusplus
extern "C" {
#endif

// y = (x - mean) * rstd * w + b, eps inside the sqrt; x fp32 [T,D], y bf16 [T,D].
int dsb_layernorm_fwd(const float* x, const float* w, const float* b, void* y_bf16, float* mean,
                      float* rstd, int T, int D, float eps, cudaStream_t stream);
// dx fp32 [T,D]; dw, db fp32 [D] are accumulated into (zero them first).
int dsb_layernorm_bwd(const void* dy_bf16, const float* x, const float* w, const float* mean,
                      const float* rstd, float* dx, float* dw, float* db, int T, int D,
                      cudaStream_t stream);
// Row statistics of fp32 logits [R, ld] with V valid columns: logsumexp, the
// label's logit (labels < 0 read column 0) and the arg-max.
int dsb_ce_fwd(const float* logits, long long ld, const long long* labels, int R, int V, float* lse,
               float* label_logit, long long* argmax, cudaStream_t stream);
// dl = scale[row] * (softmax - onehot) as bf16 [R, ldo] (columns V..ldo zeroed).
int dsb_ce_bwd(const float* logits, long long ld, const long long* labels, const float* lse,
               const float* scale, int R, int V, void* dl_bf16, long long ldo, cudaStream_t stream);
// AdamW step on one tensor; the global-norm clip factor is read from device memory.
int dsb_adamw(float* p, const float* g, float* m, float* v, long long n, const float* clip_scale,
              float lr, float b1, float b2, float eps, float wd, float bc1, float bc2,
              cudaStream_t stream);
// out[0] += sum(g^2)
int dsb_sqnorm_accumulate(const float* g, long long n, float* out, cudaStream_t stream);
// The same two operations over lists of tensors (host arrays of device pointers and element
// counts) in one launch per 160 tensors: a block takes a 64 K-element chunk of one tensor.
int dsb_adamw_multi(float* const* p, const float* const* g, float* const* m, float* const* v,
                    const long long* n, int count, const float* clip_scale, float lr, float b1,
                    float b2, float eps, float wd, float bc1, float bc2, cudaStream_t stream);
int dsb_sqnorm_multi(const float* const* g, const long long* n, int count, float* out,
                     cudaStream_t stream);

// out[t, :] = tok[ids[t], :] + pos[t % S, :]  (fp32, D % 4 == 0; ids clamped to [0, V)).
int dsb_embed_fwd(const long long* ids, const float* tok, const float* pos, float* out, int T, int S,
                  int D, int V, cudaStream_t stream);
// dtok[ids[t], :] += dy[t, :] (dtok zeroed by the caller); dpos[s, :] = sum_b dy[b*S+s, :].
int dsb_embed_bwd(const long long* ids, const float* dy, float* dtok, float* dpos, int B, int S,
                  int D, int V, cudaStream_t stream);
// total[0] += sum_{i != j} |sim_ij|; sgn (bf16 [m, ld_s]) = sign(sim) off the diagonal, 0 on it.
int dsb_offdiag_abs(const float* sim, long long ld, int m, void* sgn_bf16, long long ld_s,
                    float* total, cudaStream_t stream);
// dy_bf = bf16(dy * row_scale[t]); rowdot[t] = <dy[t], y[t]>   (dy, y fp32 [T, D], D % 4 == 0)
int dsb_route_bwd_prologue(const float* dy, const float* y, const float* row_scale,
                           void* dy_bf16, float* rowdot, int T, int D, cudaStream_t stream);

// With rs = s / max(den, 1), s = *scale_ptr or scale: dy_bf = bf16(dy * rs); with rowdot = <dy, y>:
// d_den = -rowdot / den where den > 1, else 0 (+ ext_dden, nullable); dtau = 0;
// d_scale[0] += sum_t rowdot / s (nullable; dots: T / 8 rounded up floats of scratch for it).  dy, y fp32 [T, D], D % 4 == 0, 16-byte aligned.
int dsb_route_bwd_rows(const float* dy, const float* y, const float* den, const float* scale_ptr,
                       float scale, const float* ext_dden, void* dy_bf16, float* d_den, float* dtau,
                       float* d_scale, float* dots, int T, int D, cudaStream_t stream);

// y = res + dropout(x) (res may be null: y = dropout(x)); fp32, n % 4 == 0.  An element is kept
// (and scaled by 1 / (1 - p)) iff a hash of (seed, its index) is >= p * 2^32, so the gradient
// of x is the same call with res = null on the incoming gradient.
int dsb_dropout(const float* res, const float* x, float* y, long long n, unsigned long long seed,
                float p, cudaStream_t stream);

// out[j] = sum over the rows of part [rows, n], in a fixed order; n % 4 == 0, part 16-byte aligned.
int dsb_column_sum(const float* part, int rows, int n, float* out, cudaStream_t stream);

// Gradient operand of a linear layer: dst bf16 [T, n] = bf16(sum of the up to five fp32 sources that
// cover a column: cols columns from col0, row stride ld), 0 where none does; colsum [n] (nullable) = its
// column sums, with part as scratch (dsb_linear_pack_blocks(T) * n floats, 16-byte aligned).  With p > 0 the columns [0, n_drop) are the gradient of a dropped
// [T, n_drop] tensor: the keep mask of (seed, p) is applied.  n % 8 == 0, n_drop % 4 == 0.
struct DsbPackSrc {
  const float* ptr;
  long long ld;
  int col0, cols;
  int vec;          // set by the launcher: rows may be read as float4
};
int dsb_linear_pack_blocks(int T);
int dsb_linear_pack(const struct DsbPackSrc* src, int n_src, int T, int n, void* dst_bf16, float* colsum,
                    float* part, unsigned long long seed, float p, int n_drop, cudaStream_t stream);
// Operand of a router GEMM: w bf16 [n, D] = rows of w1 [n1, D], of w2 [n2, D], zeros; b [n] likewise
// (all fp32 contiguous, n >= n1 + n2).
int dsb_router_operand(const float* w1, const float* b1, const float* w2, const float* b2, int n1, int n2,
                       int n, int D, void* w_bf16, float* b, cudaStream_t stream);
// y [T, n] = dropout(x [T, ldx]) with the mask of the contiguous tensor; n, ldx % 4 == 0.
int dsb_dropout_rows(const float* x, long long ldx, float* y, int T, int n, unsigned long long seed, float p,
                     cudaStream_t stream);

// q, k, v fp32 [B*S, H*dh] -> bf16 copies; k, v also into the fp32 caches [B, H, s_max, dh] at
// positions 0..S-1.  dh % 4 == 0, everything 16-byte aligned, S <= s_max.
int dsb_prompt_qkv(const float* q, const float* k, const float* v, void* qb, void* kb, void* vb,
                   float* cache_k, float* cache_v, int B, int S, int H, int dh, int s_max,
                   cudaStream_t stream);

// Per-token score statistics from hg = h . (E^T E) (fp32 [N, r]) and bf16 h [N, ldh]:
//   mu = <h, esum> * inv_u,  var = <hg, h> * inv_u - mu^2,  sd = sqrt(max(var, 1e-12)) + 1e-8,
//   tau = mu + off * sd,  isd = 1 / sd;  hsum[r] += column sums of h (hsum may be null).
// hg has row stride ldg; hg2 (nullable) is a second part of it, added on the fly.  Row n is token
// n % T of route n / T; its offset is off[t * o_st + route * o_sr].
int dsb_score_stats_fwd(const float* hg, const float* hg2, long long ldg, const void* h_bf16,
                        long long ldh, const float* esum, const float* off, long long o_st,
                        long long o_sr, int T, float inv_u, int N, int r, float* tau, float* isd,
                        float* mu, float* sd, float* hsum, cudaStream_t stream);
// hb[ri * T + t, :] = bf16(h[t, ri, :]) (h fp32, strides h_st, h_sr, unit inner stride, r % 8 == 0);
// z1[0 .. n1) = z2[0 .. n2) = 0.
int dsb_score_pack(const float* h, long long h_st, long long h_sr, int T, int R, int r, void* hb_bf16,
                   float* z1, int n1, float* z2, int n2, cudaStream_t stream);
// Row part of a call's backward (rows route-major, N = R * T): from dtau [N] and dh32 [N, r] of the
// gate step, the sigma path (sigma_path != 0) and the statistics: dh fp32 [T, R, r], d_off [T, R],
// w = bf16(d_var * h) [N, r] (operand of dG = w^T h * inv_u); accumulates d_esum [r].
int dsb_score_route_bwd(const float* dtau, const float* dh32, const float* d_hsum, const float* off,
                        long long o_st, long long o_sr, const float* tau, const float* isd,
                        const float* mu, const float* sd, const float* hg, const float* hg2,
                        long long ldg, const void* h_bf16, const float* esum, float inv_u,
                        int sigma_path, int T, int R, int r, float* dh, void* w_bf16, float* d_off,
                        float* d_esum, cudaStream_t stream);
// The same statistics for a handful of rows in one launch (generation), from fp32 h [T, R, r]
// (strides h_st, h_sr in elements, unit inner stride), off [T, R] (strides o_st, o_sr) and the
// fp32 Gram matrix.  Output rows are route-major: row ri * T + t; hb is bf16(h) [R * T, r].
// zero[0 .. n_zero) = 0 on the way (scratch of a later launch; may be null with n_zero = 0).
int dsb_score_stats_rows(const float* h, long long h_st, long long h_sr, const float* off,
                         long long o_st, long long o_sr, const float* gram, const float* esum,
                         float inv_u, int T, int R, int r, float* tau, float* isd, void* hb_bf16,
                         float* zero, long long n_zero, cudaStream_t stream);
// Backward of the above.  d_tau, d_isd [N], d_hsum [r], d_hb (bf16 [N, r] cotangent of the
// bf16 copy of h) may be null.  Writes dh fp32 [N, r] (all terms summed), w = bf16(d_var * h)
// [N, ldw] (operand of dG = w^T h * inv_u), d_off [N]; accumulates d_esum [r] (zero it first).
int dsb_score_stats_bwd(const float* d_tau, const float* d_isd, const float* d_hsum,
                        const void* d_hb_bf16, const float* off, const float* mu, const float* sd,
                        const float* hg, const void* h_bf16, long long ldh, const float* esum,
                        float inv_u, int N, int r, float* dh, void* w_bf16, long long ldw,
                        float* d_off, float* d_esum, cudaStream_t stream);

// Load-balance term of a pool from the column sums of h: m_u = <e_u, hsum> * inv_n [U],
//   lb = var / (mean^2 + var + 0.01) with mean = sum m_u / units, var = sum m_u^2 / units - mean^2.
// emb bf16 [U, lde], r and lde multiples of 8, r <= 512.  part: 2 * dsb_load_balance_blocks floats of
// scratch; m_u and stat [2] are kept for the backward call, which writes dmn [U] (= d m_u * inv_n)
// and d_hsum [r], with dsb_load_balance_blocks * r floats of scratch (16-byte aligned) as its part; the
// embedding gradient is dmn[u] * hsum.
int dsb_load_balance_blocks(int U, int r);
int dsb_load_balance_fwd(const void* emb_bf16, long long lde, const float* hsum, float inv_n,
                         float units, int U, int r, float* m_u, float* part, float* lb, float* stat,
                         cudaStream_t stream);
int dsb_load_balance_bwd(const void* emb_bf16, long long lde, const float* m_u, const float* stat,
                         const float* g_lb, float inv_n, float units, int U, int r, float* dmn,
                         float* d_hsum, float* part, cudaStream_t stream);
// g[u, :] += sum_l dm[l, u] * hs[l, :]  (g fp32 [U, ldg], dm [L, U], hs [L, r], r % 4 == 0).
int dsb_rank1_add(float* g, long long ldg, const float* dm, const float* hs, int L, int U, int r,
                  cudaStream_t stream);

// SRW pool op for a handful of token rows (decoding): one streaming pass over the pool.
// h [N, r], x [x_rows, D] bf16 contiguous (row n % x_rows of x belongs to row n of h), tau / isd [N];
// emb / read / write bf16 with row strides in elements (multiples of 8); unit_mask [U] or null.
// out[n, :] = (sum_u bf16(g * <x_n, r_u>) w_u) * scale / max(sum_u den_term, 1), fp32 [N, D];
// scale_ptr (device scalar) overrides scale when not null; den_out [N] may be null.
// part: dsb_srw_rows_blocks(N, D) * N * (D + 1) floats of scratch, 16-byte aligned.
// N <= dsb_srw_rows_max(D) (4 up to d_model 1280, 2 up to 2048, else 0).
int dsb_srw_rows_max(int D);
int dsb_srw_rows_blocks(int N, int D);
struct DsbGate;
int dsb_srw_rows(const void* h, const void* x, int x_rows, const float* tau, const float* isd,
                 const void* emb, long long lde, const void* read, long long ldr, const void* write,
                 long long ldw, const float* unit_mask, int N, int U, int r, int D,
                 const struct DsbGate* gate, float scale, const float* scale_ptr, float* part, float* out,
                 float* den_out, cudaStream_t stream);

// One decoded token: k, v [B, H*dh] are appended to the fp32 caches [B, H, s_max, dh] at
// position pos[0] (device scalar), out [B, H*dh] = softmax(q K^T / sqrt(dh)) V over 0..pos.
int dsb_kv_decode_attention(const float* q, const float* k, const float* v, float* cache_k,
                            float* cache_v, const long long* pos, int B, int H, int dh, int s_max,
                            float* out, cudaStream_t stream);

// y[t, n] = <x_t, W_n> + bias[n] for N <= 4 rows (decoding): x bf16 [N, K] contiguous, W bf16
// [n_out, ldw], bias fp32 [n_out] or null, y fp32 [N, ldy]; K % 8 == 0, K <= 8192.
int dsb_gemv_rows(const void* x, const void* w, long long ldw, const float* bias, float* y,
                  long long ldy, int N, int n_out, int K, cudaStream_t stream);

// Causal self-attention (tcgen05 kernels).  q, k, v, out, d_out: bf16 [B, S, H*dh]
// (head h in columns [h*dh, (h+1)*dh)); dh a multiple of 16, at most 128.
// lse, delta: fp32 [B, H, S] (delta is scratch filled by the backward call).
// Dropout on the attention weights is a hash of (seed, batch*head, query, key):
// pass the forward call's p_drop and seed to the backward call.
int dsb_attention_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B,
                      int H, int S, int dh, float p_drop, unsigned long long seed, int* status,
                      cudaStream_t stream);
// dq: fp32 [B, S, H*dh], ZEROED by the caller (query tiles are reduce-added into
// it); dk, dv: bf16 [B, S, H*dh].
int dsb_attention_bwd(const void* q, const void* k, const void* v, const void* out,
                      const void* d_out, const float* lse, float* delta, float* dq, void* dk,
                      void* dv, int B, int H, int S, int dh, float p_drop,
                      unsigned long long seed, int* status, cudaStream_t stream);

#ifdef __cplusplus
}
#endif
