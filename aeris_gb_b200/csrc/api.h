// C ABI of libaeris_b200.so. Every function returns 0 on success and a negative code on a host-side argument or
// launch error. Kernels report device-side problems (bounded waits that ran out, failed bounds checks) through
// the `status` word, which the caller owns and reads after synchronising.
#pragma once
#include <stdint.h>
#ifdef __cplusplus
extern "C" {
#endif

int aeris_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                    int a_mn, int b_mn, int epi, const void* resid, int ldr, const float* gate,
                    int rows_per_gate, void* aux, int ld_aux, int swiglu_f, int k_splits, int bn, int* status,
                    void* stream);

int aeris_gemm_bf16_2cta(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                         int a_mn, int b_mn, int epi, const void* resid, int ldr, const float* gate,
                         int rows_per_gate, void* aux, int ld_aux, int swiglu_f, int k_splits, int* status,
                         void* stream);

// The one of the two that is the faster for the shape (see gemm2.cu). bn: tile width of the one-CTA kernel (0: from N);
// allow_2cta = 0: never the other, 2: the other wherever it takes the product. ld_gate: elements from one gate row to the
// next (a multiple of 4; N where they lie without gaps).
int aeris_gemm_auto(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int a_mn,
                    int b_mn, int epi, const void* resid, int ldr, const float* gate, int rows_per_gate, int ld_gate,
                    void* aux, int ld_aux, int swiglu_f, int k_splits, int bn, int allow_2cta, int* status, void* stream);

// 1 where aeris_gemm_auto takes the two-CTA kernel, else 0; the second for weight gradients that ask for slices
// (k_splits < 0) on a device of `sms` multiprocessors.
int aeris_gemm_takes_pairs(int M, int N, int K, int epi, int allow_2cta);
int aeris_wgrad_takes_pairs(int M, int N, int K, int k_splits, int sms);

int aeris_attn_fwd(const void* q, int ldq, int q_col0, const void* k, int ldk, int k_col0, const void* v, int ldv,
                   int v_col0, void* o, int ldo, float* lse, int n_win, int N, int H, int head_dim, float scale,
                   int* status, void* stream);

int aeris_attn_bwd(const void* qkv, int ldq, int q_col0, int k_col0, int v_col0, const void* o, const void* d_o,
                   int ldo, const float* lse, float* delta, void* dqkv, int ldg, int n_win, int N, int H,
                   int head_dim, float scale, int* status, void* stream);
// 1 where aeris_attn_bwd takes these extents on a device of `sms` multiprocessors, 0 where it returns -23.
int aeris_attn_bwd_countable(int n_win, int N, int H, int head_dim, int sms);

int aeris_gemm_scatter_heads(const void* A, const void* B, int M, int N, int K, int lda, int ldb, int b_mn,
                             const void* const* peers, int sp, int sp_rank, int n_local, int L, int sec_w, int* status,
                             void* stream);
// Variant of the attention forward kernel: poly = softmax arithmetic at head_dim 64 (-1 scalar; 0 two-wide; 2 two-wide
// with two of every eight score pairs on the polynomial exp2); p_in_tmem = probabilities kept in tensor memory as the
// A operand of P V. Returns non-zero for an unknown variant.
int aeris_attn_set_fwd_variant(int poly, int p_in_tmem);
// Checking build (-DAERIS_BOUNDS_CHECK) only: status word and source rows for the gathers launched next; returns 1 when
// the library validates gather codes, 0 when it was built without the checks.
int aeris_debug_set_gather_bounds(int* status, unsigned src_rows);
int aeris_attn_fwd_push(const void* qkv, int ld, int H_local, void* o, int ldo, float* lse, int n_win, int N,
                        int head_dim, float scale, const void* const* o_peers, int sp, int n_local, int push_ld,
                        int push_col0, int* status, void* stream);
int aeris_attn_bwd_push(const void* qkv, int ld, int H_local, const void* o, const void* d_o, int ldo, const float* lse,
                        float* delta, int n_win, int N, int head_dim, float scale, const void* const* dq_peers, int sp,
                        int n_local, int push_ld, int push_sec_w, int push_col0, int* status, void* stream);

// `w` is the bf16 norm weight, or null with the fp32 weight in `w_f32`; `h_lo` (optional) receives the bf16 rounding
// residual of `h`, so that h + h_lo carries the fp32 result (used by the fp32 output head).
int aeris_modnorm_fwd(const void* x, const void* gidx, const void* const* peer_ptrs, int n_peers, void* x_out,
                      const float* scale, const float* shift, const void* w, void* h, int rows, int D, int mode,
                      float eps, const float* w_f32, void* h_lo, void* stream);
// mod_stride: elements from one sample's scale (shift) to the next, a multiple of 4
int aeris_modnorm_fwd_batch(const void* x, const void* gidx, const void* const* peer_ptrs, int n_peers, void* x_out,
                            const float* scale, const float* shift, int mod_stride, const void* w, void* h, int batch,
                            int rows, int D, int mode, float eps, const float* w_f32, void* h_lo, void* stream);
int aeris_modnorm_bwd(const void* x, const void* dh, const void* dres, const float* scale, const float* shift,
                      const void* w, void* dx, float* dscale, float* dshift, float* dw, int rows, int D, int mode,
                      float eps, const float* w_f32, void* stream);
int aeris_modnorm_fwd_f32(const void* x, const float* scale, const float* shift, const float* w_f32, float* h, int batch,
                          int rows, int D, int mode, float eps, void* stream);
int aeris_modnorm_bwd_f32(const void* x, const float* dh, const float* scale, const float* shift, const float* w_f32,
                          void* dx, float* dscale, float* dshift, float* dw, float* sums, int sum_rows, int rows, int D,
                          int mode, float eps, void* stream);
int aeris_gather_rows(const void* gidx, const void* const* peer_ptrs, int n_peers, void* out, long long rows, int D,
                      void* stream);
int aeris_swiglu_fwd(const void* u, void* act, long long rows, int F, void* stream);
int aeris_swiglu_bwd(const void* u, const void* dact, void* du, long long rows, int F, void* stream);
int aeris_scale_rows(const void* W, const float* g, void* Wg, int R, int C, void* stream);
// In-place 2-D rotary embedding of the q and k sections of qkv [rows, 3 * heads * d] (bf16); cos / sin: [L, d / 2] fp32.
int aeris_rope_qk(void* qkv, const float* cos_t, const float* sin_t, long long rows, int L, int heads, int d, int inverse,
                  void* stream);
int aeris_gate_grad_finalize(float* G, const void* W, const float* g, float* dW, float* dg, int R, int C,
                             void* stream);
int aeris_gate_prepare(const void* W2, const float* g2, void* W2g, float* G2, int C2, const void* Wo, const float* go,
                       void* Wog, float* Go, int Co, int R, float* zero, int n_zero, void* stream);
int aeris_gate_finalize_pair(float* G2, const void* W2, const float* g2, float* dW2, float* dg2, int C2, float* Go,
                             const void* Wo, const float* go, float* dWo, float* dgo, int Co, int R, void* stream);
int aeris_sumsq(const float* x, long long n, double* out, void* stream);
int aeris_adamw(float* master, float* grad, float* m, float* v, void* wbf16, float* ema, const double* norm_sq,
                long long n, float lr, float beta1, float beta2, float eps, float weight_decay, int step,
                float grad_scale, float max_norm, float ema_beta, void* stream);

int aeris_signal_barrier(const void* const* flag_ptrs, int rank, int world, unsigned epoch, int* status,
                         double timeout_s, void* stream);
int aeris_wait_flag(const void* flag, unsigned expected, int* status, double timeout_s, void* stream);
int aeris_grad_reduce_scatter(const void* const* grad_ptrs, const void* mc_grad, int world, long long lo, long long n,
                              float scale, float* out, double* sumsq, void* stream);
int aeris_shard_adamw_allgather(float* master, const float* grad, float* m, float* v, float* ema,
                                const void* const* param_ptrs, void* mc_params, int world, long long lo, long long n,
                                const double* norm_sq, float lr, float beta1, float beta2, float eps,
                                float weight_decay, int step, float max_norm, float ema_beta, void* stream);

int aeris_gemm_allgather_a(void* A, const void* const* peers, const void* const* counter_peers, int world, int rank,
                           int rows_per_rank, unsigned call_index, const void* B, void* C, int N, int K, int ldb,
                           int ldc, int b_mn, int epi, const void* resid, int ldr, void* aux, int ld_aux, int swiglu_f,
                           int* status, void* stream);
int aeris_gemm_rs_push(const void* A, const void* B, int M, int N, int K, int lda, int ldb, int b_mn,
                       const void* const* peers, int world, int rank, int rows_per_rank, int ld_dst, int* status,
                       void* stream);
int aeris_rs_finalize(const void* slots, int world, long long rows, int D, const void* resid, const float* gate,
                      void* out, void* stream);

// Geometry of one rank's token stream and image block (see csrc/diffusion.cu).
typedef struct TokGeom {
  int B, nwy_loc, nwx_loc, ws_y, ws_x, n_local, sp_rank;
  int y0, x0, H, W;
  long long sample0;
} TokGeom;
int aeris_embed_pack(const float* x_img, const float* c_img, const float* cs, const TokGeom* g, int Cx, int Cc,
                     const float* ape_y, const float* ape_x, int ape_ch, unsigned long long seed, float sd, int noise,
                     void* out, int KP, long long row0, long long rows, void* stream);
int aeris_trigflow_loss(const float* pred, int ldp, const float* x_img, const float* cs, const TokGeom* g, int Cx,
                        unsigned long long seed, float sd, const float* w_var, const float* w_lat, float inv_rows,
                        float gscale, void* dpred, int ldd, double* loss, long long row0, long long rows, void* stream);
int aeris_sampler_update(float* x_out, const float* x_base, const float* pa, const float* pb, int ldp, float ca,
                         float cb, const TokGeom* g, int Cx, void* stream);
int aeris_noise_mix(float* x, float a, float b, unsigned long long seed, const TokGeom* g, int Cx, void* stream);
int aeris_affine_channels(float* out, const float* in, const float* a, const float* b, const float* add, long long n,
                          int C, void* stream);
int aeris_gemv_bias_act(const void* W, int flags, const void* bias, const void* x, float* y, int N, int K, int B, int act,
                        int silu_in, void* stream);
int aeris_modulation_mlp(const void* W1, int flags1, const void* b1, const void* x, float* y1, int N1, int K, const void* W2,
                         int flags2, const void* b2, float* y2, int N2, int B, void* stream);
// Gradients of aeris_gemv_bias_act without `act`; added to dW, db (may be null) and dx (may be null).
int aeris_gemv_bwd(const void* W, int flags, const void* x, const float* dy, float* dW, float* db, float* dx, int N, int K,
                   int B, int silu_in, void* stream);
int aeris_modulation_mlp_bwd(const void* W1, int flags1, const void* x, float* dW1, float* db1, float* dx, int N1, int K,
                             const void* W2, int flags2, const float* y1, const float* dy, float* dW2, float* db2,
                             float* dy1, int N2, int B, void* stream);
int aeris_noise_embedding(const float* t, void* out, int out_bf16, int B, int dim, double max_period, void* stream);
// The same of 1 to 64 levels that the host knows (no copy: they travel as kernel arguments).
int aeris_noise_embedding_of(const float* levels, void* out, int out_bf16, int n, int dim, double max_period, void* stream);
int aeris_pack_embed_weights(const float* W, const float* b, void* out, int D, int Cin, int KP, void* stream);
int aeris_fold_embed_grad(const float* G, float* dW, float* db, int D, int Cin, int KP, void* stream);
int aeris_pack_head_weights(const float* W, void* out, int C, int rows, int D, void* stream);
// Slices that k_splits <= 0 stands for: `tiles` output tiles over `units` CTAs or CTA pairs (see gemm.cu).
int aeris_choose_k_splits(int tiles, int kb_total, int units, int most, int want);
int aeris_gemm_split(const void* y, const void* w, float* C, int M, int D, int lo_row, int ldc, int* status, void* stream);

// One transformer block on one GPU (csrc/block.cu; mirrored in models/block.py). Every matrix is row-major without gaps.
typedef struct AerisBlock {
  int D, F, heads, head_dim, L, mode;
  int n_win, batch;                 // windows of one sample, samples
  int step, merged;                 // windows per chunk; merged: all samples are one chunk (forward)
  int slice_windows;                // weight gradients: slices of a quarter of that many windows' rows at most, if free
  int kept, two_cta, n_peers;       // kept: the internals are full-size buffers, not workspaces of one chunk
  float eps, scale;
  long long mod_vec, mod_sample;    // element strides of `mod`: between the six vectors, between samples
  const float* mod;                 // shift1, scale1, gate1, shift2, scale2, gate2
  const void *wn1, *wqkv, *wo, *wn2, *w1, *w2;
  const float *rope_cos, *rope_sin; // null: no rotary embedding
  void *x, *y;                      // block input (with `table`: receives the gathered rows) and output
  const unsigned* table;            // null, or gather codes of the rows of x
  const void* const* peers;
  void *h1, *qkv, *o, *lse, *x1, *h2, *act, *u;
  int* status;
  void* stream;
} AerisBlock;
typedef struct AerisBlockGrad {
  const void* dy;
  void *dx, *du, *dh, *dx1, *d_o, *dqkv, *w2g, *wog;
  float *delta, *G2, *Go, *dmod;    // dmod: [batch, 6 D], overwritten
  float *n1, *to_qkv, *wo, *n2, *w1, *w2;   // weight gradients, added to
} AerisBlockGrad;
// Both return the number of kernels launched, or a negative code: -1 where `step` is not positive, else that of the launch
// that failed less 1000 times its place.
int aeris_block_forward(const AerisBlock* b);
int aeris_block_backward(const AerisBlock* b, const AerisBlockGrad* g);
// aeris_block_forward of `n` records in a row, each with `mod + mod_offset` and on `stream`; same result codes.
int aeris_blocks_forward(const AerisBlock* blocks, int n, long long mod_offset, void* stream);

#ifdef __cplusplus
}
#endif
