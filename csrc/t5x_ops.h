/* Entry points that the compiled host path (host/host_ops.cpp) calls beside those of t5x_b200.h. The
 * sources that define them include this file too, so that a changed argument list does not
 * compile on one side only. */
#ifndef T5X_OPS_H_
#define T5X_OPS_H_

#ifdef __cplusplus
extern "C" {
#endif

int t5x_rmsnorm_fwd(const void* x, const void* scale, void* y, void* rstd, int rows, int d, float eps,
                    void* stream);
long long t5x_rmsnorm_bwd_partial(int rows, int d);
int t5x_rmsnorm_bwd(const void* dy, const void* x, const void* scale, const void* rstd,
                    const void* dres, void* dx, void* dscale, void* partial, int rows, int d,
                    void* stream);
int t5x_attention_fwd(const void* q, const void* k, const void* v, void* o, void* lse, int B, int H,
                      int Lq, int Lk, long long q_sb, long long q_sl, long long q_sh, long long k_sb,
                      long long k_sl, long long k_sh, long long v_sb, long long v_sl, long long v_sh,
                      long long o_sb, long long o_sl, long long o_sh, const void* rel_bias,
                      const void* rel_bucket, int num_buckets, int nrel, int rel_off,
                      const void* key_mask, const void* q_seg, const void* kv_seg, int causal,
                      int causal_off, void* stream);
int t5x_attention_fwd_few(const void* q, const void* k, const void* v, void* o, void* lse, int B, int H,
                          int Lq, int Lk, long long q_sb, long long q_sl, long long q_sh, long long k_sb,
                          long long k_sl, long long k_sh, long long v_sb, long long v_sl, long long v_sh,
                          long long o_sb, long long o_sl, long long o_sh, const void* rel_bias,
                          const void* rel_bucket, int num_buckets, int nrel, int rel_off,
                          const void* key_mask, const void* q_seg, const void* kv_seg, int causal,
                          int causal_off, void* stream);
int t5x_attention_fwd_stream(const void* q, const void* k, const void* v, void* o, void* lse, int B,
                             int H, int Lq, int Lk, int D, long long q_sb, long long q_sl,
                             long long q_sh, long long k_sb, long long k_sl, long long k_sh,
                             long long v_sb, long long v_sl, long long v_sh, long long o_sb,
                             long long o_sl, long long o_sh, const void* rel_bias,
                             const void* rel_bucket, int num_buckets, int nrel, int rel_off,
                             const void* key_mask, const void* q_seg, const void* kv_seg, int causal,
                             int causal_off, void* stream);
int t5x_attention_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                      const void* lse, void* delta, void* dq_f32, void* dk, void* dv, int B, int H,
                      int Lq, int Lk, int D, long long q_sb, long long q_sl, long long q_sh,
                      long long k_sb, long long k_sl, long long k_sh, long long v_sb, long long v_sl,
                      long long v_sh, long long o_sb, long long o_sl, long long o_sh, long long do_sb,
                      long long do_sl, long long do_sh, long long dk_sb, long long dk_sl,
                      long long dk_sh, const void* rel_bias, const void* rel_bucket, void* d_rel_bias,
                      int num_buckets, int nrel, int rel_off, const void* key_mask, const void* q_seg,
                      const void* kv_seg, int causal, int causal_off, void* stream);
int t5x_attention_bwd_head_covers(int B, int H, int Lq, int Lk, int D, int num_buckets);
int t5x_attention_bwd_head(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                           const void* lse, void* dq, void* dk, void* dv, void* dk32, void* dv32, int B,
                           int H, int Lq, int Lk, long long q_sb, long long q_sl, long long q_sh,
                           long long k_sb, long long k_sl, long long k_sh, long long v_sb, long long v_sl,
                           long long v_sh, long long o_sb, long long o_sl, long long o_sh, long long do_sb,
                           long long do_sl, long long do_sh, long long dq_sb, long long dq_sl, long long dq_sh,
                           long long dk_sb, long long dk_sl, long long dk_sh, const void* rel_bias,
                           const void* rel_bucket, void* d_rel_bias, int num_buckets, int nrel,
                           int rel_off, const void* key_mask, const void* q_seg, const void* kv_seg,
                           int causal, int causal_off, void* stream);
int t5x_gemm_gated_grad_covers(int M, int N);
int t5x_gemm_relu_covers(int M, int N);
int t5x_gemm_relu(const void* A, const void* B, void* C, const void* positive, int M, int N, int K, long long lda,
                  long long ldb, long long ldc, long long ldp, int b_mn_major, void* stream);
int t5x_gemm_gated_grad(const void* dy, const void* B, void* h0, void* h1, int M, int N, int K, long long ld_dy,
                        long long ldb, long long ldh, int b_mn_major, void* stream);
int t5x_gated_gelu_bwd(void* dg, void* h, long long rows, int dff, long long ldh, long long ldg,
                       int write_g, void* stream);

#ifdef __cplusplus
}
#endif
#endif /* T5X_OPS_H_ */
