// Prototypes of the kernel launchers (extern "C", one per kernel family), generated by gen_protos.py.
// Every launcher enqueues on the given stream, allocates nothing and returns 0 on success, -1 for
// unsupported shapes and -2 for a launch error.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

extern "C" {

// bench_kernels.cu
int qwk_bench_chain(float *p, int n, int blocks, int pdl, cudaStream_t s);

// gdn.cu
int qwk_gdn_conv(const float *proj, int ld_proj, float *ring, const float *cw, const float *A_log, const float *dt_bias, int KL, int VL, int M, const int *slot, const int *pos, const int *run_start, const int *run_len, float *qkv, float *decay, float *beta, float eps, cudaStream_t s);
int qwk_gdn_scan(const float *qkv, const float *decay, const float *beta, const float *proj, int ld_proj, float *S, float *save, const float *norm_w, int KL, int VL, int M, const int *slot, const int *pos, const int *run_start, const int *run_len, void *o, float eps, cudaStream_t s);
int qwk_gdn_step(const float *proj, int ld_proj, float *ring, const float *cw, const float *A_log, const float *dt_bias, const float *norm_w, int KL, int VL, int M, const int *slot, const int *pos, const int *run_start, const int *run_len, float *S, float *save, float *qkv, float *decay, float *beta, void *o, float eps, cudaStream_t s);
int qwk_gdn_accept(const void *S_ptrs, const float *save, int n_layers, int max_rows, long long state, const int *pairs, int n_pairs, cudaStream_t s);

// gdn_chunk.cu
int qwk_gdn_scan_chunked(const float *qkv, const float *decay, const float *beta, const float *proj, int ld_proj, float *S, const float *norm_w, int KL, int VL, int M, const int *slot, float *scratch, void *o, float eps, cudaStream_t s);

// gemm_tc.cu
int qwk_gemm_tc_wide_min_n(int min_n);
int qwk_gemm_tc_stage_local(int on);
int qwk_gemm_tc_pair_min_n(int min_n);
int qwk_gemm_tc_exchange_nt(int nt);
int qwk_gemm_tc_exchanged(int T, int N, int K);
int qwk_gemm_tc_form(int T, int N, int K);
int qwk_gemm_bf16_tc(const void *A, const void *W, void *C, int T, int N, int K, int lda, int ldw, int ldc, int out_bf16, cudaStream_t s);
int qwk_gemm_bf16_tc_tp(void *tp_, const void *A, const void *W, void *C, int T, int N, int K, int lda, int ldw, int ldc, int out_bf16, int wait_kind, int epi_mode, int epi_kind, int ld_epi, cudaStream_t s);
int qwk_gemm_mix_tc(const void *A, const void *W, const void *xn, int SH, void *out, int ld_out, int T, int K, int lda, int ldw, cudaStream_t s);
int qwk_gemm_bf16_tc_grouped(const void *A, const void *W, void *C, const void *tiles, int max_tiles, int rows, long long w_rows, int Nw, int K, int lda, int ldw, int ldc, int out_bf16, cudaStream_t s);
int qwk_gemm_bf16_tc_splitk(const void *A, const void *W, float *C, int T, int N, int K, int lda, int ldw, int ldc, int ksplit, long long c_split, cudaStream_t s);

// gemv.cu
int qwk_gemv_bf16(const void *W, const void *x, float *y, void *y_bf16, int N, int K, int M, int ldw, int ldx, int ldy, int accumulate, int nsplit, long long w_split, long long x_split, long long y_split, cudaStream_t s);

// hc.cu
int qwk_embed_rows(const int *tokens, const void *table, int ld_table, int col0, int SH, int hc, int vocab, float *X, int M, cudaStream_t s);
int qwk_hc_pre(float *X, const float *pend, int ld_pend, const float *inj, int ld_inj, const float *w1, int SH, int hc, void *y, float *ssq, int ld_ssq, int M, cudaStream_t s);
int qwk_hc_up_mix(const float *red, int ld_red, const void *Wu, const float *X, const float *w1, int SH, int hc, int R, int n_inj, int H, float eps, int M, float *inj, int ld_inj, void *bin, int ld_bin, int bin_col0, cudaStream_t s);
int qwk_hc_down(const float *Xin, float *Xout, const float *pend, int ld_pend, const float *inj_prev, const float *w1, const void *Wd, float *send, int ld_send, int SH, int hc, int down, int M, cudaStream_t s);

// host_tier.cu
int qwk_segments_copy(const void *src, const void *dst, const long long *bytes, int n, cudaStream_t s);
int qwk_memcpy_async(void *dst, const void *src, long long bytes, int kind, cudaStream_t s);

// logits.cu
int qwk_amax_pack(const float *val, const int *idx, float *pairs, int M, int rank, int ranks, cudaStream_t s);
int qwk_amax_merge(const float *pairs, int M, int ranks, int *out_idx, float *out_val, cudaStream_t s);
int qwk_advance_rows(int *tokens, int *pos, int *ctx3, const int *next, int M, cudaStream_t s);
int qwk_row_reduce(const float *logits, int ld, int V, int idx0, int M, float *out_val, int *out_idx, float *out_max, float *out_sum, cudaStream_t s);
int qwk_merge_argmax(const float *vals, const int *idx, int ranks, int M, int stride, int *out_idx, float *out_val, cudaStream_t s);

// moe.cu
int qwk_set_moe_mma(int mask);
int qwk_moe_router(const void *Wrs, const void *x, float *rs, int nrs, int K, int M, int ldx, int E, int top_k, int F, int e_first, int e_local, int *pair_expert, float *pair_w, void *sh_h, unsigned int *ticket, const void *w13, const void *w2, long long w13_bytes, long long w2_bytes, cudaStream_t s);
int qwk_moe_route(const float *rs, int ld_rs, int M, int E, int top_k, int F, int e_first, int e_local, int *pair_expert, float *pair_w, void *sh_h, cudaStream_t s);
int qwk_moe_gate_up_pair(const void *w13, const void *s13, const void *x, int ldx, const int *pair_expert, int M, int top_k, int F, int K, void *h, cudaStream_t s);
int qwk_moe_down_combine(const void *w2, const void *s2, const void *h, const int *pair_expert, const float *pair_w, int M, int top_k, int F, int H, const void *shared_down, int ld_sd, const void *sh_h, int SF, float *out, int ldo, cudaStream_t s);

// moe_tc.cu
int qwk_gemm_q4_tc_grouped(const void *A, const void *Wq, const void *scale, void *C, const void *tiles, int max_tiles, int rows, long long w_rows, int Nw, int K, int lda, int ldc, int out_bf16, cudaStream_t s);
int qwk_gemm_q4_tc_swiglu(const void *A, const void *Wq, const void *scale, void *C, const void *tiles, int max_tiles, int rows, long long w_rows, int F, int K, int lda, int ldc, cudaStream_t s);

// mtp.cu
int qwk_mtp_norm(const float *hidden, const int *tokens, const void *embed, int vocab, const float *nh1, const float *ne1, int H, int hc, float eps, void *hn, void *en, int M, cudaStream_t s);
int qwk_mtp_add(const float *fh, const float *fe, int H, int hc, float *X, int M, cudaStream_t s);

// p2p.cu
int qwk_p2p_allreduce(const void *p2p, unsigned int k, const float *src, float *dst, int rows, int n, cudaStream_t s);
int qwk_p2p_reduce_scatter(const void *p2p, unsigned int k, const float *src, float *dst, int rows, int n, cudaStream_t s);
int qwk_p2p_allgather(const void *p2p, unsigned int k, int kind, long long off, int rows, int n, int elem, cudaStream_t s);
int qwk_fuse_next(const void *p2p, int in_kind, unsigned int in_k, int in_n, int out_kind, unsigned int out_k, int out_mode, int out_n);
int qwk_p2p_bump_base(const void *p2p, unsigned int by, cudaStream_t s);

// ple.cu
int qwk_ple_init(const unsigned long long *mult, int ngram, const unsigned long long *sizes, const long long *offsets, int heads, int eos, const float *f8_lut);
int qwk_ple_gather(const int *ctx, const void *const *shards, const void *const *scales, long long rows_per_shard, long long rows, int layout, int width, int heads, void *e, long long *ids_out, int M, cudaStream_t s);
int qwk_ple_stats(const float *kv, int ld_kv, const float *X, const float *nk1, const float *nq1, int SH, int hc, float *send, int ld_send, int M, cudaStream_t s);
int qwk_ple_apply(const float *kv, int ld_kv, const float *red, int ld_red, const float *nc1, const float *cw, int SH, int hc, int H, float eps, int taps, int dil, float *gv, float *nc, float *ring, float *X, int M, const int *slot, const int *pos, const int *run_start, const int *run_len, cudaStream_t s);

// prefill.cu
int qwk_hc_prenorm_T(float *X, const float *pend, int ld_pend, const float *inj, const float *w1, int SH, int hc, float eps, void *xn, int T, cudaStream_t s);
int qwk_hc_mid_T(const float *d, int ld_d, int R, int n_inj, int hc, void *u, float *inj, int T, int nsplit, long long split_stride, cudaStream_t s);
int qwk_q4_dequant(const void *w, const void *scale, long long rows, int K, void *out, cudaStream_t s);
int qwk_swiglu_T(const void *h13, int F, void *h, long long P, cudaStream_t s);
int qwk_moe_combine_T(const float *y, int ld_y, const int *inv, const float *pair_w, int top_k, const float *shared, int H, float *out, int T, cudaStream_t s);
int qwk_moe_sort_T(const int *pair_expert, int T, int top_k, int E, int Nw13, int Nw2, int max_tiles, int *inv, int *src_token, void *t13, void *t2, const void *x, int ldx, int H, void *xperm, cudaStream_t s);

// prefill_tp.cu
int qwk_hc_prenorm_tp(void *tp_, float *X, const float *pend_local, int ld_pend, int pend_kind, const float *inj, int SH, int hc, int T, cudaStream_t s);
int qwk_hc_norm_tp(void *tp_, const float *X, const float *w1, int SH, int hc, int H, float eps, void *xn, int T, cudaStream_t s);
int qwk_hc_mid_tp(void *tp_, int ld_d, int R, int n_inj, int hc, void *u, float *inj, int T, cudaStream_t s);
int qwk_hc_mix_tp(void *tp_, const float *g, const void *xn, int SH, int ld_bin, int T, cudaStream_t s);
int qwk_moe_combine_tp(void *tp_, const float *y, int ld_y, const int *inv, const float *pair_w, int top_k, const float *shared, int H, int T, cudaStream_t s);
int qwk_tp_push(void *tp_, int kind, const void *src, long long src_stride, int rows, int row_bytes, int mode, cudaStream_t s);
int qwk_tp_allreduce(void *tp_, int kind, const float *src, float *dst, int rows, int n, cudaStream_t s);
int qwk_tp_reduce_scatter(void *tp_, int kind, const float *src, float *dst, int rows, int n, cudaStream_t s);
int qwk_tp_allgather(void *tp_, int kind, const void *src, long long src_stride, int rows, int row_bytes, int wait, cudaStream_t s);
int qwk_tp_wait(void *tp_, int kind, cudaStream_t s);
int qwk_tp_reduce(void *tp_, int kind, float *dst, long long n, cudaStream_t s);
int qwk_copy_rows(const float *src, long long ld_src, float *dst, int n, int M, cudaStream_t s);
int qwk_embed_override(float *X, const int *rows_i, const float *emb, int ld_emb, int col0, int SH, int hc, int n, cudaStream_t s);
int qwk_mtp_ssq(const float *hidden, int n, float *ssq, int M, cudaStream_t s);
int qwk_mtp_norm_tp(void *tp_, const float *hidden, const float *ssq, const int *tokens, const void *embed, int vocab, const float *nh1, const float *ne1, int H, int hc, float eps, void *en, int M, cudaStream_t s);
int qwk_tp_argmax_send(void *tp_, const float *val, const int *idx, void *scratch16, int M, cudaStream_t s);
int qwk_tp_argmax_merge(void *tp_, int M, int *out_idx, float *out_val, cudaStream_t s);

// qsa.cu
int qwk_rope_init(double theta, int rope_dim);
int qwk_qsa_prep(const float *proj, int ld_proj, int QL, int KVL, int IH, const float *qn1, const float *kn1, const float *iqn1, const float *ikn1, int M, const int *slot, const int *pos, const int *run_start, const int *run_len, void *k_dev, void *v_dev, void *k_host, void *v_host, int n_dev_pages, const int *page_table, int max_pages, float *q, float *iq, float *raw_ring, void *ck, int ck_cap, int ratio, float eps, cudaStream_t s);
int qwk_qsa_prep_run(const float *proj, int ld_proj, int QL, int KVL, int IH, const float *qn1, const float *kn1, const float *iqn1, const float *ikn1, int M, const int *slot, const int *pos, const int *run_start, const int *run_len, void *k_dev, void *v_dev, void *k_host, void *v_host, int n_dev_pages, const int *page_table, int max_pages, float *q, float *iq, float *raw_ring, void *ck, int ck_cap, int ratio, float eps, cudaStream_t s);
int qwk_qsa_scores(const float *iq, int IH, const void *ck, int ck_cap, int M, const int *slot, const int *pos, int ratio, int topk_blocks, float *scores, int ld_scores, int max_groups, cudaStream_t s);
int qwk_qsa_select(const float *scores, int ld_scores, int M, const int *pos, int ratio, int topk, int *sel, int *sel_n, cudaStream_t s);
int qwk_qsa_attend(const float *q, int QL, int KVL, int M, const int *slot, const int *pos, void *k_dev, void *v_dev, void *k_host, void *v_host, int n_dev_pages, const int *page_table, int max_pages, const int *sel, const int *sel_n, int topk, int ratio, int nsplit, float *pm, float *pl, float *pacc, const float *proj, int ld_proj, void *o, cudaStream_t s);
int qwk_qsa_attend_mma(const float *q, int QL, int KVL, int M, const int *slot, const int *pos, void *k_dev, void *v_dev, void *k_host, void *v_host, int n_dev_pages, const int *page_table, int max_pages, const int *sel, const int *sel_n, int topk, int ratio, const float *proj, int ld_proj, void *o, cudaStream_t s);
int qwk_qsa_attend_mma_staged(const float *q, int QL, int KVL, int M, const int *slot, const int *pos, void *k_dev, void *v_dev, void *k_host, void *v_host, int n_dev_pages, const int *page_table, int max_pages, const int *sel, const int *sel_n, int topk, int ratio, const float *proj, int ld_proj, void *o, cudaStream_t s);
int qwk_set_spill_cache(void *tags, void *rows, void *miss, void *ctl, void *stats, int entries, int miss_cap);
int qwk_spill_cache_active(int unused);

// qsa_tc.cu
int qwk_qsa_takes_tc(int QL, int KVL, int M, int last_pos, int topk, int ratio, int ld_mask, int ld_proj);
int qwk_qsa_attend_tc(const float *q, int QL, int KVL, int M, int last_pos, const int *slot, const int *pos, void *k_dev, void *v_dev, void *k_host, void *v_host, int staged, int n_dev_pages, const int *page_table, int max_pages, const int *sel, const int *sel_n, int topk, void *mask, int ld_mask, const float *proj, int ld_proj, void *o, cudaStream_t s);

// sampling.cu
int qwk_sample(const float *logits, int ld, int V, int M, const void *params, const void *gen, const void *seen, void *out, cudaStream_t s);
int qwk_penalty_add(void *gen, void *seen, int V, const int *slots, const int *tokens, const int *generated, int n, cudaStream_t s);

// vision.cu
int qwk_vit_embed(float *x, const float *y, const float *bias, const float *table, const int *idx, const float *wts, int L, int D, cudaStream_t s);
int qwk_vit_layernorm(float *x, const float *y, const float *ybias, const float *w, const float *b, int L, int D, float eps, void *out, cudaStream_t s);
int qwk_vit_rope_table(const int *pos_hw, int L, float *tab, cudaStream_t s);
int qwk_vit_bias_rope(void *qkv, const float *bias, const float *tab, int L, int heads, cudaStream_t s);
int qwk_vit_bias_gelu(void *y, const float *bias, int L, int D, int tanh_form, cudaStream_t s);
int qwk_vit_residual_add(float *x, const float *y, const float *bias, int L, int D, int assign, cudaStream_t s);

// vit_attn.cu
int qwk_vit_attention_scratch(int L, int heads);
int qwk_vit_attention_split(const void *qkv, int L, int heads, void *out, void *parts, cudaStream_t s);
int qwk_vit_attention(const void *qkv, int L, int heads, void *out, cudaStream_t s);

}  // extern "C"
