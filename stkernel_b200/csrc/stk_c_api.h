// C entry points of libstk_b200.so -- generated by `python -m stkernel_b200.csrc.gen_c_api`, do not edit.
// Every function returns 0 on success (or the queried value for the few `long long` / query functions) and a
// negative code when it rejects its arguments; tensors are raw device pointers, `stream` is a cudaStream_t.
#pragma once
#include <stdint.h>
#ifdef __cplusplus
extern "C" {
#endif

// ---- attention.cu ----
long long stk_sparse_mla_workspace_bytes(int T, int nh, int D, int n_splits);
int stk_sparse_mla_pick_splits(int T, int max_rows);
int stk_sparse_mla(const void* q, long long ldt, const void* swa_cache, long long swa_stride, int swa_data_bytes, const void* comp_cache, long long comp_stride, int comp_data_bytes, int fp8, const int* swa_slots, int swa_ld, const int* swa_lens, const int* topk_slots, int topk_ld, const int* topk_lens, const float* sink, void* out, long long ldo, float* workspace, int n_splits, int T, int nh, int D, int R, int max_rows, float scale, void* stream);
int stk_sparse_mla_combine(const float* workspace, const float* sink, void* out, long long ldo, int T, int nh, int D, int n_splits, const int64_t* positions, const float* inv_freq, int R, void* stream);

// ---- attention_tc.cu ----
int stk_sparse_mla_tc(const void* q, long long ldt, const void* swa_cache, long long swa_stride, const void* comp_cache, long long comp_stride, const int* swa_slots, int swa_ld, const int* swa_lens, const int* topk_slots, int topk_ld, const int* topk_lens, float* workspace, int n_splits, int T, int nh, int D, int R, int max_rows, float scale, int* status, void* trace, void* stream);
int stk_sparse_mla_tc_out(const void* q, long long ldt, const void* swa_cache, long long swa_stride, const void* comp_cache, long long comp_stride, const int* swa_slots, int swa_ld, const int* swa_lens, const int* topk_slots, int topk_ld, const int* topk_lens, int T, int nh, int D, int R, int max_rows, float scale, void* out, long long ldo, const float* sink, const int64_t* positions, const float* inv_freq, int* status, void* stream);

// ---- elementwise.cu ----
int stk_pdl_enabled(void);
int stk_pdl_eager(void);
int stk_set_pdl_mask(int mask);
int stk_set_pdl(int on);
int stk_embed_hc(const int64_t* ids, const void* embed, void* out, int T, int H, int hc, int vocab, int vocab_start, int vocab_end, int* status, void* stream);
int stk_rmsnorm(const void* x0, long long ldx0, const void* w0, void* out0, long long ldo0, int H0, void* q0, long long ldq0, float* qs0, int qs_ld0, const void* x1, long long ldx1, const void* w1, void* out1, long long ldo1, int H1, int T, float eps, void* stream);
int stk_row_sumsq(const void* x, long long ldx, float* out, long long ldo, int T, int K, void* stream);
int stk_quant_fp8_group128(const void* x, long long ldx, void* q, long long ldq, float* scales, int scale_ld, int T, int K, void* stream);
int stk_swiglu_clamp(const void* gu, long long ldg, void* act, long long lda, int T, int I, float limit, void* q_out, long long ldq, float* q_scale, int q_scale_ld, void* stream);
int stk_moe_combine(const void* y, const float* w, const int* pair_row, const void* shared, void* out, int T, int H, int topk, const void* ll_ctx, void* stream);

// ---- ep_moe.cu ----
int stk_ep_ctx_size(void);
long long stk_ep_region_bytes(int world, int E, int e_local, int H, long long cap_rows, long long max_pairs);
int stk_ep_ctx_fill(void* ctx, const long long* bases, int rank, int world, int E, int topk, int H, long long cap_rows, long long max_pairs, int spin_budget);
long long stk_ep_ctx_offset(const void* ctx, int which);
int stk_ep_route(const void* ctx, const int* ids, int n_pairs, int* offsets_local, int* dest_base, int* cursor, int* status, void* stream);
int stk_ep_dispatch(const void* ctx, const void* x, long long ldx, const int* ids, int n_pairs, const int* dest_base, int* cursor, int* status, void* stream);
int stk_ep_return(const void* ctx, const void* y, const int* offsets_local, int max_rows, int* status, void* stream);
int stk_ep_combine(const void* ctx, const float* w, const int* ids, const void* shared, long long lds, void* out, long long ldo, int T, int* status, void* stream);

// ---- gate_cluster.cu ----
int stk_gate_route_cluster_ok(void);
int stk_gate_route_cluster(const void* W, long long ldw, const void* x, long long ldx, int T, int E, int K, const float* bias, const int* tid2eid, const int64_t* token_ids, int vocab, int* ids, float* weights, int topk, int always, int groups, int keep, int scoring, int renorm, float scaling, int* status, void* stream);

// ---- gemm_tcgen05.cu ----
int stk_gemm_pick_bt(int T, int is_fp8);
int stk_gemm_pick_splits(int T, int N, int K, int is_fp8, int sm_count);
long long stk_gemm_workspace_bytes(int T, int N, int splits);
int stk_gemm_plan(int T, int N, int K, int groups, int is_fp8, int sm_count);
int stk_gemm_token_tile_ctas(int T, int N, int K, int is_fp8, int sm_count);
int stk_gemm(const void* W, long long ldw, const void* X, long long ldx, void* out, long long ldo, int T, int N, int K, int is_fp8, int out_fp32, const float* w_scale, int w_scale_ld, const float* x_scale, int x_scale_ld, int splits, float* workspace, int* counters, int* status, int sm_count, int groups, const void* ar_ctx, void* stream);
int stk_gemm_tile(const void* W, long long ldw, const void* X, long long ldx, void* out, long long ldo, int T, int N, int K, int out_fp32, int bt, int splits, float* workspace, int* counters, int* status, int sm_count, void* stream);
int stk_gemm_gated(const void* W, long long ldw, const void* X, long long ldx, void* out, long long ldo, int T, int N, int K, int is_fp8, int out_fp32, const float* w_scale, int w_scale_ld, const float* x_scale, int x_scale_ld, int* status, int sm_count, const void* gate_ctx, int gate_rows, void* stream);
long long stk_gemm_noalloc_max_workspace_bytes(void);
int stk_gemm_noalloc_reset(void* stream);
int stk_gemm_noalloc(const void* W, long long ldw, const void* X, long long ldx, void* out, long long ldo, int T, int N, int K, int is_fp8, int out_fp32, const float* w_scale, int w_scale_ld, const float* x_scale, int x_scale_ld, int splits, int* status, int sm_count, void* stream);

// ---- grouped_attention.cu ----
int stk_grouped_prep(const void* proj, long long ldp, int q_off, int k_off, int v_off, const float* bias, int norm, float eps, float coef, float every, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, void* cache, int row, int k_col, int heads, int kv_heads, int dim, int vdim, void* q, int dp, int fp32, int T, void* stream);

// ---- hybrid_block.cu ----
int stk_xielu(const void* z, long long ldz, int ff, float a, float b, void* out, long long ldo, int width, int fp32, int T, void* stream);
int stk_embed_scaled(const int64_t* ids, const void* embed, int embed_fp32, float* x, long long ldx, int copies, int T, int W, int vocab, float scale, void* h, long long ldh, int width, int* status, void* stream);
int stk_add_layer_norm(float* x, long long ldx, const float* y, long long ldy, const float* w, void* h, int h_fp32, long long ldh, int T, int W, int width, float eps, const int64_t* rows, int center, void* stream);
int stk_join_glu(const void* proj, long long ldp, int gate_off, int up_off, int ff, void* out, long long ldo, int fp32, int mixer_dim, int ff_off, int cols, int relu, int T, void* stream);
int stk_post_norm_add(float* x, long long ldx, const float* y, long long ldy, const void* pairs, long long ldp, const int* pair_row, const float* weights, int top, const float* w, float eps, void* h, long long ldh, int W, int width, int fp32, int T, void* stream);
int stk_stream_norm(float* x, int streams, const float* y, long long ldy, const void* pairs, long long ldp, const int* pair_row, const float* weights, int top, const float* mix, const float* write, const float* read, const float* w, const float* b, float eps, void* h, long long ldh, int W, int width, int fp32, const int64_t* rows, int T, void* stream);

// ---- indexer.cu ----
int stk_indexer_scores(const void* q, const float* w, const void* kcache, long long page_stride, int k_fp8, const int* block_table, int bt_stride, const int* tok_req, const int* n_valid, float* scores, long long ld_scores, int T, int max_rows, int ih, int di, int q_fp8, void* stream);
int stk_topk_rows(const float* scores, long long ld, const int* n_valid, int* out, int out_ld, int T, int k, void* stream);
int stk_topk_to_slots(const int* topk, int k, int topk_ld, const int* block_table, int bt_stride, const int* tok_req, int* slots, int slots_ld, int* lens, int T, int max_rows, int* status, void* stream);

// ---- indexer_tc.cu ----
int stk_indexer_scores_tc(const void* q, const float* w, const void* kcache, long long page_stride, int n_pages, const int* block_table, int bt_stride, const int* tok_req, const int* n_valid, float* scores, long long ld_scores, int T, int max_rows, int ih, int di, int* status, void* stream);

// ---- kvcache.cu ----
int stk_q_norm_rope(void* q, long long ldt, const int64_t* positions, const float* inv_freq, int T, int nh, int D, int R, float eps, int do_norm, int inverse, void* stream);
int stk_kv_rope_quant_insert(const void* kv, long long ldk, const int64_t* positions, const int64_t* slots, const float* inv_freq, void* cache, long long page_stride, int data_bytes, int fp8, long long num_slots, int T, int D, int R, int* status, void* stream);
int stk_q_rope_kv_insert(void* q, long long ldt, int nh, float eps, const void* kv, long long ldk, const int64_t* positions, const int64_t* slots, const float* inv_freq, void* cache, long long page_stride, int data_bytes, int fp8, long long num_slots, int T, int D, int R, const void* kv_norm_w, int* status, void* stream);
int stk_kv_gather_dequant(const void* cache, long long page_stride, int data_bytes, int fp8, const int64_t* slots, void* out, int n, int D, int R, void* stream);
int stk_compress_windows(const float* kvs, long long kvs_ld, const float* ape, const void* norm_w, const float* inv_freq, const int64_t* positions, const int* tok_req, const int* tok_first_pos, const int* tok_last_pos, float* state, const int* block_table, int bt_stride, void* cache, long long page_stride, int data_bytes, int fp8, int idx_format, long long num_slots, int T, int D, int R, int ratio, int c, int ring, float eps, int* status, void* stream);
int stk_indexer_q_prep(const void* q, long long ldq, const float* w, long long ldw, const int64_t* positions, const float* inv_freq, void* q_out, float* w_out, int T, int ih, int d, int R, int quantize, void* stream);

// ---- latent_attention.cu ----
int stk_latent_prep(const float* p, long long ldp, int q_off, int kv_off, const float* wq, const float* wkv, float eps, int q_rank, int q_width, int kv_rank, int rot, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, void* cache, int row, int rot_off, const float* freq, void* cq, long long ldcq, int fp32, int T, void* stream);
int stk_latent_attention_simt(const void* qa, long long ldqa, int cp, const void* qr, long long ldqr, const float* gate, long long ldg, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, const void* cache, int row, int rot_off, const float* freq, int heads, int kv_rank, int rot, float scale, void* out, long long ldo, int fp32, const int* first_pos, const int* last_pos, int max_span, int T, void* stream);

// ---- latent_prompt_tc.cu ----
int stk_latent_prompt_ok(int dim, int dp, int rot, int vdim, int row, int rot_off);
int stk_latent_rows(const int* query_start, const int* req_rows, const int* start_pos, int n_req, int min_span, const int* table, int bt_stride, const void* cache, int heads, int row, void* out, long long rows, void* stream);
int stk_latent_prompt(const void* q, long long ldq, const void* qr, long long ldqr, const float* gate, long long ldg, const int* query_start, const int* start_pos, int n_req, int min_span, const void* rows, long long n_rows, int row, int rot_off, const void* kv, const float* freq, int heads, int h0, int nh, int dim, int dp, int rot, int vdim, int vp, float scale, void* out, long long ldo, int T, int* status, void* stream);
int stk_prompt_attention_ok(int dim, int dp, int vdim, int row, int k_col);
int stk_prompt_attention(const void* q, long long ldq, const int* query_start, const int* start_pos, int n_req, int min_span, const void* rows, long long n_rows, int row, int k_col, const void* gate, long long ldg, float out_scale, const float* sink, int heads, int kv_heads, int dim, int dp, int vdim, float scale, void* out, long long ldo, int T, int* status, void* stream);

// ---- latent_tokens_tc.cu ----
int stk_latent_tokens_columns(int heads, int kv_rank, int row, int max_span);
int stk_latent_tokens_splits(int T, int heads, int max_span, int context, int sm_count);
int stk_latent_tokens(const void* qa, long long ldqa, int cp, const void* qr, long long ldqr, const float* gate, long long ldg, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, const void* cache, int row, int rot_off, const float* freq, int heads, int kv_rank, int rot, float scale, void* out, long long ldo, const int* query_start, const int* req_rows, const int* start_pos, int n_req, const int* first_pos, const int* last_pos, int max_span, long long num_pages, int splits, float* part, int T, int* status, void* stream);

// ---- linear_f32.cu ----
int stk_linear_f32(const float* W, long long ldw, const float* x, long long ldx, float* out, long long ldo, int T, int N, int K, void* stream);

// ---- linear_scan.cu ----
long long stk_linear_state_slot(int dim, int vdim);
int stk_linear_chunks(const void* qh, const void* ql, const void* kh, const void* kl, long long ldqk, int step, int width, int hpg, const void* v, long long ldv, int v_off, const float* log_decay, const float* g, const float* w, const float* skip, const int* query_start, const int* req_rows, const int* start_pos, int n_req, float* S, float* o, int heads, int dim, int vdim, int min_span, float* states, int max_chunks, int T, void* stream);

// ---- mamba2.cu ----
int stk_mamba2_scan(const void* xbc, long long ld, const float* steps, const float* skip, const int* query_start, const int* req_rows, const int* start_pos, int n_req, float* S, float* o, int heads, int state, int vdim, int groups, int fp32, int min_span, int max_span, int T, void* stream);
int stk_mamba2_conv(const void* proj, long long ldp, int x_off, int dt_off, const float* taps, const float* conv_bias, int n_taps, const void* ring, const float* dt_bias, const float* neg_a, const int64_t* positions, const int* tok_req, const int* first_pos, void* out, long long ldo, float* steps, int heads, int channels, int fp32, int T, void* stream);
int stk_mamba2_finish(const float* o, const void* proj, long long ldp, int z_off, int x_off, int channels, const float* norm_w, float eps, int norm_groups, const int* tok_req, const int64_t* positions, const int* last_pos, void* ring, int n_taps, void* out, long long ldo, int cols, int fp32, int inner, int T, void* stream);

// ---- meta.cu ----
int stk_swa_indices(const int64_t* positions, const int* tok_req, const int* block_table, int bt_stride, int* slots, int ld, int* lens, int T, int window, void* stream);
int stk_swa_indices_noncausal(const int* tok_req, const int* prefix_len, const int* seq_len, const int* block_table, int bt_stride, int* slots, int ld, int* lens, int T, int window, void* stream);
int stk_compressed_valid(const int64_t* positions, int* n_valid, int T, int ratio, void* stream);
int stk_c128_indices(const int64_t* positions, const int* tok_req, const int* block_table, int bt_stride, int* slots, int ld, int* lens, int T, int ratio, int cap, void* stream);
int stk_token_maps(const int* query_start, const int* req_rows, const int* start_pos, int n_req, int* tok_req, int64_t* positions, int* first_pos, int* last_pos, const int* block_table, int bt_stride, int64_t* slot_mapping, int T_padded, void* stream);

// ---- mhc.cu ----
int stk_mhc_pick_splits(int T, int HC);
int stk_mhc_dots(const void* x, const float* fn, float* partial, int T, int H, int hc, int n_mix, int n_splits, void* stream);
int stk_mhc_finalize(const void* x, const float* partial, int n_splits, int partial_ld, int sumsq_in_partial, const float* base, const float* scale, const void* norm_w, float* post, float* comb, void* y, int T, int H, int hc, float rms_eps, float hc_eps, int sinkhorn_iters, float post_mult, int mode, void* q_out, float* q_scale, int q_scale_ld, void* stream);
int stk_mhc_finalize_rows(const void* x, const float* prod, int prod_ld, int lo_at, const float* base, const float* scale, const void* norm_w, float* post, float* comb, void* y, int T, int H, int hc, float rms_eps, float hc_eps, int sinkhorn_iters, float post_mult, void* stream);
int stk_mhc_post(const void* x, const void* res, const float* post, const float* comb, void* out, int T, int H, int hc, void* stream);
int stk_mhc_cluster(const void* x, const float* fn, const float* base, const float* scale, const void* norm_w, float* post, float* comb, void* y, int T, int H, int hc, int n_mix, float rms_eps, float hc_eps, int sinkhorn_iters, float post_mult, int mode, void* stream);
int stk_mhc_post_pre(const void* fa, const void* res_old, const float* post_old, const float* comb_old, void* x_out, const float* fn, const float* base, const float* scale, const void* norm_w, float* post, float* comb, void* y, int T, int H, int hc, int n_mix, float rms_eps, float hc_eps, int sinkhorn_iters, float post_mult, int mode, void* stream);

// ---- mhc_decode.cu ----
int stk_ll_ctx_size(void);
int stk_ll_ctx_fill(void* ctx, const long long* bases, void* counters, long long words, int rank, int world, int spin_budget);
int stk_mhc_decode(const void* x, const void* fa, const void* res_old, const float* post_old, const float* comb_old, void* x_out, const float* fn, const float* base, const float* scale, const void* norm_w, float* post, float* comb, void* y, int T, int H, float rms_eps, float hc_eps, int sinkhorn_iters, float post_mult, const void* ll_ctx, int* status, void* stream);
int stk_ll_reduce(const void* ll_ctx, void* out, long long ldo, int T, int H, int* status, void* stream);
int stk_ll_push(const void* ll_ctx, const void* in, long long ldi, int T, int H, void* stream);

// ---- mla_decode.cu ----
int stk_mla_decode_splits(int T, int nh, int max_rows, int sm_count);
int stk_sparse_mla_decode(const void* q, long long ldt, const void* swa_cache, long long swa_stride, long long swa_slots_n, const void* comp_cache, long long comp_stride, long long comp_slots_n, const int* swa_slots, int swa_ld, int swa_rows, const int* swa_lens, const int* topk_slots, int topk_ld, int topk_rows, const int* topk_lens, const float* sink, void* out, long long ldo, float* workspace, int S, int T, int nh, float scale, int prep_q, float eps, const int64_t* positions, const float* inv_freq, int out_inv_rope, const void* kv_new, long long kv_ld, const void* kv_norm_w, const int64_t* cur_slot, int* status, void* stream);

// ---- mlstm.cu ----
int stk_mlstm_scan(const void* proj, long long ldp, int q_off, int k_off, int v_off, const float* gates, const float* gate_bias, float cap, const int* query_start, const int* req_rows, const int* start_pos, int n_req, float* S, float* n, float* m, float* num, float* den, float* mt, int heads, int dim, int vdim, int fp32, int min_span, int max_span, int T, void* stream);
int stk_mlstm_gate_slot(void);
long long stk_mlstm_state_slot(int dim, int vdim);
int stk_mlstm_chunks(const void* proj, long long ldp, int q_off, int k_off, int v_off, const float* gates, const float* gate_bias, float cap, const int* query_start, const int* req_rows, const int* start_pos, int n_req, float* S, float* n, float* m, float* num, float* den, float* mt, int heads, int dim, int vdim, int min_span, float* gate_ws, float* states, int max_chunks, int T, void* stream);
int stk_mlstm_finish(const float* num, const float* den, const float* mt, float* m_state, const float* norm_w, float eps, const int* tok_req, const int64_t* positions, const int* last_pos, const void* proj, long long ldp, int g_off, void* out, long long ldo, int fp32, int heads, int vdim, int gate_off, int up_off, int ff, int ff_off, int cols, int T, void* stream);

// ---- moe.cu ----
int stk_router(const float* logits, long long ldl, const float* bias, const int* tid2eid, const int64_t* token_ids, int vocab, int* ids, float* weights, int T, int E, int topk, int always, int groups, int keep, int scoring, int renorm, float scaling, int* status, void* stream);
int stk_moe_align(const int* ids, int n_pairs, int e_start, int e_local, int* sorted, int* pair_row, int* offsets, int* sorted_expert, int* counts, void* stream);
int stk_moe_direct_blocks(int n_pairs, int width, int sm_count);
int stk_moe_expert_fc1(const void* x, long long ldx, const void* w13, const void* s13, const float* g13, const int* sorted, const int* sorted_expert, const int* offsets, int e_local, int topk, void* act, int max_rows, int H, int I, float limit, const int* direct_ids, int e_start, void* stream);
int stk_moe_expert_fc2(const void* act, const void* w2, const void* s2, const float* g2, const int* sorted_expert, const int* offsets, int e_local, void* y, int max_rows, int H, int I, const int* direct_ids, int e_start, void* stream);

// ---- moe_grouped.cu ----
int stk_moe_permute(const void* x, long long ldx, const int* sorted, const int* offsets, int e_local, int topk, void* xs, int max_rows, int H, void* stream);
int stk_moe_grouped(const void* xs, long long xs_rows, const void* w, const void* s, const float* gscale, const int* offsets, int e_local, int n_out, int K, void* out, int fc1, float limit, int bt, int* status, int sm_count, void* stream);
int stk_moe_grouped_ep(const void* xs, long long xs_rows, const void* w, const void* s, const float* gscale, const int* offsets, int e_local, int n_out, int K, void* out, int fc1, float limit, int bt, int* status, int sm_count, const void* arrived, int spin_budget, void* stream);

// ---- moe_plain.cu ----
int stk_expert_rows(const void* x, long long ldx, int div, const void* W, const int* ids, int E, void* out, long long ldo, int N, int n_pad, int K, int act, int fp32, int n_pairs, void* stream);
int stk_expert_gather(const void* x, long long ldx, const int* sorted, int topk, void* xs, int K, int n_pairs, void* stream);
int stk_experts(const void* xs, int n_pairs, const void* W, const int* offsets, int E, int N, int K, void* out, long long ldo, int act, int sm_count, int* status, void* stream);

// ---- retention.cu ----
int stk_retention_scan(const void* proj, long long ldp, int q_off, int k_off, int v_off, const float* freq, int pairs, float k_scale, const float* decay, const int* query_start, const int* req_rows, const int* start_pos, int n_req, float* S, float* o, int heads, int dim, int vdim, int fp32, int min_span, int max_span, int T, void* stream);
int stk_rotate_qk(const void* proj, long long ldp, int q_off, int k_off, const float* freq, int pairs, float k_scale, const int64_t* positions, void* out, int heads, int dim, int d8, int T, void* stream);
int stk_retention_finish(const float* o, float eps, const float* weight, const int* tok_req, const int64_t* positions, const void* proj, long long ldp, int g_off, float scale, void* out, long long ldo, int left, int col, int cols, int fp32, int heads, int vdim, int T, void* stream);

// ---- sampler.cu ----
int stk_gumbel_argmax(const void* logits, long long ld, int logits_bf16, const float* temperature, const int64_t* seed, const int64_t* pos, const int* row_group, int pos_stride, float* part_val, int* part_idx, int chunks, int64_t* out, float* processed, long long ldp, int rows, int V, const int* top_k, const float* top_p, void* thr_scratch, int v_offset, const void* ll_ctx, const int* status_in, int* agreed_status, int* status, void* stream);
int stk_coupled_accept(const int64_t* verifier, const int64_t* draft, int64_t* n_acc, int64_t* emitted, int B, int N, void* stream);
int stk_markov_topk_bias(const void* base, long long ld, int base_bf16, const void* w2, const void* embed, long long lde, float* out, long long ldo, int rows, int V, int R, int k, void* stream);
int stk_markov_chain(const int* cand_idx, const float* cand_val, const int64_t* anchors, const void* w1, const void* w2, const float* temperature, const int64_t* seed, const int64_t* pos, int64_t* out, int B, int N, int K, int R, int V, void* stream);

// ---- skinny.cu ----
int stk_skinny_linear(const void* W, long long ldw, int is_fp8, const float* w_scale, int w_scale_ld, const void* x, long long ldx, void* out, long long ldo, int T, int N, int K, int out_fp32, int sm_count, int groups, int swiglu, float limit, void* stream);
int stk_skinny_linear_fused(const void* W, long long ldw, int is_fp8, const float* w_scale, int w_scale_ld, const void* x, long long ldx, void* out, long long ldo, int T, int N, int K, int out_fp32, int sm_count, const void* norm_w, float norm_eps, const void* ll_ctx, int route, int* route_counter, const float* bias, const int* tid2eid, const int64_t* token_ids, int vocab, int* ids, float* weights, int topk, int always, int groups, int keep, int scoring, int renorm, float scaling, int* status, void* stream);

// ---- symm.cu ----
int stk_symm_alloc(long long bytes, void** out);
int stk_symm_free(void* p);
int stk_symm_export(void* p, void* handle64);
int stk_symm_import(const void* handle64, void** out);
int stk_symm_close(void* p);
int stk_symm_ctx_size(void);
int stk_symm_ctx_fill(void* ctx, const long long* bases, int rank, int world, long long off_flags, long long off_epochs, long long off_oneshot, long long oneshot_bytes, long long off_rs, long long off_ag, long long twoshot_bytes, long long off_gemm, long long gemm_bytes, int spin_budget);
int stk_oneshot_allreduce(const void* ctx, const void* in, void* out, long long n_bytes, int nblocks, int* status, void* stream);
int stk_twoshot_allreduce(const void* ctx, const void* in, void* out, long long n_bytes, int nblocks, int* status, void* stream);
int stk_symm_reduce_scatter(const void* ctx, const void* in, void* out, long long total_bytes, int nblocks, int* status, void* stream);
int stk_symm_all_gather(const void* ctx, const void* shard, void* out, long long shard_bytes, int nblocks, int* status, void* stream);
int stk_symm_ag_push(const void* ctx, const void* shard, long long shard_bytes, long long dst_off, int nblocks, int* status, void* stream);
int stk_peer_copy(const long long* dsts, const long long* srcs, int n_peers, long long bytes, int blocks_per_peer, void* stream);
int stk_peer_pingpong(void* my_flag, void* peer_flag, int initiator, int rounds, int base, int budget, int* status, void* stream);
int stk_flag_timeout_probe(const void* flag, int epoch, int budget, int* status, void* stream);

// ---- talking_attention.cu ----
int stk_talking_prep(const void* proj, long long ldp, int q_off, int k_off, int v_off, int g_off, const float* bias, const float* q_norm, const float* k_norm, float eps, const float* freq, int pairs, const float* talk, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, void* cache, int row, int k_col, int kp, int vp, int heads, int kv_heads, int dim, int vdim, void* q, float* gate, int fp32, int T, void* stream);
int stk_talking_simt(const void* q, const float* gate, const float* sink, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, const void* cache, int row, int k_col, int kp, int vp, int heads, int kv_heads, int vdim, int chunk, float scale, void* out, long long ldo, int out_cols, int fp32, const int* first_pos, const int* last_pos, int max_span, int T, void* stream);

// ---- talking_prompt_tc.cu ----
int stk_talking_prompt_ok(int heads, int kv_heads, int kp, int vp, int vdim);
int stk_talking_rows(const int* query_start, const int* req_rows, const int* start_pos, int n_req, int min_span, int chunk, const int* table, int bt_stride, const void* cache, int row, void* out, long long rows, void* stream);
int stk_talking_prompt(const void* q, const float* gate, const float* sink, const void* rows, long long n_rows, int row, int k_col, int kp, int vp, int heads, int kv_heads, int vdim, int chunk, float scale, void* out, long long ldo, int out_cols, const int* query_start, const int* start_pos, int n_req, int min_span, int T, int sm_count, int* status, void* stream);

// ---- talking_tokens_tc.cu ----
int stk_talking_tokens_ok(int heads, int kv_heads, int kp, int vp, int max_span);
int stk_talking_tokens_plan(int T, int heads, int kv_heads, int kp, int vp, int max_span, int keys, int sm_count);
int stk_talking_tokens(const void* q, const float* gate, const float* sink, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, const void* cache, int row, int k_col, int kp, int vp, int heads, int kv_heads, int vdim, int chunk, float scale, void* out, long long ldo, int out_cols, const int* query_start, const int* req_rows, const int* start_pos, int n_req, const int* first_pos, const int* last_pos, int max_span, long long num_pages, int plan, float* part, int T, int* status, void* stream);

// ---- time_mix.cu ----
int stk_time_mix_scan(const void* proj, long long ldp, int np, const float* z, long long ldz, const float* w0, const float* u, const int* query_start, const int* req_rows, const int* start_pos, int n_req, float* S, float* o, int heads, int dim, int fp32, int min_span, int max_span, int T, void* stream);
int stk_tanh_rows(const float* z, long long ldz, int n, void* out, int fp32, int T, void* stream);
int stk_time_mix_chunks_ok(int dim);
int stk_time_mix_chunks(const void* proj, long long ldp, int np, const float* z, long long ldz, const float* w0, const float* u, const int* query_start, const int* req_rows, const int* start_pos, int n_req, float* S, float* o, int heads, int dim, int min_span, void* keys, float* channel, float* states, int max_chunks, int T, void* stream);

// ---- token_shift.cu ----
int stk_embed_bigram(const int64_t* ids, const void* embed, int embed_fp32, float scale, const void* table, int buckets, int mul_prev, int mul_cur, const int* tok_req, const int64_t* positions, const int* first_pos, const int64_t* last_token, float* x, int T, int W, int vocab, int* status, void* stream);
int stk_shifted_norm(const float* x, float* x_out, const float* y0, long long ld0, const float* w0, float f0, const float* y1, long long ld1, const float* w1, float f1, const float* ff, long long ldf, const void* pairs, long long ldp, const int* pair_row, const float* weights, int top, const float* norm, float eps, const float* shift, const float* mu, int blends, void* h, void* s, void* mix, int width, int fp32, const float* now, float* then, const int* tok_req, const int64_t* positions, const int* first_pos, const int* last_pos, const int64_t* rows, float* inv, int T, int W, int decode, int sm_count, void* stream);
int stk_shift_commit(const int* query_start, const int* req_rows, int n_req, const int64_t* ids, int64_t* token, const float* then, float* now, int layers, int n_rows, int n, void* stream);

// ---- window_attention.cu ----
int stk_window_kv_insert(const void* proj, long long ldp, int q_off, int k_off, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, void* cache, int row, const float* freq, int rd, float mag, int heads, int kv_heads, int dim, int fp32, int T, void* stream);
int stk_window_attention_simt(const void* proj, long long ldp, int q_off, int k_off, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, void* cache, int row, const float* freq, int rd, float mag, int heads, int kv_heads, int dim, int k_col, int vdim, int q_step, const void* gate, long long ldg, float out_scale, int window, float scale, float softcap, const float* sink, void* out, long long ldo, int fp32, int T, void* stream);
int stk_window_attention_splits(int T, int heads, int kv_heads, int window, int sm_count);
int stk_window_attention_mma_ok(int heads, int kv_heads, int dim, int vdim, int k_col, int row);
int stk_window_attention_tokens(const void* proj, long long ldp, int q_off, int k_off, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, void* cache, int row, const float* freq, int rd, float mag, int heads, int kv_heads, int dim, int k_col, int vdim, int q_step, const void* gate, long long ldg, float out_scale, int window, float scale, float softcap, const float* sink, void* out, long long ldo, const int* first_pos, const int* last_pos, int max_span, int splits, float* part, int T, void* stream);
int stk_window_attention_tiles(const void* proj, long long ldp, int q_off, int k_off, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, void* cache, int row, const float* freq, int rd, float mag, int heads, int kv_heads, int dim, int k_col, int vdim, int q_step, const void* gate, long long ldg, float out_scale, int window, float scale, float softcap, const float* sink, void* out, long long ldo, const int* query_start, const int* req_rows, const int* start_pos, int n_req, int min_span, int max_span, int T, void* stream);

// ---- window_attention_tc.cu ----
int stk_window_attention_tc_ok(int heads, int kv_heads, int dim, int rd, int row);
int stk_window_attention_tc(const void* proj, long long ldp, int q_off, int k_off, const int64_t* positions, const int* tok_req, const int* table, int bt_stride, void* cache, int row, const float* freq, int rd, float mag, int heads, int kv_heads, int dim, int window, float scale, float softcap, const float* sink, void* out, long long ldo, const int* query_start, const int* req_rows, const int* start_pos, int n_req, int min_span, long long num_pages, int T, int* status, void* stream);

#ifdef __cplusplus
}
#endif
