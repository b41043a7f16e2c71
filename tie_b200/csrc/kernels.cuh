// Launch entry points of the kernel translation units (all enqueue on c->stream).
#pragma once
#include "common.cuh"

namespace tie {

// router.cu
struct EpPush;
int launch_router(tie_cuda_ctx *c, const float *x, const float *w, const float *bias, int n_tokens, float *logits,
		  int *topk_idx, float *topk_w, int lfm2 = 0, const EpPush *push = nullptr, bool *push_taken = nullptr,
		  const float *norm_w = nullptr, float *norm_out = nullptr);
// norm_out: x is the residual stream, its RMSNorm (weights norm_w or null) goes there and is what is routed
bool router_norm_supported(const tie_cuda_ctx *c, int n_tokens);
int router_setup(tie_cuda_ctx *c);
// decode.cu
int decode_setup(tie_cuda_ctx *c);
bool decode_supported(const tie_cuda_ctx *c, const Layer &L, int n_tokens);
// foreign_slots_ok: slots whose expert another rank owns are skipped instead of reported
int launch_decode_gate_up(tie_cuda_ctx *c, const Layer &L, const float *x, int n_tokens, bool foreign_slots_ok = false);
int launch_decode_down_peer(tie_cuda_ctx *c, const Layer &L, int n_tokens);
int launch_decode_down_combine(tie_cuda_ctx *c, const Layer &L, int n_tokens, const float *residual, float *out);
int launch_router_rows(tie_cuda_ctx *c, const float *x, const float *w, int n_rows, int in_dim, float *out);
// decode_group.cu
int decode_group_setup(tie_cuda_ctx *c);
bool decode_group_supported(const tie_cuda_ctx *c, const Layer &L, int n_tokens);
int launch_group_gate_up(tie_cuda_ctx *c, const Layer &L, const float *x, int n_tokens);
int launch_group_down(tie_cuda_ctx *c, const Layer &L, int n_tokens, float *y);
// decode_fused.cu
bool decode_fused_supported(tie_cuda_ctx *c, const Layer &L, int n_tokens);
int launch_decode_fused(tie_cuda_ctx *c, const Layer &L, const float *x, const float *bias, const float *residual, float *out,
			unsigned *host_status = nullptr);
int launch_decode_fused_blocks(tie_cuda_ctx *c, const Layer &L, int n_layers, float *hidden);
DfLayer df_layer(const Layer &L);
// sort.cu
struct SortBufs {
	int *counts, *offsets, *tile_start, *active, *n_active, *perm;
	int4 *tile_info;  // optional: one entry per token tile (expert, first sorted row, rows, 0)
	// optional: inv[row id] = where the row stands in perm (-1: nowhere), and (expert-parallel publish), with
	// owner_div = experts per GPU and top_k > 0, EP_FIRST_OF_TOKEN set in the entries of perm
	int *inv = nullptr;
	int owner_div = 0, top_k = 0;
};
int launch_sort(tie_cuda_ctx *c, const int *row_expert, int n_rows, int n_tile);
int launch_sort(tie_cuda_ctx *c, const int *row_expert, int n_rows, int n_tile, int first_expert, int n_expert,
		const SortBufs &b);
// dispatch.cu
int launch_dispatch(tie_cuda_ctx *c, const float *x, const int *row_expert, int n_src, int n_out, int n_tile, bool sums, bool after_router);
// stream.cu
bool stream_supported(const Layer &L);
int launch_stream_gate_up(tie_cuda_ctx *c, const Layer &L, const float *xin, int src_div, const int *row_expert,
			  int n_rows, int direct);
int launch_stream_down(tie_cuda_ctx *c, const Layer &L, float *y, const int *row_expert, int n_rows, int direct);
int launch_stream_matvec(tie_cuda_ctx *c, const uint8_t *wexp, WKind kind, int k, int rows_total, const float *x, float *o);
// misc.cu
int launch_rms_norm(tie_cuda_ctx *c, const float *x, const float *w, float *o, int n_tokens);
int launch_combine(tie_cuda_ctx *c, const float *y, const float *topk_w, int n_tokens, const float *residual, float *out,
		   const int *pos = nullptr, bool dependent = false);
int launch_gather_rows(tie_cuda_ctx *c, const float *x, const int *row_expert, const int *perm, int src_div, int n_rows,
		       float *rows_out, int *expert_out, int *inv);
int launch_split_rows(tie_cuda_ctx *c, const float *x, int n_src, int n_cols, __half *hi, __half *lo, __half *xq);
int launch_swiglu(tie_cuda_ctx *c, float *gate, const float *up, int n);
// tensor.cu
int tc_setup(tie_cuda_ctx *c);
int tc_make_weight_map(tie_cuda_ctx *c, DevTensor &t, bool half_tiles, int n_experts = -1);  // default: the context's local experts
bool tc_dense_supported(const tie_cuda_ctx *c, const DevTensor &t);
int tc_make_dense_view(tie_cuda_ctx *c, DevTensor &t);
int launch_tc_dense(tie_cuda_ctx *c, const DevTensor &t, int n_rows, float *y);
bool tc_supported(const tie_cuda_ctx *c, const Layer &L);
// n_tile: the token tiles of the sort, 32 or 64 rows
int launch_tc_gate_up(tie_cuda_ctx *c, const Layer &L, int n_tile);
int launch_tc_down(tie_cuda_ctx *c, const Layer &L, int n_tile, float *y, bool sorted);
int launch_tc_down_peer(tie_cuda_ctx *c, const Layer &L, const EpDst &dst);
// ep.cu
int launch_ep_signal(tie_cuda_ctx *c, int which);
int launch_ep_push_tokens(tie_cuda_ctx *c, const float *x, int n_tokens);
EpPush ep_push_args(tie_cuda_ctx *c, const float *x, int n_tokens);  // (ep_dev.cuh defines EpPush)
int launch_ep_index(tie_cuda_ctx *c);
int launch_ep_split_rows(tie_cuda_ctx *c, bool sums);
int launch_ep_combine(tie_cuda_ctx *c, int n_tokens, const float *residual, float *out);
// repack.cu
int launch_repack_q6k_r8(tie_cuda_ctx *c, const uint8_t *raw, uint8_t *dst, size_t n_rows_total, int nb);

}  // namespace tie
