// Device functions of the router shared by its kernels (router.cu) and the one-kernel decode
// step (decode_fused.cu): the AVX2 horizontal sum and the per-token selection.
#pragma once

#include "common.cuh"

namespace tie {

// hsum over the 8 lanes of one expert held in 8 consecutive threads of a warp.
__device__ __forceinline__ float hsum8_lanes(float acc)
{
	float v = __fadd_rn(acc, __shfl_down_sync(0xffffffffu, acc, 4, 8));  // lanes 0..3: l+l4
	float t = __fadd_rn(v, __shfl_down_sync(0xffffffffu, v, 1, 8));	     // lane 0: s0+s1, lane 2: s2+s3
	float r = __fadd_rn(t, __shfl_down_sync(0xffffffffu, t, 2, 8));	     // lane 0: (s0+s1)+(s2+s3)
	return r;
}

// Order-preserving map of a score to an unsigned key (larger score, larger key; -0 and +0 the same key).
__device__ __forceinline__ unsigned score_key(float v)
{
	const unsigned u = __float_as_uint(__fadd_rn(v, 0.0f));
	return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}

// The score of a key (of -0: +0).
__device__ __forceinline__ float key_score(unsigned key)
{
	return __uint_as_float(key & 0x80000000u ? key ^ 0x80000000u : ~key);
}

// find_top_k (engine.c:891-914) by one warp for NT tokens at once: key[n][i] is the key of expert
// lane + 32 i (0: none, or taken).  A round is two hardware reductions, the largest key and, among its
// holders, the lowest expert: ties keep the lower index.  Lane r < top_k ends up with the expert of
// rank r (or -1) of token n in mine[n], and its key in best[n].
template <int NT, int PER>
__device__ __forceinline__ void topk_warp(unsigned (&key)[NT][PER], int lane, int top_k, int (&mine)[NT], unsigned (&best)[NT])
{
#pragma unroll
	for (int n = 0; n < NT; n++) {
		mine[n] = -1;
		best[n] = 0u;
	}
	for (int r = 0; r < top_k; r++) {
		unsigned top[NT], e[NT];
#pragma unroll
		for (int n = 0; n < NT; n++) {
			unsigned largest = key[n][0];
#pragma unroll
			for (int i = 1; i < PER; i++)
				largest = max(largest, key[n][i]);
			top[n] = __reduce_max_sync(0xffffffffu, largest);
		}
#pragma unroll
		for (int n = 0; n < NT; n++) {
			e[n] = 0xffffffffu;
#pragma unroll
			for (int i = PER - 1; i >= 0; i--)  // (ascending experts within a lane: the last match written is the lowest)
				e[n] = key[n][i] == top[n] ? (unsigned)(lane + 32 * i) : e[n];
			e[n] = __reduce_min_sync(0xffffffffu, e[n]);
		}
#pragma unroll
		for (int n = 0; n < NT; n++) {
#pragma unroll
			for (int i = 0; i < PER; i++)
				key[n][i] = e[n] == (unsigned)(lane + 32 * i) ? 0u : key[n][i];
			if (lane == r && top[n] != 0u) {  // (0: fewer experts than top_k)
				mine[n] = (int)e[n];
				best[n] = top[n];
			}
		}
	}
}

// Selection and gate weights of tokens t .. t + n_real - 1 (n_real <= NT) by one warp; n_expert <= 32 PER.
// Qwen3-MoE: top-k of the logits, softmax of the selected ones (max-subtract, expf, sequential sum,
// multiply by 1/sum).  lfm2 (model_lfm2.c:438-473): s = sigmoid(logit) for every expert, selection on
// s + sel_bias (exp_probs_b, may be null), gates = the UNBIASED s of the selected experts, summed in
// slot order and scaled by 1/(sum + 1e-6); logits is overwritten with the sigmoid scores (the
// reference does the same to expert_scores).
template <int NT, int PER>
__device__ __forceinline__ void topk_tokens(float *__restrict__ logits, const float *__restrict__ sel_bias, int t, int n_real, int lane,
					    int n_expert, int top_k, int *__restrict__ topk_idx, float *__restrict__ topk_w, int lfm2)
{
	unsigned key[NT][PER];
#pragma unroll
	for (int n = 0; n < NT; n++)
#pragma unroll
		for (int i = 0; i < PER; i++) {
			const int e = lane + 32 * i;
			float *lg = logits + (size_t)(t + (n < n_real ? n : 0)) * n_expert + e;
			key[n][i] = 0u;
			if (e < n_expert) {
				float v = __ldcg(lg);
				if (lfm2) {
					v = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-v)));
					if (n < n_real)
						__stcg(lg, v);
					if (sel_bias)
						v = __fadd_rn(v, sel_bias[e]);
				}
				key[n][i] = score_key(v);
			}
		}
	int mine[NT];
	unsigned best[NT];
	topk_warp<NT, PER>(key, lane, top_k, mine, best);
	__syncwarp();
#pragma unroll
	for (int n = 0; n < NT; n++) {
		if (n >= n_real)
			break;
		// (a selected logit is its key again, not a load behind the selection; LFM2 gates are not what was selected on)
		float v = mine[n] < 0 ? 0.0f : (lfm2 ? __ldcg(logits + (size_t)(t + n) * n_expert + mine[n]) : key_score(best[n]));
		const float mx = __shfl_sync(0xffffffffu, v, 0);  // (scores are sorted descending: lane 0 holds the max)
		if (!lfm2)
			v = lane < top_k ? expf(__fsub_rn(v, mx)) : 0.0f;
		float sum = 0.0f;
		for (int j = 0; j < top_k; j++)
			sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, v, j));
		const float inv = __fdiv_rn(1.0f, lfm2 ? __fadd_rn(sum, 1e-6f) : sum);
		if (lane < top_k) {
			topk_idx[(size_t)(t + n) * top_k + lane] = mine[n];
			topk_w[(size_t)(t + n) * top_k + lane] = __fmul_rn(v, inv);
		}
	}
}

// One token by one warp.
__device__ __forceinline__ void topk_softmax_warp(const float *__restrict__ logits, int token, int lane, int n_expert, int top_k,
						  int *__restrict__ topk_idx, float *__restrict__ topk_w)
{
	topk_tokens<1, 8>(const_cast<float *>(logits), nullptr, token, 1, lane, n_expert, top_k, topk_idx, topk_w, 0);
}

}  // namespace tie
