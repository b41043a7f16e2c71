// Router: logits = x . W_router^T (bit-exact replay of the reference's AVX2 F32 mat-vec),
// optional bias, top-k with the reference's tie rule, softmax over the selected logits.
//
// Reference: dispatch_mat_vec on ffn_gate_inp (model_qwen3.c:431) -> mat_vec_row_f32_f32_f32_avx2
// (math_avx2.c:228-256): 8 independent lanes, lane l accumulates fma(x[8i+l], w[8i+l], acc_l)
// for i = 0..in_dim/8-1 in order, then hsum (math_avx2.c:14-21):
// ((l0+l4)+(l1+l5)) + ((l2+l6)+(l3+l7)).  Replaying that order gives bit-identical logits, which
// is what makes the top-k selection identical (the 8th/9th logit gap can be a few ulp).
// find_top_k: engine.c:891-914 (strict '>': ties keep the lower expert index, output sorted by
// score descending).  softmax: engine.c:864-888 over the k selected raw logits.
#include <mutex>

#include "common.cuh"
#include "ep_dev.cuh"
#include "kernels.cuh"

#include "router_topk.cuh"
#include "tc_ptx.cuh"

namespace tie {

// tie_cuda_route_noalloc from 9 tokens: CTA = TT tokens x EPC experts; thread = (expert, lane); router weights come
// straight from L2 (each loaded value feeds TT fused multiply-adds), x is staged in k-chunks.
template <int TT, int EPC, int KC>
__global__ void __launch_bounds__(EPC * 8) router_logits_tile(const float *__restrict__ x, const float *__restrict__ w,
							      const float *__restrict__ bias, float *__restrict__ logits,
							      int n_tokens, int hidden, int n_expert)
{
	__shared__ float xs[TT][KC];
	const int t0 = blockIdx.x * TT;
	const int e = blockIdx.y * EPC + (threadIdx.x >> 3);
	const int l = threadIdx.x & 7;
	const float *wr = w + (size_t)e * hidden;
	float acc[TT];
#pragma unroll
	for (int i = 0; i < TT; i++)
		acc[i] = 0.0f;
	for (int k0 = 0; k0 < hidden; k0 += KC) {
		__syncthreads();
		for (int i = threadIdx.x; i < TT * (KC / 4); i += EPC * 8) {
			int tt = i / (KC / 4), c = i % (KC / 4);
			float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
			if (t0 + tt < n_tokens)
				v = *reinterpret_cast<const float4 *>(x + (size_t)(t0 + tt) * hidden + k0 + 4 * c);
			*reinterpret_cast<float4 *>(&xs[tt][4 * c]) = v;
		}
		__syncthreads();
#pragma unroll 8
		for (int i = 0; i < KC / 8; i++) {
			float wv = __ldg(wr + k0 + 8 * i + l);
#pragma unroll
			for (int tt = 0; tt < TT; tt++)
				acc[tt] = __fmaf_rn(xs[tt][8 * i + l], wv, acc[tt]);
		}
	}
#pragma unroll
	for (int tt = 0; tt < TT; tt++) {
		float r = hsum8_lanes(acc[tt]);
		if (l == 0 && t0 + tt < n_tokens) {
			if (bias)
				r = __fadd_rn(r, bias[e]);
			logits[(size_t)(t0 + tt) * n_expert + e] = r;
		}
	}
}

// The router of a batch: logits, selection and softmax in one launch.
//
// Thread = one AVX2 lane l of a TPT-token x EPT-expert register tile (each of its chains a strict
// i-ascending sequence of fused multiply-adds, so the result stays bit-identical); CTA = TT tokens x TE
// experts.  The operands' rows are staged as they are, by asynchronous copies two chunks ahead; a row pitch of
// 8 words mod 32 keeps a warp's loads (8 lanes x 2 rows) free of bank conflicts.  What bounds a small batch is
// how many SMs pull the 1 MB of router weights, a large one the multiply-adds and the shared-memory loads
// beside them (wider loads move no more per cycle), so the tile grows with the batch (TIE_RT_TILES).  The
// CTA that finishes a token tile last (a counter per tile, nobody waits) selects for all its tokens.
// A small grid starts beside the kernel in front of it and fetches its first weights before it waits for the tokens.
// A copy's addresses are made once a call, not once a chunk (with the sums over the lanes below, an event on either side: 64
// tokens 16.4 us as before, 512 30.7 -> 26.7, 1000 41.1 -> 37.2, 2000 59.4 -> 52, 4096 100.4 -> 92.2).  Two AVX2 lanes per thread
// on packed multiply-adds, alone or with a loading warp in front, were equal or slower at every size.
//
// The hand-over of the tokens in an expert-parallel step rides along as one more row of CTAs, of
// which as many work as there are SMs the logits' CTAs leave free (at least 16): CTAs that share an
// SM with the logits take load/store slots from them (32 working CTAs lengthened the kernel by 10 us
// at 4 GPUs, 128 by 18 us).
constexpr int RT_NORM_SMEM = 200 * 1024;
constexpr int RT_PUSH_ROWS = 1;
static int rt_push_ctas(const tie_cuda_ctx *c, int logits_ctas, int most)
{
	int n = c->sm_count - logits_ctas;
	n = n < 16 ? 16 : n;
	return n < most ? n : most;
}

template <int TPT_, int EPT_, int TT_, int TE_, int KC_>
struct RtCfg {
	static constexpr int TPT = TPT_, EPT = EPT_, TT = TT_, TE = TE_, KC = KC_;
	static constexpr int TG = TT / TPT, EG = TE / EPT, THREADS = 8 * TG * EG;
	static constexpr int PITCH = KC + 8, STAGE = (TT + TE) * PITCH;  // floats; two rows apart by a quarter of the banks
	static constexpr int STAGES = 3, SMEM = STAGES * STAGE * (int)sizeof(float);
	static constexpr int UNROLL = TPT * EPT >= 64 ? 2 : (TPT * EPT > 8 ? 8 : 32);  // (few chains a thread: their loads go far ahead)
	static constexpr int LD = (TT + TE) * (KC / 4) / THREADS;  // 16-byte copies per thread and chunk
	// the form with the RMSNorm in front: whole rows in shared memory, and COLS float4 of each in a thread's registers
	static constexpr bool NORM = TT <= 8 && KC == 512;
	static constexpr int COLS = NORM ? 16 / TT : 0;
	static_assert(THREADS % (KC / 4) == 0 && TT % (THREADS / (KC / 4)) == 0 && (TT + TE) * (KC / 4) % THREADS == 0 && TG % 2 == 0 && EG % 2 == 0 && KC % 32 == 0, "router tile");
};

// NORM: x is the residual stream; the CTA makes the RMSNorm of its tokens itself (rms_norm_rows, the same operations in the same
// order) while the router weights arrive, and the CTAs of the first experts store it for the kernels behind.  A launch of
// its own is 3.4 us of a block of 4 tokens (8 blocks of 4 tokens 366.1 -> 356.6 us, 4 of 13 356.1 -> 349.0; with the chains' loads
// further ahead, here and in the products of the smallest tiles, another 2 and 1 %).
struct RtNorm {
	const float *w = nullptr;  // or null: weight 1
	float *out = nullptr;
	float eps = 0.f;
};
template <class C, bool NORM>
__global__ void __launch_bounds__(C::THREADS, C::THREADS >= 512 || NORM ? 1 : 2)
router_batch(const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ bias, float *__restrict__ logits,
	     int n_tokens, int hidden, int n_expert, int top_k, int *__restrict__ topk_idx, float *__restrict__ topk_w, int lfm2,
	     const float *__restrict__ sel_bias, int *__restrict__ counter, const EpPush push, const RtNorm norm)
{
	constexpr int TPT = C::TPT, EPT = C::EPT, TT = C::TT, TE = C::TE, KC = C::KC;
	extern __shared__ __align__(16) float rsm[];
	__shared__ int s_last;
	// Expert-parallel steps: RT_PUSH_ROWS more rows of CTAs (blockIdx.y past the expert tiles) store this
	// rank's tokens into every rank's memory while the others compute the logits; they share nothing
	// with them.
	if (push.x && (int)blockIdx.y * TE >= n_expert) {
		pdl_wait();
		const int row = (int)blockIdx.y - n_expert / TE, cta = row * (int)gridDim.x + (int)blockIdx.x;
		if (cta < push.n_ctas)
			ep_push_tokens_cta(push, cta, push.n_ctas);
		return;
	}
	const int t0 = blockIdx.x * TT, e0 = blockIdx.y * TE;
	// a warp is 8 lanes x 2 token groups x 2 expert groups
	const int l = threadIdx.x & 7, g4 = threadIdx.x >> 5;
	const int tg = ((threadIdx.x >> 3) & 1) + 2 * (g4 % (C::TG / 2)), eg = ((threadIdx.x >> 4) & 1) + 2 * (g4 / (C::TG / 2));
	const int n_chunks = hidden / KC;
	// what this thread copies of a chunk: 16 bytes of LD rows, ROWS apart; the addresses are made once
	constexpr int ROWS = C::THREADS / (KC / 4);
	const int row0 = threadIdx.x / (KC / 4), c4 = threadIdx.x % (KC / 4);
	const float *src[C::LD];
#pragma unroll
	for (int j = 0; j < C::LD; j++)
		src[j] = 4 * c4 + (j * ROWS < TT ? x + (size_t)min(t0 + row0 + j * ROWS, n_tokens - 1) * hidden  // (rows past the end: computed, dropped)
						 : w + (size_t)(e0 + row0 + j * ROWS - TT) * hidden);
	const uint32_t dst0 = ptx::smem_u32(rsm + row0 * C::PITCH + 4 * c4);
	auto fetch = [&](int c, bool tokens, bool weights) {
		if (c < n_chunks) {
			const uint32_t dst = dst0 + (uint32_t)((c % C::STAGES) * C::STAGE) * 4u;
#pragma unroll
			for (int j = 0; j < C::LD; j++)
				if (j * ROWS < TT ? tokens : weights)
					ptx::cp_async16(dst + (uint32_t)(j * ROWS * C::PITCH) * 4u, src[j] + (size_t)c * KC);
		}
	};
	float acc[TPT][EPT];
#pragma unroll
	for (int j = 0; j < TPT; j++)
#pragma unroll
		for (int b = 0; b < EPT; b++)
			acc[j][b] = 0.0f;
#pragma unroll
	for (int c = 0; c < C::STAGES - 1; c++)
		fetch(c, false, true);
	const int px = hidden + 8, tp = hidden / 8 + 4;	 // NORM: pitch of the rows, and of their lanes before that
	float *rows = rsm + C::STAGES * C::STAGE;
	if constexpr (NORM) {
		__shared__ float s_inv[TT];
		constexpr int COLS = C::COLS;
		float4 v[TT][COLS], g[COLS];
		auto col = [&](int k) { return threadIdx.x + k * C::THREADS; };
#pragma unroll
		for (int k = 0; k < COLS; k++)
			g[k] = norm.w && 4 * col(k) < hidden ? __ldg(reinterpret_cast<const float4 *>(norm.w) + col(k)) : make_float4(1.f, 1.f, 1.f, 1.f);
		pdl_wait();
#pragma unroll
		for (int k = 0; k < COLS; k++)
#pragma unroll
			for (int j = 0; j < TT; j++)
				if (4 * col(k) < hidden)
					v[j][k] = reinterpret_cast<const float4 *>(x + (size_t)min(t0 + j, n_tokens - 1) * hidden)[col(k)];
#pragma unroll
		for (int k = 0; k < COLS; k++)
#pragma unroll
			for (int j = 0; j < TT; j++)
				if (4 * col(k) < hidden) {  // for the sums, as [AVX2 lane][step]: four steps of a chain per load
					float *d = rows + j * (hidden + 32) + 4 * (col(k) & 1) * tp + (col(k) >> 1);
					d[0] = v[j][k].x;
					d[tp] = v[j][k].y;
					d[2 * tp] = v[j][k].z;
					d[3 * tp] = v[j][k].w;
				}
		__syncthreads();
		if (threadIdx.x < 8 * TT) {  // a thread per lane of a row's sum of squares
			const float4 *r = reinterpret_cast<const float4 *>(rows + (threadIdx.x >> 3) * (hidden + 32) + (threadIdx.x & 7) * tp);
			float a = 0.f;
#pragma unroll 16
			for (int i = 0; i < hidden / 32; i++) {
				const float4 u = r[i];
				a = __fmaf_rn(u.x, u.x, a);
				a = __fmaf_rn(u.y, u.y, a);
				a = __fmaf_rn(u.z, u.z, a);
				a = __fmaf_rn(u.w, u.w, a);
			}
			const float ss = hsum8_lanes(a);
			if ((threadIdx.x & 7) == 0)
				s_inv[threadIdx.x >> 3] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)hidden), norm.eps)));
		}
		__syncthreads();
#pragma unroll
		for (int j = 0; j < TT; j++) {
			const float inv = s_inv[j];
#pragma unroll
			for (int k = 0; k < COLS; k++)
				if (4 * col(k) < hidden) {
					const float4 a = v[j][k], b = g[k];
					const float4 o = make_float4(__fmul_rn(__fmul_rn(a.x, b.x), inv), __fmul_rn(__fmul_rn(a.y, b.y), inv),
								     __fmul_rn(__fmul_rn(a.z, b.z), inv), __fmul_rn(__fmul_rn(a.w, b.w), inv));
					*reinterpret_cast<float4 *>(rows + j * px + 4 * col(k)) = o;
					if (blockIdx.y == 0 && t0 + j < n_tokens)
						reinterpret_cast<float4 *>(norm.out + (size_t)(t0 + j) * hidden)[col(k)] = o;
				}
		}
#pragma unroll
		for (int c = 0; c < C::STAGES - 1; c++)
			ptx::cp_async_commit();  // (all the weights asked for so far are in the first group)
	} else {
		pdl_wait();	// the tokens may be the work of the kernel before this one
#pragma unroll
		for (int c = 0; c < C::STAGES - 1; c++) {
			fetch(c, true, false);
			ptx::cp_async_commit();
		}
	}
	for (int c = 0; c < n_chunks; c++) {
		ptx::cp_async_wait<C::STAGES - 2>();
		__syncthreads();  // (chunk c is here for everyone, and everyone is done with the buffer of chunk c - 1)
		fetch(c + C::STAGES - 1, !NORM, true);
		ptx::cp_async_commit();	 // (an empty group past the end)
		const float *buf = rsm + (c % C::STAGES) * C::STAGE + l, *ws = buf + (TT + eg) * C::PITCH;
		const float *xs = NORM ? rows + l + tg * px + c * KC : buf + tg * C::PITCH;
		const int xpitch = NORM ? px : C::PITCH;
#pragma unroll C::UNROLL
		for (int g = 0; g < KC / 8; g++) {
			float xv[TPT], wv[EPT];
#pragma unroll
			for (int j = 0; j < TPT; j++)
				xv[j] = xs[C::TG * j * xpitch + 8 * g];
#pragma unroll
			for (int b = 0; b < EPT; b++)
				wv[b] = ws[C::EG * b * C::PITCH + 8 * g];
#pragma unroll
			for (int b = 0; b < EPT; b++)
#pragma unroll
				for (int j = 0; j < TPT; j++)
					acc[j][b] = __fmaf_rn(xv[j], wv[b], acc[j][b]);
		}
	}
	// hsum8_lanes of every (token, expert) of the 8 threads: ((l0 + l4) + (l1 + l5)) + ((l2 + l6) + (l3 + l7)).  A thread adds
	// and passes on half of what it has per step, as far as that goes: 7/8 of a shuffle a chain instead of 3, and every thread
	// stores (4096 tokens 100.4 -> 93.5 us, 512 30.7 -> 28.8).
	constexpr int N = TPT * EPT;
	float *v = &acc[0][0];
	int at = 0;  // of the thread's sums in the flat order [j][b]
	int left = N;
#pragma unroll
	for (int step = 0; step < 3; step++) {
		const int bit = step == 0 ? 4 : (step == 1 ? 1 : 2);
		if (left > 1) {
			left /= 2;
			const bool upper = l & bit;
			at += upper ? left : 0;
#pragma unroll
			for (int n = 0; n < N / 2; n++)
				if (n < left) {
					const float keep = upper ? v[left + n] : v[n], send = upper ? v[n] : v[left + n];
					v[n] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, bit));
				}
		} else {
			v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], bit));
		}
	}
	constexpr int OUT = N >= 8 ? N / 8 : 1;
#pragma unroll
	for (int n = 0; n < OUT; n++) {
		const int j = (at + n) / EPT, b = (at + n) % EPT, t = t0 + tg + C::TG * j, e = e0 + eg + C::EG * b;
		// (fewer chains than threads: the first of those that have the same sum)
		if (t < n_tokens && (N >= 8 || (N == 4 ? !(l & 2) : (N == 2 ? !(l & 3) : l == 0)))) {
			float r = v[n];
			if (bias)
				r = __fadd_rn(r, bias[e]);
			__stcg(logits + (size_t)t * n_expert + e, r);
		}
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		// (releases the CTA's logits, which the barrier has ordered before this thread, and acquires those of the others)
		int done;
		asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(done) : "l"(counter + blockIdx.x) : "memory");
		s_last = done == n_expert / TE - 1;
	}
	__syncthreads();
	// The decode kernels' CTAs may come now and wait for this grid: before the selection, not before the products (from
	// the start of the grid a block of 6 tokens takes 69.4 us, from here 62.5, without 63.4).
	pdl_trigger();
	if (!s_last)
		return;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	// (a warp's tokens are selected for together, up to four at a time: one after the other they are a chain of
	// reductions of a microsecond each)
	constexpr int WARPS = C::THREADS / 32, TW = (TT + WARPS - 1) / WARPS, NT = TW < 4 ? TW : 4;
	const int t1 = min(t0 + TT, n_tokens);
	for (int t = t0 + warp * TW; t < min(t0 + (warp + 1) * TW, t1); t += NT) {
		const int n = min(NT, min(t0 + (warp + 1) * TW, t1) - t);
		if (n_expert <= 128)
			topk_tokens<NT, 4>(logits, sel_bias, t, n, lane, n_expert, top_k, topk_idx, topk_w, lfm2);
		else
			topk_tokens<NT, 8>(logits, sel_bias, t, n, lane, n_expert, top_k, topk_idx, topk_w, lfm2);
	}
	if (threadIdx.x == 0)
		counter[blockIdx.x] = 0;
}

// The F32 row entry and tie_cuda_route_noalloc up to 8 tokens (MoE calls of every size run on router_batch): one
// expert per CTA; the row and the tokens are staged in shared memory with wide loads, then thread (token, lane)
// runs the sequential chain.
__global__ void __launch_bounds__(64) router_logits_decode(const float *__restrict__ x, const float *__restrict__ w,
							   const float *__restrict__ bias, float *__restrict__ logits,
							   int n_tokens, int hidden, int n_expert)
{
	extern __shared__ float sm[];
	float *ws = sm;			  // [hidden]
	float *xs = sm + hidden;	  // [n_tokens][hidden + 8]  (row pad spreads tokens over banks)
	const int xstride = hidden + 8;
	const int e = blockIdx.x;
	const float4 *wr4 = reinterpret_cast<const float4 *>(w + (size_t)e * hidden);
	for (int i = threadIdx.x; i < hidden / 4; i += 64)
		reinterpret_cast<float4 *>(ws)[i] = __ldg(wr4 + i);
	for (int i = threadIdx.x; i < n_tokens * (hidden / 4); i += 64) {
		int tt = i / (hidden / 4), c4 = i % (hidden / 4);
		*reinterpret_cast<float4 *>(xs + (size_t)tt * xstride + 4 * c4) =
			*reinterpret_cast<const float4 *>(x + (size_t)tt * hidden + 4 * c4);
	}
	__syncthreads();
	const int tt = threadIdx.x >> 3, l = threadIdx.x & 7;
	float acc = 0.0f;
	if (tt < n_tokens) {
		const float *xr = xs + (size_t)tt * xstride;
#pragma unroll 16
		for (int i = 0; i < hidden / 8; i++)
			acc = __fmaf_rn(xr[8 * i + l], ws[8 * i + l], acc);
	}
	float r = hsum8_lanes(acc);
	if (l == 0 && tt < n_tokens) {
		if (bias)
			r = __fadd_rn(r, bias[e]);
		logits[(size_t)tt * n_expert + e] = r;
	}
}

__global__ void __launch_bounds__(128) router_topk(const float *__restrict__ logits, int n_tokens, int n_expert, int top_k,
						   int *__restrict__ topk_idx, float *__restrict__ topk_w)
{
	const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int lane = threadIdx.x & 31;
	if (warp >= n_tokens)
		return;
	topk_softmax_warp(logits, warp, lane, n_expert, top_k, topk_idx, topk_w);
}

// lfm2 = 0: bias (optional) is added to the logits, top-k + softmax over the selected logits
// (Qwen3-MoE).  lfm2 = 1: LFM2-MoE routing, bias (optional) is the selection bias exp_probs_b.
// push (expert-parallel steps): the kernel of the logits takes the hand-over of this rank's tokens to
// its peers along as extra CTAs where it can; *push_taken tells whether it did.
//
// The tiles, with what a launch of them takes: a + b n tenths of a microsecond when every SM has n CTAs (measured at
// 2048 inputs, 128 experts).  launch_router takes the cheapest for its batch: a tile with more products per
// operand load costs less per token, and more for the batch that leaves it half empty or one CTA over.
#define TIE_RT_TILES(X)                            \
	X(100, 820, RtCfg<8, 8, 64, 64, 64>)   \
	X(102, 410, RtCfg<8, 4, 32, 64, 64>)   \
	X(155, 212, RtCfg<4, 8, 16, 64, 64>)   \
	X(133, 130, RtCfg<4, 4, 16, 32, 64>)   \
	X(123, 101, RtCfg<2, 4, 16, 16, 256>)  \
	X(115, 69, RtCfg<2, 2, 8, 16, 256>)    \
	X(110, 51, RtCfg<1, 2, 8, 8, 512>)     \
	X(95, 28, RtCfg<1, 1, 4, 4, 512>)
static int pick_tile(const tie_cuda_ctx *c, int n_tokens)
{
	const int H = c->cfg.hidden, E = c->cfg.n_expert;
	int pick = -1, at = 0;
	long long best = 0;
#define TIE_RT_PICK(A, B, ...)                                                                             \
	{                                                                                                  \
		using C = __VA_ARGS__;                                                                     \
		const long long ctas = (long long)((n_tokens + C::TT - 1) / C::TT) * (E / C::TE);          \
		const long long cost = A + B * ((ctas + c->sm_count - 1) / c->sm_count);                   \
		if (E % C::TE == 0 && H % C::KC == 0 && (pick < 0 || cost < best)) {                       \
			pick = at;                                                                         \
			best = cost;                                                                       \
		}                                                                                          \
		at++;                                                                                      \
	}
	TIE_RT_TILES(TIE_RT_PICK)
#undef TIE_RT_PICK
	return pick;
}

// Can the router's kernel for this batch make the RMSNorm too?  (Small tiles: each CTA makes all of its tokens'.)
bool router_norm_supported(const tie_cuda_ctx *c, int n_tokens)
{
	const int H = c->cfg.hidden, pick = pick_tile(c, n_tokens);
	int at = 0;
	bool ok = false;
#define TIE_RT_NORM(A, B, ...)                                                                                              \
	if (at++ == pick) {                                                                                                 \
		using C = __VA_ARGS__;                                                                                      \
		ok = C::NORM && H / 4 <= C::COLS * C::THREADS && C::SMEM + C::TT * (H + 32) * sizeof(float) <= RT_NORM_SMEM; \
	}
	TIE_RT_TILES(TIE_RT_NORM)
#undef TIE_RT_NORM
	return ok;
}

int launch_router(tie_cuda_ctx *c, const float *x, const float *w, const float *bias, int n_tokens, float *logits,
		  int *topk_idx, float *topk_w, int lfm2, const EpPush *push, bool *push_taken, const float *norm_w, float *norm_out)
{
	const int H = c->cfg.hidden, E = c->cfg.n_expert, K = c->cfg.top_k;
	EpPush f = {};
	if (push)
		f = *push;
	if (push_taken)
		*push_taken = push != nullptr;
	const float *sel_bias = lfm2 ? bias : nullptr;
	if (lfm2)
		bias = nullptr;
	const int pick = pick_tile(c, n_tokens);
	if (pick < 0)
		return TIE_CUDA_ENOTSUP;
	int at = 0;
	RtNorm norm;
	norm.w = norm_w;
	norm.out = norm_out;
	norm.eps = c->cfg.norm_eps;
	// (dependent where it is one wave: a grid that waits beside its predecessor then takes nothing from it)
	int rc = TIE_CUDA_OK;
#define TIE_RT_RUN(A, B, ...)                                                                                              \
	if (at++ == pick) {                                                                                                \
		using C = __VA_ARGS__;                                                                                     \
		dim3 grid((n_tokens + C::TT - 1) / C::TT, E / C::TE + (push ? RT_PUSH_ROWS : 0));                          \
		f.n_ctas = rt_push_ctas(c, grid.x * (E / C::TE), grid.x * RT_PUSH_ROWS);                                   \
		const bool dependent = (int)(grid.x * grid.y) <= c->sm_count;                                              \
		auto run = [&](auto kern, size_t smem) {                                                                   \
			return launch_kernel(c, dependent, 1, kern, grid, C::THREADS, smem, x, w, bias, logits, n_tokens, H, E, K, topk_idx, topk_w, \
					     lfm2, sel_bias, c->s.route_counter, f, norm);                                 \
		};                                                                                                         \
		if constexpr (C::NORM)                                                                                     \
			rc = norm_out ? run(router_batch<C, true>, C::SMEM + C::TT * (H + 32) * sizeof(float))               \
				      : run(router_batch<C, false>, C::SMEM);                                               \
		else                                                                                                       \
			rc = norm_out ? TIE_CUDA_EINVAL : run(router_batch<C, false>, C::SMEM);                            \
	}
	TIE_RT_TILES(TIE_RT_RUN)
#undef TIE_RT_RUN
	return rc;
}

// Opt-in shared-memory sizes are set once per context (never inside a stream capture).
int router_setup(tie_cuda_ctx *c)
{
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(router_logits_decode, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
#define TIE_RT_ATTR(A, B, ...)                                                                                                               \
	{                                                                                                                                    \
		using C = __VA_ARGS__;                                                                                                       \
		TIE_CUDA_TRY(c, cudaFuncSetAttribute(router_batch<C, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));         \
		if constexpr (C::NORM)                                                                                                       \
			TIE_CUDA_TRY(c, cudaFuncSetAttribute(router_batch<C, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, RT_NORM_SMEM)); \
	}
	TIE_RT_TILES(TIE_RT_ATTR)
#undef TIE_RT_ATTR
	return TIE_CUDA_OK;
}

// Plain F32 mat-vec over the first n_rows rows of w (the math_dispatch F32 row), one vector.
int launch_router_rows(tie_cuda_ctx *c, const float *x, const float *w, int n_rows, int in_dim, float *out)
{
	size_t smem = ((size_t)in_dim + (size_t)(in_dim + 8)) * sizeof(float);
	if (smem > 200 * 1024)
		return TIE_CUDA_ENOTSUP;
	router_logits_decode<<<n_rows, 64, smem, c->stream>>>(x, w, nullptr, out, 1, in_dim, n_rows);
	TIE_CUDA_LAUNCHED(c);
	return TIE_CUDA_OK;
}

}  // namespace tie

// ---------------------------------------------------------------------------------------------
// Routing without any allocation.
//
// Some hosts of this library may not allocate device memory when they call it: a serving loop
// that forbids allocator calls once start-up is over, or an embedding application that gives the
// library a fixed memory budget and no allocator.  For them the logits scratch of the router lives in the
// library image itself: a file-scope __device__ array, present once on every GPU that loads the
// library, for as long as the process lives.
//
// TIE_ROUTE_NOALLOC_MAX_TOKENS x TIE_ROUTE_NOALLOC_MAX_EXPERTS floats = 64 KiB per GPU.
constexpr int TIE_ROUTE_NOALLOC_MAX_TOKENS = 64;
constexpr int TIE_ROUTE_NOALLOC_MAX_EXPERTS = 256;
static __device__ __align__(256) float g_route_scratch[TIE_ROUTE_NOALLOC_MAX_TOKENS * TIE_ROUTE_NOALLOC_MAX_EXPERTS];

namespace {
constexpr int NOALLOC_MAX_DEVICES = 64;
float *g_route_scratch_addr[NOALLOC_MAX_DEVICES] = {nullptr};  // device address of the array, per device
std::mutex g_route_scratch_mutex;			       // first calls of several host threads set up one at a time
}

extern "C" int tie_cuda_route_noalloc(const float *x_dev, const float *router_w_dev, const float *router_bias_dev, int n_tokens,
				      int hidden, int n_expert, int top_k, int *topk_idx_dev, float *topk_w_dev, void *cuda_stream)
{
	using namespace tie;
	if (!x_dev || !router_w_dev || !topk_idx_dev || !topk_w_dev || n_tokens <= 0 || hidden <= 0 || hidden % 8 || n_expert <= 0 ||
	    n_expert % 16 || top_k <= 0 || top_k > MAX_TOP_K || top_k > n_expert)
		return TIE_CUDA_EINVAL;
	// the kernels read x and the router matrix with 128-bit loads: an address that is not a
	// multiple of 16 bytes would be a misaligned-address fault on the device, so it is refused here
	if ((reinterpret_cast<uintptr_t>(x_dev) | reinterpret_cast<uintptr_t>(router_w_dev)) & 15u)
		return TIE_CUDA_EINVAL;
	if ((reinterpret_cast<uintptr_t>(topk_idx_dev) | reinterpret_cast<uintptr_t>(topk_w_dev) |
	     reinterpret_cast<uintptr_t>(router_bias_dev)) & 3u)
		return TIE_CUDA_EINVAL;
	if (n_tokens > TIE_ROUTE_NOALLOC_MAX_TOKENS || n_expert > TIE_ROUTE_NOALLOC_MAX_EXPERTS)
		return TIE_CUDA_ETOOBIG;
	const size_t smem = ((size_t)hidden + (size_t)n_tokens * (hidden + 8)) * sizeof(float);
	if (n_tokens <= 8 && smem > 200 * 1024)
		return TIE_CUDA_ETOOBIG;
	int dev = -1;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES)
		return TIE_CUDA_ENODEV;
	std::unique_lock<std::mutex> setup_lock(g_route_scratch_mutex);
	if (!g_route_scratch_addr[dev]) {
		// First call on this device: resolve the array's DEVICE address.  In host code the name
		// g_route_scratch is only a handle for the runtime, not an address a kernel can use.
		// (Host threads that make their first call at the same time take turns here; the lock
		// orders the set-up only, not the kernels: overlapping calls still race on the array.)
		float *p = nullptr;
		if (cudaGetSymbolAddress(reinterpret_cast<void **>(&p), g_route_scratch) != cudaSuccess || !p) {
			cudaGetLastError();
			return TIE_CUDA_ECUDA;
		}
		if (cudaFuncSetAttribute(router_logits_decode, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) !=
		    cudaSuccess) {
			cudaGetLastError();
			return TIE_CUDA_ECUDA;
		}
		g_route_scratch_addr[dev] = p;
	}
	float *logits = g_route_scratch_addr[dev];
	setup_lock.unlock();
	cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
	if (n_tokens <= 8) {
		router_logits_decode<<<n_expert, 64, smem, st>>>(x_dev, router_w_dev, router_bias_dev, logits, n_tokens, hidden, n_expert);
	} else {
		constexpr int TT = 8, EPC = 16;
		if (hidden % 256)
			return TIE_CUDA_EINVAL;
		dim3 grid((n_tokens + TT - 1) / TT, n_expert / EPC);
		router_logits_tile<TT, EPC, 256><<<grid, EPC * 8, 0, st>>>(x_dev, router_w_dev, router_bias_dev, logits, n_tokens, hidden,
									      n_expert);
	}
	if (cudaGetLastError() != cudaSuccess)
		return TIE_CUDA_ECUDA;
	router_topk<<<(n_tokens + 3) / 4, 128, 0, st>>>(logits, n_tokens, n_expert, top_k, topk_idx_dev, topk_w_dev);
	if (cudaGetLastError() != cudaSuccess)
		return TIE_CUDA_ECUDA;
	return TIE_CUDA_OK;
}
