// Decode and small batches (up to 7 tokens of this model's shape): the expert mat-vecs of every
// (token, slot) row on its own — no dispatch sort, no grouping — with the exact mma.sync products of
// mma_dot.cuh.
//
// Reference: process_expert_task (engine.c:916-964) for the selected experts of a token and the
// weighted combine (model_qwen3.c:458-467).
//
//   decode_gate_up       CTA = (a run of 16-row tiles, (token, slot)), warp = one super-block of the input row:
//                        gate and up products, summed over the warps -> SwiGLU -> h
//   decode_down_combine  CTA = (16 output rows, token), warp = one slot: the packed rows of all slots are
//                        requested (one bulk copy per slot) before the wait for h; a warp's super-blocks add up in
//                        order, the slots are combined as acc = fma(w_j, row_j, acc), j ascending from
//                        zero — the reference's combine — so no per-slot output and no combine pass exist.
//
// What bounds it: at 1-4 tokens latency (three dependent launches, 2-3 us each), above that the expansion of
// the packed weights (330 instructions per warp for 16 rows x 256 Q4_K weights, loads and all; 600 for Q6_K, and 150 for the
// image of h).  Rows that share an expert expand it once each.
#include "common.cuh"
#include "kernels.cuh"
#include "mma_dot.cuh"
#include "tc_ptx.cuh"
#include "decode_common.cuh"

namespace tie {

constexpr int DEC_MAX_NB = 8;  // super-blocks per row

// Sum of a row's products over its super-blocks, in order (decode_fused.cu adds in the same order).
// A CTA walks n_tiles row tiles of its slot: the image of x is made once, a matrix's next tile is loaded into the
// registers that its products have just left and lands under the other matrix's, and one more warp adds up a
// tile and stores h while the others are at the next.
// A block of 3 / 4 / 6 tokens 46.2 / 58.6 / 69.7 -> 44.4 / 57.2 / 64.6 us against a CTA per tile (4 tokens: 53 MB in 16 us;
// the pipes are 20 - 45 % busy, the warps wait for one another, for loads and for the products).
template <WKind KIND>
__global__ void __launch_bounds__((DEC_MAX_NB + 1) * 32, 2)
decode_gate_up(const uint8_t *__restrict__ wg, const uint8_t *__restrict__ wu, size_t expert_stride, int rows_per_expert, int nb, int n_tiles,
	       const float *__restrict__ x, int top_k, const int *__restrict__ topk_idx, float *__restrict__ h, int first_expert,
	       int n_local, const float *__restrict__ silu, unsigned *__restrict__ status, int n_expert_all)
{
	__shared__ __align__(16) uint8_t img[DEC_MAX_NB][XImage<KIND>::BYTES];
	__shared__ float red[2][DEC_MAX_NB][2][16];
	const int slot = blockIdx.y;  // (token, j)
	const int r0 = blockIdx.x * n_tiles * 16, r1 = min(r0 + n_tiles * 16, rows_per_expert);
	pdl_wait();	// the router's top-k (and x) are visible from here on
	pdl_trigger();	// the down kernel may start fetching its weights
	const int ge = topk_idx[slot];
	const int le = ge - first_expert;
	if (le < 0 || le >= n_local) {
		// n_expert_all > 0 (expert-parallel decode on replicated tokens): the slot belongs to another rank
		if (!(n_expert_all > 0 && ge >= 0 && ge < n_expert_all) && threadIdx.x == 0 && blockIdx.x == 0)
			atomicOr(status, ST_BAD_EXPERT);
		return;
	}
	const int lane = threadIdx.x & 31, b = threadIdx.x >> 5;
	if (b == nb) {
		for (int r = r0, buf = 0; r < r1; r += 16, buf ^= 1) {
			__syncthreads();
			float sum = red[buf][0][lane >> 4][lane & 15];
			for (int i = 1; i < nb; i++)
				sum = __fadd_rn(sum, red[buf][i][lane >> 4][lane & 15]);
			const float up = __shfl_down_sync(0xffffffffu, sum, 16);
			if (lane < 16)
				h[(size_t)slot * rows_per_expert + r + lane] = swiglu_lut(silu, sum, up);
		}
		return;
	}
	wg += (size_t)le * expert_stride;
	wu += (size_t)le * expert_stride;
	MmaRows<KIND> g, u;
	g.load(wg + tile_offset<KIND>(nb, r0), nb, b, lane);
	u.load(wu + tile_offset<KIND>(nb, r0), nb, b, lane);
	const float4 *xp = reinterpret_cast<const float4 *>(x + (size_t)(slot / top_k) * nb * QK_K + b * QK_K) + 2 * lane;
	const float4 x0 = xp[0], x1 = xp[1];
	const float v[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
	const float inv = x_image<KIND>(v, img[b], lane);
	for (int r = r0, buf = 0; r < r1; r += 16, buf ^= 1) {
		const bool more = r + 16 < r1;
		float2 p = dot_one(g, one_row<KIND>(img[b], lane), lane), s = g.scale(inv);
		if (more)
			g.load(wg + tile_offset<KIND>(nb, r + 16), nb, b, lane);
		if ((lane & 3) == 0) {
			red[buf][b][0][lane >> 2] = p.x * s.x;
			red[buf][b][0][(lane >> 2) + 8] = p.y * s.y;
		}
		p = dot_one(u, one_row<KIND>(img[b], lane), lane);
		s = u.scale(inv);
		if (more)
			u.load(wu + tile_offset<KIND>(nb, r + 16), nb, b, lane);
		if ((lane & 3) == 0) {
			red[buf][b][1][lane >> 2] = p.x * s.x;
			red[buf][b][1][(lane >> 2) + 8] = p.y * s.y;
		}
		__syncthreads();
	}
}

// The product of slot j's 16 staged rows with its h row, in this warp: lane (g, t = 0, 1) ends up with rows g, g + 8.
// The row's next super-block is loaded under the products of the one before, and the tile is waited for (bar;
// false in ok: it never landed) when the first image is made.  (A block of 3 / 4 tokens 40.6 / 47.3 -> 39.1 / 46.5 us against
// all warps waiting for all tiles before their first load of h.)
template <WKind KIND>
__device__ __forceinline__ float2 down_rows(const uint8_t *tile, int nb, const float *hrow, uint8_t *img, int lane, uint32_t bar,
					    unsigned *status, bool &ok)
{
	float2 out = make_float2(0.f, 0.f);
	const float4 *hp = reinterpret_cast<const float4 *>(hrow) + 2 * lane;
	float4 h0 = hp[0], h1 = hp[1];
	ok = true;
	for (int b = 0; b < nb && ok; b++) {
		const float v[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
		if (b + 1 < nb) {
			hp += QK_K / 4;
			h0 = hp[0];
			h1 = hp[1];
		}
		const float inv = x_image<KIND>(v, img, lane);
		if (b == 0)
			ok = __all_sync(0xffffffffu, dec_wait(bar, status));
		MmaRows<KIND> w;
		w.load_smem(tile, nb, b, lane);
		const float2 r = dot_one(w, one_row<KIND>(img, lane), lane), s = w.scale(inv);
		out.x = __fmaf_rn(s.x, r.x, out.x);
		out.y = __fmaf_rn(s.y, r.y, out.y);
	}
	return out;
}

// CTAS: resident per SM.  Q4_K tiles leave room for a third CTA, at 80 registers instead of 96; launch_decode_down_combine
// says where it pays.
template <WKind KIND, int CTAS = 2>
__global__ void __launch_bounds__(MAX_TOP_K * 32, CTAS)
decode_down_combine(const uint8_t *__restrict__ wd, size_t expert_stride, int rows_per_expert, int nb, const float *__restrict__ h,
		    int top_k, const int *__restrict__ topk_idx, const float *__restrict__ topk_w, const float *__restrict__ residual,
		    float *__restrict__ out, int first_expert, int n_local, unsigned *__restrict__ status)
{
	extern __shared__ __align__(128) uint8_t dsm[];
	__shared__ __align__(16) uint8_t img[MAX_TOP_K][XImage<KIND>::BYTES];
	__shared__ uint64_t bar[MAX_TOP_K];  // one per slot: a slot's rows are reduced as soon as its tile lands
	__shared__ float red[MAX_TOP_K][16];
	__shared__ int s_bad;
	const int t = blockIdx.y, r0 = blockIdx.x * 16;
	const uint32_t tile_bytes = (uint32_t)tile_offset<KIND>(nb, 16);
	const int lane = threadIdx.x & 31, j = threadIdx.x >> 5;
	// The selection was written two kernels ago and the weights never change: the tiles of all the
	// token's experts are requested BEFORE waiting for the gate/up kernel, so this fetch overlaps it.
	if (threadIdx.x == 0) {
		for (int k = 0; k < top_k; k++)
			ptx::mbar_init(ptx::smem_u32(&bar[k]), 1);
		ptx::fence_barrier_init();
		ptx::fence_proxy_async_smem();
		s_bad = 0;
	}
	__syncthreads();
	if (lane == 0) {
		const int le = topk_idx[t * top_k + j] - first_expert;
		if (le < 0 || le >= n_local) {
			s_bad = 1;
			if (blockIdx.x == 0)
				atomicOr(status, ST_BAD_EXPERT);
		} else {
			const uint32_t ba = ptx::smem_u32(&bar[j]);
			ptx::mbar_arrive_expect_tx(ba, tile_bytes);
			bulk_g2s(ptx::smem_u32(dsm + (size_t)j * tile_bytes), wd + (size_t)le * expert_stride + tile_offset<KIND>(nb, r0), tile_bytes, ba);
		}
	}
	pdl_wait();  // h of the gate/up kernel is visible from here on
	const int le = topk_idx[t * top_k + j] - first_expert;
	bool ok = true;
	if (le >= 0 && le < n_local) {
		const float2 v = down_rows<KIND>(dsm + (size_t)j * tile_bytes, nb, h + (size_t)(t * top_k + j) * nb * QK_K, img[j], lane,
						 ptx::smem_u32(&bar[j]), status, ok);
		if ((lane & 3) == 0) {
			red[j][lane >> 2] = v.x;
			red[j][(lane >> 2) + 8] = v.y;
		}
	}
	if (!__syncthreads_and(ok) || s_bad)
		return;	 // (every tile that was requested has landed, or its wait has run out)
	if (threadIdx.x < 16) {
		float acc = 0.f;
		for (int k = 0; k < top_k; k++)
			acc = __fmaf_rn(topk_w[t * top_k + k], red[k][threadIdx.x], acc);  // model_qwen3.c:458-467, slot order, from zero
		const size_t at = (size_t)t * rows_per_expert + r0 + threadIdx.x;
		if (residual)
			acc = __fadd_rn(residual[at], acc);
		out[at] = acc;
	}
}

// Expert-parallel decode on replicated tokens: every rank has routed the same tokens to the same
// experts; this rank reduces the down rows of the slots whose expert it owns and stores each
// unweighted row value into the y rows (token, slot) of EVERY rank's region (plain stores over
// NVLink, 64 bytes per tile, slot and rank).  The combine (ep_combine_rows) then runs on every rank
// over all slots in slot order — the reference's order (model_qwen3.c:458-467), so the result is
// bit-identical to the one-GPU decode kernels.  A peer's y rows of the previous step may only be
// overwritten once that peer has started this step (its pub flag): the CTA waits for all pub
// flags first (bounded; they are words of this rank's own region).
template <WKind KIND>
__global__ void __launch_bounds__(MAX_TOP_K * 32, 2)
decode_down_peer(const uint8_t *__restrict__ wd, size_t expert_stride, int rows_per_expert, int nb, const float *__restrict__ h, int top_k,
		 const int *__restrict__ topk_idx, const EpView v, const unsigned *__restrict__ step_dev, long long budget, int first_expert,
		 int n_local, unsigned *__restrict__ status)
{
	extern __shared__ __align__(128) uint8_t dsm[];
	__shared__ __align__(16) uint8_t img[MAX_TOP_K][XImage<KIND>::BYTES];
	__shared__ uint64_t bar[MAX_TOP_K];
	const int t = blockIdx.y, r0 = blockIdx.x * 16;
	const uint32_t tile_bytes = (uint32_t)tile_offset<KIND>(nb, 16);
	const int lane = threadIdx.x & 31, j = threadIdx.x >> 5;
	if (threadIdx.x == 0) {
		for (int k = 0; k < top_k; k++)
			ptx::mbar_init(ptx::smem_u32(&bar[k]), 1);
		ptx::fence_barrier_init();
		ptx::fence_proxy_async_smem();
	}
	__syncthreads();
	const int ge = topk_idx[t * top_k + j], le = ge - first_expert;
	const bool bad = ge < 0 || ge >= v.n_expert, mine = !bad && le >= 0 && le < n_local;
	if (bad && lane == 0 && blockIdx.x == 0)
		atomicOr(status, ST_BAD_EXPERT);
	if (mine && lane == 0) {
		const uint32_t ba = ptx::smem_u32(&bar[j]);
		ptx::mbar_arrive_expect_tx(ba, tile_bytes);
		bulk_g2s(ptx::smem_u32(dsm + (size_t)j * tile_bytes), wd + (size_t)le * expert_stride + tile_offset<KIND>(nb, r0), tile_bytes, ba);
	}
	pdl_wait();  // h of the gate/up kernel is visible from here on
	// every rank has started this step: its y rows of the previous step are combined and may be overwritten
	const unsigned step = *step_dev;
	bool ok = true;
	if ((int)threadIdx.x < v.n_ranks) {
		const unsigned *flag = reinterpret_cast<const unsigned *>(v.peer[v.rank] + v.off_pub) + threadIdx.x;
		const long long t0 = clock64();
		for (;;) {
			unsigned f;
			asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(f) : "l"(flag) : "memory");
			if ((int)(f - step) >= 0)
				break;
			if (clock64() - t0 > budget) {
				ok = false;
				break;
			}
			__nanosleep(100);
		}
	}
	ok = __syncthreads_and(ok);
	if (!ok && threadIdx.x == 0)
		atomicOr(status, ST_WAIT_TIMEOUT);
	// (a wait for the copies in any case: nobody leaves with copies in flight)
	const bool landed = !mine || dec_wait(ptx::smem_u32(&bar[j]), status);
	if (!__syncthreads_and(landed) || !ok || __syncthreads_or(bad))
		return;
	if (!mine)
		return;
	bool there;
	const float2 r = down_rows<KIND>(dsm + (size_t)j * tile_bytes, nb, h + (size_t)(t * top_k + j) * nb * QK_K, img[j], lane,
					 ptx::smem_u32(&bar[j]), status, there);
	// lanes of t = 0 hold row g, their neighbours of t = 1 store row g + 8
	if ((lane & 3) < 2) {
		const size_t at = (size_t)(t * top_k + j) * rows_per_expert + r0 + (lane >> 2) + 8 * (lane & 1);
		const float val = lane & 1 ? r.y : r.x;
		for (int k = 0; k < v.n_ranks; k++)
			reinterpret_cast<float *>(v.peer[k] + v.off_y)[at] = val;
	}
}

// ---- host side ----

constexpr int DEC_MAX_SMEM = 200 * 1024;

static size_t dec_down_smem(const Layer &L, int top_k)
{
	const int nb = L.down.k / QK_K;
	return (size_t)top_k * (L.down.kind == W_Q4K ? tile_offset<W_Q4K>(nb, 16) : tile_offset<W_Q6K_R8>(nb, 16));
}

bool decode_supported(const tie_cuda_ctx *c, const Layer &L, int n_tokens)
{
	// (decode_group.cu takes what it is faster at from here)
	const int n_rows = n_tokens * c->cfg.top_k;
	return (n_tokens <= 4 || 2 * n_rows <= c->n_local) && n_rows <= 65535 && L.gate.kind == L.up.kind &&
	       L.gate.k <= DEC_MAX_NB * QK_K && L.gate.rows % 16 == 0 && L.down.rows % 16 == 0 && L.down.k <= DEC_MAX_NB * QK_K &&
	       dec_down_smem(L, c->cfg.top_k) <= (size_t)DEC_MAX_SMEM;
}

// Opt-in shared-memory sizes, once per context.
int decode_setup(tie_cuda_ctx *c)
{
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(decode_down_combine<W_Q4K, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, DEC_MAX_SMEM));
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(decode_down_combine<W_Q4K>, cudaFuncAttributeMaxDynamicSharedMemorySize, DEC_MAX_SMEM));
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(decode_down_combine<W_Q6K_R8>, cudaFuncAttributeMaxDynamicSharedMemorySize, DEC_MAX_SMEM));
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(decode_down_peer<W_Q4K>, cudaFuncAttributeMaxDynamicSharedMemorySize, DEC_MAX_SMEM));
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(decode_down_peer<W_Q6K_R8>, cudaFuncAttributeMaxDynamicSharedMemorySize, DEC_MAX_SMEM));
	return TIE_CUDA_OK;
}

// x [n_tokens][hidden] -> h [(token, slot)][ffn] (sorted nowhere: rows are the top-k entries themselves)
int launch_decode_gate_up(tie_cuda_ctx *c, const Layer &L, const float *x, int n_tokens, bool foreign_slots_ok)
{
	const int n_rows = n_tokens * c->cfg.top_k, nb = L.gate.k / QK_K;
	auto kern = L.gate.kind == W_Q4K ? decode_gate_up<W_Q4K> : decode_gate_up<W_Q6K_R8>;
	// as many tiles a CTA as bring the grid to one wave of two CTAs per SM
	const int tiles = L.gate.rows / 16, n_tiles = (tiles * n_rows + 2 * c->sm_count - 1) / (2 * c->sm_count);
	return launch_kernel(c, true, 1, kern, dim3((tiles + n_tiles - 1) / n_tiles, n_rows), 32 * (nb + 1), 0, L.gate.ptr, L.up.ptr,
			  L.gate.expert_stride, L.gate.rows, nb, n_tiles, x,
			  c->cfg.top_k, c->s.topk_idx, c->s.h, c->first_expert, c->n_local, c->silu, c->s.status,
			  foreign_slots_ok ? c->cfg.n_expert : 0);
}

// h -> out [n_tokens][hidden] (= residual + sum_j w_j * down_j(h_j))
int launch_decode_down_combine(tie_cuda_ctx *c, const Layer &L, int n_tokens, const float *residual, float *out)
{
	const int top_k = c->cfg.top_k, nb = L.down.k / QK_K;
	// Q4_K: three CTAs per SM where that saves a wave (3 and 5 - 7 tokens of this model).  Blocks with such a down tensor, at 3 / 5
	// / 6 / 7 tokens: 37.8 / 51.4 / 55.8 / 63.0 -> 37.6 / 50.0 / 54.7 / 61.9 us; at 2 (one wave) 32.3 -> 33.3, at 4 (two) equal, so
	// not there.
	const long long grid = (long long)(L.down.rows / 16) * n_tokens, two = 2 * c->sm_count, three = 3 * c->sm_count;
	const bool many = (grid + three - 1) / three < (grid + two - 1) / two;
	auto kern = L.down.kind != W_Q4K ? decode_down_combine<W_Q6K_R8> : many ? decode_down_combine<W_Q4K, 3> : decode_down_combine<W_Q4K>;
	return launch_kernel(c, true, 1, kern, dim3(L.down.rows / 16, n_tokens), 32 * top_k, dec_down_smem(L, top_k), L.down.ptr, L.down.expert_stride,
			  L.down.rows, nb, c->s.h, top_k, c->s.topk_idx, c->s.topk_w, residual, out, c->first_expert, c->n_local, c->s.status);
}

// h (local slots) -> the y rows of every rank's region (expert-parallel decode on replicated tokens)
int launch_decode_down_peer(tie_cuda_ctx *c, const Layer &L, int n_tokens)
{
	const int top_k = c->cfg.top_k, nb = L.down.k / QK_K;
	auto kern = L.down.kind == W_Q4K ? decode_down_peer<W_Q4K> : decode_down_peer<W_Q6K_R8>;
	return launch_kernel(c, true, 1, kern, dim3(L.down.rows / 16, n_tokens), 32 * top_k, dec_down_smem(L, top_k), L.down.ptr, L.down.expert_stride,
			  L.down.rows, nb, c->s.h, top_k, c->s.topk_idx, c->ep.view, c->ep.step_dev, c->ep.wait_cycles, c->first_expert,
			  c->n_local, c->s.status);
}

}  // namespace tie
