// Small batches between the per-row decode kernels and the grouped tensor-core products (8 to 31 tokens of this
// model's shape): rows that share an expert share the expansion of its packed weights, on the exact mma.sync
// products of mma_dot.cuh, so that a row has the bits that the per-row kernels (decode.cu) give it.
//
// Reference: process_expert_task (engine.c:916-964) for the selected experts of a batch's tokens.
//
//   group_gate_up   item = (group of up to four rows of one expert, 16 output rows), warp = one super-block of the gate
//                   or of the up rows; one more warp adds the super-blocks up -> SwiGLU -> h
//   group_down      item = the same over the down rows, a warp per item -> y [(token, slot)][hidden]; combine_rows
//                   (misc.cu) adds the slots up
//
// Every CTA makes the list of groups from the selection itself (a microsecond; no sort, no further launch) and takes its
// share of the items, in one wave.
//
// What bounds it: the expansion (about 400 instructions per warp for 16 rows x 256 Q4_K weights with their loads and
// hand-offs, 600 for Q6_K), which an expert's every fourth row pays again.
// A block of 9 / 13 / 20 / 31 tokens with Q6_K down: 80 / 94 / 115 / 139 us (in groups of two rows 77 / 93 / 121 / 155); row by
// row 80 / 126 / 181 / 249; the grouped tensor-core products, which hold activations in 22 bits, 85 / 96 / 114 / 127.
#include "common.cuh"
#include "kernels.cuh"
#include "mma_dot.cuh"
#include "tc_ptx.cuh"
#include "decode_common.cuh"

namespace tie {

constexpr int DG_ROWS = 4;	   // rows of a group: the parts of two fit the eight columns of an MMA, and two MMAs share a fragment
constexpr int DG_MAX_TOKENS = 32;  // a bit each
constexpr int DG_MAX_ROWS = 256, DG_MAX_EXPERTS = 256;
constexpr int DG_MAX_NB = 8;  // super-blocks per row
constexpr int DG_DOWN_WARPS = 8;
// Tiles of gate/up products between the warps that make them and the one that adds them up (4: 1 % slower; a barrier per
// tile, or the last warp at a tile adding it up itself: 15 - 25 % slower).
constexpr int DG_STAGES = 8;

// What a tile of a group of one or two rows costs, and of three or four (the second MMAs and their operands).  31 tokens with 4 : 7 /
// 2 : 3 / 3 : 4 / 5 : 6: 153 / 143 / 139 / 134 us without the norm.
constexpr int DG_COST1 = 5, DG_COST2 = 6;

// The rows of a call by expert, in token order, cut in groups of DG_ROWS.
struct GroupList {
	unsigned tokens[DG_MAX_EXPERTS];  // per expert: who selected it
	uint8_t id[DG_MAX_EXPERTS][DG_MAX_TOKENS / DG_ROWS];
	uint8_t expert[DG_MAX_ROWS], size[DG_MAX_ROWS];
	uint8_t row[DG_MAX_ROWS][DG_ROWS];
	int cost[DG_MAX_ROWS];	// of a tile of every group before this one
	int first, last;	// this CTA's items, item = group * tiles + tile

	// By all threads of a CTA.  An expert occurs at most once among a token's slots (top-k), so a row's place among
	// its expert's is the number of earlier tokens that selected the expert.
	__device__ __forceinline__ void make(const int *topk_idx, int n_rows, int top_k, int first_expert, int n_local, int tiles,
					     unsigned *status)
	{
		for (int e = threadIdx.x; e < n_local; e += blockDim.x)
			tokens[e] = 0;
		__syncthreads();
		for (int i = threadIdx.x; i < n_rows; i += blockDim.x) {
			const int e = topk_idx[i] - first_expert;
			if (e >= 0 && e < n_local)
				atomicOr(&tokens[e], 1u << (i / top_k));
			else if (blockIdx.x == 0)
				atomicOr(status, ST_BAD_EXPERT);
		}
		__syncthreads();
		if (threadIdx.x < 32) {
			int made = 0, total = 0;
			for (int i0 = 0; i0 < n_rows; i0 += 32) {
				const int i = i0 + threadIdx.x, e = i < n_rows ? topk_idx[i] - first_expert : -1;
				const bool on = e >= 0 && e < n_local;
				const int place = on ? __popc(tokens[e] & ((1u << (i / top_k)) - 1u)) : 0;
				const bool lead = on && place % DG_ROWS == 0;
				const int size_here = lead ? min(DG_ROWS, __popc(tokens[e]) - place) : 0;
				const unsigned firsts = __ballot_sync(0xffffffffu, lead), wide = __ballot_sync(0xffffffffu, size_here > 2);
				if (lead) {
					const unsigned below = (1u << threadIdx.x) - 1u;
					const int g = made + __popc(firsts & below);
					id[e][place / DG_ROWS] = (uint8_t)g;
					expert[g] = (uint8_t)e;
					size[g] = (uint8_t)size_here;
					cost[g] = total + DG_COST1 * __popc(firsts & below) + (DG_COST2 - DG_COST1) * __popc(wide & below);
				}
				made += __popc(firsts);
				total += DG_COST1 * __popc(firsts) + (DG_COST2 - DG_COST1) * __popc(wide);
				__syncwarp();
				if (on)	 // (the group's first row is an earlier one: same or earlier round)
					row[id[e][place / DG_ROWS]][place % DG_ROWS] = (uint8_t)i;
			}
			// the CTA's share of the items: what starts between two equal steps of their cost
			int bound[2];
			for (int k = 0; k < 2; k++) {
				const int c = (int)((long long)total * tiles * (blockIdx.x + k) / gridDim.x);
				int g = -1;  // the last group that starts at or before c
				for (int g0 = 0; g0 < made; g0 += 32)
					g += __popc(__ballot_sync(0xffffffffu, g0 + (int)threadIdx.x < made && cost[g0 + threadIdx.x] * tiles <= c));
				const int w = g < 0 ? 1 : (size[g] > 2 ? DG_COST2 : DG_COST1);
				bound[k] = g < 0 ? 0 : g * tiles + min(tiles, (c - cost[g] * tiles + w - 1) / w);
			}
			if (threadIdx.x == 0) {
				first = bound[0];
				last = bound[1];
			}
		}
		__syncthreads();
	}
};

// One super-block of a 16-row tile, 16 bytes a piece: rows of a chunk are contiguous (144 or 208 bytes: the fragment
// loads have no bank conflicts).
template <WKind KIND>
struct ChunkCopy {
	static constexpr int ROW = KIND == W_Q4K ? Q4K_BYTES : Q6K_RECORD, PIECES = ROW / 16, BYTES = 16 * ROW;
	static constexpr int PER_LANE = (16 * PIECES + 31) / 32;
	uint32_t from[PER_LANE];
	__device__ __forceinline__ void init(int nb, int b, int lane)
	{
#pragma unroll
		for (int k = 0; k < PER_LANE; k++) {
			const int i = lane + 32 * k, row = i / PIECES, piece = i - row * PIECES;
			from[k] = (uint32_t)(KIND == W_Q4K ? (row * nb + b) * Q4K_BYTES
							   : (row >> 3) * (int)q6k_r8_group_bytes(nb) + ((row & 7) * nb + b) * Q6K_RECORD) +
				  16 * piece;
		}
	}
	__device__ __forceinline__ void start(uint32_t dst, const uint8_t *tile, int lane) const
	{
#pragma unroll
		for (int k = 0; k < PER_LANE; k++)
			if (32 * (k + 1) <= 16 * PIECES || lane + 32 * k < 16 * PIECES)
				ptx::cp_async16(dst + 16 * (lane + 32 * k), tile + from[k]);
	}
};

template <WKind KIND>
struct GuCfg {
	static constexpr int IMG = DG_ROWS * XImage<KIND>::BYTES, CHUNKS = 2 * ChunkCopy<KIND>::BYTES;
	static constexpr int RED = DG_STAGES * DG_ROWS * 16 * (int)sizeof(float);  // per warp
	static size_t smem(int nb) { return (size_t)nb * (IMG + 2 * (CHUNKS + RED)); }
};

// The tiles of a run of items, one after the other.
template <WKind KIND>
struct TileCursor {
	const uint8_t *tile;
	int g, left;  // group; its tiles from this one on
	__device__ __forceinline__ void set(const GroupList &gl, const uint8_t *w, size_t expert_stride, int nb, int tiles, int it)
	{
		g = it / tiles;
		left = (g + 1) * tiles - it;
		tile = w + (size_t)gl.expert[g] * expert_stride + tile_offset<KIND>(nb, (tiles - left) * 16);
	}
	// (there is a next tile)
	__device__ __forceinline__ void next(const GroupList &gl, const uint8_t *w, size_t expert_stride, int nb, int tiles)
	{
		if (--left) {
			tile += tile_offset<KIND>(nb, 16);
		} else {
			tile = w + (size_t)gl.expert[++g] * expert_stride;
			left = tiles;
		}
	}
};

// h of a group's rows (ROWS at most) from a tile's products p, which lie [gate, up by half-warp][super-block][row][16]: all rows
// together, as one after the other their sums and table look-ups take longer than a tile (31 tokens 159 -> 139 us).
template <int ROWS>
__device__ __forceinline__ void group_h(const float *p, int nb, int n, const uint8_t *row, float *h, int rows_per_expert, const float *silu, int lane)
{
	float sum[ROWS], act[ROWS];
#pragma unroll
	for (int m = 0; m < ROWS; m++)
		sum[m] = p[m * 16];
	for (int i = 1; i < nb; i++)
#pragma unroll
		for (int m = 0; m < ROWS; m++)
			sum[m] = __fadd_rn(sum[m], p[(i * DG_ROWS + m) * 16]);
#pragma unroll
	for (int m = 0; m < ROWS; m++) {
		const float up = __shfl_down_sync(0xffffffffu, sum[m], 16);
		act[m] = m < n ? swiglu_lut(silu, sum[m], up) : 0.f;
	}
	if (lane < 16)
#pragma unroll
		for (int m = 0; m < ROWS; m++)
			if (m < n)
				h[(size_t)row[m] * rows_per_expert] = act[m];
}

template <WKind KIND>
__global__ void __launch_bounds__((2 * DG_MAX_NB + 1) * 32, 1)
group_gate_up(const uint8_t *__restrict__ wg, const uint8_t *__restrict__ wu, size_t expert_stride, int rows_per_expert, int nb,
	      const float *__restrict__ x, int top_k, int n_rows, const int *__restrict__ topk_idx, float *__restrict__ h, int first_expert,
	      int n_local, const float *__restrict__ silu, unsigned *__restrict__ status)
{
	using C = GuCfg<KIND>;
	extern __shared__ __align__(128) uint8_t dsm[];	 // images of x [super-block][row of the group], chunks [warp][slot], products
	__shared__ GroupList gl;
	__shared__ float inv[DG_MAX_NB][DG_ROWS];
	__shared__ uint64_t full[DG_STAGES], empty[DG_STAGES];
	__shared__ __align__(16) uint8_t zeros[XImage<KIND>::PART];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tiles = rows_per_expert / 16;
	float *red = reinterpret_cast<float *>(dsm + (size_t)nb * (C::IMG + 2 * C::CHUNKS));  // [stage][gate, up][super-block][row][16]
	constexpr int RED_ROWS = DG_ROWS * 16;
	if (threadIdx.x == 0) {
		for (int i = 0; i < DG_STAGES; i++) {
			ptx::mbar_init(ptx::smem_u32(&full[i]), 2 * nb);
			ptx::mbar_init(ptx::smem_u32(&empty[i]), 1);
		}
		ptx::fence_barrier_init();
	}
	for (int i = threadIdx.x; i < XImage<KIND>::PART / 4; i += blockDim.x)
		reinterpret_cast<uint32_t *>(zeros)[i] = 0;
	pdl_wait();	// the router's top-k (and x) are visible from here on
	pdl_trigger();	// the down kernel may make its list
	gl.make(topk_idx, n_rows, top_k, first_expert, n_local, tiles, status);
	const int2 items = make_int2(gl.first, gl.last);
	bool ok = true;	 // (a wait that ran out: on without waiting, the status word is set)
	if (warp == 2 * nb) {
		int g = items.x / tiles, r0 = (items.x - g * tiles) * 16, st = 0;
		uint32_t parity = 0;
		for (int it = items.x; it < items.y; it++) {
			const int n = gl.size[g];
			ok = ok && dec_wait(ptx::smem_u32(&full[st]), status, parity);
			const float *p = red + ((size_t)st * 2 + (lane >> 4)) * nb * RED_ROWS + (lane & 15);
			float *hp = h + r0 + lane;
			if (n <= 2)
				group_h<2>(p, nb, n, gl.row[g], hp, rows_per_expert, silu, lane);
			else
				group_h<DG_ROWS>(p, nb, n, gl.row[g], hp, rows_per_expert, silu, lane);
			__syncwarp();
			if (lane == 0)
				ptx::mbar_arrive(ptx::smem_u32(&empty[st]));
			if (++st == DG_STAGES) {
				st = 0;
				parity ^= 1;
			}
			if ((r0 += 16) == rows_per_expert) {
				r0 = 0;
				g++;
			}
		}
		return;
	}
	const int mat = warp >= nb, b = mat ? warp - nb : warp;
	const uint8_t *w = mat ? wu : wg;
	uint8_t *img = dsm + b * C::IMG, *chunks = dsm + (size_t)nb * C::IMG + warp * C::CHUNKS;
	const uint32_t slots = ptx::smem_u32(chunks);
	ChunkCopy<KIND> copy;
	copy.init(nb, b, lane);
	TileCursor<KIND> now;
	if (items.x < items.y) {
		now.set(gl, w, expert_stride, nb, tiles, items.x);
		copy.start(slots, now.tile, lane);
	}
	ptx::cp_async_commit();
	int n = 0, slot = 0, st = 0;
	uint32_t parity = 1;  // of the stage: the first round finds every one empty
	MmaCol<true> col[2];
	for (int it = items.x; it < items.y; it++) {
		if (it == items.x || now.left == tiles) {  // another group: the gate and the up warp of a super-block make its images together
			n = gl.size[now.g];
			asm volatile("bar.sync %0, 64;" ::"r"(1 + b) : "memory");
			for (int m = mat; m < n; m += 2) {
				const float4 *xp = reinterpret_cast<const float4 *>(x + (size_t)(gl.row[now.g][m] / top_k) * nb * QK_K + b * QK_K) + 2 * lane;
				const float4 x0 = xp[0], x1 = xp[1];
				const float v[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
				const float f = x_image<KIND>(v, img + m * XImage<KIND>::BYTES, lane);
				if (lane == 0)
					inv[b][m] = f;
			}
			asm volatile("bar.sync %0, 64;" ::"r"(1 + b) : "memory");
			col[0] = two_rows<KIND>(img, XImage<KIND>::BYTES, 0, n, zeros, lane);
			col[1] = two_rows<KIND>(img, XImage<KIND>::BYTES, 2, n, zeros, lane);
		}
		ptx::cp_async_wait<0>();
		__syncwarp();  // (everybody's pieces are there, and everybody is done with the other slot)
		TileCursor<KIND> next = now;
		if (it + 1 < items.y) {
			next.next(gl, w, expert_stride, nb, tiles);
			copy.start(slots + (slot ^ 1) * ChunkCopy<KIND>::BYTES, next.tile, lane);
		}
		ptx::cp_async_commit();
		MmaRows<KIND> wr;
		wr.load_chunk(chunks + slot * ChunkCopy<KIND>::BYTES, now.tile, nb, b, lane);
		ok = ok && dec_wait(ptx::smem_u32(&empty[st]), status, parity);
		float *dst = red + ((size_t)(st * 2 + mat) * nb + b) * RED_ROWS;
		float2 r[2];
		if (n > 2)
			wr.dot(col, lane, r);
		else
			r[0] = r[1] = dot_one(wr, col[0], lane);
		if ((lane & 1) == 0) {	// lanes t = 0 of a quad have the first row of a pair, t = 2 the second
#pragma unroll
			for (int p = 0; p < 2; p++) {
				const int m = 2 * p + (lane >> 1 & 1);
				if (m < n) {
					const float2 f = wr.scale(inv[b][m]);
					dst[m * 16 + (lane >> 2)] = r[p].x * f.x;
					dst[m * 16 + (lane >> 2) + 8] = r[p].y * f.y;
				}
			}
		}
		__syncwarp();
		if (lane == 0)
			ptx::mbar_arrive(ptx::smem_u32(&full[st]));
		slot ^= 1;
		if (++st == DG_STAGES) {
			st = 0;
			parity ^= 1;
		}
		now = next;
	}
	ptx::cp_async_wait<0>();
}

// A warp owns one staged tile: the next one is requested as soon as the last super-block's weights are in registers
// and arrives under their products.  (Three CTAs per SM for Q4_K, at 80 registers: 13 tokens 85.4 -> 88.6 us.)
template <WKind KIND>
__global__ void __launch_bounds__(DG_DOWN_WARPS * 32, 2)
group_down(const uint8_t *__restrict__ wd, size_t expert_stride, int rows_per_expert, int nb, const float *__restrict__ h, int top_k, int n_rows,
	   const int *__restrict__ topk_idx, float *__restrict__ y, int first_expert, int n_local, unsigned *__restrict__ status)
{
	extern __shared__ __align__(128) uint8_t dsm[];	 // a tile per warp, then the images of h: [row of the group][super-block]
	__shared__ GroupList gl;
	__shared__ float inv[DG_ROWS][DG_MAX_NB];
	__shared__ uint64_t bar[DG_DOWN_WARPS];
	__shared__ __align__(16) uint8_t zeros[XImage<KIND>::PART];
	constexpr int STRIDE = XImage<KIND>::BYTES;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tiles = rows_per_expert / 16;
	const uint32_t tile_bytes = (uint32_t)tile_offset<KIND>(nb, 16), ba = ptx::smem_u32(&bar[warp]);
	uint8_t *tile = dsm + (size_t)warp * tile_bytes, *img = dsm + (size_t)DG_DOWN_WARPS * tile_bytes;
	if (lane == 0) {
		ptx::mbar_init(ba, 1);
		ptx::fence_barrier_init();
		ptx::fence_proxy_async_smem();
	}
	for (int i = threadIdx.x; i < XImage<KIND>::PART / 4; i += blockDim.x)
		reinterpret_cast<uint32_t *>(zeros)[i] = 0;
	// (the selection was written two kernels ago, the weights never change: neither waits for h)
	gl.make(topk_idx, n_rows, top_k, first_expert, n_local, tiles, status);
	const int2 items = make_int2(gl.first, gl.last);
	auto request = [&](int it) {  // one lane
		const int g = it / tiles;
		ptx::mbar_arrive_expect_tx(ba, tile_bytes);
		bulk_g2s(ptx::smem_u32(tile), wd + (size_t)gl.expert[g] * expert_stride + tile_offset<KIND>(nb, (it - g * tiles) * 16), tile_bytes, ba);
	};
	// a warp takes every eighth of the CTA's items in a group, then of those in the next: end: where that group ends
	auto settle = [&](int &it, int &end) {
		while (it >= end && end < items.y) {
			it = end + warp;
			end = min(items.y, end + tiles);
		}
	};
	int it = items.x + warp, end = min(items.y, (items.x / tiles + 1) * tiles);
	settle(it, end);
	if (lane == 0 && it < items.y)
		request(it);
	const int m = lane >> 1 & 1;  // of a pair of the group's rows
	uint32_t parity = 0;
	bool ok = true;
	pdl_wait();  // h of the gate/up kernel is visible from here on
	pdl_trigger();	// (the combine comes as the last CTAs leave: a block of 13 tokens 87.3 -> 86.0 us; behind the grouped GEMM it costs 1 - 2 us)
	for (int s0 = items.x, s1; s0 < items.y; s0 = s1) {
		const int g = s0 / tiles, n = gl.size[g];
		s1 = min(items.y, (g + 1) * tiles);
		__syncthreads();  // (the images of the group before are done with)
		for (int j = warp; j < n * nb; j += DG_DOWN_WARPS) {
			const int k = j / nb, b = j - k * nb;
			const float4 *hp = reinterpret_cast<const float4 *>(h + ((size_t)gl.row[g][k] * nb + b) * QK_K) + 2 * lane;
			const float4 h0 = hp[0], h1 = hp[1];
			const float v[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
			const float f = x_image<KIND>(v, img + (size_t)j * STRIDE, lane);
			if (lane == 0)
				inv[k][b] = f;
		}
		__syncthreads();
		while (it < s1) {
			const int r0 = (it - g * tiles) * 16;
			it += DG_DOWN_WARPS;
			settle(it, end);  // (the next item from here on)
			ok = ok && __all_sync(0xffffffffu, dec_wait(ba, status, parity));
			parity ^= 1;
			float2 out[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
			for (int b = 0; b < nb && ok; b++) {
				MmaRows<KIND> w;
				w.load_smem(tile, nb, b, lane);
				if (b == nb - 1) {
					__syncwarp();
					if (lane == 0 && it < items.y) {
						ptx::fence_proxy_async_smem();
						request(it);
					}
				}
				const MmaCol<true> col[2] = {two_rows<KIND>(img + b * STRIDE, nb * STRIDE, 0, n, zeros, lane),
							     two_rows<KIND>(img + b * STRIDE, nb * STRIDE, 2, n, zeros, lane)};
				float2 r[2];
				if (n > 2)
					w.dot(col, lane, r);
				else
					r[0] = r[1] = dot_one(w, col[0], lane);
#pragma unroll
				for (int p = 0; p < 2; p++) {
					const float2 f = w.scale(inv[2 * p + m][b]);
					out[p].x = __fmaf_rn(f.x, r[p].x, out[p].x);
					out[p].y = __fmaf_rn(f.y, r[p].y, out[p].y);
				}
			}
			// lanes t = 0, 1 of a quad hold rows g and g + 8 of the first row of a pair, t = 2, 3 of the second
#pragma unroll
			for (int p = 0; p < 2; p++)
				if (ok && 2 * p + m < n)
					y[(size_t)gl.row[g][2 * p + m] * rows_per_expert + r0 + (lane >> 2) + 8 * (lane & 1)] = lane & 1 ? out[p].y : out[p].x;
		}
	}
}

// ---- host side ----

constexpr int DG_MAX_SMEM = 200 * 1024;

static size_t group_gate_up_smem(const DevTensor &t)
{
	return t.kind == W_Q4K ? GuCfg<W_Q4K>::smem(t.k / QK_K) : GuCfg<W_Q6K_R8>::smem(t.k / QK_K);
}

static size_t group_down_smem(const DevTensor &t)
{
	const int nb = t.k / QK_K;
	return t.kind == W_Q4K ? DG_DOWN_WARPS * tile_offset<W_Q4K>(nb, 16) + (size_t)nb * DG_ROWS * XImage<W_Q4K>::BYTES
			       : DG_DOWN_WARPS * tile_offset<W_Q6K_R8>(nb, 16) + (size_t)nb * DG_ROWS * XImage<W_Q6K_R8>::BYTES;
}

bool decode_group_supported(const tie_cuda_ctx *c, const Layer &L, int n_tokens)
{
	// from where few rows have their expert to themselves: 7 / 8 tokens of this model's shape 68.9 / 74.1 us a block here, 67.7 /
	// 78.9 row by row (decode.cu); up to where the tensor path takes over (run_experts)
	const int n_rows = n_tokens * c->cfg.top_k;
	return n_tokens > 4 && 16 * n_rows > 7 * c->n_local && n_tokens <= DG_MAX_TOKENS && n_rows <= DG_MAX_ROWS && n_rows < 2 * c->n_local && c->n_local <= DG_MAX_EXPERTS &&
	       L.gate.kind == L.up.kind && L.gate.k <= DG_MAX_NB * QK_K && L.gate.rows % 16 == 0 && L.down.rows % 16 == 0 &&
	       L.down.k <= DG_MAX_NB * QK_K && group_down_smem(L.down) <= (size_t)DG_MAX_SMEM && group_gate_up_smem(L.gate) <= (size_t)DG_MAX_SMEM;
}

int decode_group_setup(tie_cuda_ctx *c)
{
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(group_gate_up<W_Q4K>, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_MAX_SMEM));
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(group_gate_up<W_Q6K_R8>, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_MAX_SMEM));
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(group_down<W_Q4K>, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_MAX_SMEM));
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(group_down<W_Q6K_R8>, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_MAX_SMEM));
	return TIE_CUDA_OK;
}

// x [n_tokens][hidden] -> h [(token, slot)][ffn]
int launch_group_gate_up(tie_cuda_ctx *c, const Layer &L, const float *x, int n_tokens)
{
	const int nb = L.gate.k / QK_K;
	auto kern = L.gate.kind == W_Q4K ? group_gate_up<W_Q4K> : group_gate_up<W_Q6K_R8>;
	return launch_kernel(c, true, 1, kern, dim3(c->sm_count * (DG_MAX_NB / nb)), 32 * (2 * nb + 1), group_gate_up_smem(L.gate), L.gate.ptr, L.up.ptr,
			     L.gate.expert_stride, L.gate.rows, nb, x, c->cfg.top_k, n_tokens * c->cfg.top_k, c->s.topk_idx, c->s.h, c->first_expert,
			     c->n_local, c->silu, c->s.status);
}

// h -> y [(token, slot)][hidden], unweighted
int launch_group_down(tie_cuda_ctx *c, const Layer &L, int n_tokens, float *y)
{
	auto kern = L.down.kind == W_Q4K ? group_down<W_Q4K> : group_down<W_Q6K_R8>;
	return launch_kernel(c, true, 1, kern, dim3(2 * c->sm_count), 32 * DG_DOWN_WARPS, group_down_smem(L.down), L.down.ptr, L.down.expert_stride,
			     L.down.rows, L.down.k / QK_K, c->s.h, c->cfg.top_k, n_tokens * c->cfg.top_k, c->s.topk_idx, y, c->first_expert, c->n_local,
			     c->s.status);
}

}  // namespace tie
