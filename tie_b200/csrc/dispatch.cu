// Token-to-expert dispatch of the grouped products in one launch: the counting sort of the rows by expert and the split of
// their inputs into the token operand, in sorted order.
//
// A call's rows are (source, slot): row r belongs to source r / n_out (the token; n_out = top_k).  Every CTA takes a run of
// sources.  It needs to know where its rows of each expert start, so it counts the rows of every expert itself, all of
// them and those in front of its own (counters in shared memory: integer sums, whatever order they are made in), scans the
// totals over the experts, ranks its own rows (rows of one expert keep their order) and then reads each of its sources
// once, splits it and stores it at its n_out places.  The first CTA writes the tables that the products read.
//
// The count is 128 KB of ids a CTA at 4096 tokens of 8 experts, from L2, where a sort of its own was one or two launches in
// front of the split: latency for small batches, where nothing else runs.  Sort and split -> this, 64 tokens 8.2 + 8.2 ->
// 13.2 us, 512 13.3 + 12.3 -> 17.4, 1000 13.3 + 16.4 -> 23.5, 4096 17.4 + 53.3 -> 70.6 (an event between them in all of
// these).  The stores bound it from some 1000 tokens on (276 MB at 4096).
#include "common.cuh"
#include "kernels.cuh"
#include "split8.cuh"

namespace tie {

constexpr int DISP_THREADS = 1024, DISP_WARPS = DISP_THREADS / 32, DISP_MAX_E = 256, DISP_E_WARPS = DISP_MAX_E / 32;

struct DispatchOut {
	int *counts, *offsets, *tile_start, *active, *n_active, *perm, *inv;
	int4 *tile_info;
	__half *hi, *lo, *xq;
	int q_cols;
};

template <int STEPS>
__global__ void __launch_bounds__(DISP_THREADS, 1)
dispatch_rows(const float *__restrict__ x, int n_cols, const int *__restrict__ row_expert, int n_src, int n_out, int first_expert, int n_local,
	      int n_tile, const DispatchOut o, unsigned *__restrict__ status)
{
	__shared__ int hist[2][DISP_MAX_E];	      // rows in front of this CTA's, and the others
	__shared__ int start[DISP_WARPS][DISP_MAX_E];  // rows of expert e in warp w's 32 rows; then: where they start
	__shared__ int base[DISP_MAX_E];	      // where the CTA's next rows of expert e start
	__shared__ int place[DISP_THREADS];
	__shared__ int wsum[3][DISP_E_WARPS];
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int per = (n_src + gridDim.x - 1) / gridDim.x, src0 = min(n_src, (int)blockIdx.x * per), src1 = min(n_src, src0 + per);
	const int n_rows = n_src * n_out, mine0 = src0 * n_out;
	if (tid < 2 * DISP_MAX_E)
		(&hist[0][0])[tid] = 0;
	__syncthreads();
	pdl_wait();
	pdl_trigger();	// (the gate/up product sets itself up meanwhile)
	constexpr int AHEAD = 8;
	for (int r0 = warp * 32; r0 < n_rows; r0 += AHEAD * DISP_THREADS) {
		int le[AHEAD];
#pragma unroll
		for (int i = 0; i < AHEAD; i++) {
			const int r = r0 + i * DISP_THREADS + lane;
			le[i] = r < n_rows ? row_expert[r] - first_expert : -1;
		}
#pragma unroll
		for (int i = 0; i < AHEAD; i++) {
			const int r = r0 + i * DISP_THREADS + lane;
			if (r - lane >= n_rows)
				break;
			// (a warp whose rows are all of one expert, as rows that come grouped are, adds once)
			int *cell = (unsigned)le[i] < (unsigned)n_local ? &hist[r >= mine0][le[i]] : nullptr;
			const unsigned long long c0 = __shfl_sync(0xffffffffu, (unsigned long long)cell, 0);
			if (__all_sync(0xffffffffu, (unsigned long long)cell == c0)) {
				if (lane == 0 && cell)
					atomicAdd(cell, 32);
			} else if (cell) {
				atomicAdd(cell, 1);
			}
		}
	}
	__syncthreads();
	// exclusive scans over the experts: rows, token tiles, experts with rows (thread e stands for expert e)
	int before = 0, total = 0, v[3] = {0, 0, 0}, incl[3] = {0, 0, 0};
	if (tid < DISP_MAX_E) {
		before = hist[0][tid];
		total = before + hist[1][tid];
		v[0] = total;
		v[1] = (total + n_tile - 1) / n_tile;
		v[2] = total > 0 ? 1 : 0;
#pragma unroll
		for (int k = 0; k < 3; k++) {
			incl[k] = v[k];
#pragma unroll
			for (int d = 1; d < 32; d <<= 1) {
				const int t = __shfl_up_sync(0xffffffffu, incl[k], d);
				if (lane >= d)
					incl[k] += t;
			}
			if (lane == 31)
				wsum[k][warp] = incl[k];
		}
	}
	__syncthreads();
	if (tid < DISP_MAX_E) {
		int excl[3], all[3];
#pragma unroll
		for (int k = 0; k < 3; k++) {
			int bw = 0, a = 0;
#pragma unroll
			for (int i = 0; i < DISP_E_WARPS; i++) {
				const int w = wsum[k][i];
				bw += i < warp ? w : 0;
				a += w;
			}
			excl[k] = bw + incl[k] - v[k];
			all[k] = a;
		}
		base[tid] = excl[0] + before;
		if (blockIdx.x == 0 && tid < n_local) {
			o.counts[tid] = total;
			o.offsets[tid] = excl[0];
			o.tile_start[tid] = excl[1];
			if (total > 0)
				o.active[excl[2]] = tid;
			for (int j = 0; j * n_tile < total; j++)
				o.tile_info[excl[1] + j] = make_int4(tid, excl[0] + j * n_tile, min(n_tile, total - j * n_tile), 0);
		}
		if (blockIdx.x == 0 && tid == 0) {
			o.offsets[n_local] = all[0];
			o.tile_start[n_local] = all[1];
			*o.n_active = all[2];
		}
	}
	// the CTA's sources, as many at a time as have a thread for each of their rows
	const int chunk = DISP_THREADS / n_out, upr = (n_cols + STEPS * 256 - 1) / (STEPS * 256);
	for (int s0 = src0; s0 < src1; s0 += chunk) {
		const int ns = min(chunk, src1 - s0), nr = ns * n_out, n_warps = (nr + 31) / 32;
		for (int i = tid; i < n_warps * DISP_MAX_E; i += DISP_THREADS)
			(&start[0][0])[i] = 0;
		const int r = s0 * n_out + tid;
		int le = -1;
		if (tid < nr) {
			le = row_expert[r] - first_expert;
			if ((unsigned)le >= (unsigned)n_local) {
				le = -1;
				atomicOr(status, ST_BAD_EXPERT);
			}
		}
		__syncthreads();  // (also: base is written; the places of the sources before are read)
		unsigned same = 0;
		if (warp < n_warps) {
			same = __match_any_sync(0xffffffffu, le);
			if (le >= 0 && (same & ((1u << lane) - 1u)) == 0)
				start[warp][le] = __popc(same);
		}
		__syncthreads();
		if (tid < DISP_MAX_E) {
			int at = base[tid];
			for (int w = 0; w < n_warps; w++) {
				const int n = start[w][tid];
				start[w][tid] = at;
				at += n;
			}
			base[tid] = at;
		}
		__syncthreads();
		if (tid < nr) {
			const int pos = le >= 0 ? start[warp][le] + __popc(same & ((1u << lane) - 1u)) : -1;
			place[tid] = pos;
			o.inv[r] = pos;
			if (pos >= 0)
				o.perm[pos] = r;
		}
		__syncthreads();
		for (int un = warp; un < ns * upr; un += DISP_WARPS) {
			const int s = un / upr;
			SplitUnit<STEPS> u;
			u.load(x + (size_t)(s0 + s) * n_cols, (un - s * upr) * STEPS * 256 + lane * 8, n_cols);
			u.split(o.xq != nullptr);
			for (int j = 0; j < n_out; j++) {
				const int at = place[s * n_out + j];
				if (at >= 0)
					u.store(o.hi + (size_t)at * n_cols, o.lo + (size_t)at * n_cols, o.xq ? o.xq + (size_t)at * o.q_cols : nullptr, lane);
			}
		}
	}
}

// x: n_src rows of the hidden size; row r of row_expert is a row of source r / n_out.  after_router: the launch right in front
// is the router's (which lets its successors in early).
int launch_dispatch(tie_cuda_ctx *c, const float *x, const int *row_expert, int n_src, int n_out, int n_tile, bool sums, bool after_router)
{
	Scratch &s = c->s;
	const int H = c->cfg.hidden;
	if (c->n_local > DISP_MAX_E || H % 256 || n_out <= 0 || n_out > 32)
		return TIE_CUDA_ENOTSUP;
	if (n_src <= 0)
		return TIE_CUDA_EINVAL;
	DispatchOut o = {s.counts, s.offsets, s.tile_start, s.active, s.n_active, s.perm, s.inv, s.tile_info, s.xs_hi, s.xs_lo, sums ? s.xq : nullptr,
			 xq_cols(H)};
	const int per = (n_src + c->sm_count - 1) / c->sm_count, grid = (n_src + per - 1) / per;
	// units of 512 columns where the warps of a CTA have one each, else of 256
	const bool wide = per * ((H + 511) / 512) >= DISP_WARPS;
	return launch_kernel(c, after_router, 1, wide ? dispatch_rows<2> : dispatch_rows<1>, dim3(grid), DISP_THREADS, 0, x, H, row_expert, n_src, n_out,
			     c->first_expert, c->n_local, n_tile, o, s.status);
}

}  // namespace tie
