// Decode of ONE token as ONE kernel: router, selection, gate/up + SwiGLU, down + combine.
//
// Reference: the is_moe branch of transformer_layer_qwen3 for batch_len == 1
// (model_qwen3.c:403-471).  The three-kernel decode path (decode.cu) pays three launches and
// cannot keep the down tiles in flight under the gate/up kernel (the two kernels do not fit one
// SM together).  Here one cooperative grid (one CTA per SM, all co-resident) walks the phases
// with grid-wide barriers between them, two in a block and one behind it:
//
//   R  CTA e < n_expert: logit e by warp 0, the AVX2 lane order replayed (8 chains of sequential fused
//      multiply-adds, hsum tree: bit-exact, as router_batch); other warps meanwhile make the
//      images of x (mma_dot.cuh) for its gate/up tile
//   -- barrier --
//      every CTA selects the experts itself from the logits (one warp, hardware max/min reductions:
//      cheaper than a broadcast), then requests its gate and up tiles and, once those land, the down
//      tiles of all selected experts for its 16 output rows (bulk copies, ~190 KB per SM, one issuing
//      thread per copy group); the gate weights are computed while the tiles are on their way
//   G  CTA (slot, row tile): a warp takes 16 rows x one super-block of gate or up; table SwiGLU -> h
//   -- barrier --
//   D  CTA (row tile): a warp takes one (slot, super-block); the products meet in shared memory and are
//      added up per slot in super-block order, then over the slots from zero,
//      acc = fma(w_j, v_j, acc) (model_qwen3.c:458-467), + residual
//   -- barrier, the next block of a stack --
//
// A stack of blocks is one launch (the blocks may differ in the kind of the down tensor): a third barrier costs less
// than the end of a grid and the start of the next, 22.7 -> 21.1 us a block, 20.2 with the norm weights loaded beside the row instead of behind its sum.
//
// Bound by latency: of 23.5 us for one block with its weights in HBM, 4.0 are RMSNorm + router chains, 1.4 and 1.9 the
// two grid barriers, 1.5 the selection, 3.0 the first tile's arrival, 4.5 gate/up, 3.3 the down products, 0.6 the combine, 3.3
// launch and tail (the 25.5 MB themselves would take 3.9).
//
// The barriers count arrivals in a device word that only grows (targets are relative to an epoch
// the last CTA of every launch advances), so the launch arguments never change and the kernel
// replays from a CUDA graph.  Every spin is bounded; a CTA that gives up flags the status word,
// waits (bounded) for its own copies in flight and returns.
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "mma_dot.cuh"
#include "tc_ptx.cuh"
#include "decode_common.cuh"
#include "router_topk.cuh"

namespace tie {

constexpr int DF_THREADS = 768;	// 24 warps: two products of 16 rows x one super-block each for gate/up, one for down
constexpr int DF_WARPS = DF_THREADS / 32;
constexpr int DF_MAX_CHUNKS = 8;
constexpr long long DF_WAIT_CYCLES = 1ll << 30;

struct DfShared {
	uint64_t bar_gu[DF_MAX_CHUNKS];
	uint64_t bar_dn[MAX_TOP_K];
	int idx[MAX_TOP_K];
	float w[MAX_TOP_K];
	unsigned base;
	int ok;
	int dn_req[MAX_TOP_K];	// the down tile of slot j has been requested
	float inv;  // 1 / rms of the row (RMSNorm in the kernel)
	float x_inv[8];	 // per super-block of x: the factor that undoes its image's scaling
	DfLayer lay;
};

struct DfArgs {
	DfLayer first;		  // the (first) block's weights
	const DfLayer *layers;	  // n_layers > 1: all of them, and x == residual == out
	int n_layers;
	size_t stride_gu;  // bytes per expert
	const float *x, *bias, *residual, *silu;
	float norm_eps;	 // >= 0: x is the un-normed hidden row, RMSNorm (weights norm_w or 1) happens in the kernel
	float *logits, *h, *out, *topk_w;
	int *topk_idx;
	unsigned *status, *sync;  // sync[0]: arrivals, sync[1]: epoch
	unsigned *host_status;	  // or null: out is host memory; the status word goes here once all of out is there
	int n_expert, top_k, first_expert, n_local;
	int rpt_gu, tiles_gu, rpt_dn, tiles_dn;
	uint32_t off_b, off_c, off_v, off_n;  // shared-memory offsets: down tiles, images of x, products, normed x
};

__device__ __forceinline__ unsigned df_ld_acquire(const unsigned *p)
{
	unsigned v;
	asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}

// All CTAs of the (cooperative, co-resident) grid arrive; returns false after DF_WAIT_CYCLES.
__device__ __forceinline__ bool df_grid_barrier(unsigned *counter, unsigned target, DfShared *sh, unsigned *status)
{
	__syncthreads();
	if (threadIdx.x == 0) {
		// (release: what the CTA wrote before its barrier above is visible to whoever sees the count)
		asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
		const long long t0 = clock64();
		int ok = 1;
		while ((int)(df_ld_acquire(counter) - target) < 0) {
			if (clock64() - t0 > DF_WAIT_CYCLES) {
				atomicOr(status, ST_WAIT_TIMEOUT);
				ok = 0;
				break;
			}
		}
		sh->ok = ok;
	}
	__syncthreads();
	return sh->ok != 0;
}

// D, its products: a job is (slot, super-block); the gate/up tiles are done with, their space takes the images of h.
template <WKind KD, int F>
__device__ __forceinline__ bool df_down(uint8_t *dsm, const uint8_t *sd, float *prod, const float *h, int top_k, uint32_t tile_dn, int warp,
					int lane, DfShared &sh, unsigned *status, uint32_t parity)
{
	constexpr int NBF = F / QK_K;
	uint8_t *himg = dsm + warp * XImage<KD>::BYTES;
	for (int i = warp; i < top_k * NBF; i += DF_WARPS) {
		const int j = i / NBF, b = i % NBF;
		const float4 *hp = reinterpret_cast<const float4 *>(h + (size_t)j * F + b * QK_K) + 2 * lane;
		const float4 h0 = __ldcg(hp), h1 = __ldcg(hp + 1);  // (written by other CTAs of this grid)
		const float v[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
		const float inv = x_image<KD>(v, himg, lane);
		if (!__all_sync(0xffffffffu, dec_wait(ptx::smem_u32(&sh.bar_dn[j]), status, parity)))
			return false;
		MmaRows<KD> w;
		w.load_smem(sd + (size_t)j * tile_dn, NBF, b, lane);
		const float2 r = dot_one(w, one_row<KD>(himg, lane), lane), s = w.scale(inv);
		if ((lane & 3) == 0) {
			float2 *d = reinterpret_cast<float2 *>(prod) + i * 16 + (lane >> 2);
			d[0] = make_float2(r.x, s.x);
			d[8] = make_float2(r.y, s.y);
		}
	}
	return true;
}

template <WKind KG, int K, int F>
__global__ void __launch_bounds__(DF_THREADS, 1) decode1_fused(const DfArgs a)
{
	constexpr int NBK = K / QK_K, NBF = F / QK_K;
	constexpr int CH = 16;	// rows per gate/up copy chunk (own barrier): one MMA tile
	extern __shared__ __align__(128) uint8_t dsm[];
	__shared__ DfShared sh;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int cta = blockIdx.x, G = gridDim.x;
	const int top_k = a.top_k;
	uint8_t *ximg = dsm + a.off_c;			    // images of x's super-blocks, for gate/up
	float *prod = reinterpret_cast<float *>(dsm + a.off_v);	 // products before they are added up

	const bool gu_role = cta < top_k * a.tiles_gu, dn_role = cta < a.tiles_dn;
	const int slot = cta / a.tiles_gu;
	const int g0 = (cta % a.tiles_gu) * a.rpt_gu, g1 = min(g0 + a.rpt_gu, F);
	const int d0 = cta * a.rpt_dn, d1 = min(d0 + a.rpt_dn, K);
	const int n_chunks = gu_role ? (g1 - g0 + CH - 1) / CH : 0;
	const uint32_t tile_gu = (uint32_t)(tile_offset<KG>(NBK, g1) - tile_offset<KG>(NBK, g0));

	if (tid == DF_THREADS - 1) {  // (not in a warp that the norm or the router waits for)
		for (int c = 0; c < DF_MAX_CHUNKS; c++)
			ptx::mbar_init(ptx::smem_u32(&sh.bar_gu[c]), 1);
		for (int j = 0; j < MAX_TOP_K; j++) {
			ptx::mbar_init(ptx::smem_u32(&sh.bar_dn[j]), 1);
			sh.dn_req[j] = 0;
		}
		ptx::fence_barrier_init();
		sh.lay = a.first;
		sh.base = df_ld_acquire(a.sync + 1);
	}
	unsigned target = 0;  // grid barriers, relative to the epoch
	bool alive = true;
	for (int layer = 0;; layer++) {
		const uint32_t parity = (uint32_t)layer & 1u;  // (every copy barrier completes once a layer)

		// The row, its norm weights and the CTA's row of the router matrix are on their way before anything is computed.
		// For the sequential chains both lie as [AVX2 lane][step] too: a thread of a chain gets four steps per load (one each:
		// 16 blocks 320 us, so 305, with the two lines on the barrier and the selection; the tile area is free until the selection).
		constexpr int TP = K / 8 + 4;
		float *wt = reinterpret_cast<float *>(dsm), *xt = wt + 8 * TP, *xn = reinterpret_cast<float *>(dsm + a.off_n);
		auto transposed = [&](float *t, const float4 &v) {  // 4 tid .. of the row
			float *d = t + 4 * (tid & 1) * TP + (tid >> 1);
			d[0] = v.x;
			d[TP] = v.y;
			d[2 * TP] = v.z;
			d[3 * TP] = v.w;
		};
		static_assert(K / 4 <= DF_THREADS, "one 16-byte load per thread");
		const float *router_w = layer ? sh.lay.router_w : a.first.router_w, *norm_w = layer ? sh.lay.norm_w : a.first.norm_w;
		float4 xv = make_float4(0.f, 0.f, 0.f, 0.f), nv = make_float4(1.f, 1.f, 1.f, 1.f);
		if (tid < K / 4) {
			xv = __ldcg(reinterpret_cast<const float4 *>(a.x) + tid);	// (the row is overwritten in place at the end)
			float4 wv = make_float4(0.f, 0.f, 0.f, 0.f);
			if (cta < a.n_expert)
				wv = __ldg(reinterpret_cast<const float4 *>(router_w + (size_t)cta * K) + tid);
			if (a.norm_eps >= 0.0f && norm_w)
				nv = __ldg(reinterpret_cast<const float4 *>(norm_w) + tid);
			reinterpret_cast<float4 *>(xn)[tid] = xv;
			transposed(xt, xv);
			transposed(wt, wv);
		}
		__syncthreads();
		if (layer == 0)
			target = sh.base;
		// ---------------- (RMSNorm of the row, every CTA for itself: rms_norm_f32_f32_f32_avx2, math_avx2.c:56-97) ----------------
		if (a.norm_eps >= 0.0f) {
			if (warp == 0) {
				float acc = 0.0f;
				if (lane < 8) {
					const float4 *t = reinterpret_cast<const float4 *>(xt + lane * TP);
#pragma unroll 16
					for (int i = 0; i < K / 32; i++) {
						const float4 v = t[i];
						acc = __fmaf_rn(v.x, v.x, acc);
						acc = __fmaf_rn(v.y, v.y, acc);
						acc = __fmaf_rn(v.z, v.z, acc);
						acc = __fmaf_rn(v.w, v.w, acc);
					}
				}
				const float ss = hsum8_lanes(acc);  // (l + l4), then + 1, then + 2: the reference's tree
				if (lane == 0)
					sh.inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), a.norm_eps)));
			}
			__syncthreads();
			const float inv = sh.inv;
			if (tid < K / 4) {
				const float4 o = make_float4(__fmul_rn(__fmul_rn(xv.x, nv.x), inv), __fmul_rn(__fmul_rn(xv.y, nv.y), inv),
							     __fmul_rn(__fmul_rn(xv.z, nv.z), inv), __fmul_rn(__fmul_rn(xv.w, nv.w), inv));
				reinterpret_cast<float4 *>(xn)[tid] = o;
				transposed(xt, o);
			}
			__syncthreads();
		}

		// ---------------- R: one router logit per CTA (warp 0), the images of x beside it ----------------
		if (warp == 0 && cta < a.n_expert) {
			float acc = 0.0f;
			if (lane < 8) {
				const float4 *tx = reinterpret_cast<const float4 *>(xt + lane * TP), *tw = reinterpret_cast<const float4 *>(wt + lane * TP);
#pragma unroll 16
				for (int i = 0; i < K / 32; i++) {
					const float4 u = tx[i], v = tw[i];
					acc = __fmaf_rn(u.x, v.x, acc);
					acc = __fmaf_rn(u.y, v.y, acc);
					acc = __fmaf_rn(u.z, v.z, acc);
					acc = __fmaf_rn(u.w, v.w, acc);
				}
			}
			float r = hsum8_lanes(acc);
			if (lane == 0) {
				if (a.bias)
					r = __fadd_rn(r, a.bias[cta]);
				__stcg(a.logits + cta, r);
			}
		}
		if (gu_role && warp >= 8 && warp < 8 + NBK) {
			const int b = warp - 8;
			const float4 *xp = reinterpret_cast<const float4 *>(xn + b * QK_K) + 2 * lane;
			const float4 x0 = xp[0], x1 = xp[1];
			const float v[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
			const float inv = x_image<KG>(v, ximg + b * XImage<KG>::BYTES, lane);
			if (lane == 0)
				sh.x_inv[b] = inv;
		}
		if (!df_grid_barrier(a.sync, target += (unsigned)G, &sh, a.status))
			return;	 // nothing of this CTA is in flight yet

		// ---------------- selection (every CTA for itself) and all weight requests ----------------
		if (warp == 0) {
			auto select = [&](auto per) {
				unsigned key[1][per.value];
#pragma unroll
				for (int i = 0; i < per.value; i++)
					key[0][i] = lane + 32 * i < a.n_expert ? score_key(__ldcg(a.logits + lane + 32 * i)) : 0u;
				int mine[1];
				unsigned best[1];
				topk_warp<1, per.value>(key, lane, top_k, mine, best);
				if (lane < top_k)
					sh.idx[lane] = mine[0];
			};
			if (a.n_expert <= 128)
				select(std::integral_constant<int, 4>());
			else
				select(std::integral_constant<int, 8>());
		}
		__syncthreads();
		bool bad = false;
		for (int j = 0; j < top_k; j++) {
			const int le = sh.idx[j] - a.first_expert;
			bad |= (le < 0 || le >= a.n_local);
		}
		if (bad && cta == 0 && tid == 0)
			atomicOr(a.status, ST_BAD_EXPERT);
		const bool dn_q6k = sh.lay.down_q6k;
		const uint32_t tile_dn = !dn_role ? 0
						  : (uint32_t)(dn_q6k ? tile_offset<W_Q6K_R8>(NBF, d1) - tile_offset<W_Q6K_R8>(NBF, d0)
								      : tile_offset<W_Q4K>(NBF, d1) - tile_offset<W_Q4K>(NBF, d0));
		uint8_t *sg = dsm, *su = dsm + tile_gu, *sd = dsm + a.off_b;
		// one issuing thread per copy group (issuing a bulk copy costs ~100 cycles): warp c < 8 the
		// gate/up chunk c, warp 8 + j the down tile of slot j.  The down tiles are requested when the warp's
		// last gate/up chunk has landed: asked for earlier they share the HBM bandwidth with the gate/up
		// tiles, and they still have a product, a grid barrier and the image of h to arrive in.
		auto request_down = [&]() {  // lane 0 of warp 8 + j
			const int j = warp - DF_MAX_CHUNKS;
			if (dn_role && j >= 0 && j < top_k) {
				const uint32_t ba = ptx::smem_u32(&sh.bar_dn[j]);
				sh.dn_req[j] = 1;
				ptx::fence_proxy_async_smem();
				ptx::mbar_arrive_expect_tx(ba, tile_dn);
				bulk_g2s(ptx::smem_u32(sd + (size_t)j * tile_dn),
					 sh.lay.wd + (size_t)(sh.idx[j] - a.first_expert) * sh.lay.stride_dn +
						 (dn_q6k ? tile_offset<W_Q6K_R8>(NBF, d0) : tile_offset<W_Q4K>(NBF, d0)),
					 tile_dn, ba);
			}
		};
		if (lane == 0 && !bad) {
			ptx::fence_proxy_async_smem();	// the tile area held the router's staging
			if (warp < DF_MAX_CHUNKS) {
				const int c = warp;
				if (gu_role && c < n_chunks) {
					const size_t eb = (size_t)(sh.idx[slot] - a.first_expert) * a.stride_gu;
					const int c0 = g0 + c * CH, c1 = min(c0 + CH, g1);
					const size_t o0 = tile_offset<KG>(NBK, c0), o1 = tile_offset<KG>(NBK, c1);
					const uint32_t bytes = (uint32_t)(o1 - o0), rel = (uint32_t)(o0 - tile_offset<KG>(NBK, g0));
					const uint32_t ba = ptx::smem_u32(&sh.bar_gu[c]);
					ptx::mbar_arrive_expect_tx(ba, 2 * bytes);
					bulk_g2s(ptx::smem_u32(sg + rel), sh.lay.wg + eb + o0, bytes, ba);
					bulk_g2s(ptx::smem_u32(su + rel), sh.lay.wu + eb + o0, bytes, ba);
				}
			} else if (!gu_role) {
				request_down();	 // (a CTA without gate/up rows: nothing to wait for)
			}
		}
		if (warp == DF_WARPS - 1) {  // softmax (engine.c:864-888) with the arithmetic of topk_tokens, while the tiles are on their way
			const int e = lane < top_k ? sh.idx[lane] : -1;
			const float score = e >= 0 ? __ldcg(a.logits + e) : 0.0f;
			const float mx = __shfl_sync(0xffffffffu, score, 0);
			const float ex = (lane < top_k) ? expf(__fsub_rn(score, mx)) : 0.0f;
			float sum = 0.0f;
			for (int j = 0; j < top_k; j++)
				sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, ex, j));
			const float w = __fmul_rn(ex, __fdiv_rn(1.0f, sum));
			if (lane < top_k) {
				sh.w[lane] = w;
				if (cta == 0) {
					a.topk_idx[lane] = e;
					a.topk_w[lane] = w;
				}
			}
		}
		// waits (bounded) for every copy this CTA requested: before it gives up, and harmless otherwise
		auto drain = [&]() {
			if (bad)
				return;
			for (int c = 0; c < n_chunks; c++)
				dec_wait(ptx::smem_u32(&sh.bar_gu[c]), a.status, parity);
			if (dn_role)
				for (int j = 0; j < top_k; j++)
					if (sh.dn_req[j])
						dec_wait(ptx::smem_u32(&sh.bar_dn[j]), a.status, parity);
		};

		// ---------------- G: gate, up, SwiGLU ----------------
		if (gu_role && !bad) {
			// a job is (chunk of 16 rows, matrix, super-block); the products of a row's super-blocks are added up in order
			const int jobs = n_chunks * 2 * NBK;
			for (int i = warp; i < jobs && alive; i += DF_WARPS) {
				const int chunk = i / (2 * NBK), mat = i % 2, b = (i % (2 * NBK)) >> 1;
				alive = __all_sync(0xffffffffu, dec_wait(ptx::smem_u32(&sh.bar_gu[chunk]), a.status, parity));
				if (!alive)
					break;
				if (i + DF_WARPS >= jobs && lane == 0)	// the warp's last
					request_down();
				MmaRows<KG> w;
				w.load_smem((mat ? su : sg) + tile_offset<KG>(NBK, chunk * CH), NBK, b, lane);
				const float2 r = dot_one(w, one_row<KG>(ximg + b * XImage<KG>::BYTES, lane), lane), s = w.scale(sh.x_inv[b]);
				if ((lane & 3) == 0) {
					float *d = prod + ((chunk * 2 + mat) * NBK + b) * 16 + (lane >> 2);
					d[0] = r.x * s.x;
					d[8] = r.y * s.y;
				}
			}
			if (warp >= jobs && lane == 0)
				request_down();
			alive = __syncthreads_and(alive);
			if (alive && tid < g1 - g0) {
				const float *pg = prod + (tid >> 4) * 2 * NBK * 16 + (tid & 15), *pu = pg + NBK * 16;
				float g = pg[0], u = pu[0];
				for (int b = 1; b < NBK; b++) {
					g = __fadd_rn(g, pg[b * 16]);
					u = __fadd_rn(u, pu[b * 16]);
				}
				__stcg(a.h + (size_t)slot * F + g0 + tid, swiglu_lut(a.silu, g, u));
			}
		}
		alive = __syncthreads_and(alive);
		if (!alive) {  // a copy never landed: leave, but not with copies in flight
			if (tid == 0)
				drain();
			return;
		}
		if (!df_grid_barrier(a.sync, target += (unsigned)G, &sh, a.status)) {
			if (tid == 0)
				drain();
			return;
		}

		// ---------------- D: down + combine ----------------
		const bool more = layer + 1 < a.n_layers && !bad;  // (bad is the same in every CTA: they all selected alike)
		if (more && tid == 0) {	 // this CTA's share of the next block's router matrix -> L2
			const uint32_t bytes = (uint32_t)a.n_expert * K * sizeof(float), per = ((bytes + G - 1) / G + 15u) & ~15u, o = per * (uint32_t)cta;
			if (o < bytes) {
				const uint32_t n = min(per, bytes - o);
				asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<const uint8_t *>(a.layers[layer + 1].router_w) + o), "r"(n)
					     : "memory");
			}
			if (cta == 0 && a.layers[layer + 1].norm_w)
				asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.layers[layer + 1].norm_w), "r"(K * 4) : "memory");
		}
		if (dn_role && !bad) {
			alive = dn_q6k ? df_down<W_Q6K_R8, F>(dsm, sd, prod, a.h, top_k, tile_dn, warp, lane, sh, a.status, parity)
				       : df_down<W_Q4K, F>(dsm, sd, prod, a.h, top_k, tile_dn, warp, lane, sh, a.status, parity);
			alive = __syncthreads_and(alive);
			if (alive) {
				for (int lr = tid; lr < d1 - d0; lr += DF_THREADS) {
					float acc = 0.f;
					for (int j = 0; j < top_k; j++) {
						float v = 0.f;
						for (int b = 0; b < NBF; b++) {
							const float2 e = reinterpret_cast<const float2 *>(prod)[(j * NBF + b) * 16 + lr];
							v = __fmaf_rn(e.y, e.x, v);
						}
						acc = __fmaf_rn(sh.w[j], v, acc);  // slot order, from zero
					}
					if (a.residual)
						acc = __fadd_rn(__ldcg(a.residual + d0 + lr), acc);
					__stcg(a.out + d0 + lr, acc);
				}
			}
		}
		__syncthreads();
		if (!alive || !more) {
			if (tid == 0) {
				drain();
				// the last CTA out advances the epoch for the next launch
				target += (unsigned)G;
				if (a.host_status)
					__threadfence_system();
				if (alive && atomicAdd(a.sync, 1u) == target - 1u) {
					atomicExch(a.sync + 1, target);
					if (a.host_status) {
						const unsigned st = *(volatile unsigned *)a.status;
						__threadfence_system();
						*(volatile unsigned *)a.host_status = st;
					}
				}
			}
			return;
		}
		if (tid == DF_THREADS - 1) {
			sh.lay = a.layers[layer + 1];
			for (int j = 0; j < MAX_TOP_K; j++)
				sh.dn_req[j] = 0;
		}
		// the row is complete, and the next block may overwrite h, the logits and the tiles
		if (!df_grid_barrier(a.sync, target += (unsigned)G, &sh, a.status))
			return;	 // (every copy of this CTA has been waited for)
	}
}

// ---- host side ----

template <WKind KIND>
static size_t df_row_bytes(int k)
{
	return (size_t)(k / QK_K) * (KIND == W_Q4K ? Q4K_BYTES : Q6K_BYTES);
}

struct DfPlan {
	int rpt_gu, tiles_gu, rpt_dn, tiles_dn, grid;
	size_t smem, off_b, off_c, off_v, off_n;
	bool ok;
};

template <WKind KG, int K, int F>
static DfPlan df_plan(const tie_cuda_ctx *c)
{
	DfPlan p = {};
	const int top_k = c->cfg.top_k, sms = c->sm_count;
	const int want_gu = sms / top_k;
	if (want_gu < 1)
		return p;
	p.rpt_gu = ((F + want_gu - 1) / want_gu + 15) / 16 * 16;
	p.tiles_gu = (F + p.rpt_gu - 1) / p.rpt_gu;
	p.rpt_dn = 16;	// one MMA tile
	p.tiles_dn = (K + p.rpt_dn - 1) / p.rpt_dn;
	constexpr int NBK = K / QK_K, NBF = F / QK_K;
	if (p.rpt_gu / 16 > DF_MAX_CHUNKS || NBK > 8 || F % 16 || K % 16)
		return p;
	p.grid = max(c->cfg.n_expert, max(top_k * p.tiles_gu, p.tiles_dn));
	if (p.grid > sms)
		return p;
	const size_t tile_gu = (size_t)p.rpt_gu * df_row_bytes<KG>(K), tile_dn = (size_t)p.rpt_dn * df_row_bytes<W_Q6K_R8>(F);  // (the larger kind)
	size_t area_a = 2 * tile_gu;
	area_a = max(area_a, (size_t)2 * (K + 32) * sizeof(float));			 // the row and the router row, by AVX2 lane
	area_a = max(area_a, (size_t)DF_WARPS * max(XImage<W_Q4K>::BYTES, XImage<W_Q6K_R8>::BYTES));  // images of h
	p.off_b = (area_a + 127) / 128 * 128;
	p.off_c = (p.off_b + (size_t)top_k * tile_dn + 127) / 128 * 128;
	p.off_v = p.off_c + (size_t)NBK * XImage<KG>::BYTES;
	p.off_n = (p.off_v + max((size_t)p.rpt_gu * 2 * NBK, (size_t)top_k * NBF * 16 * 2) * sizeof(float) + 15) / 16 * 16;
	p.smem = p.off_n + (size_t)K * sizeof(float);
	p.ok = p.smem <= 220 * 1024;
	return p;
}

DfLayer df_layer(const Layer &L)
{
	return {L.gate.ptr, L.up.ptr, L.down.ptr, L.router_w, L.norm_w, L.down.expert_stride, L.down.kind == W_Q6K_R8};
}

template <WKind KG, int K, int F>
static int df_launch(tie_cuda_ctx *c, const Layer &L, int n_layers, const float *x, const float *bias, const float *residual, float *out,
		     bool query_only, bool norm, unsigned *host_status)
{
	const DfPlan p = df_plan<KG, K, F>(c);
	if (!p.ok)
		return TIE_CUDA_ENOTSUP;
	if (query_only)
		return TIE_CUDA_OK;
	Scratch &s = c->s;
	DfArgs a = {};
	a.first = df_layer(L);
	a.layers = c->df_table + (&L - c->layers);
	a.n_layers = n_layers;
	a.stride_gu = L.gate.expert_stride;
	a.x = x;
	a.bias = bias;
	a.residual = residual;
	a.silu = c->silu;
	a.logits = s.logits;
	a.h = s.h;
	a.out = out;
	a.topk_w = s.topk_w;
	a.topk_idx = s.topk_idx;
	a.status = s.status;
	a.sync = s.dec_sync;
	a.n_expert = c->cfg.n_expert;
	a.top_k = c->cfg.top_k;
	a.first_expert = c->first_expert;
	a.n_local = c->n_local;
	a.rpt_gu = p.rpt_gu;
	a.tiles_gu = p.tiles_gu;
	a.rpt_dn = p.rpt_dn;
	a.tiles_dn = p.tiles_dn;
	a.off_b = (uint32_t)p.off_b;
	a.off_c = (uint32_t)p.off_c;
	a.off_v = (uint32_t)p.off_v;
	a.off_n = (uint32_t)p.off_n;
	a.norm_eps = norm ? c->cfg.norm_eps : -1.0f;
	a.host_status = host_status;
	auto kern = decode1_fused<KG, K, F>;
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(p.grid);
	cfg.blockDim = dim3(DF_THREADS);
	cfg.dynamicSmemBytes = p.smem;
	cfg.stream = c->stream;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeCooperative;  // all CTAs co-resident: they wait on one another
	attr[0].val.cooperative = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
	if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
		// the grid cannot be co-resident here (a shared or partitioned GPU): the caller takes the chain
		cudaGetLastError();
		c->coop_ok = false;
		return TIE_CUDA_ENOTSUP;
	}
	TIE_CUDA_TRY(c, e);
	c->launches++;
	return TIE_CUDA_OK;
}

// The (hidden, ffn_dim) pairs the one-kernel step is built for.
#define TIE_DF_SHAPES(X) X(2048, 768) X(512, 256)

static int df_dispatch(tie_cuda_ctx *c, const Layer &L, int n_layers, const float *x, const float *bias, const float *residual, float *out,
		       bool query_only, bool norm, unsigned *host_status)
{
	if (L.gate.kind != L.up.kind)
		return TIE_CUDA_ENOTSUP;
	const int K = c->cfg.hidden, F = c->cfg.ffn_dim;
#define X(KK, FF)                                                                                                               \
	if (K == KK && F == FF)                                                                                                 \
		return L.gate.kind == W_Q4K ? df_launch<W_Q4K, KK, FF>(c, L, n_layers, x, bias, residual, out, query_only, norm, host_status) \
					    : df_launch<W_Q6K_R8, KK, FF>(c, L, n_layers, x, bias, residual, out, query_only, norm, host_status);
	TIE_DF_SHAPES(X)
#undef X
	return TIE_CUDA_ENOTSUP;
}

bool decode_fused_supported(tie_cuda_ctx *c, const Layer &L, int n_tokens)
{
	if (n_tokens != 1 || !c->coop_ok || c->cfg.top_k > MAX_TOP_K || c->cfg.n_expert > 256)
		return false;
	return df_dispatch(c, L, 1, nullptr, nullptr, nullptr, nullptr, true, false, nullptr) == TIE_CUDA_OK;
}

// host_status: out is pinned host memory, and the status word follows it there when the row is complete.
int launch_decode_fused(tie_cuda_ctx *c, const Layer &L, const float *x, const float *bias, const float *residual, float *out,
			unsigned *host_status)
{
	return df_dispatch(c, L, 1, x, bias, residual, out, false, false, host_status);
}

// hidden += block(RMSNorm(hidden)), for n_layers consecutive blocks from L on (same gate / up kind, decode_fused_supported).
int launch_decode_fused_blocks(tie_cuda_ctx *c, const Layer &L, int n_layers, float *hidden)
{
	return df_dispatch(c, L, n_layers, hidden, nullptr, hidden, hidden, false, true, nullptr);
}

}  // namespace tie
