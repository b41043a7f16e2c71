// Small element-wise kernels around the expert products: RMSNorm, weighted combine (+ residual),
// the fp16 hi/lo split of activations for the tensor-core path, and the table SwiGLU on its own.
#include "common.cuh"
#include "kernels.cuh"
#include "split8.cuh"

namespace tie {

// rms_norm_f32_f32_f32_avx2 (math_avx2.c:56-97): 8 lanes of sequential fma(x,x,acc), hsum tree,
// inv = 1/sqrtf(ss/n + eps), o = (x*w)*inv.  One CTA per token: lane l < 8 of warp 0 runs lane l's chain
// over a shared-memory copy of the row (bit-identical sum of squares).  Bound by latency at a few tokens: the row and
// the weights are loaded together by all threads, not by a warp per token, the weights behind the sum.
// A block of 2 / 4 / 13 tokens 35.8 / 50.6 / 96.4 -> 32.4 / 47.3 / 93.5 us.
constexpr int NORM_THREADS = 256, NORM_REGS = 2;  // float4 of row and weights a thread keeps (rows up to 2048)
__global__ void __launch_bounds__(NORM_THREADS) rms_norm_rows(const float *__restrict__ x, const float *__restrict__ w,
							      float *__restrict__ o, int n, float eps)
{
	extern __shared__ float xs[];
	__shared__ float s_inv;
	const float4 *xr = reinterpret_cast<const float4 *>(x + (size_t)blockIdx.x * n), *w4 = reinterpret_cast<const float4 *>(w);
	float4 *orow = reinterpret_cast<float4 *>(o + (size_t)blockIdx.x * n), *xs4 = reinterpret_cast<float4 *>(xs);
	float4 v[NORM_REGS], g[NORM_REGS];
#pragma unroll
	for (int j = 0; j < NORM_REGS; j++) {
		const int i = threadIdx.x + j * NORM_THREADS;
		g[j] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
		if (i < n / 4) {
			v[j] = xr[i];
			if (w)
				g[j] = __ldg(w4 + i);
		}
	}
#pragma unroll
	for (int j = 0; j < NORM_REGS; j++)
		if (threadIdx.x + j * NORM_THREADS < n / 4)
			xs4[threadIdx.x + j * NORM_THREADS] = v[j];
	for (int i = threadIdx.x + NORM_REGS * NORM_THREADS; i < n / 4; i += NORM_THREADS)
		xs4[i] = xr[i];
	__syncthreads();
	if (threadIdx.x < 32) {
		const int lane = threadIdx.x;
		float acc = 0.f;
		if (lane < 8) {
#pragma unroll 32
			for (int i = 0; i < n / 8; i++) {
				const float a = xs[8 * i + lane];
				acc = __fmaf_rn(a, a, acc);
			}
		}
		const float v4 = __fadd_rn(acc, __shfl_down_sync(0xffffffffu, acc, 4));
		const float t2 = __fadd_rn(v4, __shfl_down_sync(0xffffffffu, v4, 1));
		const float ss = __fadd_rn(t2, __shfl_down_sync(0xffffffffu, t2, 2));
		if (lane == 0)
			s_inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)n), eps)));
	}
	__syncthreads();
	pdl_trigger();	// the router may come and fetch its first weights (from the start of the grid: 512 tokens 199 -> 210 us)
	const float inv = s_inv;
	auto put = [&](int i, const float4 &a, const float4 &b) {
		orow[i] = make_float4(__fmul_rn(__fmul_rn(a.x, b.x), inv), __fmul_rn(__fmul_rn(a.y, b.y), inv),
				      __fmul_rn(__fmul_rn(a.z, b.z), inv), __fmul_rn(__fmul_rn(a.w, b.w), inv));
	};
#pragma unroll
	for (int j = 0; j < NORM_REGS; j++)
		if (threadIdx.x + j * NORM_THREADS < n / 4)
			put(threadIdx.x + j * NORM_THREADS, v[j], g[j]);
	for (int i = threadIdx.x + NORM_REGS * NORM_THREADS; i < n / 4; i += NORM_THREADS)
		put(i, xs4[i], w ? __ldg(w4 + i) : make_float4(1.0f, 1.0f, 1.0f, 1.0f));
}

// model_qwen3.c:458-467: acc = 0; acc += w_j * y_j, j ascending (fused multiply-add, as the
// reference compiles it).  residual != null: out = residual + acc (math_avx2.c:731-751).
// pos != null: the row of (t, j) is y[pos[t*top_k + j]] instead of y[t*top_k + j] (< 0, after a call that reports an
// expert out of range: any row).
__global__ void __launch_bounds__(512) combine_rows(const float *__restrict__ y, const float *__restrict__ topk_w, int top_k,
						    int hidden, const float *__restrict__ residual, float *__restrict__ out,
						    const int *__restrict__ pos)
{
	const int t = blockIdx.x;
	pdl_wait();
	float wj[MAX_TOP_K];
	size_t yrow[MAX_TOP_K];
#pragma unroll
	for (int j = 0; j < MAX_TOP_K; j++) {
		wj[j] = (j < top_k) ? topk_w[(size_t)t * top_k + j] : 0.f;
		yrow[j] = (j < top_k) ? (size_t)(pos ? max(pos[(size_t)t * top_k + j], 0) : t * top_k + j) * hidden : 0;
	}
	for (int k = threadIdx.x * 4; k < hidden; k += blockDim.x * 4) {
		float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
		for (int j = 0; j < MAX_TOP_K; j++) {
			if (j < top_k) {
				float4 v = *reinterpret_cast<const float4 *>(y + yrow[j] + k);
				acc.x = __fmaf_rn(wj[j], v.x, acc.x);
				acc.y = __fmaf_rn(wj[j], v.y, acc.y);
				acc.z = __fmaf_rn(wj[j], v.z, acc.z);
				acc.w = __fmaf_rn(wj[j], v.w, acc.w);
			}
		}
		if (residual) {
			float4 r = *reinterpret_cast<const float4 *>(residual + (size_t)t * hidden + k);
			acc.x = __fadd_rn(r.x, acc.x);
			acc.y = __fadd_rn(r.y, acc.y);
			acc.z = __fadd_rn(r.z, acc.z);
			acc.w = __fadd_rn(r.w, acc.w);
		}
		*reinterpret_cast<float4 *>(out + (size_t)t * hidden + k) = acc;
	}
}

constexpr int ROWS_WARPS = 8;  // warps per CTA of the row passes: one row per warp at a time

// The rows of a dense product's batch, split (Split8), and their sub-block sums (xq, optional, q_cols per row: the Q4_K
// "min" term).  A warp takes STEPS x 256 columns of a row, eight values per lane and step (16-byte loads and
// stores); n_cols must be a multiple of 256.
template <int STEPS>
__global__ void __launch_bounds__(ROWS_WARPS * 32) split_rows(const float *__restrict__ x, int n_src, int n_cols, __half *__restrict__ hi,
							      __half *__restrict__ lo, __half *__restrict__ xq, int q_cols)
{
	pdl_trigger();	// (the product sets itself up meanwhile)
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int upr = (n_cols + STEPS * 256 - 1) / (STEPS * 256);  // units per row
	for (int un = blockIdx.x * ROWS_WARPS + warp; un < n_src * upr; un += gridDim.x * ROWS_WARPS) {
		const int t = un / upr;
		SplitUnit<STEPS> u;
		u.load(x + (size_t)t * n_cols, (un - t * upr) * STEPS * 256 + lane * 8, n_cols);
		u.split(xq != nullptr);
		u.store(hi + (size_t)t * n_cols, lo + (size_t)t * n_cols, xq ? xq + (size_t)t * q_cols : nullptr, lane);
	}
}

// Expert-parallel dispatch payload: rows in expert-sorted order, their expert ids, and the
// inverse permutation (row id -> sorted position) for the combine on the way back.
__global__ void __launch_bounds__(256) gather_rows(const float *__restrict__ x, const int *__restrict__ row_expert,
						   const int *__restrict__ perm, int src_div, int n_cols,
						   float *__restrict__ rows_out, int *__restrict__ expert_out, int *__restrict__ inv)
{
	const int p = blockIdx.x;
	int rid = perm[p];
	if ((unsigned)rid >= gridDim.x)  // stale entry behind the rows the sort placed (an expert id was out of range)
		rid = 0;
	const float4 *xr = reinterpret_cast<const float4 *>(x + (size_t)(rid / src_div) * n_cols);
	float4 *orow = reinterpret_cast<float4 *>(rows_out + (size_t)p * n_cols);
	for (int k = threadIdx.x; k < n_cols / 4; k += blockDim.x)
		orow[k] = xr[k];
	if (threadIdx.x == 0) {
		expert_out[p] = row_expert[rid];
		inv[rid] = p;
	}
}

__global__ void __launch_bounds__(256) swiglu_kernel(float *__restrict__ gate, const float *__restrict__ up, int n,
						     const float *__restrict__ silu)
{
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n)
		gate[i] = swiglu_lut(silu, gate[i], up[i]);
}

int launch_rms_norm(tie_cuda_ctx *c, const float *x, const float *w, float *o, int n_tokens)
{
	const int H = c->cfg.hidden;
	const size_t smem = (size_t)H * sizeof(float);
	if (smem > 47 * 1024)  // the kernel runs within the default dynamic shared-memory limit
		return TIE_CUDA_ENOTSUP;
	rms_norm_rows<<<n_tokens, NORM_THREADS, smem, c->stream>>>(x, w, o, H, c->cfg.norm_eps);
	TIE_CUDA_LAUNCHED(c);
	return TIE_CUDA_OK;
}

int launch_combine(tie_cuda_ctx *c, const float *y, const float *topk_w, int n_tokens, const float *residual, float *out,
		   const int *pos, bool dependent)
{
	// Few tokens: a thread per 16 bytes of the row, so that nothing comes in turn (64 tokens a step 124.3 -> 123.0 us, 13 84.7 ->
	// 83.4); from two CTAs per SM on 256 threads (4096 tokens 59 us, with 512 72).
	const int threads = n_tokens < 2 * c->sm_count && c->cfg.hidden >= 2048 ? 512 : 256;
	return launch_kernel(c, dependent, 1, combine_rows, dim3(n_tokens), threads, 0, y, topk_w, c->cfg.top_k, c->cfg.hidden, residual, out, pos);
}

int launch_split_rows(tie_cuda_ctx *c, const float *x, int n_src, int n_cols, __half *hi, __half *lo, __half *xq)
{
	if (n_cols % 256)
		return TIE_CUDA_ENOTSUP;
	if (n_src <= 0)
		return TIE_CUDA_OK;
	// units of 1024 columns where they are enough to fill the SMs a few times over, else of 256
	const bool wide = (long long)n_src * ((n_cols + 1023) / 1024) >= 4ll * ROWS_WARPS * c->sm_count;
	const long long units = (long long)n_src * (wide ? (n_cols + 1023) / 1024 : n_cols / 256), cap = c->sm_count * 8;
	const long long want = (units + ROWS_WARPS - 1) / ROWS_WARPS;
	auto kern = wide ? split_rows<4> : split_rows<1>;
	kern<<<(int)(want < cap ? want : cap), ROWS_WARPS * 32, 0, c->stream>>>(x, n_src, n_cols, hi, lo, xq, xq_cols(n_cols));
	TIE_CUDA_LAUNCHED(c);
	return TIE_CUDA_OK;
}

int launch_gather_rows(tie_cuda_ctx *c, const float *x, const int *row_expert, const int *perm, int src_div, int n_rows,
		       float *rows_out, int *expert_out, int *inv)
{
	gather_rows<<<n_rows, 256, 0, c->stream>>>(x, row_expert, perm, src_div, c->cfg.hidden, rows_out, expert_out, inv);
	TIE_CUDA_LAUNCHED(c);
	return TIE_CUDA_OK;
}

int launch_swiglu(tie_cuda_ctx *c, float *gate, const float *up, int n)
{
	swiglu_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(gate, up, n, c->silu);
	TIE_CUDA_LAUNCHED(c);
	return TIE_CUDA_OK;
}

}  // namespace tie
