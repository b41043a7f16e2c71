// fp32 activations as the tensor-core path's token operand: fp16 hi + lo halves and sub-block sums.
#pragma once

#include "common.cuh"

namespace tie {

// Eight consecutive values v[0..7] (k = k0 .. k0+7, k0 a multiple of 8) as their fp16 hi and lo
// halves (hi = rn16(v), lo = rn16(v - hi)) in the operand order [k0, k2, k1, k3] per group of 4, and the
// sum over the 32-wide sub-block they belong to (four neighbouring lanes hold one), split the same way.
struct Split8 {
	uint4 hi, lo;
	__half sum_hi, sum_lo;
	__device__ __forceinline__ void make(const float v[8], bool sums)
	{
		uint32_t h[4], l[4];
#pragma unroll
		for (int g = 0; g < 2; g++) {
			const float a = v[4 * g], b = v[4 * g + 1], c = v[4 * g + 2], d = v[4 * g + 3];
			const __half2 h0 = __floats2half2_rn(a, c), h1 = __floats2half2_rn(b, d);
			const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
			const __half2 l0 = __floats2half2_rn(a - f0.x, c - f0.y), l1 = __floats2half2_rn(b - f1.x, d - f1.y);
			h[2 * g] = *reinterpret_cast<const uint32_t *>(&h0);
			h[2 * g + 1] = *reinterpret_cast<const uint32_t *>(&h1);
			l[2 * g] = *reinterpret_cast<const uint32_t *>(&l0);
			l[2 * g + 1] = *reinterpret_cast<const uint32_t *>(&l1);
		}
		hi = make_uint4(h[0], h[1], h[2], h[3]);
		lo = make_uint4(l[0], l[1], l[2], l[3]);
		if (sums) {
			float sum = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
			sum += __shfl_xor_sync(0xffffffffu, sum, 1);
			sum += __shfl_xor_sync(0xffffffffu, sum, 2);
			sum_hi = __float2half_rn(sum);
			sum_lo = __float2half_rn(sum - __half2float(sum_hi));
		}
	}
	__device__ __forceinline__ void store(int k0, __half *__restrict__ hi_row, __half *__restrict__ lo_row, __half *__restrict__ q_row,
					      int lane) const
	{
		*reinterpret_cast<uint4 *>(hi_row + k0) = hi;
		*reinterpret_cast<uint4 *>(lo_row + k0) = lo;
		if (q_row && (lane & 3) == 0) {
			q_row[xq_index(k0 >> 5)] = sum_hi;
			q_row[xq_index(k0 >> 5) + 8] = sum_lo;
		}
	}
};

// A warp's STEPS x 256 columns of a row (k: the lane's first), read and split once and stored at any number of places.
template <int STEPS>
struct SplitUnit {
	float4 v[STEPS][2];
	Split8 p[STEPS];
	int k, n_cols;
	__device__ __forceinline__ void load(const float *__restrict__ row, int k_, int n_cols_)
	{
		k = k_;
		n_cols = n_cols_;
#pragma unroll
		for (int i = 0; i < STEPS; i++)
			if (k + i * 256 < n_cols) {  // (uniform over the warp: n_cols is a multiple of 256)
				v[i][0] = *reinterpret_cast<const float4 *>(row + k + i * 256);
				v[i][1] = *reinterpret_cast<const float4 *>(row + k + i * 256 + 4);
			}
	}
	__device__ __forceinline__ void split(bool sums)
	{
#pragma unroll
		for (int i = 0; i < STEPS; i++)
			if (k + i * 256 < n_cols) {
				const float f[8] = {v[i][0].x, v[i][0].y, v[i][0].z, v[i][0].w, v[i][1].x, v[i][1].y, v[i][1].z, v[i][1].w};
				p[i].make(f, sums);
			}
	}
	__device__ __forceinline__ void store(__half *__restrict__ hi_row, __half *__restrict__ lo_row, __half *__restrict__ q_row, int lane) const
	{
#pragma unroll
		for (int i = 0; i < STEPS; i++)
			if (k + i * 256 < n_cols)
				p[i].store(k + i * 256, hi_row, lo_row, q_row, lane);
	}
};

}  // namespace tie
