// Warp-level products of 16 packed weight rows x one super-block with ONE activation row on the
// mma.sync tensor path, exact to fp32: the building block of the decode kernels (decode.cu,
// decode_group.cu, decode_fused.cu), which stay bit-identical to one another because they share it.
//
// An activation row enters as THREE fp16 parts (hi, mid, lo: 33 significand bits after a power-of-two
// scaling of the super-block: fp32 values down to 2^-10 of the super-block's largest are represented exactly,
// smaller ones to 2^-34 of the largest) that sit in columns 0, 1, 2 of the MMA's 8 (a second row's in 4, 5, 6):
// one m16n8k16 covers 16 rows x 16 k of all three, and the columns are added in fp32 at the end.  The weights
// are exact small integers in fp16 (tc_dequant.cuh): sc*q for Q4_K, q - 32 for Q6_K, whose 16-wide scale groups are one MMA each and are scaled in fp32 afterwards (their
// products sc*(q-32) would not always fit 11 bits).  A lane therefore expands packed words straight into its
// fragment registers, 4.5 (Q4_K) to 7 (Q6_K) instructions per 4 weights where a scalar reduction needs 12 to
// 16, needs no activations in registers, and the k order inside a super-block is free: lane t of a
// quad takes sub-blocks 2t and 2t+1 (Q4_K) resp. the 4 weights 4t .. 4t+3 of each scale group (Q6_K).
#pragma once

#include "common.cuh"
#include "tc_dequant.cuh"

namespace tie {

// Shared-memory image of one super-block (256 values) of an activation row: parts[p] in the order
// [k0, k2, k1, k3] of every group of 4, blocks of 64 values PAD bytes apart so that the fragment loads have no
// bank conflicts, then the parts of the 8 sub-block sums (Q4_K).
template <WKind KIND>
struct XImage {
	static constexpr int BLK = KIND == W_Q4K ? 144 : 128;	       // bytes from one block of 64 values to the next
	static constexpr int PART = KIND == W_Q4K ? 4 * 144 : 512 + 32;  // ... from one part to the next
	static constexpr int SUMS = 3 * PART;
	static constexpr int BYTES = SUMS + (KIND == W_Q4K ? 3 * 16 : 0);
	static_assert(BYTES % 16 == 0, "image size");
};

// A float rounded to a multiple of the last bit of c = 1.5 x 2^n (it has to be below 2^(n-1)).
__device__ __forceinline__ float on_grid(float v, float c)
{
	return __fsub_rn(__fadd_rn(v, c), c);
}

// One warp: 8 consecutive values per lane -> the image; returns the factor that undoes the scaling.
// The values are scaled by a power of two so that the largest lies in [2^9, 2^10): sums of 32 stay
// inside fp16, and a part's last bit is 2^-24.
// The parts lie on fixed grids, multiples of 2^-1 and of 2^-12 (sums of 32: 2^4, 2^-7) and what is left: the tensor
// cores cut the low bits off a sum at every step, always towards zero, and on a grid the products (at most 21 bits) add
// up to what 24 bits hold, nearly always.  (Parts rounded each to its own 11 bits: a block of 1 - 8 tokens was 2.9e-7 -
// 4.5e-7 from 64-bit arithmetic, in fp32 throughout 0.6e-7 - 2.9e-7.)
template <WKind KIND>
__device__ __forceinline__ float x_image(const float (&v)[8], uint8_t *img, int lane)
{
	unsigned m = 0;
#pragma unroll
	for (int i = 0; i < 8; i++)
		m = max(m, __float_as_uint(v[i]) & 0x7fffffffu);
	m = __reduce_max_sync(0xffffffffu, m);
	int e = (int)(m >> 23);		    // biased exponent of the largest magnitude
	e = e == 255 ? 136 : max(e, 20);    // (inf / nan: unscaled; zeros and denormals: any scale whose inverse is a number)
	const float s = __uint_as_float((unsigned)(127 + 136 - e) << 23), inv = __uint_as_float((unsigned)(127 - 136 + e) << 23);
	uint32_t part[3][4];
	float sum = 0.0f;
#pragma unroll
	for (int g = 0; g < 2; g++) {
		const float a[4] = {v[4 * g] * s, v[4 * g + 2] * s, v[4 * g + 1] * s, v[4 * g + 3] * s};
		sum += (a[0] + a[2]) + (a[1] + a[3]);
#pragma unroll
		for (int h = 0; h < 2; h++) {
			float r0 = a[2 * h], r1 = a[2 * h + 1];
#pragma unroll
			for (int p = 0; p < 3; p++) {
				const float c = p == 0 ? 0x1.8p22f : 0x1.8p11f, q0 = p < 2 ? on_grid(r0, c) : r0, q1 = p < 2 ? on_grid(r1, c) : r1;
				part[p][2 * g + h] = h2_bits(__floats2half2_rn(q0, q1));
				r0 -= q0;
				r1 -= q1;
			}
		}
	}
	__syncwarp();  // (the image may still be read as the previous one)
	uint8_t *d = img + (lane >> 3) * XImage<KIND>::BLK + (lane & 7) * 16;
#pragma unroll
	for (int p = 0; p < 3; p++)
		*reinterpret_cast<uint4 *>(d + p * XImage<KIND>::PART) = make_uint4(part[p][0], part[p][1], part[p][2], part[p][3]);
	if (KIND == W_Q4K) {
		sum += __shfl_xor_sync(0xffffffffu, sum, 1);
		sum += __shfl_xor_sync(0xffffffffu, sum, 2);
		if ((lane & 3) == 0) {
#pragma unroll
			for (int p = 0; p < 3; p++) {
				const float q = p < 2 ? on_grid(sum, p == 0 ? 0x1.8p27f : 0x1.8p16f) : sum;
				reinterpret_cast<__half *>(img + XImage<KIND>::SUMS + 16 * p)[lane >> 2] = __float2half_rn(q);
				sum -= q;
			}
		}
	}
	__syncwarp();
	return inv;
}

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
	asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
	    : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
	    : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_1688(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0)
{
	asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
	    : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
	    : "r"(a0), "r"(a1), "r"(b0));
}

// Where a lane's column of the MMA (column g = lane / 4) has its activations: a part of an image, and that part's sums.
// A column that carries nothing reads zeros (ALL) or is off.
template <bool ALL>
struct MmaCol {
	const uint8_t *x, *sums;
	bool on;
	__device__ __forceinline__ bool reads() const { return ALL || on; }
};
// one activation row: columns 0, 1, 2 are its parts
template <WKind KIND>
__device__ __forceinline__ MmaCol<false> one_row(const uint8_t *img, int lane)
{
	const int g = lane >> 2;
	return {img + g * XImage<KIND>::PART, img + XImage<KIND>::SUMS + 16 * g, g < 3};
}
// rows m0 and m0 + 1 of n_rows (their images `stride` bytes apart): columns 0 .. 2 and 4 .. 6
template <WKind KIND>
__device__ __forceinline__ MmaCol<true> two_rows(const uint8_t *img, int stride, int m0, int n_rows, const uint8_t *zeros, int lane)
{
	const int part = (lane >> 2) & 3, m = m0 + (lane >> 4);
	if (part == 3 || m >= n_rows)
		return {zeros, zeros, false};
	img += m * stride;
	return {img + part * XImage<KIND>::PART, img + XImage<KIND>::SUMS + 16 * part, true};
}

// What lane (g = lane / 4, t = lane % 4) holds of the packed rows g and g + 8 of a 16-row tile.
template <WKind KIND>
struct MmaRows;

// The products of a super-block: c[0] + c[1] is row g's, c[2] + c[3] row g + 8's, over two lanes of the quad.
__device__ __forceinline__ float2 quad_rows(const float (&c)[4])
{
	float r0 = c[0] + c[1], r1 = c[2] + c[3];  // lane t = 0: columns 0, 1 (hi, mid); t = 1: 2 (lo), 3 (nothing); t = 2, 3: the second row's
	r0 += __shfl_xor_sync(0xffffffffu, r0, 1);
	r1 += __shfl_xor_sync(0xffffffffu, r1, 1);
	return make_float2(r0, r1);  // (valid in lanes t = 0, 1; two_rows: the second row's in t = 2, 3)
}

template <>
struct MmaRows<W_Q4K> {
	uint4 hdr[2], q[2][2];
	// rows: address of row 0 of the tile at super-block b (row stride in bytes); SMEM: staged there
	__device__ __forceinline__ void load(const uint8_t *tile, int nb, int b, int lane)
	{
		const int g = lane >> 2, t = lane & 3;
#pragma unroll
		for (int r = 0; r < 2; r++) {
			const uint8_t *blk = tile + ((size_t)(g + 8 * r) * nb + b) * Q4K_BYTES;
			hdr[r] = __ldg(reinterpret_cast<const uint4 *>(blk));
			q[r][0] = __ldg(reinterpret_cast<const uint4 *>(blk + 16 + 32 * t));
			q[r][1] = __ldg(reinterpret_cast<const uint4 *>(blk + 32 + 32 * t));
		}
	}
	// the same from a tile staged in shared memory (rows of 128-byte multiples: odd rows take their halves in
	// the other order, so that a quarter of the warp covers all banks)
	__device__ __forceinline__ void load_smem(const uint8_t *tile, int nb, int b, int lane)
	{
		const int g = lane >> 2, t = lane & 3, odd = g & 1;
#pragma unroll
		for (int r = 0; r < 2; r++) {
			const uint8_t *blk = tile + ((size_t)(g + 8 * r) * nb + b) * Q4K_BYTES;
			hdr[r] = *reinterpret_cast<const uint4 *>(blk);
			const uint4 u = *reinterpret_cast<const uint4 *>(blk + 16 + 32 * t + 16 * odd);
			const uint4 v = *reinterpret_cast<const uint4 *>(blk + 16 + 32 * t + 16 * (odd ^ 1));
			q[r][0] = odd ? v : u;
			q[r][1] = odd ? u : v;
		}
	}
	// the same from super-block b of a tile staged by itself (ChunkCopy)
	__device__ __forceinline__ void load_chunk(const uint8_t *chunk, const uint8_t *, int, int, int lane)
	{
		const int g = lane >> 2, t = lane & 3;
#pragma unroll
		for (int r = 0; r < 2; r++) {
			const uint8_t *blk = chunk + (g + 8 * r) * Q4K_BYTES;
			hdr[r] = *reinterpret_cast<const uint4 *>(blk);
			q[r][0] = *reinterpret_cast<const uint4 *>(blk + 16 + 32 * t);
			q[r][1] = *reinterpret_cast<const uint4 *>(blk + 32 + 32 * t);
		}
	}
	__device__ __forceinline__ float2 scale(float inv) const { return make_float2(inv, inv); }
	// the tile's products with a row are scale(inv).x * r.x (row g) and scale(inv).y * r.y (row g + 8); NP MMAs, of one or two
	// rows each, share the expanded weights
	template <int NP, bool ALL>
	__device__ __forceinline__ void dot(const MmaCol<ALL> (&col)[NP], int lane, float2 (&r)[NP]) const
	{
		const int t = lane & 3;
		const __half2 k1024 = __float2half2_rn(1024.0f);
		Q4kConsts c[2];
		uint32_t mins[2];
#pragma unroll
		for (int w = 0; w < 2; w++) {
			// scales and mins of sub-blocks 2t, 2t + 1 (get_scale_min_k4, math_scalar.c:91-100)
			const uint4 h = hdr[w];
			const uint32_t sc8 = t & 2 ? and_or(h.y >> 2, 0x30303030u, h.w & 0x0F0F0F0Fu) : h.y & 0x3F3F3F3Fu;
			const uint32_t mn8 = t & 2 ? and_or(h.z >> 2, 0x30303030u, (h.w >> 4) & 0x0F0F0F0Fu) : h.z & 0x3F3F3F3Fu;
			const uint32_t sc = sc8 >> (16 * (t & 1)), mn = mn8 >> (16 * (t & 1));
			const __half2 s_lo = __hsub2(bits_h2(__byte_perm(sc, 0x64006400u, 0x7050u)), k1024);
			const __half2 s_hi = __hsub2(bits_h2(__byte_perm(sc, 0x64006400u, 0x7151u)), k1024);
			c[w].sl = s_lo;
			c[w].cl = __hmul2(s_lo, __float2half2_rn(-1024.0f));
			c[w].sh = __hmul2(s_hi, __float2half2_rn(0.0625f));
			c[w].ch = __hmul2(s_hi, __float2half2_rn(-64.0f));
			mins[w] = h2_bits(__hsub2(bits_h2(__byte_perm(mn, 0x64006400u, 0x7170u)), k1024));
		}
		float lo[NP][4], hi[NP][4], mm[NP][4];
#pragma unroll
		for (int p = 0; p < NP; p++) {
#pragma unroll
			for (int i = 0; i < 4; i++)
				lo[p][i] = hi[p][i] = mm[p][i] = 0.f;
			mma_1688(mm[p], mins[0], mins[1], col[p].reads() ? *reinterpret_cast<const uint32_t *>(col[p].sums + 4 * t) : 0u);
		}
#pragma unroll
		for (int i2 = 0; i2 < 4; i2++) {  // two words: 8 k of either sub-block
			uint4 bl[NP], bh[NP];
#pragma unroll
			for (int p = 0; p < NP; p++) {
				const uint8_t *xp = col[p].x + t * XImage<W_Q4K>::BLK;
				bl[p] = bh[p] = make_uint4(0, 0, 0, 0);
				if (col[p].reads()) {
					bl[p] = *reinterpret_cast<const uint4 *>(xp + 16 * i2);
					bh[p] = *reinterpret_cast<const uint4 *>(xp + 64 + 16 * i2);
				}
			}
			const uint4 w0 = q[0][i2 >> 1], w1 = q[1][i2 >> 1];
			const uint32_t wa[2] = {i2 & 1 ? w0.z : w0.x, i2 & 1 ? w0.w : w0.y}, wb[2] = {i2 & 1 ? w1.z : w1.x, i2 & 1 ? w1.w : w1.y};
#pragma unroll
			for (int j = 0; j < 2; j++) {
				uint32_t l0[2], h0[2], l1[2], h1[2];
				q4k_int_word(wa[j], c[0], l0, h0);
				q4k_int_word(wb[j], c[1], l1, h1);
#pragma unroll
				for (int p = 0; p < NP; p++) {
					mma_16816(lo[p], l0[0], l1[0], l0[1], l1[1], j ? bl[p].z : bl[p].x, j ? bl[p].w : bl[p].y);
					mma_16816(hi[p], h0[0], h1[0], h0[1], h1[1], j ? bh[p].z : bh[p].x, j ? bh[p].w : bh[p].y);
				}
			}
		}
#pragma unroll
		for (int p = 0; p < NP; p++) {
			float s[4];
#pragma unroll
			for (int i = 0; i < 4; i++) {
				const uint32_t h = hdr[i >> 1].x;
				s[i] = half_bits_to_float(h & 0xffffu) * (lo[p][i] + hi[p][i]) - half_bits_to_float(h >> 16) * mm[p][i];
			}
			r[p] = quad_rows(s);
		}
	}
};

template <>
struct MmaRows<W_Q6K_R8> {
	uint32_t a[2][4], b[2][4], h[2][4], sc[2][4];
	float d[2];
	// tile: first of the two R8 groups of 8 rows (each q6k_r8_group_bytes(nb) long)
	// chunk != null: the records lie there by themselves (ChunkCopy), only d is fetched from the tile
	template <bool SMEM, bool CHUNK = false>
	__device__ __forceinline__ void load_t(const uint8_t *tile, int nb, int blk, int lane, const uint8_t *chunk = nullptr)
	{
		const int g = lane >> 2, t = lane & 3;
#pragma unroll
		for (int r = 0; r < 2; r++) {
			const uint8_t *grp = tile + r * q6k_r8_group_bytes(nb);
			const uint8_t *rec = CHUNK ? chunk + (g + 8 * r) * Q6K_RECORD : grp + (size_t)(g * nb + blk) * Q6K_RECORD;
#pragma unroll
			for (int pp = 0; pp < 4; pp++) {
				const uint32_t *p = reinterpret_cast<const uint32_t *>(rec + 48 * pp + 4 * t);
				const uint32_t *ps = reinterpret_cast<const uint32_t *>(rec + 192 + 4 * pp);
				a[r][pp] = SMEM ? p[0] : __ldg(p);
				b[r][pp] = SMEM ? p[4] : __ldg(p + 4);
				h[r][pp] = SMEM ? p[8] : __ldg(p + 8);
				sc[r][pp] = SMEM ? *ps : __ldg(ps);
			}
			const unsigned short *pd = reinterpret_cast<const unsigned short *>(grp + q6k_r8_d_off(nb, g, blk));
			d[r] = half_bits_to_float(SMEM && !CHUNK ? *pd : __ldg(pd));
		}
	}
	__device__ __forceinline__ void load(const uint8_t *tile, int nb, int blk, int lane) { load_t<false>(tile, nb, blk, lane); }
	__device__ __forceinline__ void load_smem(const uint8_t *tile, int nb, int blk, int lane) { load_t<true>(tile, nb, blk, lane); }
	__device__ __forceinline__ void load_chunk(const uint8_t *chunk, const uint8_t *tile, int nb, int blk, int lane)
	{
		load_t<true, true>(tile, nb, blk, lane, chunk);
	}
	__device__ __forceinline__ float2 scale(float inv) const { return make_float2(d[0] * inv, d[1] * inv); }
	template <int NP, bool ALL>
	__device__ __forceinline__ void dot(const MmaCol<ALL> (&col)[NP], int lane, float2 (&r)[NP]) const
	{
		const int t = lane & 3;
		const __half2 k1056 = __float2half2_rn(1056.0f), k16th = __float2half2_rn(0.0625f), km96 = __float2half2_rn(-96.0f);
		float s[NP][4];
#pragma unroll
		for (int n = 0; n < NP; n++)
#pragma unroll
			for (int i = 0; i < 4; i++)
				s[n][i] = 0.f;
#pragma unroll
		for (int pp = 0; pp < 4; pp++) {
			const uint32_t sx[2] = {sc[0][pp] ^ 0x80808080u, sc[1][pp] ^ 0x80808080u};
			uint32_t w[4][2][2];  // [q][row]
#pragma unroll
			for (int i = 0; i < 2; i++) {
				q6k_word<4>(a[i][pp], h[i][pp], w[0][i], w[2][i]);
				q6k_word<2>(b[i][pp], h[i][pp], w[1][i], w[3][i]);
#pragma unroll
				for (int e = 0; e < 2; e++) {
					w[0][i][e] = h2_bits(__hsub2(bits_h2(w[0][i][e]), k1056));
					w[1][i][e] = h2_bits(__hsub2(bits_h2(w[1][i][e]), k1056));
					w[2][i][e] = h2_bits(__hfma2(bits_h2(w[2][i][e]), k16th, km96));
					w[3][i][e] = h2_bits(__hfma2(bits_h2(w[3][i][e]), k16th, km96));
				}
			}
#pragma unroll
			for (int q = 0; q < 4; q++) {  // 16 weights: l + 32 q of the half, one scale
				// int8 scale -> float: 2^23 + (s + 128), less 2^23 + 128
				const float s0 = __uint_as_float(__byte_perm(sx[0], 0x4B000000u, 0x7650u | q)) - 8388736.0f;
				const float s1 = __uint_as_float(__byte_perm(sx[1], 0x4B000000u, 0x7650u | q)) - 8388736.0f;
#pragma unroll
				for (int n = 0; n < NP; n++) {
					uint2 x = make_uint2(0, 0);
					if (col[n].reads())
						x = *reinterpret_cast<const uint2 *>(col[n].x + 8 * t + 2 * (128 * (pp >> 1) + 16 * (pp & 1) + 32 * q));
					float p[4] = {0.f, 0.f, 0.f, 0.f};
					mma_16816(p, w[q][0][0], w[q][1][0], w[q][0][1], w[q][1][1], x.x, x.y);
					s[n][0] = __fmaf_rn(s0, p[0], s[n][0]);
					s[n][1] = __fmaf_rn(s0, p[1], s[n][1]);
					s[n][2] = __fmaf_rn(s1, p[2], s[n][2]);
					s[n][3] = __fmaf_rn(s1, p[3], s[n][3]);
				}
			}
		}
#pragma unroll
		for (int n = 0; n < NP; n++)
			r[n] = quad_rows(s[n]);
	}
};

template <WKind KIND, bool ALL>
__device__ __forceinline__ float2 dot_one(const MmaRows<KIND> &w, const MmaCol<ALL> &col, int lane)
{
	const MmaCol<ALL> c[1] = {col};
	float2 r[1];
	w.dot(c, lane, r);
	return r[0];
}

}  // namespace tie
