// Packed Q4_K / Q6_K quants -> exact small-integer fp16 MMA operands, in packed half2 arithmetic.
//
// A weight of a super-block (256 k) factors as
//   Q4_K: w = d * (sc_b * q) - dmin * m_b      (sc_b, m_b 6-bit, q 4-bit)   math_scalar.c:216-255
//   Q6_K: w = d * (sc_b * (q - 32))            (sc_b int8, q 6-bit)         math_scalar.c:257-287
// with d, dmin constant over the super-block.  The integer products sc_b*q (<= 945) and
// sc_b*(q-32) are what the tensor cores multiply: they are EXACT in fp16 up to 2048 (the Q6_K
// product can reach 4096; above 2048 an odd product is off by 1, at most 2^-11 of that one
// weight).  The fp32 factors d and dmin are applied when a super-block's partial sums are
// taken out of tensor memory, so no low-order operand is needed for the weights.
//
// Quants become halves without conversion instructions: a 16-bit field 0x6400 | q is the half
// 1024 + q, 0x6400 | (q << 4) is 1024 + 16 q (q < 64); one HFMA2 with a per-sub-block scale and
// offset then yields sc*q for two weights (the offset is a half and the product inside the fused
// multiply-add is exact, so the result is the integer, rounded once where it has more than 11
// bits).  The same for sc*(q-32) from 1024 + 16 q, whose offset -96 sc is a half; from 1024 + q it would
// be -1056 sc, which is none, so 1056 is subtracted first (exactly) and the product rounds.  The two halves of
// such a pair come from bytes 0 and 2 (or 1 and 3) of a 32-bit word, so within every group of 4
// consecutive k the operand tiles hold the order [k0, k2, k1, k3]; the token operand is written in
// the same order (split_rows, the gate/up epilogue), so the contraction is unchanged.
#pragma once

#include "common.cuh"

namespace tie {

__device__ __forceinline__ uint32_t h2_bits(__half2 v)
{
	return *reinterpret_cast<uint32_t *>(&v);
}
__device__ __forceinline__ __half2 bits_h2(uint32_t v)
{
	return *reinterpret_cast<__half2 *>(&v);
}

// (w & mask) | magic in ONE logic instruction.  Two literal constants do not fit one instruction, and left
// to itself the compiler spends two; the expansion is bound by the logic pipe.
__device__ __forceinline__ uint32_t and_or(uint32_t w, uint32_t mask, uint32_t magic)
{
	uint32_t r;
	asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "r"(mask), "r"(magic));
	return r;
}

// Scale constants of one Q4_K sub-block pair (low nibbles: sub-block 2p, high nibbles: 2p+1).
struct Q4kConsts {
	__half2 sl, cl;	 // low nibbles:  (1024 + q)    * s      - 1024 s
	__half2 sh, ch;	 // high nibbles: (1024 + 16 q) * (s/16) -   64 s
};

// One 32-bit word of Q4_K quants (4 bytes = 4 low + 4 high nibbles) -> sc*q as half2 pairs:
// lo[0] = bytes (0, 2), lo[1] = bytes (1, 3) of the low nibbles; hi[] the same of the high ones.
__device__ __forceinline__ void q4k_int_word(uint32_t w, const Q4kConsts &c, uint32_t lo[2], uint32_t hi[2])
{
	const uint32_t w8 = w >> 8;
	lo[0] = h2_bits(__hfma2(bits_h2(and_or(w, 0x000F000Fu, 0x64006400u)), c.sl, c.cl));
	lo[1] = h2_bits(__hfma2(bits_h2(and_or(w8, 0x000F000Fu, 0x64006400u)), c.sl, c.cl));
	hi[0] = h2_bits(__hfma2(bits_h2(and_or(w, 0x00F000F0u, 0x64006400u)), c.sh, c.ch));
	hi[1] = h2_bits(__hfma2(bits_h2(and_or(w8, 0x00F000F0u, 0x64006400u)), c.sh, c.ch));
}

// Eight 6-bit quants: their low four bits are the bytes' low (first four) and high nibbles of a, their high two bits lie
// in the bytes of h, SHIFT bits below bit 4 and below bit 8.  Both are ORed into mantissas where they stand, with
// one shift of a and two of h for all eight (joined into bytes first, 18 instructions of the logic pipe instead of 11):
// lo[0] = 1024 + q of bytes (0, 2), lo[1] of bytes (1, 3), hi[] = 1024 + 16 q.
template <int SHIFT>
__device__ __forceinline__ void q6k_word(uint32_t a, uint32_t h, uint32_t lo[2], uint32_t hi[2])
{
	const uint32_t a8 = a >> 8, hl = h << SHIFT, hr = h >> (8 - SHIFT);
	lo[0] = and_or(hl, 0x00300030u, and_or(a, 0x000F000Fu, 0x64006400u));
	lo[1] = and_or(hr, 0x00300030u, and_or(a8, 0x000F000Fu, 0x64006400u));
	hi[0] = and_or(hl, 0x03000300u, and_or(a, 0x00F000F0u, 0x64006400u));
	hi[1] = and_or(hr, 0x03000300u, and_or(a8, 0x00F000F0u, 0x64006400u));
}

}  // namespace tie
