// Grouped expert GEMMs for prefill on the 5th-generation tensor cores (tcgen05.mma with the
// weight operand and the accumulators in tensor memory), fed from packed Q4_K / Q6_K super-blocks.
//
// Reference: the same arithmetic as process_expert_task (engine.c:916-964) — gate/up products
// (math_avx2.c:535-604, 753-769), down product (math_avx2.c:411-495, 771-787) — but for all tokens
// routed to an expert at once instead of one token at a time (model_qwen3.c:415).
//
// Formulation: out^T = W . x^T.  Weight rows fill the 128-row M dimension of the MMA (expert row
// counts are multiples of 128), the ragged token count of an expert is the N dimension (tiles of
// up to 64 tokens).  A weight of a 256-wide super-block is d * (integer) - dmin * (integer)
// (tc_dequant.cuh), so the tensor cores multiply integer fp16 weights, exact up to 2048, with the
// activations (split into fp16 hi + lo: 22 significand bits; one fp16 is not accurate enough
// for the 1e-3 parity bound) and the fp32 block factors are applied once per super-block:
//   out[r][n] = sum_B d[r][B] * sum_{k in B} (sc*q)[r][k] * x[n][k]  -  sum_b (dmin*m)[r][b] * xsum[n][b]
// where xsum[n][b] is the sum of x[n] over the 32-wide sub-block b (Q4_K only).  The second term
// is one extra 16-deep MMA step per half super-block into an accumulator of its own: its weights
// dmin*m (17 significant bits) are split into fp16 hi (first half) + lo (second half), the block's 8
// sums lie beside one another as 8 hi + 8 lo halves.
//
// The kernel is persistent: one CTA per SM walks (token tile, 128-row tile) work items.  Roles:
//   * a weight loader thread brings the packed blocks of one super-block x 128 rows into shared
//     memory with TMA (three or four super-blocks in flight: the HBM latency is hidden by the
//     hardware, not by registers, and no thread issues scattered 16-byte loads);
//   * producer warps, in four (or two: TcRoles) groups of 128 threads (one per weight row), expand them (one HFMA2 per two
//     weights) and write the A tiles to TENSOR MEMORY (tcgen05.st) into a ring of four units of half a
//     super-block;
//   * a token loader thread issues TMA tile loads of the token operand (hi/lo fp16, expert-sorted
//     rows: only rows the expert really has) and of the sub-block sums, into rings of their own;
//   * one MMA issuer thread walks the super-blocks: P += A.B_lo over the block's 16-wide k steps, then
//     P += A.B_hi into the same accumulator columns (one column per token; tiles that half fill the
//     columns: one MMA over hi and lo rows, into columns side by side), a super-block per accumulator
//     buffer, two buffers of 64 columns in turn (NT = 32, launches of narrow tiles: four of 32), and the block's min sums into a
//     buffer of their own;
//   * drain warps take a finished super-block out of tensor memory (tcgen05.ld), hand the buffer back
//     at once, fold the values into fp32 registers with d (-1 for the min sums), and after the last
//     super-block of a work item finish and store the rows — while the MMAs of the next super-blocks / work
//     item already run.
// All hand-offs go through mbarriers (tcgen05.commit on the MMA side).  Every wait
// is bounded: on a timeout the CTA raises ST_WAIT_TIMEOUT in the status word, all roles leave their
// loops, tensor memory is released and the kernel returns.
//
// PAIR: the kernel runs as clusters of two CTAs (two SMs) that share a token tile and take two
// neighbouring 128-row weight tiles.  Each CTA loads, expands and drains its own weight tile as
// above, but the MMAs are issued once for both by the even-ranked CTA (tcgen05.mma.cta_group::2,
// M = 256), and the token operand is split between the two CTAs' shared memories: each holds the hi
// and lo rows of half of the tile's tokens, so it fetches half of the operand bytes.
// Barriers that collect arrivals from both CTAs live in the leader (remote mbarrier arrivals; TMA
// loads of the peer count their bytes there); the MMA completions are committed to both CTAs at
// once.  No copy is delivered to more than one CTA.
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "tc_dequant.cuh"
#include "tc_ptx.cuh"

namespace tie {

constexpr int TC_BM = 128;
constexpr int TC_BK = 64;
constexpr int TC_SPB = QK_K / TC_BK;	  // stages per super-block
constexpr int TC_THREADS = (16 + 8 + 3) * 32;  // producer and drain warps (TcRoles), MMA issuer, token loader, weight loader
// Narrow tiles (up to 32 tokens): four groups of producer warps, whose expansion paces them, and two sets of four drain
// warps.  The sets take the work items in turn, so that one finishes its rows while the other folds the next item's super-blocks.
// Wide tiles: eight drain warps a set, half of the tokens for each four.  Gate and up, whose rows take longest to
// finish, have two such sets and two producer groups (4096 tokens 422 -> 387 us, 512 98 -> 90); the others one set and four groups
// (down product of 4096 tokens 217 us, in the form of gate and up 233).
// Registers: the kernel is launched with 72 per thread; the producers give of theirs to the drain warps,
// whose 32 sums per thread otherwise spill (gate/up at 512 tokens 96 -> 90 us, at 4096 414 -> 385 us).
constexpr int TC_LREGS = 72;
template <bool GU, int NT>
struct TcRoles {
	static constexpr int PGROUPS = GU && NT > 32 ? 2 : 4, PWARPS = 4 * PGROUPS, DWARPS = 24 - PWARPS;
	static constexpr int NSETS = GU || NT == 32 ? 2 : 1, SET = DWARPS / NSETS;
	static constexpr int PARTS = SET / 4;  // how many ways a set splits the tokens
	static constexpr int PREGS = PGROUPS == 4 ? 64 : 56, DREGS = PGROUPS == 4 ? 88 : 80;
	static_assert(PARTS == (NT == 32 ? 1 : 2) && PWARPS * PREGS + DWARPS * DREGS <= 24 * TC_LREGS, "roles");
};
constexpr int TC_UNITS = 4;  // slots of the weight ring in tensor memory: half a super-block each
// Super-blocks whose MMAs are in flight or waited for, at most: who waits for one has seen those TC_DONE and more before
// it retire, and none TC_DONE after it can before the wait is over (a phase parity tells neighbouring phases apart, no more).
constexpr int TC_DONE = 8;
constexpr int TC_NDS = 8;    // block-factor hand-off buffers (producers -> drain warps)
constexpr long long TC_WAIT_CYCLES = 1ll << 30;	 // about half a second of SM clocks
constexpr float TC_H_SCALE = 1.0f / 256.0f;	 // keeps SwiGLU outputs inside fp16 range; exact (power of two)

// Tensor-memory columns.  NT: tokens per tile (N of the MMAs, at most), 32 or 64 by the rows per expert
// (run_experts).  What paces narrow tiles is the round trip of an accumulator (MMA, commit, drain, hand-back:
// about 1800 cycles) and the drain's row stores at the end of an item, so tiles of up to 32 tokens get four
// accumulators, and their items go to two sets of drain warps in turn (64 tokens: gate/up 76 -> 71 us, down
// 56 -> 50).
constexpr uint32_t TC_TMEM_COLS = 512;
constexpr int TC_NBUF_MAX = 4;
template <WKind KIND, int NT>
struct TcCols {
	static constexpr bool Q4 = KIND == W_Q4K;
	static constexpr int NBUF = NT == 32 || !Q4 ? 4 : 2;  // accumulators of one super-block
	static constexpr int NM = NT == 32 ? 2 : 1;	      // ... of the min sums of a work item (Q4_K)
	static constexpr uint32_t UNIT = 64 + (Q4 ? 8 : 0);   // one unit of the weight ring
	static constexpr uint32_t M = NBUF * NT, A = M + (Q4 ? NM * NT : 0);
	static_assert(A + TC_UNITS * UNIT <= TC_TMEM_COLS, "tensor memory budget");
};

// shared memory
constexpr int TC_B_BYTES = 128 * 1024;	// token ring: groups of four stages of (hi, lo) x 64 k x the CTA's token rows
constexpr int TC_BG_MAX = 8;
template <bool PAIR, int NT>
struct TcRing {
	static constexpr int ROWS = PAIR ? NT / 2 : NT;			// token rows a CTA holds, at most
	static constexpr int GROUP = TC_SPB * 2 * ROWS * TC_BK * 2;	// 16 .. 64 KB
	static constexpr int GROUPS = TC_B_BYTES / GROUP;
	static_assert(GROUPS <= TC_BG_MAX && GROUPS <= TC_DONE && (GROUPS & (GROUPS - 1)) == 0, "token ring");
};
// packed super-block of 128 rows: the 144-byte Q4_K blocks resp. the 208-byte Q6_K records
// (192 bytes of quants + 16 bytes of scales) of the rows back to back, one TMA box.  Row strides
// of 9 and 13 x 16 bytes: 16-byte reads by 32 consecutive rows are bank-conflict free.
constexpr int TC_Q6_ROW = Q6K_RECORD;
constexpr int TC_NWB_MAX = 4, TC_NWF_MAX = 6;
template <WKind KIND, bool GU, bool PAIR, int NT>
struct TcSmem {
	static constexpr bool Q4 = KIND == W_Q4K;
	static constexpr int NWB = Q4 && PAIR ? 4 : 3;	// packed super-blocks in flight
	// A barrier's phase parity tells neighbouring phases apart, no more: a role may not skip uses of one.  The
	// producer groups take every other super-block, so an odd number of buffers gets two barriers each.
	static constexpr int NWF = NWB % 2 ? 2 * NWB : NWB;
	static constexpr int WBUF = TC_BM * (Q4 ? Q4K_BYTES : TC_Q6_ROW);
	static constexpr int XQ = Q4 ? 2 * TcRing<PAIR, NT>::ROWS * 128 : 0;  // sub-block sums of a work item (Q4_K): two 64-wide tiles
	static constexpr int OFF_W = TC_B_BYTES;
	static constexpr int OFF_XQ = OFF_W + NWB * WBUF;
	static constexpr int OFF_DS = OFF_XQ + 2 * XQ;	// block factors (Q4_K)
	static constexpr int OFF_PSUM = OFF_DS + (Q4 ? TC_NDS * TC_BM * 4 : 0);	 // gate and up: sums handed from drain warp to drain warp
	static constexpr int OFF_BAR = OFF_PSUM + (GU ? 8 * 32 * 4 : 0);
	static constexpr int SMEM = OFF_BAR + 512 + 1024 /* alignment slack */;
	static_assert(WBUF % 1024 == 0 && NWB <= TC_NWB_MAX, "packed super-block buffers");
	static_assert(SMEM <= 226 * 1024, "shared memory budget");  // (1 KB is left to the static variables)
};

struct TcShared {
	uint64_t full[2];		// both units of a super-block written by their producer groups
	uint64_t bfull[TC_BG_MAX];	// token tiles of a super-block (and a segment of sums) landed (TMA transaction bytes)
	uint64_t done[TC_DONE];		// MMAs of a super-block retired: weight units, token tiles and sums are free, its accumulator is complete
	uint64_t wfull[TC_NWF_MAX];	// packed super-block landed
	uint64_t wempty[TC_NWB_MAX];	// ... and expanded
	uint64_t pfull[2][TC_NBUF_MAX];	// accumulator complete, per set of drain warps (where there are two)
	uint64_t pempty[TC_NBUF_MAX];	// accumulator read out by the drain warps
	uint64_t mempty[2];		// min sums of a work item read out by the drain warps
	uint64_t sfull[8], sempty[8];	// gate and up: half a sub-block's sums handed to the warp of the other half, and taken
	uint64_t fin;			// every commit has landed
	uint32_t tmem_base;
	uint32_t abort;
};
static_assert(sizeof(TcShared) <= 512, "barrier block");

// Bounded wait: false (and the abort flag raised) when the barrier does not flip in time or
// another role / CTA has already reported a timeout.  After a first miss the thread lets the
// hardware suspend it between polls, so that waiting roles do not take issue slots from the
// producers.
// BACKOFF_NS > 0: roles that can afford a few hundred cycles of extra latency also sleep between polls.
template <int BACKOFF_NS = 0>
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, volatile uint32_t *abort_flag, unsigned *status)
{
	if (ptx::mbar_try_wait(bar, parity))
		return true;
	const long long t0 = clock64();
	uint32_t spins = 0;
	while (!ptx::mbar_try_wait_suspend(bar, parity, 20000u)) {
		if (BACKOFF_NS > 0)
			__nanosleep(BACKOFF_NS);
		if (*abort_flag)
			return false;
		if (clock64() - t0 > TC_WAIT_CYCLES || ((++spins & 255u) == 0 && (*(volatile unsigned *)status & ST_WAIT_TIMEOUT))) {
			atomicOr(status, ST_WAIT_TIMEOUT);
			*abort_flag = 1;
			return false;
		}
	}
	return true;
}

// A whole warp waits: every lane tests the barrier (no divergence around the wait — a single
// polling lane with a broadcast was measured 5 % slower over the whole kernel) and the warp votes.
template <int BACKOFF_NS = 0>
__device__ __forceinline__ bool tc_wait_warp(uint32_t bar, uint32_t parity, volatile uint32_t *abort_flag, unsigned *status, int lane)
{
	(void)lane;
	return __all_sync(0xffffffffu, tc_wait<BACKOFF_NS>(bar, parity, abort_flag, status));
}

// A work item: a token tile (expert le, sorted rows [row0, row0 + n_valid)) x a 128-row tile (GU: 64 rows of either matrix).
struct TcItem {
	int le, row0, n_valid, n_mma;  // n_mma: n_valid rounded up to 16, the N of the MMAs
	int box;	  // 0, 1, 2: the tile's token boxes hold 16, 32 or 64 rows (half of that per CTA of a pair)
	int m0;	      // first row of the matrix
	int part;     // SPLIT: which part of the rows' super-blocks (else 0)
};

// The first TC_ITEMS work items of a CTA are decoded into shared memory when the kernel starts, all at
// once: every role needs every item, and the two integer divisions of a decode in front of each item
// cost each role about a thousand cycles per item (measured: gate/up at 512 tokens 90 -> 88 us).
constexpr int TC_ITEMS = 128;
// m_items: work items per token tile (128-row tiles, or pairs of them); a CTA of a pair takes the
// tile 2 * item + its rank.  tile_rows: rows of the matrix a tile takes.  Packed: expert, first row, rows, first weight row.
// SPLIT (dense only): n_parts neighbouring items are the parts of one tile; the part stands in place of the expert.
template <bool PAIR, int NT, bool SPLIT>
__device__ __forceinline__ int4 tc_decode(int t, int m_items, const int4 *__restrict__ tile_info, int n_rows, int tile_rows, uint32_t rank,
					  int n_parts)
{
	int part = 0;
	if (SPLIT) {
		part = t % n_parts;
		t /= n_parts;
	}
	const int slot = t / m_items, mi = t - slot * m_items;
	const int4 ti = tile_info ? __ldg(tile_info + slot) : make_int4(0, slot * NT, min(NT, n_rows - slot * NT), 0);
	return make_int4(SPLIT ? part : ti.x, ti.y, ti.z, (PAIR ? 2 * mi + (int)rank : mi) * tile_rows);
}
template <bool PAIR, int NT, bool SPLIT>
__device__ __forceinline__ TcItem tc_item(int t, int tl, const int4 *s_items, int m_items, const int4 *__restrict__ tile_info,
					  int n_rows, int tile_rows, uint32_t rank, int n_parts)
{
	const int4 ti = tl < TC_ITEMS ? s_items[tl] : tc_decode<PAIR, NT, SPLIT>(t, m_items, tile_info, n_rows, tile_rows, rank, n_parts);
	TcItem it;
	it.le = SPLIT ? 0 : ti.x;
	it.part = SPLIT ? ti.x : 0;
	it.row0 = ti.y;
	it.n_valid = ti.z;
	it.n_mma = (ti.z + 15) & ~15;
	it.box = ti.z <= 16 ? 0 : (ti.z <= 32 ? 1 : 2);
	it.m0 = ti.w;
	return it;
}

__device__ __forceinline__ uint4 lds128(uint32_t addr)
{
	uint4 v;
	asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
	return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr)
{
	uint2 v;
	asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
	return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr)
{
	uint32_t v;
	asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
	return v;
}

// half2 (1024 + b_i, 1024 + b_j) from two bytes of a word: each byte becomes the low mantissa
// bits of 0x6400 | byte.  selector 0x7i5j picks bytes j (low half) and i (high half).
__device__ __forceinline__ __half2 byte_pair_1024(uint32_t w, uint32_t selector)
{
	return bits_h2(__byte_perm(w, 0x64006400u, selector));
}

// Expansion of half a packed super-block (already in shared memory) by the producer thread of a row:
// prepare() once, then four pieces of 32 weights.  Q4_K: piece(2q + i) makes columns 8i .. 8i+7 and 16 + 8i .. of the
// half's stage q.  (Pieces of 16 registers: a whole stage at a time spills at the 72 registers 27 warps leave each thread.)
template <WKind KIND>
struct Expander;

template <>
struct Expander<W_Q4K> {
	uint32_t qaddr;	 // the half's quants: 64 bytes
	uint4 hdr;	 // the block's first 16 bytes: d | dmin, packed 6-bit scales and mins
	uint32_t sc8;	 // the half's four scales as bytes (get_scale_min_k4, math_scalar.c:91-100)
	__device__ __forceinline__ void prepare(uint32_t wbuf, int row, int half)
	{
		const uint32_t blk = wbuf + (uint32_t)row * Q4K_BYTES;
		qaddr = blk + 16u + 64u * half;
		hdr = lds128(blk);
		sc8 = half ? and_or(hdr.y >> 2, 0x30303030u, hdr.w & 0x0F0F0F0Fu) : hdr.y & 0x3F3F3F3Fu;
	}
	__device__ __forceinline__ float d() const { return half_bits_to_float(hdr.x & 0xffffu); }
	__device__ __forceinline__ void piece(int i, uint32_t a[8], uint32_t b[8]) const
	{
		const __half2 k1024 = __float2half2_rn(1024.0f);
		const __half2 s_lo = __hsub2(byte_pair_1024(sc8, (i & 2) ? 0x7252u : 0x7050u), k1024);
		const __half2 s_hi = __hsub2(byte_pair_1024(sc8, (i & 2) ? 0x7353u : 0x7151u), k1024);
		Q4kConsts c;
		c.sl = s_lo;
		c.cl = __hmul2(s_lo, __float2half2_rn(-1024.0f));
		c.sh = __hmul2(s_hi, __float2half2_rn(0.0625f));
		c.ch = __hmul2(s_hi, __float2half2_rn(-64.0f));
		const uint4 q = lds128(qaddr + 16u * i);
		const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
		for (int k = 0; k < 4; k++)  // k = 16 i + 4k .. (low nibbles), 32 + 16 i + 4k .. (high nibbles) of the stage
			q4k_int_word(w[k], c, a + 2 * k, b + 2 * k);
	}
	// The products dmin * m of the block's 8 sub-blocks, split into fp16 hi + lo: four columns of the hi part
	// (lo_part false) or of the lo part.  The half products round once (hi) and the fused remainder is
	// exact before its rounding (lo): 17 bits of an 11 x 6 bit product.
	__device__ __forceinline__ void min_columns(bool lo_part, uint32_t v[4]) const
	{
		const __half2 k1024 = __float2half2_rn(1024.0f);
		const __half2 dmin = bits_h2(__byte_perm(hdr.x, 0u, 0x3232u));
		const uint32_t mn[2] = {hdr.z & 0x3F3F3F3Fu, and_or(hdr.z >> 2, 0x30303030u, (hdr.w >> 4) & 0x0F0F0F0Fu)};
#pragma unroll
		for (int j = 0; j < 4; j++) {
			const __half2 m = __hsub2(byte_pair_1024(mn[j >> 1], (j & 1) ? 0x7372u : 0x7170u), k1024);
			const __half2 h = __hmul2(dmin, m);
			v[j] = h2_bits(lo_part ? __hfma2(dmin, m, __hneg2(h)) : h);
		}
	}
};

template <>
struct Expander<W_Q6K_R8> {
	uint32_t qaddr, saddr;	// the half's 2 x 48 bytes of quants, its 8 scale bytes
	__device__ __forceinline__ void prepare(uint32_t wbuf, int row, int half)
	{
		const uint32_t rec = wbuf + (uint32_t)row * TC_Q6_ROW;
		qaddr = rec + 96u * half;
		saddr = rec + 192u + 8u * half;
	}
	// sixteen weights of each stage: v[stage][0 .. 3] columns 8 hs + 4 k .. (k = i & 1), v[stage][4 .. 7] the same + 16.
	// Low nibbles: 1056 is subtracted in front of the product.  sc * 1056 behind it is no half, nor a sixteenth of it for odd
	// scales from 63 up, whose weights were off by up to half a step.  High nibbles: 96 * sc has 9 bits.
	__device__ __forceinline__ void piece(int i, uint32_t v[2][8]) const
	{
		const int hs = i >> 1, k = i & 1;
		const __half2 k1152 = __float2half2_rn(1152.0f), k1056 = __float2half2_rn(1056.0f);
		const uint32_t chunk = qaddr + 48u * hs + 8u * k;
		const uint2 w[2] = {lds64(chunk), lds64(chunk + 16u)}, h = lds64(chunk + 32u);
		const uint32_t scx = lds32(saddr + 4u * hs) ^ 0x80808080u;  // int8 -> half as 1024 + (s ^ 0x80) - 1152
#pragma unroll
		for (int ab = 0; ab < 2; ab++) {
			const __half2 s0 = __hsub2(byte_pair_1024(scx, ab ? 0x7151u : 0x7050u), k1152), s1 = __hsub2(byte_pair_1024(scx, ab ? 0x7353u : 0x7252u), k1152);
			const __half2 f1 = __hmul2(s1, __float2half2_rn(0.0625f)), c1 = __hmul2(s1, __float2half2_rn(-96.0f));
			const uint32_t a2[2] = {w[ab].x, w[ab].y}, h2[2] = {h.x, h.y};
#pragma unroll
			for (int j = 0; j < 2; j++) {
				uint32_t lo[2], hi[2];
				if (ab)
					q6k_word<2>(a2[j], h2[j], lo, hi);
				else
					q6k_word<4>(a2[j], h2[j], lo, hi);
#pragma unroll
				for (int e = 0; e < 2; e++) {
					v[0][4 * ab + 2 * j + e] = h2_bits(__hmul2(__hsub2(bits_h2(lo[e]), k1056), s0));
					v[1][4 * ab + 2 * j + e] = h2_bits(__hfma2(bits_h2(hi[e]), f1, c1));
				}
			}
		}
	}
};

// GU (gate and up): a tile is 64 rows of w0 and the same of w1, sixteen of each in the tensor-memory lanes of a
// warp, so that the SwiGLU of a row is one shuffle away in the drain: h * out_scale, split into fp16 hi + lo, goes to the down
// product's operand (and its sub-block sums, where that is Q4_K).  The products themselves stay on the chip: as
// fp32 rows for a pass of its own they were 2 x 200 MB at 4096 tokens.  (Products and pass -> product with SwiGLU: 64 tokens
// 69 + 10 -> 70 us, 512 86 + 13 -> 90, 4096 368 + 57 -> 387.)  The table is read through the 28 KB of L1 that shared memory
// leaves; its middle 20 KB in shared memory took a weight buffer's place, 64 tokens 70 -> 76 us.
// Otherwise (down, dense) products times out_scale (a power of two) are stored in sorted order, or, with perm, in
// the order of the rows y[perm[row0 + n]].
// tm0/1/2: maps of the split token operand ([hi | lo][rows][k], box 64 k x 16/32/64 rows x 2; half
// of the rows for a CTA of a pair); tq0/1/2: the same of its sub-block sums; tw0 / tw1: byte maps of
// the two weight tensors, box = packed super-block x 128 rows.
//
// Every role walks the same sequence of super-blocks, numbered through the work items of the CTA: n % 2
// selects the accumulator buffer and the pair of ring slots.
//
// The sub-block sums (Q4_K) come in segments of 8 super-blocks: the expert products have one per work item, a
// dense tensor with more than 2048 inputs several.  tile_info null (dense tensors): no tables, the
// token tiles are n_local rows cut in order.
//
// PEER (expert parallelism over peer memory, down product only): sorted row p belongs to row
// dst.row[p] & 0xFFFFFF of rank dst.row[p] >> 24 and is stored there, into that rank's memory
// (dst.y[rank], plain stores over NVLink, 128 contiguous bytes per warp and row).
struct GuOut {
	__half *hi = nullptr;	 // [rows][rows of the matrix], the k order of the operand tiles
	size_t lo = 0;		 // the lo halves lie so many values behind
	__half *sums = nullptr;	 // [rows][sum_cols] or null
	int sum_cols = 0;
	const float *silu = nullptr;
};
// SPLIT: a dense product whose tiles leave most of the device idle (2048 -> 512 of 37 tokens: 8 tiles) divides the super-blocks of a
// row among the n_parts CTAs of a cluster, one work item each.  They leave their sums in shared memory, and each adds up its
// share of the tile's tokens from all of them, in the order of the parts.  (Through global memory, the last to come adding
// up, 37 tokens took 27 us instead of 15.)
template <WKind KIND, bool GU, bool PEER = false, bool PAIR = false, int NT = TC_TOKEN_TILE, bool SPLIT = false>
__global__ void __launch_bounds__(TC_THREADS, 1)
grouped_gemm_sb(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1,
		const __grid_constant__ CUtensorMap tm2, const __grid_constant__ CUtensorMap tq0,
		const __grid_constant__ CUtensorMap tq1, const __grid_constant__ CUtensorMap tq2,
		const __grid_constant__ CUtensorMap tw0, const __grid_constant__ CUtensorMap tw1, const uint8_t *__restrict__ w0,
		const uint8_t *__restrict__ w1, size_t expert_stride, int k_dim, const int4 *__restrict__ tile_info,
		const int *__restrict__ tile_start, int n_local, int m_tiles, float *__restrict__ y, const int *__restrict__ perm,
		int out_stride, float out_scale, unsigned *__restrict__ status, int rows_per_matrix, const EpDst dst,
		const int xq_depth, const GuOut gu, const int n_parts)
{
	static_assert(!SPLIT || (!GU && !PEER && !PAIR && NT == 32), "parts of plain products in narrow tiles only");
	static_assert(!(GU && PEER), "peer destinations exist for the down product only");
	using Sm = TcSmem<KIND, GU, PAIR, NT>;
	constexpr int TILE_ROWS = GU ? TC_BM / 2 : TC_BM;  // of a matrix
	using Ring = TcRing<PAIR, NT>;
	using Cols = TcCols<KIND, NT>;
	constexpr int NBUF = Cols::NBUF;
	using Roles = TcRoles<GU, NT>;
	constexpr int PARTS = Roles::PARTS;
	constexpr int FOLDERS = Roles::SET;  // drain warps that read an accumulator
	constexpr bool Q4 = KIND == W_Q4K;
	constexpr uint32_t UNIT = Cols::UNIT;
	extern __shared__ uint8_t smem_raw[];
	__shared__ int s_total;
	__shared__ int4 s_items[TC_ITEMS];
	// a pair walks the work items together: its index among the pairs, and this CTA's rank in it
	const uint32_t rank = PAIR ? ptx::cluster_ctarank() : 0u;
	const int walker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
	const int stride_t = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
	const int m_items = PAIR ? m_tiles / 2 : m_tiles;
	const int nb = k_dim / QK_K, nbl = SPLIT ? nb / n_parts : nb;  // super-blocks of a row, and of a work item

	const uint32_t raw = ptx::smem_u32(smem_raw);
	const uint32_t tiles = (raw + 1023u) & ~1023u;
	uint8_t *smem = smem_raw + (tiles - raw);
	TcShared *sh = reinterpret_cast<TcShared *>(smem + Sm::OFF_BAR);
	float *ds = reinterpret_cast<float *>(smem + Sm::OFF_DS);  // [TC_NDS][128] d of the rows (Q4_K)
	float *psum = reinterpret_cast<float *>(smem + Sm::OFF_PSUM);
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

	// token tiles of a super-block: four stages of the CTA's hi rows followed by its lo rows
	auto b_group = [&](uint32_t q) -> uint32_t { return tiles + q * Ring::GROUP; };
	auto xq_buf = [&](uint32_t i) -> uint32_t { return tiles + Sm::OFF_XQ + i * Sm::XQ; };
	auto w_buf = [&](int wb) -> uint32_t { return tiles + Sm::OFF_W + wb * Sm::WBUF; };

	if (threadIdx.x == 0) {
		for (int s = 0; s < 2; s++)
			ptx::mbar_init(ptx::smem_u32(&sh->full[s]), (PAIR ? 2 : 1) * 8);
		for (int s = 0; s < TC_BG_MAX; s++)
			ptx::mbar_init(ptx::smem_u32(&sh->bfull[s]), 1);
		for (int s = 0; s < TC_DONE; s++)
			ptx::mbar_init(ptx::smem_u32(&sh->done[s]), 1);
		for (int s = 0; s < Sm::NWF; s++)
			ptx::mbar_init(ptx::smem_u32(&sh->wfull[s]), 1);
		for (int s = 0; s < Sm::NWB; s++)
			ptx::mbar_init(ptx::smem_u32(&sh->wempty[s]), 8);
		for (int s = 0; s < NBUF; s++) {
			ptx::mbar_init(ptx::smem_u32(&sh->pfull[0][s]), 1);
			ptx::mbar_init(ptx::smem_u32(&sh->pfull[1][s]), 1);
			ptx::mbar_init(ptx::smem_u32(&sh->pempty[s]), (PAIR ? 2 : 1) * FOLDERS);
		}
		for (int s = 0; s < 2; s++)
			ptx::mbar_init(ptx::smem_u32(&sh->mempty[s]), (PAIR ? 2 : 1) * FOLDERS);
		for (int s = 0; s < 8; s++) {
			ptx::mbar_init(ptx::smem_u32(&sh->sfull[s]), 1);
			ptx::mbar_init(ptx::smem_u32(&sh->sempty[s]), 1);
		}
		ptx::mbar_init(ptx::smem_u32(&sh->fin), 1);
		sh->abort = 0;
		ptx::fence_barrier_init();
		ptx::fence_proxy_async_smem();
	}
	constexpr int W_MMA = Roles::PWARPS + Roles::DWARPS, W_TOK = W_MMA + 1, W_WGT = W_TOK + 1;
	if (warp == W_MMA) {  // the MMA warp owns the tensor-memory allocation (pairs: one warp of each CTA, together)
		if (PAIR) {
			ptx::tmem_alloc_pair(ptx::smem_u32(&sh->tmem_base), TC_TMEM_COLS);
			ptx::tmem_relinquish_pair();
		} else {
			ptx::tmem_alloc(ptx::smem_u32(&sh->tmem_base), TC_TMEM_COLS);
			ptx::tmem_relinquish();
		}
	}
	if (warp == W_TOK && lane == 0) {
		ptx::prefetch_tmap(&tm0);
		ptx::prefetch_tmap(&tm1);
		ptx::prefetch_tmap(&tm2);
		if (Q4) {
			ptx::prefetch_tmap(&tq0);
			ptx::prefetch_tmap(&tq1);
			ptx::prefetch_tmap(&tq2);
		}
	}
	if (warp == W_WGT && lane == 0) {
		ptx::prefetch_tmap(&tw0);
		if (GU)
			ptx::prefetch_tmap(&tw1);
	}
	if (GU)
		pdl_trigger();	// (the down product sets itself up as the SMs fall idle)
	pdl_wait();  // what the kernels before this one wrote is visible from here on
	if (threadIdx.x == 0)
		s_total = (*(volatile unsigned *)status & ST_WAIT_TIMEOUT) ? 0 : (tile_info ? tile_start[n_local] : (n_local + NT - 1) / NT) * m_items * (SPLIT ? n_parts : 1);
	ptx::tc_fence_before();
	__syncthreads();
	const int total = s_total;  // (a CTA without work items goes through the motions: it holds tensor memory, its peer waits for it)
	if (threadIdx.x < TC_ITEMS) {
		const int t = walker + threadIdx.x * stride_t;
		if (t < total)
			s_items[threadIdx.x] = tc_decode<PAIR, NT, SPLIT>(t, m_items, tile_info, n_local, TILE_ROWS, rank, n_parts);
	}
	__syncthreads();
	if (PAIR)
		ptx::cluster_sync_all();  // both CTAs' barriers are initialised before either signals the other's
	ptx::tc_fence_after();
	const uint32_t tmem = sh->tmem_base;
	volatile uint32_t *abort_flag = &sh->abort;
	// arrival on a barrier that the MMA issuer (in the leader CTA of a pair) waits on
	auto arrive_issuer = [&](uint64_t *bar) {
		if (PAIR)
			ptx::mbar_arrive_leader(ptx::smem_u32(bar));
		else
			ptx::mbar_arrive(ptx::smem_u32(bar));
	};

	if (warp < Roles::PWARPS) {
		// ================= producers: packed blocks (shared memory) -> integer A tiles (tensor memory) =================
		// Groups of four warps (one warp per 32-row quadrant of tensor memory).  A unit is half a
		// super-block: two 64-k stages and, for Q4_K, the hi (first half) or lo columns of its dmin * m
		// products.  Group j makes half j & 1 of every super-block (four groups: of every other); a
		// first piece is expanded in registers BEFORE the slot is waited for.
		ptx::setmaxnreg_dec<Roles::PREGS>();
		constexpr uint32_t STEP = Roles::PGROUPS / 2;
		const int row = threadIdx.x & 127, grp = threadIdx.x >> 7, half = grp & 1;
		// (GU: lanes 0 - 15 of a warp take rows of the gate box, 16 - 31 the same rows of the up box behind it)
		const int wrow = GU ? ((row & 16) << 2) + ((row >> 5) << 4) + (row & 15) : row;
		const uint32_t slot0 = tmem + ((uint32_t)((warp & 3) * 32) << 16) + Cols::A + UNIT * (STEP == 2 ? grp : half);
		const uint32_t n_sb = walker < total ? (uint32_t)((total - 1 - walker) / stride_t + 1) * (uint32_t)nbl : 0u;
		bool alive = true;
		for (uint32_t n = STEP == 2 ? grp >> 1 : 0; n < n_sb; n += STEP) {
			const uint32_t wb = n % Sm::NWB, slot = slot0 + (STEP == 1 ? 2 * UNIT * (n & 1u) : 0u);
			if (!tc_wait_warp(ptx::smem_u32(&sh->wfull[n % Sm::NWF]), (n / Sm::NWF) & 1u, abort_flag, status, lane))
				break;
			Expander<KIND> ex;
			ex.prepare(w_buf(wb), wrow, half);
			if constexpr (Q4) {
				if (half == 0)
					ds[(n & (TC_NDS - 1)) * TC_BM + row] = ex.d();
			}
#pragma unroll
			for (int i = 0; i < 4; i++) {
				uint32_t v[2][8];
				if constexpr (Q4)
					ex.piece(i, v[0], v[1]);
				else
					ex.piece(i, v);
				if (i == 0) {
					const uint32_t m = n - 2u;  // the slot's last user
					if (n >= 2 && !tc_wait_warp(ptx::smem_u32(&sh->done[m % TC_DONE]), (m / TC_DONE) & 1u, abort_flag, status, lane)) {
						alive = false;
						break;
					}
					ptx::tc_fence_after();
				}
				if constexpr (Q4) {
					ptx::tmem_st8(slot + 32u * (i >> 1) + 8u * (i & 1), v[0]);
					ptx::tmem_st8(slot + 32u * (i >> 1) + 8u * (i & 1) + 16u, v[1]);
				} else {
#pragma unroll
					for (int c = 0; c < 4; c++)
						ptx::tmem_st4(slot + 32u * (c >> 1) + 8u * (i >> 1) + 4u * (i & 1) + 16u * (c & 1), v[c >> 1] + 4 * (c & 1));
				}
			}
			if (!alive)
				break;
			if constexpr (Q4) {
				uint32_t v[4];
				ex.min_columns(half != 0, v);
				ptx::tmem_st4(slot + 64u, v);  // (twice: once for the hi, once for the lo sums of the tokens)
				ptx::tmem_st4(slot + 68u, v);
			}
			ptx::tmem_st_wait();
			ptx::tc_fence_before();
			__syncwarp();
			if (lane == 0) {
				arrive_issuer(&sh->full[STEP == 2 ? grp >> 1 : n & 1u]);
				// this warp's half of the packed super-block is expanded: the buffer goes back to the weight loader
				ptx::mbar_arrive(ptx::smem_u32(&sh->wempty[wb]));
			}
		}
	} else if (warp < W_MMA) {
		// ================= drain warps: partial sums of a super-block -> fp32 rows =================
		ptx::setmaxnreg_inc<Roles::DREGS>();
		const int dw = warp - Roles::PWARPS, quad = warp & 3, part = (dw >> 2) % PARTS, set = Roles::NSETS == 2 ? dw / Roles::SET : 0;
		const int lrow = quad * 32 + lane;
		const uint32_t tlane = tmem + ((uint32_t)(quad * 32) << 16);
		const bool upper = GU && (lane & 16);  // a lane of up rows
		uint32_t handed = 0;		       // GU: sums handed over (or taken) so far
		uint32_t n = 0;	   // super-blocks so far
		uint32_t pph = 0;  // per accumulator: parity of this set's next wait (it takes only its items' uses)
		bool alive = true;
		int dtl = 0;
		for (int t = walker; t < total && alive; t += stride_t, dtl++) {
			if (Roles::NSETS == 2 && (dtl & 1) != set) {  // the other set's item
				n += nbl;
				continue;
			}
			const TcItem item = tc_item<PAIR, NT, SPLIT>(t, dtl, s_items, m_items, tile_info, n_local, TILE_ROWS, rank, n_parts);
			const int mrow = item.m0 + (GU ? quad * 16 + (lane & 15) : lrow);
			// tokens of this warp: the whole tile, or half of it (the first or the second by part).
			// Where twice the columns fit an accumulator, the hi and lo products have columns of their own (one MMA
			// for both), which for a pair lie [hi lo] per CTA's half of the tokens.
			const bool stacked = 2 * item.n_mma <= NT;
			const int ntok = PARTS == 1 ? item.n_mma : (item.n_mma > 32 ? 32 : item.n_mma >> 1);
			const int tok0 = part * ntok;
			const bool two = ntok == 32;
			const uint32_t c_hi = PAIR ? part * item.n_mma : tok0, c_lo = PAIR ? c_hi + ntok : item.n_mma + tok0;  // (two parts)
			float acc[32];
#pragma unroll
			for (int j = 0; j < 32; j++)
				acc[j] = 0.0f;
			// acc += scale * the warp's columns of an accumulator; the buffer is handed back once they are in registers
			// (columns past the warp's tokens are read along and dropped)
			auto fold = [&](uint32_t col, bool both, float scale, uint64_t *bar) {
				uint32_t v[16];
				if (two) {
					ptx::tmem_ld16(tlane + col + tok0, v);
					ptx::tmem_ld_wait();
#pragma unroll
					for (int j = 0; j < 16; j++)
						acc[j] = __fmaf_rn(scale, __uint_as_float(v[j]), acc[j]);
					ptx::tmem_ld16(tlane + col + tok0 + 16, v);
					ptx::tmem_ld_wait();
				} else if (both) {
					uint32_t u[16];
					ptx::tmem_ld16(tlane + col + (PARTS == 1 ? 0u : c_hi), v);
					ptx::tmem_ld16(tlane + col + (PARTS == 1 ? 16u : c_lo), u);
					ptx::tmem_ld_wait();
					if (PARTS == 1 && PAIR) {  // [hi lo] of tokens 0 .. 7, then of 8 .. 15
#pragma unroll
						for (int j = 0; j < 8; j++) {
							v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(v[8 + j]));
							v[8 + j] = __float_as_uint(__uint_as_float(u[j]) + __uint_as_float(u[8 + j]));
						}
					} else {
#pragma unroll
						for (int j = 0; j < 16; j++)
							v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(u[j]));
					}
				} else {
					ptx::tmem_ld16(tlane + col + tok0, v);
					ptx::tmem_ld_wait();
				}
				ptx::tc_fence_before();
				__syncwarp();
				if (lane == 0)
					arrive_issuer(bar);
				if (two) {
#pragma unroll
					for (int j = 0; j < 16; j++)
						acc[16 + j] = __fmaf_rn(scale, __uint_as_float(v[j]), acc[16 + j]);
				} else {
#pragma unroll
					for (int j = 0; j < 16; j++)
						acc[j] = __fmaf_rn(scale, __uint_as_float(v[j]), acc[j]);
				}
			};
			// Q6_K: d of (row, super-block) straight from global memory, one super-block ahead
			const int sb0 = item.part * nbl;
			const uint8_t *grp = nullptr;
			float dnext = 0.0f;
			if (!Q4) {
				grp = (upper ? w1 : w0) + (size_t)item.le * expert_stride + (size_t)(mrow >> 3) * q6k_r8_group_bytes(nb);
				dnext = half_bits_to_float(__ldg(reinterpret_cast<const unsigned short *>(grp + q6k_r8_d_off(nb, mrow & 7, sb0))));
			}
			for (int sbi = 0; sbi < nbl; sbi++, n++) {
				float scale = (GU ? 1.0f : out_scale) * dnext;
				if (!Q4 && sbi + 1 < nbl)
					dnext = half_bits_to_float(
						__ldg(reinterpret_cast<const unsigned short *>(grp + q6k_r8_d_off(nb, mrow & 7, sb0 + sbi + 1))));
				const uint32_t buf = n % NBUF;
				if (!tc_wait_warp(ptx::smem_u32(Roles::NSETS == 2 ? &sh->pfull[set][buf] : &sh->done[n % TC_DONE]),
						  Roles::NSETS == 2 ? (pph >> buf) & 1u : (n / TC_DONE) & 1u, abort_flag, status, lane)) {
					alive = false;
					break;
				}
				if (Roles::NSETS == 2)
					pph ^= 1u << buf;
				ptx::tc_fence_after();
				if (Q4)
					scale = (GU ? 1.0f : out_scale) * ds[(n & (TC_NDS - 1)) * TC_BM + lrow];
				fold(NT * buf, stacked, scale, &sh->pempty[buf]);
			}
			if (!alive)
				break;
			// the min sums (Q4_K) were complete with the last super-block
			if (Q4)
				fold(Cols::M + NT * (set % Cols::NM), false, GU ? -1.0f : -out_scale, &sh->mempty[set % Cols::NM]);
			const int n_rows = min(ntok, item.n_valid - tok0);
			const int p0 = item.row0 + tok0;  // sorted position of the first row
			if constexpr (GU) {
				// Lane l holds gate (l < 16) or up rows of all the warp's tokens and makes h of row l & 15 for half of them.
				auto finish = [&](auto half_tokens) {
					constexpr int H = half_tokens.value;
					const int j0 = upper ? H : 0;
					// (the order [k0, k2, k1, k3] of every group of 4)
					const int k = (mrow & ~3) | (mrow & 1) << 1 | (mrow >> 1 & 1);
					__half *hp = gu.hi + (size_t)(p0 + j0) * rows_per_matrix + k;
					float h[H];
#pragma unroll
					for (int j = 0; j < H; j++) {
						const float other = __shfl_xor_sync(0xffffffffu, upper ? acc[j] : acc[H + j], 16);
						const float mine = upper ? acc[H + j] : acc[j];
						h[j] = swiglu_lut(gu.silu, upper ? other : mine, upper ? mine : other) * out_scale;
					}
#pragma unroll
					for (int j = 0; j < H; j++) {
						if (j0 + j < n_rows) {
							const __half hi = __float2half_rn(h[j]);
							hp[0] = hi;
							hp[gu.lo] = __float2half_rn(h[j] - __half2float(hi));
						}
						hp += rows_per_matrix;
					}
					if (gu.sums) {
						// sums over the warp's 16 rows (a token each for lane & (H - 1)), added to those of the sub-block's other 16
#pragma unroll
						for (int w = 8; w >= 1; w >>= 1) {
							if (w >= H) {
#pragma unroll
								for (int j = 0; j < H; j++)
									h[j] += __shfl_xor_sync(0xffffffffu, h[j], w);
								continue;
							}
							const bool keep_hi = lane & w;
#pragma unroll
							for (int j = 0; j < w; j++) {
								const float send = keep_hi ? h[j] : h[w + j], keep = keep_hi ? h[w + j] : h[j];
								h[j] = keep + __shfl_xor_sync(0xffffffffu, send, w);
							}
						}
						const int tok = j0 + (lane & (H - 1)), pair = (dw >> 2) * 2 + (quad >> 1);
						const uint32_t sf = ptx::smem_u32(&sh->sfull[pair]), se = ptx::smem_u32(&sh->sempty[pair]);
						float *ps = psum + pair * 32 + lane;
						if (quad & 1) {
							alive = tc_wait_warp(se, (handed & 1u) ^ 1u, abort_flag, status, lane);
							*ps = h[0];
							__syncwarp();
							if (lane == 0)
								ptx::mbar_arrive(sf);
						} else {
							alive = tc_wait_warp(sf, handed & 1u, abort_flag, status, lane);
							const float sum = h[0] + *ps;
							__syncwarp();
							if (lane == 0)
								ptx::mbar_arrive(se);
							if (alive && tok < n_rows && (lane & 15) < H) {
								const __half hi = __float2half_rn(sum);
								__half *q = gu.sums + (size_t)(p0 + tok) * gu.sum_cols + xq_index(mrow >> 5);
								q[0] = hi;
								q[8] = __float2half_rn(sum - __half2float(hi));
							}
						}
						handed++;
					}
				};
				if (two)
					finish(std::integral_constant<int, 16>());
				else
					finish(std::integral_constant<int, 8>());
				continue;
			}
			// rows of this work item: lanes hold consecutive output columns (coalesced 128-byte stores)
			// (in sorted order a tile's stores go to neighbouring rows: scattered to the rows' own places, 8 KB apart in 268 MB
			// at 4096 tokens, the down product took 238 us there instead of 217, 61 instead of 55 at 512)
			if (!PEER && !perm) {
				// (SPLIT: [token][128 rows] in the token ring, which the item's MMAs are done with)
				float *yr = SPLIT ? reinterpret_cast<float *>(smem) + tok0 * TC_BM + lrow : y + (size_t)p0 * out_stride + mrow;
				const unsigned ystep = SPLIT ? TC_BM : out_stride;
#pragma unroll
				for (int j0 = 0; j0 < 32; j0 += 8) {
					if (j0 + 8 <= n_rows) {
#pragma unroll
						for (int j = 0; j < 8; j++)
							yr[(size_t)(unsigned)j * ystep] = acc[j0 + j];
					} else {
#pragma unroll
						for (int j = 0; j < 8; j++)
							if (j0 + j < n_rows)
								yr[(size_t)(unsigned)j * ystep] = acc[j0 + j];
					}
					yr += 8 * (size_t)ystep;
					asm volatile("" ::: "memory");	// (the addresses of eight rows at a time: hoisted together they spill)
				}
			} else {
				int rid = 0;
				if (lane < n_rows)
					rid = PEER ? (int)dst.row[p0 + lane] : perm[p0 + lane];
#pragma unroll
				for (int j = 0; j < 32; j++) {
					const int rj = __shfl_sync(0xffffffffu, rid, j);
					if (j < n_rows) {
						float *yr = PEER ? dst.y[(unsigned)rj >> 24] + (size_t)(rj & 0xFFFFFF) * out_stride : y + (size_t)rj * out_stride;
						yr[mrow] = acc[j];
					}
					asm volatile("" ::: "memory");	// (one row's address at a time: hoisted together they spill)
				}
			}
		}
	} else if (warp == W_MMA) {
		// ================= MMA issuer (pairs: in the leader, for both CTAs) =================
		// One thread, one super-block at a time: the barriers it needs are tested together and branched on once
		// — a wait in front of every stage cost this thread more than the stage's MMAs (8 MMAs of N = 16 take 93
		// cycles to issue, 107 with the commit, 260 behind a test-and-branch; four stages behind one, 130 each).
		// One commit tells everybody who waits for the super-block (a barrier each for the units, the token tiles and the
		// accumulator were four, and the sums' barriers two more: prompt of 512 212.2 -> 210.5 us, 4096 -> 2048 projection of
		// 512 tokens 24.4 -> 23.7).
		if (rank == 0 && ptx::elect_one()) {
			auto mma = [&](uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc) {
				if (PAIR)
					ptx::mma_f16_ts_pair(d, a, b, idesc, acc);
				else
					ptx::mma_f16_ts(d, a, b, idesc, acc);
			};
			auto commit = [&](uint64_t *bar) {
				if (PAIR)
					ptx::mma_commit_pair(ptx::smem_u32(bar));
				else
					ptx::mma_commit(ptx::smem_u32(bar));
			};
			uint32_t n = 0, tl = 0, xs_n = 0;  // super-blocks, work items, segments of sums so far
			bool alive = true;
			auto wait = [&](uint32_t bar, uint32_t parity) {
				alive = alive && tc_wait(bar, parity, abort_flag, status);
			};
			for (int t = walker; t < total && alive; t += stride_t, tl++) {
				const TcItem item = tc_item<PAIR, NT, SPLIT>(t, (int)tl, s_items, m_items, tile_info, n_local, TILE_ROWS, rank, n_parts);
				const uint32_t idesc = ptx::umma_idesc_f16(PAIR ? 2 * TC_BM : TC_BM, item.n_mma);
				const uint32_t idesc2 = ptx::umma_idesc_f16(PAIR ? 2 * TC_BM : TC_BM, 2 * item.n_mma);
				const uint32_t lo_off = (uint32_t)((PAIR ? 8 : 16) << item.box) * 128u;
				// a tile whose hi and lo products fit an accumulator side by side fills its box, so the lo rows follow the
				// hi rows and one MMA of twice the columns takes both
				const bool stacked = 2 * item.n_mma <= NT;
				const uint32_t dset = Roles::NSETS == 2 ? tl & 1u : 0u, mset = Cols::NM == 2 ? dset : 0u;  // the set of drain warps that takes the item, its min sums
				for (int sbi = 0; sbi < nbl; sbi++, n++) {
					const int g = item.part * nbl + sbi;  // of the row
					const uint32_t buf = n % NBUF, j0 = 2u * (n & 1u);
					const uint32_t q = n & (Ring::GROUPS - 1);
					const uint32_t fb = ptx::smem_u32(&sh->bfull[q]), fu = ptx::smem_u32(&sh->full[n & 1u]), pe = ptx::smem_u32(&sh->pempty[buf]);
					// (the phase before a barrier's first counts as complete: the first uses of an accumulator do not wait)
					const uint32_t fb_ph = (n / Ring::GROUPS) & 1u, fu_ph = (n >> 1) & 1u, pe_ph = ((n / NBUF) & 1u) ^ 1u;
					if (!ptx::mbar_try_wait3(fb, fb_ph, fu, fu_ph, pe, pe_ph)) {
						wait(fb, fb_ph);
						wait(pe, pe_ph);
						wait(fu, fu_ph);
						if (!alive)
							break;
					}
					ptx::tc_fence_after();
					const uint32_t dP = tmem + NT * buf, bt = b_group(q);
					const uint32_t xs = ptx::umma_desc_lo(xq_buf(xs_n & 1u) + (uint32_t)((g >> 2) & 1) * lo_off) + 2u * (g & 3);
					auto stages = [&](auto both) {
						auto a_of = [&](int q4) { return tmem + Cols::A + UNIT * (j0 + (q4 >> 1)) + 32u * (q4 & 1); };
						auto b_of = [&](int q4) { return ptx::umma_desc_lo(bt + q4 * 2u * lo_off); };
						// The lo products first: the tensor cores cut the low bits off a sum at every step, which costs next to
						// nothing while the sum is that of the lo halves (in turn with the hi products: error of a dense row of
						// 4096 inputs 2.9e-7 -> 6.0e-7).  The weights' units are held for longer: 4096 tokens 990 -> 1000 us.
						if (!both.value) {
#pragma unroll
							for (int q4 = 0; q4 < TC_SPB; q4++)
#pragma unroll
								for (int kk = 0; kk < TC_BK / 16; kk++)
									mma(dP, a_of(q4) + 8 * kk, b_of(q4) + (lo_off >> 4) + 2 * kk, idesc, (q4 > 0 || kk > 0) ? 1u : 0u);
						}
#pragma unroll
						for (int q4 = 0; q4 < TC_SPB; q4++)
#pragma unroll
							for (int kk = 0; kk < TC_BK / 16; kk++)
								mma(dP, a_of(q4) + 8 * kk, b_of(q4) + 2 * kk, both.value ? idesc2 : idesc,
								    (!both.value || q4 > 0 || kk > 0) ? 1u : 0u);
					};
					if (stacked)
						stages(std::true_type());
					else
						stages(std::false_type());
					if (Q4) {
						// (dmin m)_hi (first unit), (dmin m)_lo (second) times the block's sums, hi and lo side by side in k; an item's
						// first ones behind its first stages, so that the drain of its accumulator's last item holds those up no more
						if (sbi == 0) {
							wait(ptx::smem_u32(&sh->mempty[mset]), ((tl / Cols::NM) & 1u) ^ 1u);
							if (!alive)
								break;
							ptx::tc_fence_after();
						}
						const uint32_t dM = tmem + Cols::M + NT * mset, aM = tmem + Cols::A + UNIT * j0 + 64u;
						mma(dM, aM, xs, idesc, sbi > 0 ? 1u : 0u);
						mma(dM, aM + UNIT, xs, idesc, 1u);
						if ((g & 7) == 7 || sbi == nbl - 1)
							xs_n++;
					}
					commit(&sh->done[n % TC_DONE]);
					if (Roles::NSETS == 2)
						commit(&sh->pfull[dset][buf]);
				}
			}
			// the last commits have to land in both CTAs' barriers before either CTA may leave
			commit(&sh->fin);
		}
		__syncwarp();
		tc_wait_warp(ptx::smem_u32(&sh->fin), 0, abort_flag, status, lane);
	} else if (warp == W_TOK) {
		// ================= token loader: token operand and sub-block sums (TMA) =================
		if (ptx::elect_one()) {
			uint32_t tl = 0, n = 0, xs_n = 0, x_end = 0;  // x_end: where the segment of sums before the current one ended
			bool alive = true;
			for (int t = walker; t < total && alive; t += stride_t, tl++) {
				const TcItem item = tc_item<PAIR, NT, SPLIT>(t, (int)tl, s_items, m_items, tile_info, n_local, TILE_ROWS, rank, n_parts);
				// one box per super-block: four stages of 64 k x (hi, lo) x the CTA's token rows.  The CTAs of a pair
				// take the first and the second half of the tile's n_mma columns; all the bytes are counted on
				// the leader's barrier, whose token loader announces them.
				const uint32_t row_bytes = (uint32_t)(16 << item.box) * 128u;  // of one 64-wide column tile, both CTAs
				const int row0 = item.row0 + (PAIR ? (int)rank * (item.n_mma >> 1) : 0);
				const CUtensorMap *tmp = item.box == 0 ? &tm0 : (item.box == 1 ? &tm1 : &tm2);
				auto wait_done = [&](uint32_t m) {
					return tc_wait<100>(ptx::smem_u32(&sh->done[m % TC_DONE]), (m / TC_DONE) & 1u, abort_flag, status);
				};
				for (int sbi = 0; sbi < nbl; sbi++, n++) {
					const int g = item.part * nbl + sbi;
					const bool sums = Q4 && (sbi == 0 || (g & 7) == 0);
					const uint32_t q = n & (Ring::GROUPS - 1);
					if (n >= (uint32_t)Ring::GROUPS && !wait_done(n - Ring::GROUPS)) {
						alive = false;
						break;
					}
					const uint32_t fb = ptx::smem_u32(&sh->bfull[q]);
					uint32_t bytes = 2u * TC_SPB * row_bytes;
					if (sums) {
						// a segment of the sub-block sums comes with its first super-block (two buffers; the segment before the
						// last one is over with the super-block in front of x_end, of which the wait above may have told)
						if (xs_n >= 2u && x_end + Ring::GROUPS > n + 1u && !wait_done(x_end - 1u)) {
							alive = false;
							break;
						}
						x_end = n;
						bytes += (uint32_t)xq_depth * row_bytes;
					}
					if (rank == 0)
						ptx::mbar_arrive_expect_tx(fb, bytes);
					if (sums) {
						const uint32_t xi = xs_n & 1u;
						const CUtensorMap *tqp = item.box == 0 ? &tq0 : (item.box == 1 ? &tq1 : &tq2);
						if (PAIR)
							ptx::tma_load_3d_pair(xq_buf(xi), tqp, fb, 0, row0, (g >> 3) * 2);
						else
							ptx::tma_load_3d(xq_buf(xi), tqp, fb, 0, row0, (g >> 3) * 2);
						xs_n++;
					}
					if (PAIR)
						ptx::tma_load_4d_pair(b_group(q), tmp, fb, 0, row0, 0, g * TC_SPB);
					else
						ptx::tma_load_4d(b_group(q), tmp, fb, 0, row0, 0, g * TC_SPB);
				}
			}
		}
	} else {
		// ================= weight loader: packed super-blocks -> shared memory =================
		int wb = 0;
		uint32_t wph = 0, wc = 0;
		bool alive = true;
		int wtl = 0;
		for (int t = walker; t < total && alive; t += stride_t, wtl++) {
			const TcItem item = tc_item<PAIR, NT, SPLIT>(t, wtl, s_items, m_items, tile_info, n_local, TILE_ROWS, rank, n_parts);
			for (int sbi = 0; sbi < nbl; sbi++) {
				const int g = item.part * nbl + sbi;
				if (wc >= (uint32_t)Sm::NWB && !tc_wait_warp<100>(ptx::smem_u32(&sh->wempty[wb]), wph ^ 1u, abort_flag, status, lane)) {
					alive = false;
					break;
				}
				const uint32_t bar = ptx::smem_u32(&sh->wfull[wc % Sm::NWF]);
				if (ptx::elect_one()) {
					ptx::mbar_arrive_expect_tx(bar, Sm::WBUF);
					const int row = item.le * rows_per_matrix + item.m0;
#pragma unroll
					for (int m = 0; m < (GU ? 2 : 1); m++) {
						const CUtensorMap *tw = m ? &tw1 : &tw0;
						const uint32_t at = w_buf(wb) + m * (Sm::WBUF / 2);
						if (Q4)	 // box = (one block, 128 or 64 rows)
							ptx::tma_load_2d(at, tw, bar, g * Q4K_BYTES, row);
						else  // box = (one record, 8 rows of a group, 16 or 8 groups)
							ptx::tma_load_3d(at, tw, bar, g * TC_Q6_ROW, 0, row >> 3);
					}
				}
				wc++;
				if (++wb == Sm::NWB) {
					wb = 0;
					wph ^= 1u;
				}
			}
		}
	}

	if (*abort_flag) {
		// give copies that may still be in flight time to land before the CTA's memory is released
		for (int i = 0; i < 200; i++)
			__nanosleep(1000);
	}
	ptx::tc_fence_before();
	__syncthreads();
	if constexpr (SPLIT) {
		ptx::cluster_sync_all();
		const int4 it = s_items[0];  // (one item a CTA; the parts of a tile differ in the part only)
		const uint32_t me = ptx::cluster_ctarank();
		for (int i = threadIdx.x; total > 0 && i < (it.z - (int)me + n_parts - 1) / n_parts * (TC_BM / 4); i += TC_THREADS) {
			const int tok = (int)me + i / (TC_BM / 4) * n_parts, col = i % (TC_BM / 4) * 4;
			float4 v[TC_MAX_PARTS];
#pragma unroll
			for (int k = 0; k < TC_MAX_PARTS; k++)
				if (k < n_parts)
					v[k] = ptx::ld_cluster(ptx::cluster_addr(tiles + (uint32_t)(tok * TC_BM + col) * 4u, k));
#pragma unroll
			for (int k = 1; k < TC_MAX_PARTS; k++)
				if (k < n_parts)
					v[0] = make_float4(__fadd_rn(v[0].x, v[k].x), __fadd_rn(v[0].y, v[k].y), __fadd_rn(v[0].z, v[k].z), __fadd_rn(v[0].w, v[k].w));
			*reinterpret_cast<float4 *>(y + (size_t)(it.y + tok) * out_stride + it.w + col) = v[0];
		}
		ptx::cluster_sync_all();  // (nobody's shared memory goes while it is read)
	}
	if (PAIR)
		ptx::cluster_sync_all();  // neither CTA leaves while its peer may still signal its barriers or read its memories
	if (warp == W_MMA) {
		if (PAIR)
			ptx::tmem_dealloc_pair(tmem, TC_TMEM_COLS);
		else
			ptx::tmem_dealloc(tmem, TC_TMEM_COLS);
	}
}

// ---- host side ----

typedef CUresult (*PFN_encodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
				    const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
				    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static PFN_encodeTiled get_encode_fn()
{
	static PFN_encodeTiled fn = nullptr;
	if (!fn) {
		void *p = nullptr;
		cudaDriverEntryPointQueryResult qres;
		if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
		    qres == cudaDriverEntryPointSuccess)
			fn = reinterpret_cast<PFN_encodeTiled>(p);
	}
	return fn;
}

static int encode_2d(tie_cuda_ctx *c, CUtensorMap *tm, CUtensorMapDataType type, size_t elem, void *base, size_t rows, size_t cols,
		     unsigned box_cols, unsigned box_rows, CUtensorMapSwizzle swz)
{
	PFN_encodeTiled enc = get_encode_fn();
	if (!enc) {
		snprintf(c->cuda_err, sizeof(c->cuda_err), "cuTensorMapEncodeTiled entry point not found");
		return TIE_CUDA_ECUDA;
	}
	cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
	cuuint64_t strides[1] = {(cuuint64_t)cols * elem};
	cuuint32_t box[2] = {box_cols, box_rows};
	cuuint32_t estr[2] = {1, 1};
	CUresult r = enc(tm, type, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
			 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	if (r != CUDA_SUCCESS) {
		snprintf(c->cuda_err, sizeof(c->cuda_err), "cuTensorMapEncodeTiled failed: %d", (int)r);
		return TIE_CUDA_ECUDA;
	}
	return TIE_CUDA_OK;
}

static int encode_map(tie_cuda_ctx *c, CUtensorMap *tm, void *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
		      const cuuint32_t *box)
{
	PFN_encodeTiled enc = get_encode_fn();
	if (!enc) {
		snprintf(c->cuda_err, sizeof(c->cuda_err), "cuTensorMapEncodeTiled entry point not found");
		return TIE_CUDA_ECUDA;
	}
	cuuint32_t estr[4] = {1, 1, 1, 1};
	CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, rank, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
			 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	if (r != CUDA_SUCCESS) {
		snprintf(c->cuda_err, sizeof(c->cuda_err), "cuTensorMapEncodeTiled (token operand) failed: %d", (int)r);
		return TIE_CUDA_ECUDA;
	}
	return TIE_CUDA_OK;
}

// Split fp16 operand [hi | lo][rows][cols] (lo array right behind hi), 128-byte swizzle.  A box is one
// super-block: 4 tiles of 64 columns, of each the box_rows hi rows, then the box_rows lo rows.
// A CTA of a pair fetches half of a token tile's rows: boxes of 8, 16, 32 rows instead of 16, 32, 64.
static int make_tmap(tie_cuda_ctx *c, CUtensorMap *tm, void *base, size_t rows, size_t cols, unsigned box_rows)
{
	cuuint64_t dims[4] = {TC_BK, (cuuint64_t)rows, 2, (cuuint64_t)cols / TC_BK};
	cuuint64_t strides[3] = {(cuuint64_t)cols * 2, (cuuint64_t)rows * cols * 2, TC_BK * 2};
	cuuint32_t box[4] = {TC_BK, box_rows, 2, TC_SPB};
	return encode_map(c, tm, base, 4, dims, strides, box);
}

// Their sub-block sums [rows][cols] (16 columns per super-block): a box is up to two tiles of 64 columns,
// the most a launch needs.
static int xq_depth(size_t cols)
{
	return cols > 64 ? 2 : 1;
}
static int make_sums_tmap(tie_cuda_ctx *c, CUtensorMap *tm, void *base, size_t rows, size_t cols, unsigned box_rows)
{
	cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)cols / 64};
	cuuint64_t strides[2] = {(cuuint64_t)cols * 2, 128};
	cuuint32_t box[3] = {64, box_rows, (cuuint32_t)xq_depth(cols)};
	return encode_map(c, tm, base, 3, dims, strides, box);
}

// Byte map of an expert tensor for the weight loader.  Q4_K: [experts x rows][row bytes], box = one
// 144-byte block x 128 rows.  Q6_K: [groups][8 rows][row records], box = one 208-byte record x 8 x 16.  half_tiles: boxes of
// half the rows (gate and up, which share a tile).
int tc_make_weight_map(tie_cuda_ctx *c, DevTensor &t, bool half_tiles, int n_experts)
{
	if (n_experts <= 0)
		n_experts = c->n_local;
	t.has_map = false;
	if (t.rows % TC_BM || t.k % QK_K)
		return TIE_CUDA_OK;
	const int nb = t.k / QK_K;
	const unsigned box_rows = half_tiles ? TC_BM / 2 : TC_BM;
	if (t.kind == W_Q4K) {
		int rc = encode_2d(c, &t.map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, t.ptr, (size_t)t.rows * n_experts, (size_t)nb * Q4K_BYTES,
				   Q4K_BYTES, box_rows, CU_TENSOR_MAP_SWIZZLE_NONE);
		if (rc)
			return rc;
	} else {
		PFN_encodeTiled enc = get_encode_fn();
		if (!enc) {
			snprintf(c->cuda_err, sizeof(c->cuda_err), "cuTensorMapEncodeTiled entry point not found");
			return TIE_CUDA_ECUDA;
		}
		cuuint64_t dims[3] = {(cuuint64_t)nb * Q6K_RECORD, 8, (cuuint64_t)t.rows * n_experts / 8};
		cuuint64_t strides[2] = {(cuuint64_t)nb * Q6K_RECORD, (cuuint64_t)q6k_r8_group_bytes(nb)};
		cuuint32_t box[3] = {Q6K_RECORD, 8, box_rows / 8};
		cuuint32_t estr[3] = {1, 1, 1};
		CUresult r = enc(&t.map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, t.ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
				 CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
		if (r != CUDA_SUCCESS) {
			snprintf(c->cuda_err, sizeof(c->cuda_err), "cuTensorMapEncodeTiled (Q6_K weights) failed: %d", (int)r);
			return TIE_CUDA_ECUDA;
		}
	}
	t.has_map = true;
	return TIE_CUDA_OK;
}

int tc_setup(tie_cuda_ctx *c)
{
	Scratch &s = c->s;
	const size_t H = c->cfg.hidden, F = c->cfg.ffn_dim;
	// tmap[array * 3 + box]: array 0 = x, 1 = h, 2 = sums of x, 3 = sums of h; box rows 16, 32, 64
	void *bases[4] = {s.xs_hi, s.hs_hi, s.xq, s.hq};
	size_t cols[4] = {H, F, (size_t)xq_cols((int)H), (size_t)xq_cols((int)F)};
	for (int a = 0; a < 4; a++)
		for (int b = 0; b < 3; b++) {
			auto make = a < 2 ? make_tmap : make_sums_tmap;
			int rc = make(c, &c->tmap[a * 3 + b], bases[a], s.rows_pad, cols[a], 16u << b);
			if (!rc)
				rc = make(c, &c->tmap_half[a * 3 + b], bases[a], s.rows_pad, cols[a], 8u << b);
			if (rc)
				return rc;
		}
#define TC_ATTR(KIND, GU) \
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(grouped_gemm_sb<KIND, GU>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcSmem<KIND, GU, false, 64>::SMEM)); \
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(grouped_gemm_sb<KIND, GU, false, false, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize,               \
					     TcSmem<KIND, GU, false, 32>::SMEM));                                                                         \
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(grouped_gemm_sb<KIND, GU, false, true, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize,                \
					     TcSmem<KIND, GU, true, 32>::SMEM))
	TC_ATTR(W_Q4K, false);
	TC_ATTR(W_Q4K, true);
	TC_ATTR(W_Q6K_R8, false);
	TC_ATTR(W_Q6K_R8, true);
#undef TC_ATTR
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(grouped_gemm_sb<W_Q4K, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
					     TcSmem<W_Q4K, false, false, 64>::SMEM));
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(grouped_gemm_sb<W_Q6K_R8, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
					     TcSmem<W_Q6K_R8, false, false, 64>::SMEM));
	// the forms that split a dense product's rows (narrow tiles only: launch_tc_dense)
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(grouped_gemm_sb<W_Q4K, false, false, false, 32, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
					     TcSmem<W_Q4K, false, false, 32>::SMEM));
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(grouped_gemm_sb<W_Q6K_R8, false, false, false, 32, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
					     TcSmem<W_Q6K_R8, false, false, 32>::SMEM));
	// the CTA-pair forms; how many pairs the device holds at once sizes their (persistent) grids
#define TC_ATTR_PAIR(KIND, GU, PEER)                                                                                          \
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(grouped_gemm_sb<KIND, GU, PEER, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
					     TcSmem<KIND, GU, true, 64>::SMEM));                                                   \
	TIE_CUDA_TRY(c, cudaFuncSetAttribute(grouped_gemm_sb<KIND, GU, PEER, true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 0))
	TC_ATTR_PAIR(W_Q4K, false, false);
	TC_ATTR_PAIR(W_Q4K, true, false);
	TC_ATTR_PAIR(W_Q4K, false, true);
	TC_ATTR_PAIR(W_Q6K_R8, false, false);
	TC_ATTR_PAIR(W_Q6K_R8, true, false);
	TC_ATTR_PAIR(W_Q6K_R8, false, true);
#undef TC_ATTR_PAIR
	{
		cudaLaunchConfig_t cfg = {};
		cfg.gridDim = dim3(c->sm_count & ~1);
		cfg.blockDim = dim3(TC_THREADS);
		cfg.dynamicSmemBytes = TcSmem<W_Q4K, true, true, 64>::SMEM;
		cudaLaunchAttribute attr[1];
		attr[0].id = cudaLaunchAttributeClusterDimension;
		attr[0].val.clusterDim.x = 2;
		attr[0].val.clusterDim.y = 1;
		attr[0].val.clusterDim.z = 1;
		cfg.attrs = attr;
		cfg.numAttrs = 1;
		int n_clusters = 0;
		if (cudaOccupancyMaxActiveClusters(&n_clusters, grouped_gemm_sb<W_Q4K, true, false, true>, &cfg) != cudaSuccess) {
			cudaGetLastError();
			n_clusters = 0;
		}
		c->tc_pairs = n_clusters < c->sm_count / 2 ? n_clusters : c->sm_count / 2;
	}
	// and how many clusters of n CTAs, for products whose rows are split (the SMs of a GPC are not a multiple of every n; either
	// kind of weights takes an SM per CTA)
	for (int n = 2; n <= TC_MAX_PARTS; n++) {
		cudaLaunchConfig_t cfg = {};
		cfg.gridDim = dim3(c->sm_count / n * n);
		cfg.blockDim = dim3(TC_THREADS);
		cfg.dynamicSmemBytes = TcSmem<W_Q4K, false, false, 32>::SMEM;
		cudaLaunchAttribute attr[1];
		attr[0].id = cudaLaunchAttributeClusterDimension;
		attr[0].val.clusterDim.x = n;
		attr[0].val.clusterDim.y = 1;
		attr[0].val.clusterDim.z = 1;
		cfg.attrs = attr;
		cfg.numAttrs = 1;
		if (cudaOccupancyMaxActiveClusters(&c->tc_clusters[n], grouped_gemm_sb<W_Q4K, false, false, false, 32, true>, &cfg) != cudaSuccess) {
			cudaGetLastError();
			c->tc_clusters[n] = 0;
		}
	}
	c->tmaps_ok = true;
	return TIE_CUDA_OK;
}

static bool tc_paired(const tie_cuda_ctx *c, int m_tiles, int k_dim, int min_blocks)
{
	return c->tc_pairs > 0 && !c->tc_no_pair && m_tiles % 2 == 0 && k_dim >= min_blocks * QK_K;
}

// arr: 0 = the split inputs x (gate/up), 1 = the split activations h (down).
template <WKind KIND, bool GU, bool PEER = false, int NT = TC_TOKEN_TILE, bool SPLIT = false>
static int launch_tc_t(tie_cuda_ctx *c, const DevTensor &t0, const DevTensor *t1, int arr, float *y, float out_scale,
		       bool sorted_out = false, const EpDst *dst = nullptr, int dense_rows = 0, const DenseView *view = nullptr,
		       const GuOut &gu = GuOut(), int n_parts = 1)
{
	Scratch &s = c->s;
	const int4 *tile_info = dense_rows ? nullptr : s.tile_info;
	const int n_experts = dense_rows ? dense_rows : c->n_local;
	const int m_tiles = (GU ? 2 : 1) * t0.rows / TC_BM;
	const CUtensorMap &w0m = t0.map;
	const CUtensorMap &w1m = GU ? t1->map : t0.map;
	const uint8_t *w1p = t1 ? t1->ptr : nullptr;
	const int *perm = sorted_out ? nullptr : s.perm;
	const int out_stride = t0.rows;
	const EpDst d = dst ? *dst : EpDst();
	const int k_dim = t0.k;
	const int xqd = xq_depth((size_t)xq_cols(t0.k));
	// a dense tensor brings the maps of its own view of the operand scratch (entries 0-2 operand, 3-5 sums)
	const CUtensorMap *mh = view ? view->half : c->tmap_half + arr * 3, *mhq = view ? view->half + 3 : c->tmap_half + (2 + arr) * 3;
	const CUtensorMap *mf = view ? view->full : c->tmap + arr * 3, *mfq = view ? view->full + 3 : c->tmap + (2 + arr) * 3;
	// pairs of CTAs (one MMA issue for two 128-row tiles) where the 128-row tiles pair up and a work item has at
	// least 4 super-blocks.  Measured at 64 / 512 / 4096 tokens: rows of 8 super-blocks (gate/up) 68 / 79 / 355 us
	// paired, 70 / 92 / 410 single (a pair fetches half the token bytes per CTA); rows of 3 (down) 59 / 73 / 310
	// paired, 55 / 70 / 294 single (the hand-offs between two SMs are not amortised over so few).  Wide tiles of Q6_K rows, which
	// expand longest, from 3 on: since their rows are stored in order, 512 / 1000 / 4096 tokens 56.3 / 76.8 / 228 paired,
	// 56.3 / 78.8 / 236 single (narrow, 64: 50.2 and 48.2; wide Q4_K 52 / 73.7 / 224 and 50.2 / 72.7 / 225).
	const int min_blocks = KIND == W_Q6K_R8 && NT > 32 && !PEER ? 3 : 4;
	// Set up beside the kernel in front: a CTA needs a whole SM, so they come as SMs fall idle (9 tokens 84.3 -> 82.3 us, 64 137.5 ->
	// 135.4; since no pass stands between the two products wide tiles gain too: a step of 400 / 512 / 4096 tokens 167.1 / 188.7 /
	// 929 -> 164.8 / 183.5 / 926).
	const int items = dense_rows ? (dense_rows + NT - 1) / NT * m_tiles * n_parts : 1 << 30;	// (known for a dense tensor: no idle CTAs)
	if constexpr (!SPLIT) {
		if (tc_paired(c, m_tiles, k_dim, min_blocks))
			return launch_kernel(c, true, 2, grouped_gemm_sb<KIND, GU, PEER, true, NT>, dim3(2 * min(c->tc_pairs, items / 2)), TC_THREADS,
				     TcSmem<KIND, GU, true, NT>::SMEM, mh[0], mh[1], mh[2], mhq[0], mhq[1], mhq[2], w0m, w1m, t0.ptr, w1p,
				     t0.expert_stride, k_dim, tile_info, s.tile_start, n_experts, m_tiles, y, perm, out_stride, out_scale,
				     s.status, t0.rows, d, xqd, gu, n_parts);
	}
	return launch_kernel(c, true, n_parts, grouped_gemm_sb<KIND, GU, PEER, false, NT, SPLIT>, dim3(min(c->sm_count, items)), TC_THREADS,
			     TcSmem<KIND, GU, false, NT>::SMEM, mf[0], mf[1], mf[2], mfq[0], mfq[1], mfq[2], w0m, w1m, t0.ptr, w1p,
			     t0.expert_stride, k_dim, tile_info, s.tile_start, n_experts, m_tiles, y, perm, out_stride, out_scale, s.status,
			     t0.rows, d, xqd, gu, n_parts);
}

static bool tc_tensor_ok(const DevTensor &t)
{
	return t.has_map && t.rows % TC_BM == 0 && t.k % QK_K == 0;
}

bool tc_supported(const tie_cuda_ctx *c, const Layer &L)
{
	return c->tmaps_ok && L.gate.kind == L.up.kind && tc_tensor_ok(L.gate) && tc_tensor_ok(L.up) && tc_tensor_ok(L.down);
}

// xs_hi/xs_lo (and xq for Q4_K) must hold the split inputs in sorted order; the sort must
// have been run with n_tile (32 or 64).  Leaves the SwiGLU outputs, scaled and split, in hs_hi/hs_lo (and their sums in hq
// where the down matrix is Q4_K).
int launch_tc_gate_up(tie_cuda_ctx *c, const Layer &L, int n_tile)
{
	Scratch &s = c->s;
	GuOut gu;
	gu.hi = s.hs_hi;
	gu.lo = (size_t)(s.hs_lo - s.hs_hi);
	gu.sums = L.down.kind == W_Q4K ? s.hq : nullptr;
	gu.sum_cols = xq_cols(L.gate.rows);
	gu.silu = c->silu;
	auto launch = n_tile == 32 ? (L.gate.kind == W_Q4K ? launch_tc_t<W_Q4K, true, false, 32> : launch_tc_t<W_Q6K_R8, true, false, 32>)
				   : (L.gate.kind == W_Q4K ? launch_tc_t<W_Q4K, true> : launch_tc_t<W_Q6K_R8, true>);
	return launch(c, L.gate, &L.up, 0, nullptr, TC_H_SCALE, true, nullptr, 0, nullptr, gu, 1);
}

// reads hs_hi/hs_lo; writes y in sorted order or (sorted false) y[perm[p]].
int launch_tc_down(tie_cuda_ctx *c, const Layer &L, int n_tile, float *y, bool sorted)
{
	const float scale = 1.0f / TC_H_SCALE;
	if (n_tile == 32)
		return L.down.kind == W_Q4K ? launch_tc_t<W_Q4K, false, false, 32>(c, L.down, nullptr, 1, y, scale, sorted)
					    : launch_tc_t<W_Q6K_R8, false, false, 32>(c, L.down, nullptr, 1, y, scale, sorted);
	return L.down.kind == W_Q4K ? launch_tc_t<W_Q4K, false>(c, L.down, nullptr, 1, y, scale, sorted)
				    : launch_tc_t<W_Q6K_R8, false>(c, L.down, nullptr, 1, y, scale, sorted);
}

// A dense tensor (one "expert") on the grouped product: y[p][row] = sum_k w[row][k] x[p][k].  The
// split operand of the batch lives in the context's x arrays, VIEWED with the tensor's own row
// length k (any multiple of 256): hi rows at the array's start, lo rows rows_view * k behind, the
// sub-block sums likewise in the sums array; the tensor carries the tensor maps of that view.
bool tc_dense_supported(const tie_cuda_ctx *c, const DevTensor &t)
{
	return c->tmaps_ok && t.has_map && t.view && t.rows % TC_BM == 0 && t.k % QK_K == 0;
}

int tc_make_dense_view(tie_cuda_ctx *c, DevTensor &t)
{
	Scratch &s = c->s;
	const size_t H = c->cfg.hidden, K = t.k, XH = xq_cols((int)H), XK = xq_cols((int)K);
	DenseView *v = new (std::nothrow) DenseView();
	if (!v)
		return TIE_CUDA_ENOMEM;
	const size_t rows_x = s.rows_pad * H / K, rows_q = s.rows_pad * XH / XK;
	v->rows = rows_x < rows_q ? rows_x : rows_q;
	v->lo_off = v->rows * K;
	for (int b = 0; b < 3 && v->rows >= 64; b++) {
		int rc = make_tmap(c, &v->full[b], s.xs_hi, v->rows, K, 16u << b);
		if (!rc)
			rc = make_tmap(c, &v->half[b], s.xs_hi, v->rows, K, 8u << b);
		if (!rc)
			rc = make_sums_tmap(c, &v->full[3 + b], s.xq, v->rows, XK, 16u << b);
		if (!rc)
			rc = make_sums_tmap(c, &v->half[3 + b], s.xq, v->rows, XK, 8u << b);
		if (rc) {
			delete v;
			return rc;
		}
	}
	if (v->rows < 64) {  // the scratch of this context cannot hold a single tile of such rows
		delete v;
		return TIE_CUDA_OK;
	}
	t.view = v;
	return TIE_CUDA_OK;
}

int launch_tc_dense(tie_cuda_ctx *c, const DevTensor &t, int n_rows, float *y)
{
	// tiles of 64 rows share a weight tile's expansion; tiles of 32 where those leave SMs idle
	const int m_tiles = t.rows / TC_BM, nb = t.k / QK_K;
	const bool narrow = (n_rows + 63) / 64 * m_tiles <= c->sm_count / 2;
	const int tiles = (narrow ? (n_rows + 31) / 32 : (n_rows + 63) / 64) * m_tiles;
	// As many parts of a row as divide it and fit the device at once.  2048 -> 512 of 37 tokens 14.8 -> 10.9 us, 4096 -> 2048 of 64
	// 19.6 -> 12.9; a second wave of clusters costs more than the parts give (2048 -> 512 of 100 tokens, 16 clusters of 8: 16.9).
	// (Clusters of two and more are half as many as SMs at the most, so tiles of 64 are never split: these are more.)
	int parts = 1;
	for (int n = 2; narrow && n <= TC_MAX_PARTS; n++)
		if (nb % n == 0 && tiles <= c->tc_clusters[n])
			parts = n;
	auto run = [&](auto launch) { return launch(c, t, nullptr, 0, y, 1.0f, true, nullptr, n_rows, t.view, GuOut(), parts); };
	const bool q4 = t.kind == W_Q4K;
	if (parts > 1)
		return q4 ? run(launch_tc_t<W_Q4K, false, false, 32, true>) : run(launch_tc_t<W_Q6K_R8, false, false, 32, true>);
	if (narrow)
		return q4 ? run(launch_tc_t<W_Q4K, false, false, 32>) : run(launch_tc_t<W_Q6K_R8, false, false, 32>);
	return q4 ? run(launch_tc_t<W_Q4K, false>) : run(launch_tc_t<W_Q6K_R8, false>);
}

// The down product of an expert-parallel step: row p goes to the rank and row dst->row[p] names.
int launch_tc_down_peer(tie_cuda_ctx *c, const Layer &L, const EpDst &dst)
{
	if (L.down.kind == W_Q4K)
		return launch_tc_t<W_Q4K, false, true>(c, L.down, nullptr, 1, nullptr, 1.0f / TC_H_SCALE, true, &dst);
	return launch_tc_t<W_Q6K_R8, false, true>(c, L.down, nullptr, 1, nullptr, 1.0f / TC_H_SCALE, true, &dst);
}

}  // namespace tie
