// Integer keys for the arg-min over approximate squared distances, shared by the tensor-core and
// the CUDA-core fast passes: values that all lie in one binade are turned into (value, column)
// keys whose unsigned order is the order of (value, column), and chunks of 32 keys are reduced to
// the smallest and the second smallest with plain integer minima.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "common.cuh"

namespace bkm {

__device__ __forceinline__ uint32_t umin3(uint32_t a, uint32_t b, uint32_t c) { return __vimin3_u32(a, b, c); }

// Keys of accumulator values.  The kernel adds a constant to every value so that
// all of them are positive floats with the SAME exponent; their bit patterns then order like the
// values, the upper exponent bits carry no information, and bits * M + column (M odd, > column:
// one integer multiply-add, off the min/max pipe) is a key that keeps the full 23-bit mantissa
// and carries the column position.
// Smallest of 32 keys with three-input minima (16 instructions).
__device__ __forceinline__ uint32_t min_of_32(const uint32_t (&p)[32])
{
	uint32_t a[12];
	#pragma unroll
	for (int i = 0; i < 10; ++i) a[i] = umin3(p[3 * i], p[3 * i + 1], p[3 * i + 2]);
	a[10] = p[30];
	a[11] = p[31];
	uint32_t c[4];
	#pragma unroll
	for (int i = 0; i < 4; ++i) c[i] = umin3(a[3 * i], a[3 * i + 1], a[3 * i + 2]);
	return min(umin3(c[0], c[1], c[2]), c[3]);
}

// Smallest of 16 values (8 instructions).
__device__ __forceinline__ uint32_t min_of_16(const uint32_t* p)
{
	const uint32_t a0 = umin3(p[0], p[1], p[2]), a1 = umin3(p[3], p[4], p[5]), a2 = umin3(p[6], p[7], p[8]);
	const uint32_t a3 = umin3(p[9], p[10], p[11]), a4 = umin3(p[12], p[13], p[14]);
	return min(umin3(a0, a1, a2), umin3(a3, a4, p[15]));
}

__device__ __forceinline__ uint32_t min_of(const uint32_t (&p)[16]) { return min_of_16(p); }
__device__ __forceinline__ uint32_t min_of(const uint32_t (&p)[32]) { return min_of_32(p); }

// The two smallest of N distinct keys: key - (smallest + 1) wraps to the top of the unsigned range for the smallest only, and the
// minimum of these differences belongs to the second smallest.
template<int N>
__device__ __forceinline__ void two_smallest(const uint32_t (&p)[N], uint32_t& best, uint32_t& second)
{
	best = min_of(p);
	const uint32_t shift = ~best;                  // -(smallest + 1)
	uint32_t r0 = p[0] + shift, r1 = p[1] + shift, r2 = p[2] + shift, r3 = p[3] + shift;
	#pragma unroll
	for (uint32_t t = 4; t < N; t += 4) {
		r0 = __viaddmin_u32(p[t], shift, r0);
		r1 = __viaddmin_u32(p[t + 1], shift, r1);
		r2 = __viaddmin_u32(p[t + 2], shift, r2);
		r3 = __viaddmin_u32(p[t + 3], shift, r3);
	}
	second = min(umin3(r0, r1, r2), r3) - shift;
}

// The two smallest values of a point's row, and the column of the smallest, from minima alone.  The
// columns are partitioned twice: by their position (column mod 16) and into groups of 16 neighbours.  Two
// columns of one position lie in different groups, so the second smallest value of the row is the
// second smallest of the 16 position minima or the second smallest of the group minima, whichever is
// less; the smallest one has its position from the one partition and its group from the other.  A value thus
// takes part in two three-input minima (which each take in two values) and needs no key of its own: 32 of them
// for a chunk of 32 columns and nine instructions to rank its two groups, where 32 keys with a pass for
// the smallest and one for the second took 88 (and no final ranking of positions, about 60 per row and warp).  The
// epilogues are bound by the ALU pipe (two clocks per instruction): 2^26 x 16 against 256 means 3.35 -> 2.82 ms,
// 2^21 x 32 against 1024 with update sums 0.510 -> 0.419 ms.  Equal values give a difference of zero, a near-tie.
// Positions and groups become keys of the usual form (bits * M + column) only for ranking.
struct RowMin {
	uint32_t position[16];
	uint32_t best, second;      // the two smallest group minima so far, as keys bits * M + group within the chunk
	uint32_t chunk;             // chunk (of 32 columns) of the first

	__device__ __forceinline__ void reset()
	{
		#pragma unroll
		for (int t = 0; t < 16; ++t) position[t] = 0xFFFFFFFFu;
		best = second = 0xFFFFFFFFu;
		chunk = 0;
	}

	// Ranks the minima of the two groups of a chunk.
	__device__ __forceinline__ void take_groups(uint32_t g0, uint32_t g1, uint32_t key_mult, uint32_t chunk_id)
	{
		const uint32_t k0 = g0 * key_mult, k1 = g1 * key_mult + 1u;
		const uint32_t lo = min(k0, k1), hi = max(k0, k1);
		second = umin3(second, hi, max(best, lo));
		chunk = lo < best ? chunk_id : chunk;
		best = min(best, lo);
	}

	// One chunk of 32 columns.
	__device__ __forceinline__ void take_chunk(const uint32_t (&v)[32], uint32_t key_mult, uint32_t chunk_id)
	{
		#pragma unroll
		for (int t = 0; t < 16; ++t) position[t] = umin3(position[t], v[t], v[t + 16]);
		take_groups(min_of_16(v), min_of_16(v + 16), key_mult, chunk_id);
	}

	// (best, second, chunk of best) with keys bits * M + column within the chunk.  What stands for "nothing" -
	// padding, or no second column at all - lies above every key of a value.  Values outside the binade (means
	// beyond what the pass can hold) give meaningless, but harmless keys.
	__device__ __forceinline__ void finish(uint32_t key_base, uint32_t key_mult, uint32_t key_magic, uint32_t& best_out, uint32_t& second_out, uint32_t& chunk_out) const;
};

// The three smallest keys of a point so far, with the chunks (of 32 columns) of the first two.  A point
// whose third smallest is far enough from the smallest has only two candidates for the exact re-check.
struct BestThree {
	uint32_t best = 0xFFFFFFFFu, second = 0xFFFFFFFFu, third = 0xFFFFFFFFu, best_chunk = 0, second_chunk = 0;

	// Takes in another such triple, b <= s <= t.  Where keys of different chunks are equal, either may be
	// called the second: the other is then the third and as close.
	__device__ __forceinline__ void merge(uint32_t b, uint32_t s, uint32_t t, uint32_t b_chunk, uint32_t s_chunk)
	{
		const bool wins = b < best;
		const uint32_t loser = max(best, b), loser_chunk = wins ? best_chunk : b_chunk;
		const uint32_t middle = max(min(second, s), min(max(second, s), loser));      // second smallest of the three that are left
		const uint32_t next = umin3(second, s, loser);
		third = umin3(third, t, middle);
		second_chunk = next == loser ? loser_chunk : (next == second ? second_chunk : s_chunk);
		second = next;
		best_chunk = wins ? b_chunk : best_chunk;
		best = min(best, b);
	}
};

// Takes a chunk of 32 columns into the three smallest keys.  Plain minima instead of a tournament: the keys are
// distinct (they carry the column), so key - (smallest + 1) wraps to the top of the unsigned range for the
// smallest key only, and the minimum of these differences - 28 fused add-and-minimum instructions in four
// independent chains - belongs to the second smallest; once more from there for the third.
__device__ __forceinline__ void chunk_update3(const uint32_t (&v)[32], uint32_t key_mult, uint32_t chunk_id, BestThree& state)
{
	uint32_t p[32];
	#pragma unroll
	for (uint32_t t = 0; t < 32; ++t) p[t] = v[t] * key_mult + t;
	auto min_above = [&p](uint32_t key) {          // the smallest key above `key`
		const uint32_t shift = ~key;               // -(key + 1)
		uint32_t r0 = p[0] + shift, r1 = p[1] + shift, r2 = p[2] + shift, r3 = p[3] + shift;
		#pragma unroll
		for (uint32_t t = 4; t < 32; t += 4) {
			r0 = __viaddmin_u32(p[t], shift, r0);
			r1 = __viaddmin_u32(p[t + 1], shift, r1);
			r2 = __viaddmin_u32(p[t + 2], shift, r2);
			r3 = __viaddmin_u32(p[t + 3], shift, r3);
		}
		return min(umin3(r0, r1, r2), r3) - shift;
	};
	const uint32_t b = min_of_32(p), s = min_above(b);
	state.merge(b, s, min_above(s), chunk_id, chunk_id);
}


// The constants that turn accumulator values into integer keys.
struct KeyConsts {
	float pow2;          // P: every accumulator value lies in [P, 2P)
	float offset_c;      // constant added to every |c|^2 - 2 x.c by the extra K step
	uint32_t key_mult;   // M
	uint32_t key_base;   // M * (bit pattern of P) mod 2^32
	uint32_t key_magic;  // multiplier of div_key for this M
};

// Offset constant: every value |c|^2 - 2 x.c lies in [-X2, X2 + 2*C2] (X2, C2 = largest |x|^2,
// |c|^2 after centring), an interval of width 2*(X2+C2); with P a power of two >= 1.25 times
// that width, value + P + X2 + P/32 stays inside [P, 2P) with P/32 of head-room on both
// sides for the rounding of the pass: one exponent for all values.
// Key of a value with bit pattern v in column t: v * M + t (mod 2^32) = key_base + M * mantissa + t.
// M is an odd number >= 33 chosen so that the largest key stays below 2^32: keys then order like
// (value, column).  A multiplier that is not a power of two keeps the multiply-add on the FMA
// pipe; the min/max tournament owns the ALU pipe.
__device__ __forceinline__ KeyConsts make_key_consts(float x2max, float c2max)
{
	KeyConsts kc;
	const float span = 1.25f * (2.0f * (x2max + c2max)) + 1.0e-30f;
	int e;
	frexpf(span, &e);                       // span = m * 2^e, m in [0.5, 1)
	kc.pow2 = ldexpf(1.0f, e);              // >= span
	kc.offset_c = kc.pow2 + x2max + kc.pow2 * (1.0f / 32.0f);
	kc.key_mult = 33;
	const uint32_t eb = __float_as_uint(kc.pow2) >> 23;
	while (kc.key_mult < 63 && ((kc.key_mult * eb) & 511u) > 510u - kc.key_mult) kc.key_mult += 2;
	kc.key_base = kc.key_mult * __float_as_uint(kc.pow2);
	kc.key_magic = (uint32_t)((((unsigned long long)(64u - kc.key_mult)) << 32) / kc.key_mult) + 1u;
	return kc;
}

// x / M for the key multipliers (33 <= M <= 63) without the integer-division sequence: with
// magic = floor(2^32 * (64 - M) / M) + 1 and t = high word of magic * x, the quotient is
// (t + (x - t) / 2) / 32, exact for every 32-bit x (division by an invariant, round-up method).
__device__ __forceinline__ uint32_t div_key(uint32_t x, uint32_t magic)
{
	const uint32_t t = __umulhi(magic, x);
	return (t + ((x - t) >> 1)) >> 5;
}

// Index of the mean that a key stands for.
__device__ __forceinline__ uint32_t key_column(uint32_t key, uint32_t chunk, uint32_t key_base, uint32_t key_mult, uint32_t key_magic)
{
	const uint32_t x = key - key_base;
	return chunk * 32u + (x - div_key(x, key_magic) * key_mult);
}

__device__ __forceinline__ void RowMin::finish(uint32_t key_base, uint32_t key_mult, uint32_t key_magic, uint32_t& best_out, uint32_t& second_out, uint32_t& chunk_out) const
{
	uint32_t p[16];
	#pragma unroll
	for (uint32_t t = 0; t < 16; ++t) p[t] = position[t] * key_mult + t;
	uint32_t b, next;
	two_smallest(p, b, next);
	second_out = min(next, second);
	// both smallest keys have the same value part: what is left of the group's key is its number
	const uint32_t value = div_key(b - key_base, key_magic) * key_mult + key_base;
	best_out = b + ((best - value) & 1u) * 16u;
	chunk_out = chunk;
}

// Appends the points whose `flag` is set to the near-tie list with ONE atomic per warp (a counter
// that every flagged point bumps by itself is a serial bottleneck once a few per cent of the points
// are flagged).  All 32 lanes of the warp must call it together.
__device__ __forceinline__ void append_flagged(bool flag, uint32_t point, Control* __restrict__ ctl, uint32_t* __restrict__ flag_list, uint64_t n)
{
	const uint32_t mask = __ballot_sync(0xffffffffu, flag);
	if (mask == 0) return;
	const uint32_t lane = threadIdx.x & 31u;
	const int leader = __ffs(mask) - 1;
	uint32_t base = 0;
	if ((int)lane == leader) base = atomicAdd(&ctl->flag_count, (uint32_t)__popc(mask));
	base = __shfl_sync(0xffffffffu, base, leader);
	if (flag) {
		const uint32_t pos = base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
		if ((uint64_t)pos < n) flag_list[pos] = point;
		else atomicOr(&ctl->status, (uint32_t)STATUS_LIST_OVERFLOW);
	}
}

// The same through a small buffer in shared memory that belongs to one warp: flagged points collect
// there and go out FLAG_BUFFER entries at a time, so that the round trip of the global counter is
// paid once per buffer instead of once per call (a warp that waits for it does nothing else).
// `cnt` lives in a register and is the same in all lanes.  All 32 lanes call together; the warp
// calls flush_flag_buffer once more when it is done.
constexpr uint32_t FLAG_BUFFER = 64;

__device__ __forceinline__ void flush_flag_buffer(uint32_t* buf, uint32_t& cnt, Control* __restrict__ ctl, uint32_t* __restrict__ flag_list, uint64_t n)
{
	if (cnt == 0) return;
	const uint32_t lane = threadIdx.x & 31u;
	uint32_t base = 0;
	if (lane == 0) base = atomicAdd(&ctl->flag_count, cnt);
	base = __shfl_sync(0xffffffffu, base, 0);
	for (uint32_t e = lane; e < cnt; e += 32) {
		if ((uint64_t)(base + e) < n) flag_list[base + e] = buf[e];
		else atomicOr(&ctl->status, (uint32_t)STATUS_LIST_OVERFLOW);
	}
	__syncwarp();
	cnt = 0;
}

__device__ __forceinline__ void buffered_append(bool flag, uint32_t point, uint32_t* buf, uint32_t& cnt, Control* __restrict__ ctl,
	uint32_t* __restrict__ flag_list, uint64_t n)
{
	const uint32_t mask = __ballot_sync(0xffffffffu, flag);
	if (mask == 0) return;
	const uint32_t m = (uint32_t)__popc(mask);
	if (cnt + m > FLAG_BUFFER) flush_flag_buffer(buf, cnt, ctl, flag_list, n);
	const uint32_t lane = threadIdx.x & 31u;
	if (flag) buf[cnt + (uint32_t)__popc(mask & ((1u << lane) - 1u))] = point;
	cnt += m;
	__syncwarp();
}

} // namespace bkm
