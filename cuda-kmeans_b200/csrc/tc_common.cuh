// Device helpers shared by the tensor-core assignment kernels: shared-memory operand descriptors
// for tcgen05.mma, the bounded wait, and the arg-min over accumulator columns on integer keys.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"
#include "keys.cuh"
#include "tc_split.cuh"

namespace bkm {

constexpr uint32_t TC_MA = 2;            // point tiles per block (= TMEM accumulators)
constexpr uint32_t TC_NB = 2;            // centroid-tile stages
constexpr uint32_t TC_NT_MAX = 256;      // centroids per tile (the widest MMA: N = 256)
constexpr uint32_t TC_EPI_WARPS = 16;          // four per TMEM lane quarter, each a quarter of the columns
constexpr uint32_t TC_THREADS = (2 + TC_EPI_WARPS) * 32;
constexpr uint32_t TC_MAX_KPAD = 1u << 20;
constexpr uint32_t TC_TMEM_COLS = 512;


// Bounded wait that also gives up when another role already failed.  try_wait suspends the
// thread for a while by itself but comes back early often, so the loop around it decides how
// much the waiting warps take from the warps that work.  SLEEP_NS = 0: look at the abort flag
// and the clock in every round (the clock read is slow and paces the loop).  SLEEP_NS > 0:
// sleep between rounds and look at flag and clock every 256th round only.  LEAN: the 256 rounds
// run as one six-instruction loop (the CTA-pair kernel gained 1.4 % from it, the one-CTA kernel
// lost 2 %: measured, not explained).
template<uint32_t SLEEP_NS = 0, bool LEAN = false>
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag)
{
	if (ptx::mbar_try_wait(bar, parity)) return true;
	if (SLEEP_NS != 0 && LEAN) {
		uint64_t t0 = 0;
		while (true) {
			if (ptx::mbar_poll_round<SLEEP_NS>(bar, parity, 256)) return true;
			if (*abort_flag) return false;
			const uint64_t now = ptx::globaltimer_ns();
			if (t0 == 0) t0 = now;
			else if (now - t0 > ptx::WAIT_LIMIT_NS) break;
		}
	} else if (SLEEP_NS == 0) {
		const uint64_t t0 = ptx::globaltimer_ns();
		while (true) {
			if (ptx::mbar_try_wait(bar, parity)) return true;
			if (*abort_flag) return false;
			if (ptx::globaltimer_ns() - t0 > ptx::WAIT_LIMIT_NS) break;
		}
	} else {
		uint32_t spins = 0;
		uint64_t t0 = 0;
		while (true) {
			if (ptx::mbar_try_wait(bar, parity)) return true;
			__nanosleep(SLEEP_NS);
			if ((++spins & 255u) == 0) {
				if (*abort_flag) return false;
				const uint64_t now = ptx::globaltimer_ns();
				if (t0 == 0) t0 = now;
				else if (now - t0 > ptx::WAIT_LIMIT_NS) break;
			}
		}
	}
	*abort_flag = 1;
	return false;
}

// Like wait_or_abort, and a wait that runs out also raises the flag of the other CTA.
template<uint32_t SLEEP_NS = 100>
__device__ __forceinline__ bool pair_wait(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t peer_abort_addr)
{
	if (wait_or_abort<SLEEP_NS, true>(bar, parity, abort_flag)) return true;
	ptx::st_cluster_u32(peer_abort_addr, 1u);
	return false;
}

// Place in a ring of buffers.  (Counted up with a wrap: remainder and quotient by a ring size that is known at run time cost the
// loading lane of the screening pass 800 clocks per slice, beside four busy warps, where a slice's multiplication takes 512.)
struct RingPos {
	uint32_t slot = 0, phase = 0;
	__device__ __forceinline__ void next(uint32_t slots) { if (++slot == slots) { slot = 0; phase ^= 1u; } }
};

// K-major operand, 64-byte swizzle: rows of 64 B, 8-row groups 512 B apart.
__device__ __forceinline__ uint64_t make_desc_sw64(uint32_t smem_addr)
{
	return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | (1ull << 16) | (32ull << 32) | (1ull << 46) | (4ull << 61);
}

// K-major operand without swizzle, one K step (16 fp16 = two 16-byte chunks) wide: 8x16-byte core
// matrices; the two chunks of a row group are 128 B apart, row groups 256 B apart.
__device__ __forceinline__ uint64_t make_desc_aug(uint32_t smem_addr)
{
	return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | (8ull << 16) | (16ull << 32) | (1ull << 46);
}

// The two 32-bit halves of such descriptors: the low half holds the address field (>> 4) and the
// leading byte offset, the high half is a constant of the layout.
constexpr uint32_t DESC_HI_SW128 = 64u | (1u << 14) | (2u << 29);     // 128-byte swizzle, 8-row groups 1024 B apart
constexpr uint32_t DESC_HI_AUG = 16u | (1u << 14);                    // no swizzle, row groups 256 B apart
constexpr uint32_t DESC_HI_SW64 = 32u | (1u << 14) | (4u << 29);      // 64-byte swizzle, 8-row groups 512 B apart
__device__ __forceinline__ uint32_t desc_lo_sw128(uint32_t smem_addr) { return ((smem_addr >> 4) & 0x3FFFu) | (1u << 16); }
__device__ __forceinline__ uint32_t desc_lo_aug(uint32_t smem_addr) { return ((smem_addr >> 4) & 0x3FFFu) | (8u << 16); }

// The constant A operand of the extra K step (128 rows, no-swizzle layout): see tc_aug_row.  Padding columns get the value
// 2P - P/32 (and the rounding of two fp16 values), above every real value (at most 1.83 P) and inside [P, 2P), so
// that the arg-min needs no column masks.
__device__ __forceinline__ void fill_a_aug(uint8_t* a_aug, const KeyConsts& kc, float x2max, uint32_t tid, uint32_t nthreads)
{
	const float offset_c = kc.offset_c, padding = kc.pow2 - fmaxf(x2max, 1.0f) - kc.pow2 * (1.0f / 16.0f);     // (the offset takes the norm as at least 1, too)
	const __half a0 = __float2half_rn(TC_AUG_A0), a1 = __float2half_rn(TC_AUG_A1), a2 = __float2half_rn(TC_AUG_A2);
	const __half a3 = __float2half_rn(offset_c * (1.0f / TC_AUG_B3)), a4 = __float2half_rn(padding * (1.0f / TC_AUG_B3));
	const uint4 row = make_uint4((uint32_t)__half_as_ushort(a0) | ((uint32_t)__half_as_ushort(a1) << 16),
		(uint32_t)__half_as_ushort(a2) | ((uint32_t)__half_as_ushort(a3) << 16), (uint32_t)__half_as_ushort(a4), 0u);
	uint32_t* words = reinterpret_cast<uint32_t*>(a_aug);
	for (uint32_t r = tid; r < TC_MTILE; r += nthreads) {
		*reinterpret_cast<uint4*>(words + aug_offset(r, 0)) = row;
		*reinterpret_cast<uint4*>(words + aug_offset(r, 1)) = make_uint4(0u, 0u, 0u, 0u);
	}
}

// Key constants of the scaled values.  The norms are taken as at least 1 so that the offset constant
// is a normal fp16 value; that it is rounded to 11 bits there (P / 1024 at most) is covered by the
// head-room of P / 32.
__device__ __forceinline__ KeyConsts tc_key_consts(float x2max, float c2max) { return make_key_consts(fmaxf(x2max, 1.0f), c2max); }

// The part of the near-tie band that does not depend on the point: four value spacings, plus what the
// absolute 2^-25 of small operand values can move a product sum by (2 * 2^-25 * sqrt(dim) * (|x| + |c|)
// for each side), plus what the reference's own squares lose where they are subnormal: half of 2^-149
// for each dimension and distance, so dim * 2^-149 for a difference of two, twice that taken, in units of
// `scale` squared (the values of this pass are scaled to the data, the reference's are not: where they
// vanish its distances tie).
// It is infinite - every point goes to the exact kernel - where the means lie beyond what the operands
// hold, and where a squared distance of the reference, at most 2 * (|x|^2 + |c|^2) before the scaling, can
// pass half the largest float: its distances are then infinite and tie.  (A point beyond the operands'
// range has an infinite |x|^2, which does the same for that point.)
__device__ __forceinline__ float tc_margin_floor(float ulp, float x2max, float c2max, float sqrt_dim, float scale)
{
	const float s63 = scale * 9.223372e18f, s_74 = scale * 5.293956e-23f;            // scale * 2^63, scale * 2^-74
	if (!(c2max <= TC_NORM2_MAX) || x2max + c2max >= s63 * s63) return INFINITY;
	return 4.0f * ulp + 2.4e-7f * sqrt_dim * sqrtf(x2max + c2max) + (sqrt_dim * s_74) * (sqrt_dim * s_74);
}

// The three products of one operand-tile pair over KS steps of 16 dimensions: the small cross
// terms lo*hi and hi*lo first, then the dominant hi*hi.  Operands are the low halves of the
// descriptors (+2 in the address field = 32 bytes = one K step), `hi_word` their common high half.
// `acc_first` = accumulate the very first product onto the destination.
template<uint32_t KS>
__device__ __forceinline__ void issue_products(uint32_t d_tmem, uint32_t a_hi, uint32_t a_lo, uint32_t b_hi, uint32_t b_lo,
	uint32_t hi_word, uint32_t idesc, uint32_t acc_first)
{
	ptx::mma_f16_halves(d_tmem, a_lo, hi_word, b_hi, hi_word, idesc, acc_first);
	#pragma unroll
	for (uint32_t ks = 1; ks < KS; ++ks)
		ptx::mma_f16_halves(d_tmem, a_lo + 2 * ks, hi_word, b_hi + 2 * ks, hi_word, idesc, 1);
	#pragma unroll
	for (uint32_t ks = 0; ks < KS; ++ks)
		ptx::mma_f16_halves(d_tmem, a_hi + 2 * ks, hi_word, b_lo + 2 * ks, hi_word, idesc, 1);
	#pragma unroll
	for (uint32_t ks = 0; ks < KS; ++ks)
		ptx::mma_f16_halves(d_tmem, a_hi + 2 * ks, hi_word, b_hi + 2 * ks, hi_word, idesc, 1);
}

// The end of a point's arg-min: decode the winning key (key - key_base = M * mantissa + column) and
// write the assignment.  Returns whether best and second are closer than `margin`, i.e. whether
// the point has to be queued for the exact kernel (the caller appends, a warp at a time).
__device__ __forceinline__ bool finish_point(uint32_t best, uint32_t second, uint32_t bchunk, uint32_t key_base, uint32_t key_mult, uint32_t key_magic,
	float ulp, float margin, uint32_t k, uint64_t p, uint32_t* __restrict__ asg)
{
	const uint32_t bm = div_key(best - key_base, key_magic);
	// (with means beyond the operands' range the keys mean nothing: any index, the exact kernel follows)
	asg[p] = min(bchunk * 32u + ((best - key_base) - bm * key_mult), k - 1);
	// keys are (mantissa * M + column): the difference of the quotients counts value spacings
	const float gap = second == 0xFFFFFFFFu ? INFINITY : (float)(div_key(second - key_base, key_magic) - bm) * ulp;
	return !(gap > margin);                  // (a margin that is not a number sends the point to the exact kernel as well)
}

// ---- the CTA-pair kernel (assign_tc_pair.cu), used through the plan of assign_tc.cu ----
bool assign_tc_pair_supported(uint32_t k, uint32_t k_pad, uint32_t dim, uint32_t d_pad, uint32_t nt_cols, int sm_count);
bool assign_tc_pair_can_fuse(uint32_t k_pad, uint32_t dim, uint32_t d_pad);
cudaError_t assign_tc_pair_prepare(int sm_count, int* max_pairs);
cudaError_t launch_assign_tc_pair(const CUtensorMap& a_hi, const CUtensorMap& a_lo, const CUtensorMap& b_hi, const CUtensorMap& b_lo,
	const float* b_aug, const float* xnorm, uint32_t* asg, uint64_t n, uint32_t n_tiles, uint32_t k, uint32_t k_pad, uint32_t d_pad,
	uint32_t ksteps, int max_pairs, Control* ctl, int slot, uint32_t* flag_list, float margin_coef, float sqrt_dim, cudaStream_t stream,
	const FusedAcc* fused, uint32_t dim, uint32_t step_begin = 0, uint32_t step_end = 0);

// ---- the screening pass (assign_tc_screen.cu), likewise ----
cudaError_t assign_tc_screen_prepare(int sm_count, int* max_pairs);
cudaError_t launch_assign_tc_screen(const CUtensorMap& a_hi, const CUtensorMap& b_hi, const CUtensorMap& b_aug, const TcPoints& tp, uint32_t* asg,
	uint64_t n, uint32_t k, uint32_t k_pad, uint32_t dim, int max_pairs, Control* ctl, int slot, float margin_coef, float margin_scale, float sqrt_dim,
	cudaStream_t stream);

} // namespace bkm
