// The fp16 operands of the tensor-core assignment: a (scaled, centred) coordinate as the sum of two
// fp16 values, and a mean's |c|^2 as the sum of three products of powers of two and fp16 values.
#pragma once

#include <cuda_fp16.h>
#include <cstdint>

#include "common.cuh"

namespace bkm {

// x = hi + lo to 22 bits (2^-25 absolute for |x| < 2^-2, where lo is subnormal); values that fp16
// cannot hold stay finite, which keeps |hi + lo| <= |x|.
__device__ __forceinline__ void tc_split(float x, __half& hi, __half& lo)
{
	const float c = fminf(fmaxf(x, -65504.0f), 65504.0f);
	hi = __float2half_rn(c);
	lo = __float2half_rn(c - __half2float(hi));
}

// Two neighbouring dimensions as the words of the two planes; what the high parts leave over is added to `rest2`, squared.
__device__ __forceinline__ void tc_split2(float x0, float x1, uint32_t& hi, uint32_t& lo, float& rest2)
{
	__half h0, l0, h1, l1;
	tc_split(x0, h0, l0);
	tc_split(x1, h1, l1);
	const float r0 = x0 - __half2float(h0), r1 = x1 - __half2float(h1);
	rest2 = fmaf(r0, r0, fmaf(r1, r1, rest2));
	hi = (uint32_t)__half_as_ushort(h0) | ((uint32_t)__half_as_ushort(h1) << 16);
	lo = (uint32_t)__half_as_ushort(l0) | ((uint32_t)__half_as_ushort(l1) << 16);
}

// The extra K step.  Columns 0..2 carry v = |c|^2 (at most TC_NORM2_MAX): fp16 values on the mean's
// side against 2^15, 2^4 and 2^-7 on the points' side, exact to 33 bits; column 3 carries the offset
// constant of the keys as an fp16 value on the points' side against 2^15 on the mean's side.  Column 4 is for the padding
// rows behind the last mean: 2^15 there and 0 for the means, against what puts their value above that of every mean.
constexpr float TC_AUG_A0 = 32768.0f, TC_AUG_A1 = 16.0f, TC_AUG_A2 = 0.0078125f, TC_AUG_B3 = 32768.0f;

__device__ __forceinline__ uint4 tc_aug_row(float v)
{
	v = fminf(v, 2.0f * 1073741824.0f - 4194304.0f);
	const __half b0 = __float2half_rn(v * (1.0f / TC_AUG_A0));
	const float r1 = v - __half2float(b0) * TC_AUG_A0;
	const __half b1 = __float2half_rn(r1 * (1.0f / TC_AUG_A1));
	const float r2 = r1 - __half2float(b1) * TC_AUG_A1;
	const __half b2 = __float2half_rn(r2 * (1.0f / TC_AUG_A2));
	return make_uint4((uint32_t)__half_as_ushort(b0) | ((uint32_t)__half_as_ushort(b1) << 16),
		(uint32_t)__half_as_ushort(b2) | ((uint32_t)__half_as_ushort(__float2half_rn(TC_AUG_B3)) << 16), 0u, 0u);
}

__device__ __forceinline__ uint4 tc_aug_padding_row()
{
	const uint32_t b = (uint32_t)__half_as_ushort(__float2half_rn(TC_AUG_B3));
	return make_uint4(0u, b << 16, b, 0u);
}

} // namespace bkm
