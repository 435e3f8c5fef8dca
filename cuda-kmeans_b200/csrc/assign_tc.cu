// Assignment on the 5th-generation tensor cores (tcgen05 + TMEM), GEMM form.
//
//   |x - c|^2 = |x|^2 + ( |c|^2 - 2 x.c )          argmin over c ignores |x|^2
//
// The x.c contraction runs on fp16 pairs: every fp32 operand, centred and multiplied by a power of
// two of the data set (tc_scale), is split once into an fp16 high part and an fp16 low part
// (x = xh + xl, 22 bits as with tf32 pairs), and xl*ch + xh*cl + xh*ch is accumulated in fp32 in
// tensor memory, which restores fp32-level accuracy of the products.  A K step holds 16 dimensions
// where tf32 has 8 at the same cost, so the three products take half the tensor time and the operands
// half the bytes.  |c|^2 and an offset constant enter the same accumulator through one more K step
// whose A operand is a constant tile, so the accumulator holds |c|^2 - 2 x.c + C, all values positive with one exponent, and
// the epilogue is a pure arg-min on integer keys.  The N x k distance
// matrix never exists in HBM.  Because the GEMM form cancels, a point whose best and
// second-best values are closer than the error band of this formulation is queued for the
// exact CUDA-core kernel, so the final assignment equals the reference arithmetic
// (headers/serial.hpp:21-35 of krulis-martin/cuda-kmeans) for every point.  The kernel covers
// the shape range of the reference's cachedRegsAssignmentKernel (kernels/kernels.cu:548-661).
//
// Kernel organisation (one persistent CTA per SM, 18 warps):
//   warp 0      : TMA producer.  dim <= 64: point tiles (128 points, hi and lo plane) go through a
//                 ring and stay for all mean tiles; mean tiles (up to 256 means, hi and lo, plus
//                 their |c|^2 K step) stream through a 2-stage ring, or stay when there is only
//                 one.  dim > 64: both operands stream in 32-dimension slices.
//   warp 1      : allocates the 512 TMEM columns and issues the tcgen05.mma instructions
//                 (kind::f16, M=128, N<=256, K=16) into two accumulators, one per point tile of
//                 a block.  The whole warp walks the loop; one elected lane issues.
//   warps 2..17 : epilogue.  Eight warps per accumulator (TMEM lane quarter x column half), so
//                 that one accumulator is reduced while the other is being multiplied.  A warp
//                 reads its columns with tcgen05.ld two 32-column chunks at a time, hands the
//                 accumulator back after its last load, and reduces each chunk with integer minima
//                 (RowMin); what it keeps per point stays in registers across all mean tiles and
//                 is merged through shared memory at the end.
// Mean sets of 2..4 tiles of 256 with 17 <= dim <= 64 run on CTA pairs instead, with all means
// resident in shared memory (assign_tc_pair.cu).
// All mbarrier waits are bounded; a wait that runs out sets STATUS_WAIT_TIMEOUT and lets every
// role fall through to the end, where TMEM is released.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "../../include/bkm.h"
#include "kernels.cuh"
#include "ptx.cuh"
#include "tc_common.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <new>

namespace bkm {

constexpr uint32_t A_PLANE_BYTES = TC_MTILE * TC_KCHUNK * 4;     // 16 KiB: 128 rows x 128 B
constexpr uint32_t B_PLANE_BYTES = TC_NT_MAX * TC_KCHUNK * 4;    // 32 KiB: 256 rows x 128 B
constexpr uint32_t A_TILE_BYTES = 2 * A_PLANE_BYTES;             // hi + lo
constexpr uint32_t B_STAGE_BYTES = 2 * B_PLANE_BYTES;
constexpr uint32_t AUG_BYTES = TC_NT_MAX * 8 * 4;                // 8 KiB: 256 rows x one K step of 16 fp16
// K-loop mode (dim > 64): both operands stream in 32-dimension slices (16 words = rows of 64 B,
// 64-byte swizzle).  A stage holds the slice of BOTH point tiles of the block and of one mean tile:
// [A0 hi | A0 lo | A1 hi | A1 lo | B hi | B lo], and feeds both accumulators, so every byte of
// the mean tile that crosses from L2 is used for 256 points.  Three stages; the |c|^2 steps of
// the current and the next mean tile sit behind them.
constexpr uint32_t KL_KW = 16;
constexpr uint32_t KL_STAGES = 3;
constexpr uint32_t KL_A_PLANE = TC_MTILE * KL_KW * 4;            // 8 KiB
constexpr uint32_t KL_B_PLANE = TC_NT_MAX * KL_KW * 4;           // 16 KiB
constexpr uint32_t KL_A1_OFF = 2 * KL_A_PLANE, KL_B_OFF = 4 * KL_A_PLANE;
constexpr uint32_t KL_STAGE_BYTES = KL_B_OFF + 2 * KL_B_PLANE;   // 64 KiB
constexpr uint32_t KL_AUG_OFF = KL_STAGES * KL_STAGE_BYTES;      // two |c|^2 steps of 8 KiB
constexpr uint32_t SM_A_OFF = 0;
constexpr uint32_t SM_B_OFF = SM_A_OFF + TC_MA * A_TILE_BYTES;
constexpr uint32_t SM_BAUG_OFF = SM_B_OFF + TC_NB * B_STAGE_BYTES; // |c|^2 K step per stage
constexpr uint32_t SM_AAUG_OFF = SM_BAUG_OFF + TC_NB * AUG_BYTES;  // constant ones tile (128 rows)
constexpr uint32_t SM_MERGE_OFF = SM_AAUG_OFF + TC_MTILE * 8 * 4;
// (with THREE the same slots hold five words and extend over the flag buffers, which that form does not use)
constexpr uint32_t MERGE_BYTES = 2 * 3 * TC_MA * TC_MTILE * 4;   // (best, second, chunk) of the upper column half, two slots
constexpr uint32_t SM_FLAG_OFF = SM_MERGE_OFF + MERGE_BYTES;       // per epilogue warp: near-ties on their way to the list
constexpr uint32_t SM_BAR_OFF = SM_FLAG_OFF + TC_EPI_WARPS * FLAG_BUFFER * 4;
constexpr uint32_t SM_TOTAL = SM_BAR_OFF + 256;
constexpr uint32_t SM_ALLOC = SM_TOTAL + 1024;                   // slack for 1024-byte alignment

uint32_t tc_nt_cols(uint32_t k) { return k >= TC_NT_MAX ? TC_NT_MAX : round_up(k, 32); }
uint32_t tc_kpad(uint32_t k) { return round_up(k, tc_nt_cols(k)); }

// The three-key form costs the epilogue a third more minima; it pays where the multiplication is long
// enough to make that small and the exact pass over all means long enough to matter (2^20 x 512 against
// 4096: the pass 8.70 -> 9.06 ms, the re-check of 4400 points 1.49 -> 0.09 ms).
uint32_t tc_partial_words(uint32_t k, uint32_t dim)
{
	if (tc_dpad(dim) <= TC_KCHUNK || tc_kpad(k) / tc_nt_cols(k) < 2 * TC_JSPLIT) return 0;
	return dim >= 256 ? 5 : 3;
}

bool assign_tc_supported(const Shape& s)
{
	return s.dim <= 4096 && tc_kpad(s.k) <= TC_MAX_KPAD && s.n < (1ull << 32) - 1024;
}

// ------------------------------------------------------------------------------------------
// one-off split of the points
// ------------------------------------------------------------------------------------------

// Largest |x|^2 of a block's points -> ctl->xmax2, one atomic per block: one per warp kept the line that
// every block reads its scale from busy (82 us for 100 003 points of 128 dimensions).
__device__ __forceinline__ void block_norm_max(float local_max, Control* __restrict__ ctl)
{
	__shared__ float warp_max[8];
	#pragma unroll
	for (int off = 16; off > 0; off >>= 1) local_max = fmaxf(local_max, __shfl_xor_sync(0xffffffffu, local_max, off));
	if ((threadIdx.x & 31u) == 0) warp_max[threadIdx.x >> 5] = local_max;
	__syncthreads();
	if (threadIdx.x != 0) return;
	#pragma unroll
	for (int w = 1; w < 8; ++w) local_max = fmaxf(local_max, warp_max[w]);
	// non-negative floats order like their bit patterns
	atomicMax(reinterpret_cast<int*>(&ctl->xmax2), __float_as_int(local_max));
}

// Row-major points: a lane per operand word (two dimensions), 16 or 32 lanes per row, so that reads and
// writes are coalesced; a warp has the words of SPLIT_ROWS (pairs of) rows in flight.  Rows
// [p_begin, p_end) of the planes (both multiples of 32); rows at or behind n are padding.
constexpr uint32_t SPLIT_ROWS = 4;

__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ pts, uint32_t* __restrict__ a_hi,
	uint32_t* __restrict__ a_lo, float* __restrict__ xnorm, float* __restrict__ xlow, uint64_t n, uint64_t p_begin, uint64_t p_end, uint32_t d, uint32_t d_pad, int vec,
	const float* __restrict__ center, Control* __restrict__ ctl, const uint32_t* __restrict__ skip_if)
{
	if (skip_if && *skip_if) return;
	const float scale = tc_scale(ctl->xdev);
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	const uint32_t lanes = d_pad == 16 ? 16u : 32u, word = lane & (lanes - 1u);
	const uint32_t per_warp = SPLIT_ROWS * (32u / lanes);                // 4 or 8 rows
	float local_max = 0.0f;
	for (uint64_t r0 = p_begin + ((uint64_t)blockIdx.x * 8 + warp) * per_warp; r0 < p_end; r0 += (uint64_t)gridDim.x * 8 * per_warp) {
		const uint64_t first = r0 + (lane >= lanes ? SPLIT_ROWS : 0u);
		float norm[SPLIT_ROWS] = {}, rest[SPLIT_ROWS] = {};
		for (uint32_t w = word; w < d_pad; w += lanes) {
			const uint32_t j = 2 * w;
			const float c0 = j < d ? center[j] : 0.0f, c1 = j + 1 < d ? center[j + 1] : 0.0f;
			float x0[SPLIT_ROWS], x1[SPLIT_ROWS];
			#pragma unroll
			for (uint32_t u = 0; u < SPLIT_ROWS; ++u) {
				const uint64_t p = first + u;
				const float* src = pts + (size_t)p * d + j;
				x0[u] = c0; x1[u] = c1;
				if (p < n && vec && j < d) {                                 // rows on 8-byte boundaries, dim even
					const float2 v = *reinterpret_cast<const float2*>(src);
					x0[u] = v.x; x1[u] = v.y;
				} else if (p < n) {
					if (j < d) x0[u] = src[0];
					if (j + 1 < d) x1[u] = src[1];
				}
			}
			#pragma unroll
			for (uint32_t u = 0; u < SPLIT_ROWS; ++u) {
				const float y0 = (x0[u] - c0) * scale, y1 = (x1[u] - c1) * scale;
				uint32_t hi, lo;
				tc_split2(y0, y1, hi, lo, rest[u]);
				const size_t o = (size_t)(first + u) * d_pad + w;
				a_hi[o] = hi;
				a_lo[o] = lo;
				norm[u] = fmaf(y0, y0, fmaf(y1, y1, norm[u]));
			}
		}
		#pragma unroll
		for (uint32_t u = 0; u < SPLIT_ROWS; ++u) {
			float s = norm[u];
			#pragma unroll
			for (uint32_t off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
			const float other = __shfl_xor_sync(0xffffffffu, s, 16);
			if (lanes == 32) s += other;
			if (xlow) {                                  // (rows of 32 lanes, see tc_screen_fits)
				float r = rest[u];
				#pragma unroll
				for (uint32_t off = 16; off > 0; off >>= 1) r += __shfl_xor_sync(0xffffffffu, r, off);
				if (lane == 0) xlow[first + u] = sqrtf(r);
			}
			if (!(s <= TC_NORM2_MAX)) {
				// beyond what the planes hold, or not a number: a zero row whose |x|^2 sends the point to the exact kernel
				s = INFINITY;
				for (uint32_t w = word; w < d_pad; w += lanes) { a_hi[(size_t)(first + u) * d_pad + w] = 0u; a_lo[(size_t)(first + u) * d_pad + w] = 0u; }
				if (word == 0) atomicAdd(&ctl->beyond, 1u);
			} else {
				local_max = fmaxf(local_max, s);
			}
			if (word == 0) xnorm[first + u] = s;
		}
	}
	block_norm_max(local_max, ctl);
}

// Dimension-major points: a lane per point (reads coalesced along the points), 32 dimensions in flight.
// The 64-byte slices of a warp's 32 points pass through shared memory (16-byte pieces, swizzled so that
// neither side meets a bank twice) and leave as whole rows: written straight from the lanes, 16 bytes
// every 64, the stores cost 1.3 ms for 2^21 points of 32 dimensions.
__global__ void __launch_bounds__(256) split_columns_kernel(const float* __restrict__ pts, uint32_t* __restrict__ a_hi,
	uint32_t* __restrict__ a_lo, float* __restrict__ xnorm, float* __restrict__ xlow, uint64_t n, uint64_t p_begin, uint64_t p_end, uint32_t d, uint32_t d_pad,
	const float* __restrict__ center, Control* __restrict__ ctl, const uint32_t* __restrict__ skip_if)
{
	if (skip_if && *skip_if) return;
	__shared__ uint4 s_hi[8][128], s_lo[8][128];
	const float scale = tc_scale(ctl->xdev);
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	float local_max = 0.0f;
	for (uint64_t p0 = p_begin + ((uint64_t)blockIdx.x * 8 + warp) * 32; p0 < p_end; p0 += (uint64_t)gridDim.x * 256) {
		const uint64_t p = p0 + lane;
		uint4* out_hi = reinterpret_cast<uint4*>(a_hi + (size_t)p0 * d_pad);
		uint4* out_lo = reinterpret_cast<uint4*>(a_lo + (size_t)p0 * d_pad);
		const uint32_t pitch = d_pad / 4;           // 16-byte pieces of a row
		float s = 0.0f, rest = 0.0f;
		for (uint32_t w0 = 0; w0 < d_pad; w0 += 16) {
			float x[32];
			#pragma unroll
			for (uint32_t i = 0; i < 32; ++i) {
				const uint32_t j = 2 * w0 + i;
				x[i] = (p < n && j < d) ? pts[(size_t)j * n + p] : 0.0f;
			}
			#pragma unroll
			for (uint32_t i = 0; i < 32; ++i) {
				const uint32_t j = 2 * w0 + i;
				x[i] = (p < n && j < d) ? (x[i] - center[j]) * scale : 0.0f;
				s = fmaf(x[i], x[i], s);
			}
			__syncwarp();                           // the previous slice has been read
			#pragma unroll
			for (uint32_t q = 0; q < 4; ++q) {
				uint4 hi, lo;
				tc_split2(x[8 * q + 0], x[8 * q + 1], hi.x, lo.x, rest);
				tc_split2(x[8 * q + 2], x[8 * q + 3], hi.y, lo.y, rest);
				tc_split2(x[8 * q + 4], x[8 * q + 5], hi.z, lo.z, rest);
				tc_split2(x[8 * q + 6], x[8 * q + 7], hi.w, lo.w, rest);
				const uint32_t e = lane * 4 + (q ^ ((lane >> 1) & 3u));
				s_hi[warp][e] = hi;
				s_lo[warp][e] = lo;
			}
			__syncwarp();
			#pragma unroll
			for (uint32_t r = 0; r < 4; ++r) {
				const uint32_t row = r * 8 + (lane >> 2), q = lane & 3u, e = row * 4 + (q ^ ((row >> 1) & 3u));
				out_hi[(size_t)row * pitch + w0 / 4 + q] = s_hi[warp][e];
				out_lo[(size_t)row * pitch + w0 / 4 + q] = s_lo[warp][e];
			}
		}
		if (!(s <= TC_NORM2_MAX)) s = INFINITY;     // (as above)
		else local_max = fmaxf(local_max, s);
		__syncwarp();
		if (s == INFINITY) {
			for (uint32_t q = 0; q < pitch; ++q) { out_hi[(size_t)lane * pitch + q] = make_uint4(0u, 0u, 0u, 0u); out_lo[(size_t)lane * pitch + q] = make_uint4(0u, 0u, 0u, 0u); }
			atomicAdd(&ctl->beyond, 1u);
		}
		xnorm[p] = s;
		if (xlow) xlow[p] = sqrtf(rest);
	}
	block_norm_max(local_max, ctl);
}

// One block per dimension: mean of that coordinate over at most 8192 evenly spaced points (any vector
// near the points serves), and the sample's largest distance from it.  Bound by the latency of strided
// reads: a thread has all of its samples in flight together (65536 samples in a loop of 256 threads
// took 28-39 us per new batch of a stateless call).
constexpr uint32_t CENTER_THREADS = 1024, CENTER_PER_THREAD = 8;

template<bool SOA>
__global__ void __launch_bounds__(CENTER_THREADS) compute_center_kernel(const float* __restrict__ pts, float* __restrict__ center,
	uint64_t n, uint64_t n_sampled, uint32_t d, Control* __restrict__ ctl, const uint32_t* __restrict__ skip_if)
{
	if (skip_if && *skip_if) return;
	__shared__ float part[4][CENTER_THREADS / 32];
	const uint32_t j = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	// the sample is taken from the first n_sampled points
	constexpr uint32_t MAX_SAMPLES = CENTER_THREADS * CENTER_PER_THREAD;
	const uint32_t samples = n_sampled < MAX_SAMPLES ? (uint32_t)n_sampled : MAX_SAMPLES;
	float x[CENTER_PER_THREAD];
	#pragma unroll
	for (uint32_t r = 0; r < CENTER_PER_THREAD; ++r) {
		const uint32_t t = threadIdx.x + r * CENTER_THREADS;
		const uint64_t i = samples == MAX_SAMPLES ? (uint64_t)t * n_sampled / MAX_SAMPLES : (t < samples ? t : 0u);
		x[r] = SOA ? pts[(size_t)j * n + i] : pts[(size_t)i * d + j];
	}
	// (values that are not finite are left out: one of them must not spoil the centre for all points)
	float sum = 0.0f, cnt = 0.0f, mn = INFINITY, mx = -INFINITY;
	#pragma unroll
	for (uint32_t r = 0; r < CENTER_PER_THREAD; ++r) {
		if (threadIdx.x + r * CENTER_THREADS < samples && fabsf(x[r]) < INFINITY) {
			sum += x[r];
			cnt += 1.0f;
			mn = fminf(mn, x[r]);
			mx = fmaxf(mx, x[r]);
		}
	}
	#pragma unroll
	for (int off = 16; off > 0; off >>= 1) {
		sum += __shfl_xor_sync(0xffffffffu, sum, off);
		cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
		mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
		mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
	}
	if (lane == 0) { part[0][warp] = sum; part[1][warp] = mn; part[2][warp] = mx; part[3][warp] = cnt; }
	__syncthreads();
	if (warp != 0) return;
	sum = part[0][lane]; mn = part[1][lane]; mx = part[2][lane]; cnt = part[3][lane];
	#pragma unroll
	for (int off = 16; off > 0; off >>= 1) {
		sum += __shfl_xor_sync(0xffffffffu, sum, off);
		cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
		mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
		mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
	}
	if (lane == 0) {
		float c = sum / cnt;
		if (!(fabsf(c) < INFINITY)) c = 0.0f;
		center[j] = c;
		const float dev = fmaxf(fmaxf(mx - c, c - mn), 0.0f);
		if (dev < 3.0e38f) atomicMax(reinterpret_cast<int*>(&ctl->xdev), __float_as_int(dev));
	}
}

cudaError_t launch_compute_center(const float* pts, const Shape& s, float* center, Control* ctl, cudaStream_t stream, const uint32_t* skip_if,
	uint64_t n_sampled)
{
	if (n_sampled == 0 || n_sampled > s.n) n_sampled = s.n;
	if (s.soa) compute_center_kernel<true><<<s.dim, CENTER_THREADS, 0, stream>>>(pts, center, s.n, n_sampled, s.dim, ctl, skip_if);
	else compute_center_kernel<false><<<s.dim, CENTER_THREADS, 0, stream>>>(pts, center, s.n, n_sampled, s.dim, ctl, skip_if);
	return cudaGetLastError();
}

cudaError_t launch_split_points(const float* pts, const Shape& s, const TcPoints& tp, const float* center, Control* ctl, cudaStream_t stream,
	const uint32_t* skip_if, uint64_t p_begin, uint64_t p_end)
{
	if (p_end == 0 || p_end > tp.n_pad) p_end = tp.n_pad;
	if ((p_begin & 31u) != 0 || (p_end & 31u) != 0 || p_begin >= p_end) return cudaErrorInvalidValue;
	uint32_t* a_hi = reinterpret_cast<uint32_t*>(tp.a_hi);
	uint32_t* a_lo = reinterpret_cast<uint32_t*>(tp.a_lo);
	const uint64_t rows_pb = s.soa ? 256 : 8 * SPLIT_ROWS * (tp.d_pad == 16 ? 2 : 1);
	const uint32_t grid = (uint32_t)std::min<uint64_t>((p_end - p_begin + rows_pb - 1) / rows_pb, (uint64_t)current_sm_count() * 8);
	const int vec = s.dim % 2 == 0 && (reinterpret_cast<uintptr_t>(pts) & 7u) == 0 ? 1 : 0;
	if (s.soa) split_columns_kernel<<<grid, 256, 0, stream>>>(pts, a_hi, a_lo, tp.xnorm, tp.xlow, s.n, p_begin, p_end, s.dim, tp.d_pad, center, ctl, skip_if);
	else split_rows_kernel<<<grid, 256, 0, stream>>>(pts, a_hi, a_lo, tp.xnorm, tp.xlow, s.n, p_begin, p_end, s.dim, tp.d_pad, vec, center, ctl, skip_if);
	return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------
// the assignment kernel
// ------------------------------------------------------------------------------------------

constexpr uint32_t TC_NA_MAX = 8;        // most point-tile buffers (single resident centroid tile, 16-float rows)

struct TcBars {
	uint64_t a_full[TC_NA_MAX];
	uint64_t a_empty[TC_NA_MAX];
	uint64_t b_full[KL_STAGES];      // TC_NB of them in the resident-points modes
	uint64_t b_empty[KL_STAGES];
	uint64_t aug_full[2];            // K-loop mode: |c|^2 step of a mean tile has landed
	uint64_t aug_empty[2];
	uint64_t acc_full[TC_MA];
	uint64_t acc_empty[TC_MA];
	uint32_t tmem_slot;
	uint32_t abort_flag;
};
static_assert(sizeof(TcBars) <= 256, "barrier block too large");
static_assert(SM_ALLOC <= 227 * 1024, "shared memory budget exceeded");
static_assert(2 * 5 * TC_MA * TC_MTILE * 4 <= SM_BAR_OFF - SM_MERGE_OFF, "merge slots of five words");
static_assert(KL_AUG_OFF + 2 * AUG_BYTES <= SM_AAUG_OFF, "K-loop stages overlap the constant tile");

// What an epilogue warp keeps of a point's row: the two smallest values, or (THREE) the three smallest.
template<bool THREE> struct RowState;
template<> struct RowState<false> {
	RowMin row;
	__device__ __forceinline__ void reset() { row.reset(); }
	__device__ __forceinline__ void take_chunk(const uint32_t (&v)[32], uint32_t key_mult, uint32_t chunk_id) { row.take_chunk(v, key_mult, chunk_id); }
	__device__ __forceinline__ void finish(uint32_t key_base, uint32_t key_mult, uint32_t key_magic, BestThree& st) const { row.finish(key_base, key_mult, key_magic, st.best, st.second, st.best_chunk); }
};
template<> struct RowState<true> {
	BestThree three;
	__device__ __forceinline__ void reset() { three = BestThree(); }
	__device__ __forceinline__ void take_chunk(const uint32_t (&v)[32], uint32_t key_mult, uint32_t chunk_id) { chunk_update3(v, key_mult, chunk_id, three); }
	__device__ __forceinline__ void finish(uint32_t, uint32_t, uint32_t, BestThree& st) const { st = three; }
};

// Combines the partial arg-min results of the CTAs that shared the mean tiles of a point block.
// THREE: the partial results carry the third smallest key, and a near-tie between two means only goes
// to the list of pairs.
// LIST: the points are list[0 .. *list_count) (the partial results lie in the order of the list).
template<bool THREE, bool LIST>
__global__ void __launch_bounds__(256) merge_partials_kernel(const uint32_t* __restrict__ partial, uint64_t partial_stride, uint32_t parts,
	const float* __restrict__ xnorm, uint32_t* __restrict__ asg, uint64_t n, uint32_t k, Control* __restrict__ ctl, int slot,
	uint32_t* __restrict__ flag_list, float margin_coef, float sqrt_dim, uint32_t* __restrict__ pairs, const uint32_t* __restrict__ list)
{
	constexpr uint32_t WORDS = THREE ? 5 : 3;
	const uint64_t total = LIST ? min((uint64_t)ctl->screen_count, n) : n;
	const float x2max = ctl->xmax2, c2max = ctl->mean_max[slot].c2;
	const KeyConsts kc = tc_key_consts(x2max, c2max);
	const float ulp = kc.pow2 * 1.1920929e-07f;
	const float margin_floor = tc_margin_floor(ulp, x2max, c2max, sqrt_dim, tc_scale(ctl->xdev));
	const uint32_t lane = threadIdx.x & 31u;
	const uint64_t n32 = (total + 31) & ~(uint64_t)31;  // whole warps walk the loop together (the append is a warp operation)
	for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n32; p += (uint64_t)gridDim.x * blockDim.x) {
		bool flag = false, two = false;
		uint32_t other = 0, i = 0;
		if (p < total) {
			i = LIST ? list[p] : (uint32_t)p;
			BestThree st;
			for (uint32_t part = 0; part < parts; ++part) {
				const uint32_t* src = partial + (size_t)part * WORDS * partial_stride + p;
				const uint32_t ob = src[0], os = src[partial_stride], oc = src[2 * partial_stride];
				if (THREE) st.merge(ob, os, src[3 * partial_stride], oc, src[4 * partial_stride]);
				else st.merge(ob, os, 0xFFFFFFFFu, oc, 0u);
			}
			const float margin = margin_coef * (xnorm[i] + c2max) + margin_floor;
			flag = finish_point(st.best, st.second, st.best_chunk, kc.key_base, kc.key_mult, kc.key_magic, ulp, margin, k, i, asg);
			if (THREE && flag && st.second != 0xFFFFFFFFu) {
				const uint32_t bm = div_key(st.best - kc.key_base, kc.key_magic);
				const float gap3 = st.third == 0xFFFFFFFFu ? INFINITY : (float)(div_key(st.third - kc.key_base, kc.key_magic) - bm) * ulp;
				other = key_column(st.second, st.second_chunk, kc.key_base, kc.key_mult, kc.key_magic);
				two = margin < INFINITY && gap3 > margin && other < k;
				flag = !two;
			}
		}
		append_flagged(flag, i, ctl, flag_list, n);
		if (THREE) {
			const uint32_t mask = __ballot_sync(0xffffffffu, two);
			if (mask != 0) {
				uint32_t base = 0;
				if (lane == 0) base = atomicAdd(&ctl->pair_count, (uint32_t)__popc(mask));
				base = __shfl_sync(0xffffffffu, base, 0) + (uint32_t)__popc(mask & ((1u << lane) - 1u));
				if (two) {
					if ((uint64_t)base < n) { pairs[base] = i; pairs[n + base] = other; }
					else atomicOr(&ctl->status, (uint32_t)STATUS_LIST_OVERFLOW);
				}
			}
		}
	}
}

// EVEN: mean tiles of 128 or 256 columns, so every warp takes its columns in pairs of 32-column chunks and the
// epilogue runs without the odd-chunk branches.
// THREE (K loop with jsplit > 1): the partial results carry the three smallest keys.
// LIST (K loop): the points are list[0 .. ctl->screen_count), and their rows (of row_words words) are gathered from the planes.
template<bool EVEN, bool THREE, bool LIST>
__global__ void __launch_bounds__(TC_THREADS, 1) assign_tc_kernel(
	const __grid_constant__ CUtensorMap tm_a_hi, const __grid_constant__ CUtensorMap tm_a_lo,
	const __grid_constant__ CUtensorMap tm_b_hi, const __grid_constant__ CUtensorMap tm_b_lo,
	const float* __restrict__ b_aug, const float* __restrict__ xnorm, uint32_t* __restrict__ asg,
	uint64_t n_all, uint32_t n_tiles, uint32_t k, uint32_t k_pad, uint32_t nt_cols, uint32_t kw, uint32_t kchunks, uint32_t ksteps, uint32_t idesc,
	Control* __restrict__ ctl, int slot, uint32_t* __restrict__ flag_list, float margin_coef, float sqrt_dim,
	uint32_t jsplit, uint32_t* __restrict__ partial, uint64_t partial_stride, const uint32_t* __restrict__ list,
	const float* __restrict__ a_hi, const float* __restrict__ a_lo, uint32_t row_words)
{
	const uint64_t n = LIST ? min((uint64_t)ctl->screen_count, n_all) : n_all;
	if (LIST) {
		n_tiles = (uint32_t)((n + TC_MTILE - 1) / TC_MTILE);
		if ((blockIdx.x / jsplit) * TC_MA >= n_tiles) return;     // nothing to do for this block (most of them, with a short list)
	}
	extern __shared__ uint8_t smem_raw[];
	// (an offset from the array, so that the compiler still knows it for shared memory: 32-bit addresses in the epilogue)
	uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
	TcBars* bars = reinterpret_cast<TcBars*>(smem + SM_BAR_OFF);
	uint32_t* mg_state = reinterpret_cast<uint32_t*>(smem + SM_MERGE_OFF);
	volatile uint32_t* abort_flag = &bars->abort_flag;

	const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
	const uint32_t n_ctiles = k_pad / nt_cols;
	const uint32_t nblocks = (n_tiles + TC_MA - 1) / TC_MA;
	// With jsplit > 1, `jsplit` neighbouring CTAs work on the same block of points and share the
	// mean tiles among them (K loop with many mean tiles: the point tiles are re-read for every mean
	// tile, and fewer distinct point blocks in flight keep those re-reads in L2).  Each writes its
	// partial arg-min; merge_partials_kernel combines them.
	const uint32_t jpart = blockIdx.x % jsplit, bid = blockIdx.x / jsplit, nbid = gridDim.x / jsplit;
	const uint32_t jper = (n_ctiles + jsplit - 1) / jsplit;
	const uint32_t j_begin = min(n_ctiles, jpart * jper), j_end = min(n_ctiles, j_begin + jper);
	// Resident-points layout (dim <= 64).  With a single centroid tile (k <= 256) that tile is loaded
	// once and stays, and the space of the second stage holds two more point tiles, so that the
	// next block's points arrive while this block is still being multiplied.
	// Rows are kw = 32 words (128 B) or, for dim <= 32, kw = 16 words (64 B): half-size tiles.
	const bool b_resident = n_ctiles == 1;
	const uint32_t a_plane = TC_MTILE * kw * 4, a_tile = 2 * a_plane;
	const uint32_t b_plane = TC_NT_MAX * kw * 4, b_stage = 2 * b_plane;
	const uint32_t n_bstage = b_resident ? 1u : TC_NB;
	const uint32_t n_abuf = min(TC_NA_MAX, (SM_AAUG_OFF - n_bstage * (b_stage + AUG_BYTES)) / a_tile);
	const uint32_t sm_b_off = n_abuf * a_tile;
	const uint32_t sm_baug_off = sm_b_off + n_bstage * b_stage;

	if (threadIdx.x == 0) {
		for (uint32_t i = 0; i < TC_NA_MAX; ++i) {
			ptx::mbar_init(&bars->a_full[i], 1);
			ptx::mbar_init(&bars->a_empty[i], 1);
		}
		for (uint32_t i = 0; i < TC_MA; ++i) {
			ptx::mbar_init(&bars->acc_full[i], 1);
			ptx::mbar_init(&bars->acc_empty[i], TC_EPI_WARPS / TC_MA);
		}
		for (uint32_t i = 0; i < KL_STAGES; ++i) {
			ptx::mbar_init(&bars->b_full[i], LIST ? 33 : 1);     // (and the lanes that gather)
			ptx::mbar_init(&bars->b_empty[i], 1);
		}
		for (uint32_t i = 0; i < 2; ++i) {
			ptx::mbar_init(&bars->aug_full[i], 1);
			ptx::mbar_init(&bars->aug_empty[i], 1);
		}
		bars->abort_flag = 0;
		ptx::fence_mbar_init();
	}
	if (warp == 1) {
		ptx::tmem_alloc(&bars->tmem_slot, TC_TMEM_COLS);
		ptx::tmem_relinquish();
	}
	const float x2max = ctl->xmax2, c2max = ctl->mean_max[slot].c2;
	const KeyConsts kc = tc_key_consts(x2max, c2max);
	const float pow2 = kc.pow2;
	const uint32_t key_mult = kc.key_mult, key_base = kc.key_base, key_magic = kc.key_magic;
	fill_a_aug(smem + SM_AAUG_OFF, kc, x2max, threadIdx.x, TC_THREADS);
	ptx::fence_proxy_async();
	ptx::tc_fence_before();
	__syncthreads();
	ptx::tc_fence_after();
	const uint32_t tmem_base = bars->tmem_slot;

	if (warp == 0) {
		// ---------------- TMA producer ----------------
		if (LIST) {
			// The whole warp gathers the rows of the listed points with asynchronous 16-byte copies, in the swizzle
			// that the tensor maps give the other operands; the first lane loads the means.  Row piece lane % 4 of the
			// rows lane / 4, + 8, + 16 ..  (Gathering by TMA, four rows of 64 bytes an instruction, took 68
			// clocks each: 18 900 points of 512 dimensions against 4096 means 600 us, a quarter of that now.)
			uint32_t b_count = 0, aug_count = 0;
			bool ok = true;
			const uint32_t sub = lane >> 2, piece = lane & 3u;
			const uint32_t swizzled = sub * (KL_KW * 4) + ((piece ^ ((sub >> 1) & 3u)) * 16);
			auto landed = [&](uint32_t count) {
				// this lane's copies of stage `count` are complete: visible to the tensor cores, then announced
				ptx::fence_proxy_async();
				ptx::mbar_arrive(&bars->b_full[count % KL_STAGES]);
			};
			for (uint32_t blk = bid; blk < nblocks && ok; blk += nbid) {
				const uint32_t tiles = min(TC_MA, n_tiles - blk * TC_MA);
				uint32_t row[TC_MA][TC_MTILE / 8];
				#pragma unroll
				for (uint32_t t = 0; t < TC_MA; ++t)
					#pragma unroll
					for (uint32_t r = 0; r < TC_MTILE / 8; ++r) {
						const uint64_t e = (uint64_t)(blk * TC_MA + t) * TC_MTILE + r * 8 + sub;
						row[t][r] = list[e < n ? e : n - 1];       // (rows behind the last point repeat it)
					}
				for (uint32_t j = j_begin; j < j_end && ok; ++j) {
					const uint32_t as = aug_count & 1u;
					ok = __all_sync(0xffffffffu, wait_or_abort<100>(&bars->aug_empty[as], ((aug_count >> 1) & 1u) ^ 1u, abort_flag)) != 0;
					if (!ok) break;
					if (lane == 0) {
						ptx::mbar_arrive_expect_tx(&bars->aug_full[as], nt_cols * 8 * 4);
						ptx::bulk_g2s(smem + KL_AUG_OFF + as * AUG_BYTES, b_aug + (size_t)j * nt_cols * 8, nt_cols * 8 * 4, &bars->aug_full[as]);
					}
					++aug_count;
					for (uint32_t kc = 0; kc < kchunks; ++kc) {
						const uint32_t s = b_count % KL_STAGES, u = b_count / KL_STAGES;
						ok = __all_sync(0xffffffffu, wait_or_abort<100>(&bars->b_empty[s], (u & 1u) ^ 1u, abort_flag)) != 0;
						if (!ok) break;
						uint8_t* dst = smem + s * KL_STAGE_BYTES;
						if (lane == 0) {
							const int32_t x = (int32_t)(kc * KL_KW);
							ptx::mbar_arrive_expect_tx(&bars->b_full[s], 2 * nt_cols * KL_KW * 4);
							ptx::tma_load_2d(dst + KL_B_OFF, &tm_b_hi, x, (int32_t)(j * nt_cols), &bars->b_full[s]);
							ptx::tma_load_2d(dst + KL_B_OFF + KL_B_PLANE, &tm_b_lo, x, (int32_t)(j * nt_cols), &bars->b_full[s]);
						}
						const uint32_t at = ptx::smem_u32(dst) + swizzled;
						const size_t column = (size_t)kc * KL_KW + piece * 4;
						#pragma unroll
						for (uint32_t t = 0; t < TC_MA; ++t) {
							if (t >= tiles) break;
							#pragma unroll
							for (uint32_t r = 0; r < TC_MTILE / 8; ++r) {
								const size_t o = (size_t)row[t][r] * row_words + column;
								ptx::cp_async16(at + t * KL_A1_OFF + r * (8 * KL_KW * 4), a_hi + o);
								ptx::cp_async16(at + t * KL_A1_OFF + KL_A_PLANE + r * (8 * KL_KW * 4), a_lo + o);
							}
						}
						ptx::cp_async_commit();
						if (b_count != 0) { ptx::cp_async_wait_all_but_one(); landed(b_count - 1); }
						++b_count;
					}
				}
			}
			ptx::cp_async_wait_all();
			if (b_count != 0) landed(b_count - 1);
			// (do not leave while an own copy may still be in flight)
			__syncwarp();
			for (uint32_t back = 0; back < KL_STAGES && back < b_count; ++back) {
				const uint32_t c = b_count - 1 - back;
				ptx::mbar_wait(&bars->b_full[c % KL_STAGES], (c / KL_STAGES) & 1u);
			}
			for (uint32_t back = 0; back < 2 && back < aug_count; ++back) {
				const uint32_t c = aug_count - 1 - back;
				ptx::mbar_wait(&bars->aug_full[c & 1u], (c >> 1) & 1u);
			}
		} else if (lane == 0) {
			ptx::prefetch_tmap(&tm_a_hi); ptx::prefetch_tmap(&tm_a_lo);
			ptx::prefetch_tmap(&tm_b_hi); ptx::prefetch_tmap(&tm_b_lo);
			uint32_t a_use[TC_NA_MAX] = {0, 0, 0, 0, 0, 0, 0, 0};
			uint32_t b_count = 0;
			bool ok = true;
			uint32_t aug_count = 0;
			if (kchunks > 1) {
				// K-loop mode: one (block of two point tiles, mean tile, 32-dimension slice) per stage
				for (uint32_t blk = bid; blk < nblocks && ok; blk += nbid) {
					const uint32_t tiles = min(TC_MA, n_tiles - blk * TC_MA);
					for (uint32_t j = j_begin; j < j_end && ok; ++j) {
						{
							const uint32_t as = aug_count & 1u, au = aug_count >> 1;
							ok = wait_or_abort<400>(&bars->aug_empty[as], (au & 1u) ^ 1u, abort_flag);
							if (!ok) break;
							ptx::mbar_arrive_expect_tx(&bars->aug_full[as], nt_cols * 8 * 4);
							ptx::bulk_g2s(smem + KL_AUG_OFF + as * AUG_BYTES, b_aug + (size_t)j * nt_cols * 8, nt_cols * 8 * 4, &bars->aug_full[as]);
							++aug_count;
						}
						for (uint32_t kc = 0; kc < kchunks; ++kc) {
							const uint32_t s = b_count % KL_STAGES, u = b_count / KL_STAGES;
							ok = wait_or_abort<400>(&bars->b_empty[s], (u & 1u) ^ 1u, abort_flag);
							if (!ok) break;
							uint8_t* dst = smem + s * KL_STAGE_BYTES;
							const int32_t row = (int32_t)(blk * TC_MA * TC_MTILE), x = (int32_t)(kc * KL_KW);
							ptx::mbar_arrive_expect_tx(&bars->b_full[s], tiles * 2 * KL_A_PLANE + 2 * nt_cols * KL_KW * 4);
							ptx::tma_load_2d(dst, &tm_a_hi, x, row, &bars->b_full[s]);
							ptx::tma_load_2d(dst + KL_A_PLANE, &tm_a_lo, x, row, &bars->b_full[s]);
							if (tiles > 1) {
								ptx::tma_load_2d(dst + KL_A1_OFF, &tm_a_hi, x, row + (int32_t)TC_MTILE, &bars->b_full[s]);
								ptx::tma_load_2d(dst + KL_A1_OFF + KL_A_PLANE, &tm_a_lo, x, row + (int32_t)TC_MTILE, &bars->b_full[s]);
							}
							ptx::tma_load_2d(dst + KL_B_OFF, &tm_b_hi, x, (int32_t)(j * nt_cols), &bars->b_full[s]);
							ptx::tma_load_2d(dst + KL_B_OFF + KL_B_PLANE, &tm_b_lo, x, (int32_t)(j * nt_cols), &bars->b_full[s]);
							++b_count;
						}
					}
				}
			} else {
				uint32_t g = 0;                       // running count of point tiles = position in the A ring
				bool b_loaded = false;
				for (uint32_t blk = bid; blk < nblocks && ok; blk += nbid) {
					const uint32_t tiles = min(TC_MA, n_tiles - blk * TC_MA);
					for (uint32_t i = 0; i < tiles && ok; ++i, ++g) {
						const uint32_t buf = g % n_abuf, u = g / n_abuf;
						ok = wait_or_abort<400>(&bars->a_empty[buf], (u & 1u) ^ 1u, abort_flag);
						if (!ok) break;
						uint8_t* dst = smem + SM_A_OFF + buf * a_tile;
						const int32_t row = (int32_t)((blk * TC_MA + i) * TC_MTILE);
						ptx::mbar_arrive_expect_tx(&bars->a_full[buf], a_tile);
						ptx::tma_load_2d(dst, &tm_a_hi, 0, row, &bars->a_full[buf]);
						ptx::tma_load_2d(dst + a_plane, &tm_a_lo, 0, row, &bars->a_full[buf]);
						++a_use[buf];
					}
					for (uint32_t j = j_begin; j < j_end && ok; ++j) {
						if (b_resident && b_loaded) break;
						const uint32_t s = b_count % TC_NB, u = b_count / TC_NB;
						ok = wait_or_abort<400>(&bars->b_empty[s], (u & 1u) ^ 1u, abort_flag);
						if (!ok) break;
						uint8_t* dst = smem + sm_b_off + s * b_stage;
						const uint32_t aug_bytes = nt_cols * 8 * 4;
						ptx::mbar_arrive_expect_tx(&bars->b_full[s], 2 * nt_cols * kw * 4 + aug_bytes);
						ptx::tma_load_2d(dst, &tm_b_hi, 0, (int32_t)(j * nt_cols), &bars->b_full[s]);
						ptx::tma_load_2d(dst + b_plane, &tm_b_lo, 0, (int32_t)(j * nt_cols), &bars->b_full[s]);
						ptx::bulk_g2s(smem + sm_baug_off + s * AUG_BYTES, b_aug + (size_t)j * nt_cols * 8, aug_bytes, &bars->b_full[s]);
						++b_count;
						b_loaded = true;
					}
				}
			}
			// Do not leave while an own copy may still be in flight towards this CTA's shared memory.
			for (uint32_t i = 0; i < TC_NA_MAX; ++i)
				if (a_use[i]) ptx::mbar_wait(&bars->a_full[i], (a_use[i] - 1) & 1u);
			const uint32_t ring = kchunks > 1 ? KL_STAGES : TC_NB;
			for (uint32_t back = 0; back < ring && back < b_count; ++back) {
				const uint32_t c = b_count - 1 - back;
				ptx::mbar_wait(&bars->b_full[c % ring], (c / ring) & 1u);
			}
			for (uint32_t back = 0; back < 2 && back < aug_count; ++back) {
				const uint32_t c = aug_count - 1 - back;
				ptx::mbar_wait(&bars->aug_full[c & 1u], (c >> 1) & 1u);
			}
		}
	} else if (warp == 1) {
		// ---------------- MMA issuer ----------------
		// The whole warp walks the loop (so that the address arithmetic is warp-uniform and stays
		// off the vector ALU, which the epilogue warps of the same scheduler keep busy); one
		// elected lane issues the tensor-core instructions.
		{
			uint32_t acc_use[TC_MA] = {0, 0};
			uint32_t b_count = 0;
			bool ok = true;
			const uint32_t a_aug_lo = desc_lo_aug(ptx::smem_u32(smem + SM_AAUG_OFF));
			const uint32_t desc_hi = kw == 32 ? DESC_HI_SW128 : DESC_HI_SW64;
			if (kchunks > 1) {
				// K-loop mode: both accumulators of the block collect the slices of one mean tile together
				uint32_t aug_count = 0;
				for (uint32_t blk = bid; blk < nblocks && ok; blk += nbid) {
					const uint32_t tiles = min(TC_MA, n_tiles - blk * TC_MA);
					for (uint32_t j = j_begin; j < j_end && ok; ++j) {
						for (uint32_t i = 0; i < tiles && ok; ++i) {
							ok = wait_or_abort<200>(&bars->acc_empty[i], (acc_use[i] & 1u) ^ 1u, abort_flag);
							++acc_use[i];
						}
						if (!ok) break;
						ptx::tc_fence_after();
						for (uint32_t kc = 0; kc < kchunks; ++kc) {
							const uint32_t s = b_count % KL_STAGES, u = b_count / KL_STAGES;
							ok = wait_or_abort<100>(&bars->b_full[s], u & 1u, abort_flag);
							if (!ok) break;
							const bool last = kc == kchunks - 1;
							const uint32_t as = aug_count & 1u;
							if (last) {
								ok = wait_or_abort<100>(&bars->aug_full[as], (aug_count >> 1) & 1u, abort_flag);
								if (!ok) break;
							}
							ptx::tc_fence_after();
							const uint32_t base = ptx::smem_u32(smem + s * KL_STAGE_BYTES);
							const uint64_t b_hi = make_desc_sw64(base + KL_B_OFF), b_lo = make_desc_sw64(base + KL_B_OFF + KL_B_PLANE);
							const uint32_t steps = last ? ksteps : 2u;
							if (ptx::elect_one()) {
								for (uint32_t i = 0; i < tiles; ++i) {
									const uint32_t d_tmem = tmem_base + i * TC_NT_MAX;
									const uint64_t a_hi = make_desc_sw64(base + i * KL_A1_OFF), a_lo = make_desc_sw64(base + i * KL_A1_OFF + KL_A_PLANE);
									#pragma unroll
									for (uint32_t ks = 0; ks < 2; ++ks)
										if (ks < steps) ptx::mma_f16(d_tmem, a_lo + 2 * ks, b_hi + 2 * ks, idesc, (kc | ks) > 0);
									#pragma unroll
									for (uint32_t ks = 0; ks < 2; ++ks)
										if (ks < steps) ptx::mma_f16(d_tmem, a_hi + 2 * ks, b_lo + 2 * ks, idesc, 1);
									#pragma unroll
									for (uint32_t ks = 0; ks < 2; ++ks)
										if (ks < steps) ptx::mma_f16(d_tmem, a_hi + 2 * ks, b_hi + 2 * ks, idesc, 1);
									if (last) {
										ptx::mma_f16(d_tmem, make_desc_aug(ptx::smem_u32(smem + SM_AAUG_OFF)), make_desc_aug(ptx::smem_u32(smem + KL_AUG_OFF + as * AUG_BYTES)), idesc, 1);
										ptx::mma_commit(&bars->acc_full[i]);
									}
								}
								ptx::mma_commit(&bars->b_empty[s]);
								if (last) ptx::mma_commit(&bars->aug_empty[as]);
							}
							__syncwarp();
							++b_count;
						}
						++aug_count;
					}
				}
			} else {
				RingPos ring;                         // of point tiles: the block's first
				bool b_ready = false;
				for (uint32_t blk = bid; blk < nblocks && ok; blk += nbid) {
					const uint32_t tiles = min(TC_MA, n_tiles - blk * TC_MA);
					for (uint32_t j = j_begin; j < j_end && ok; ++j) {
						const uint32_t s = b_resident ? 0u : b_count % TC_NB, u = b_count / TC_NB;
						if (!(b_resident && b_ready)) {
							ok = wait_or_abort<100>(&bars->b_full[s], u & 1u, abort_flag);
							if (!ok) break;
							b_ready = true;
						}
						const uint32_t b_addr = ptx::smem_u32(smem + sm_b_off + s * b_stage);
						const uint32_t b_hi = desc_lo_sw128(b_addr), b_lo = desc_lo_sw128(b_addr + b_plane);
						const uint32_t b_aug_lo = desc_lo_aug(ptx::smem_u32(smem + sm_baug_off + s * AUG_BYTES));
						RingPos tile = ring;
						for (uint32_t i = 0; i < tiles; ++i, tile.next(n_abuf)) {
							const uint32_t buf = tile.slot, ua = tile.phase;
							if (j == j_begin) {
								ok = wait_or_abort<100>(&bars->a_full[buf], ua & 1u, abort_flag);
								if (!ok) break;
							}
							ok = wait_or_abort<200>(&bars->acc_empty[i], (acc_use[i] & 1u) ^ 1u, abort_flag);
							if (!ok) break;
							ptx::tc_fence_after();
							const uint32_t a_addr = ptx::smem_u32(smem + SM_A_OFF + buf * a_tile);
							const uint32_t a_hi = desc_lo_sw128(a_addr), a_lo = desc_lo_sw128(a_addr + a_plane);
							const uint32_t d_tmem = tmem_base + i * TC_NT_MAX;
							if (ptx::elect_one()) {
								switch (ksteps) {
								case 4: issue_products<4>(d_tmem, a_hi, a_lo, b_hi, b_lo, desc_hi, idesc, 0); break;
								case 3: issue_products<3>(d_tmem, a_hi, a_lo, b_hi, b_lo, desc_hi, idesc, 0); break;
								case 2: issue_products<2>(d_tmem, a_hi, a_lo, b_hi, b_lo, desc_hi, idesc, 0); break;
								default: issue_products<1>(d_tmem, a_hi, a_lo, b_hi, b_lo, desc_hi, idesc, 0); break;
								}
								ptx::mma_f16_halves(d_tmem, a_aug_lo, DESC_HI_AUG, b_aug_lo, DESC_HI_AUG, idesc, 1);
								ptx::mma_commit(&bars->acc_full[i]);
								if (j == j_end - 1) ptx::mma_commit(&bars->a_empty[buf]);
							}
							__syncwarp();
							++acc_use[i];
						}
						if (!ok) break;
						if (!b_resident) {
							if (ptx::elect_one()) ptx::mma_commit(&bars->b_empty[s]);
							__syncwarp();
							++b_count;
						}
					}
					for (uint32_t i = 0; i < tiles; ++i) ring.next(n_abuf);
				}
			}
		}
	} else {
		// ---------------- epilogue ----------------
		// Warp (q, half, i): TMEM lane quarter q (the only lanes the warp may read), column half
		// `half` of accumulator i.  The eight warps of one accumulator work while the other
		// accumulator is being multiplied, so on every scheduler two warps read tensor memory while
		// the other two keep the integer pipes busy.  A warp takes its columns two 32-column chunks
		// at a time into registers and hands the accumulator back after its last load.
		// The loops are kept rolled on purpose: unrolled, the arg-min code outgrows the instruction
		// cache and the warps starve on instruction fetch.
		const uint32_t q = warp & 3u;
		const uint32_t part = (warp - 2) >> 2;     // 0..3
		const uint32_t i = part >> 1;              // accumulator = point tile within the block
		const uint32_t half = part & 1u;
		const uint32_t row = q * 32 + lane;
		const float ulp = pow2 * 1.1920929e-07f;   // spacing of the values inside [P, 2P)
		const float margin_floor = tc_margin_floor(ulp, x2max, c2max, sqrt_dim, tc_scale(ctl->xdev));
		const uint32_t chunks_total = nt_cols >> 5;                    // 1..8
		const uint32_t per_half = (chunks_total + 1) / 2;              // 1..4
		const uint32_t first_chunk = half * per_half;
		const uint32_t nchunks = first_chunk >= chunks_total ? 0u : min(per_half, chunks_total - first_chunk);
		const uint32_t bar_id = 1u + i * 4u + q;   // named barrier of the two warps that share these rows
		uint32_t* flag_buf = reinterpret_cast<uint32_t*>(smem + SM_FLAG_OFF) + (warp - 2) * FLAG_BUFFER;
		uint32_t flag_cnt = 0;
		uint32_t acc_use = 0, blk_count = 0;
		bool ok = true;
		for (uint32_t blk = bid; blk < nblocks; blk += nbid, ++blk_count) {
			const uint32_t tiles = min(TC_MA, n_tiles - blk * TC_MA);
			if (i >= tiles) continue;              // odd tail: this accumulator is not used in the last block
			RowState<THREE> rows;
			rows.reset();
			const uint64_t p = (uint64_t)(blk * TC_MA + i) * TC_MTILE + row;
			float xn = 0.0f;                       // |x|^2 of this thread's point, needed at the end of the block
			uint32_t point = (uint32_t)p;
			#pragma unroll 1
			for (uint32_t j = j_begin; j < j_end; ++j) {
				// the whole warp polls (one warp instruction either way, and no divergent region around it)
				if (ok) ok = __all_sync(0xffffffffu, wait_or_abort<100>(&bars->acc_full[i], acc_use & 1u, abort_flag)) != 0;
				++acc_use;
				if (ok && nchunks > 0) {
					ptx::tc_fence_after();
					#pragma unroll 1
					for (uint32_t c = 0; c < nchunks; c += 2) {
						const uint32_t colbase = (first_chunk + c) * 32u;
						const uint32_t taddr = tmem_base + ((q * 32u) << 16) + i * TC_NT_MAX + colbase;
						const uint32_t chunk0 = (j * nt_cols + colbase) >> 5;
						const bool two = EVEN ? true : c + 1 < nchunks;
						uint32_t v0[32], v1[32];
						// the second chunk travels from tensor memory while the first is reduced
						ptx::tmem_ld32(taddr, v0);
						ptx::tmem_ld_wait();
						ptx::tmem_ld32(taddr + 32, v1);            // (a chunk that is not there lies inside the accumulator's columns, and is not used)
						rows.take_chunk(v0, key_mult, chunk0);
						ptx::tmem_ld_wait();
						if (c + 2 >= nchunks) {
							// last load: the tensor cores may fill this accumulator again
							ptx::tc_fence_before();
							__syncwarp();
							if (lane == 0) ptx::mbar_arrive(&bars->acc_empty[i]);
							// fetched behind the hand-back of the block's last accumulator: the arithmetic on
							// the chunks just loaded covers the latency
							if (j == j_end - 1 && half == 0 && p < n) {
								if (LIST) point = list[p];
								xn = xnorm[LIST ? point : p];
							}
						}
						if (two) rows.take_chunk(v1, key_mult, chunk0 + 1);
					}
				} else {
					__syncwarp();
					if (lane == 0) ptx::mbar_arrive(&bars->acc_empty[i]);
				}
			}
			// The upper column half hands its state to the lower one through shared memory.  The slots
			// alternate with the block count, so one barrier per block is enough: a slot is written
			// again only after its reader has passed the barrier of the block in between.
			BestThree st;
			rows.finish(key_base, key_mult, key_magic, st);
			constexpr uint32_t WORDS = THREE ? 5 : 3;
			uint32_t* mg = mg_state + ((blk_count & 1u) * TC_MA + i) * (WORDS * TC_MTILE);
			if (half == 1) {
				mg[row] = st.best; mg[TC_MTILE + row] = st.second; mg[2 * TC_MTILE + row] = st.best_chunk;
				if (THREE) { mg[3 * TC_MTILE + row] = st.third; mg[4 * TC_MTILE + row] = st.second_chunk; }
			}
			asm volatile("bar.sync %0, 64;" :: "r"(bar_id) : "memory");
			bool flag = false;
			if (half == 0 && p < n && ok) {
				const uint32_t ob = mg[row], os = mg[TC_MTILE + row], oc = mg[2 * TC_MTILE + row];
				if (THREE) st.merge(ob, os, mg[3 * TC_MTILE + row], oc, mg[4 * TC_MTILE + row]);
				else st.merge(ob, os, 0xFFFFFFFFu, oc, 0u);
				if (partial != nullptr) {
					// this CTA saw only its share of the mean tiles: the keys go out as they are
					uint32_t* dst = partial + (size_t)jpart * WORDS * partial_stride + p;
					dst[0] = st.best; dst[partial_stride] = st.second; dst[2 * partial_stride] = st.best_chunk;
					if (THREE) { dst[3 * partial_stride] = st.third; dst[4 * partial_stride] = st.second_chunk; }
				} else {
					flag = finish_point(st.best, st.second, st.best_chunk, key_base, key_mult, key_magic, ulp, margin_coef * (xn + c2max) + margin_floor, k, LIST ? point : p, asg);
				}
			}
			if (half == 0 && partial == nullptr) buffered_append(flag, point, flag_buf, flag_cnt, ctl, flag_list, n_all);
		}
		flush_flag_buffer(flag_buf, flag_cnt, ctl, flag_list, n_all);
	}

	ptx::tc_fence_before();
	__syncthreads();
	if (warp == 1) {
		__syncwarp();
		ptx::tc_fence_after();
		ptx::tmem_dealloc(tmem_base, TC_TMEM_COLS);
	}
	if (threadIdx.x == 0 && bars->abort_flag) atomicOr(&ctl->status, (uint32_t)STATUS_WAIT_TIMEOUT);
}

// ------------------------------------------------------------------------------------------
// self-test of the bounded wait
// ------------------------------------------------------------------------------------------

// One thread waits for a barrier phase that nothing will ever complete, with a short limit, and
// reports through the status word exactly as the assignment kernels do when a wait runs out.
__global__ void wait_timeout_selftest_kernel(Control* ctl, uint64_t limit_ns)
{
	__shared__ uint64_t bar;
	if (threadIdx.x == 0) {
		ptx::mbar_init(&bar, 1);
		ptx::fence_mbar_init();
		if (!ptx::mbar_wait(&bar, 0, limit_ns)) atomicOr(&ctl->status, (uint32_t)STATUS_WAIT_TIMEOUT);
	}
}

cudaError_t launch_wait_timeout_selftest(Control* ctl, uint64_t limit_ns, cudaStream_t stream)
{
	wait_timeout_selftest_kernel<<<1, 32, 0, stream>>>(ctl, limit_ns);
	return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------

struct TcPlan {
	CUtensorMap a_hi, a_lo, b_hi, b_lo;
	CUtensorMap bh_hi, bh_lo;       // the means in boxes of 128 rows: one CTA's half of a tile (pair kernel)
	bool pair_ok;                   // the CTA-pair kernel covers this shape
	bool pair_allowed;
	int max_pairs;                  // CTA pairs the device holds at once
	CUtensorMap as_hi, bs_hi, bs_aug;   // screening pass: planes of high parts in slices of 32 words, |c|^2 steps of 128 means
	bool screen_ok;                 // ... can run
	int screen_mode;                // see tc_plan_screen
	int screen_pairs;               // CTA pairs of the screening pass the device holds at once
	Shape s;
	TcPoints tp;
	TcMeans tm;
	uint32_t nt_cols;
	uint32_t idesc;
	int sm_count;
};

static PFN_cuTensorMapEncodeTiled_v12000 get_encode()
{
	static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
	static bool tried = false;
	if (!tried) {
		tried = true;
		void* p = nullptr;
		cudaDriverEntryPointQueryResult qres;
		if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
			qres == cudaDriverEntryPointSuccess)
			fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
	}
	return fn;
}

// [rows][cols] 32-bit words (two fp16 each) row-major, box = box_rows x 32 columns with 128-byte
// swizzle, or, when the rows are only 16 words long or the K loop runs (rows longer than 32 words,
// 16-word slices), box_rows x 16 columns with 64-byte swizzle.
static bool encode_plane(CUtensorMap* out, const float* base, uint64_t rows, uint32_t cols, uint32_t box_rows, uint32_t kw = 0, bool swizzle = true)
{
	if (kw == 0) kw = (cols == 16 || cols > TC_KCHUNK) ? 16u : TC_KCHUNK;
	auto enc = get_encode();
	if (!enc) return false;
	cuuint64_t dims[2] = {cols, rows};
	cuuint64_t strides[1] = {(cuuint64_t)cols * sizeof(float)};
	cuuint32_t box[2] = {kw, box_rows};
	cuuint32_t estr[2] = {1, 1};
	CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
		CU_TENSOR_MAP_INTERLEAVE_NONE, !swizzle ? CU_TENSOR_MAP_SWIZZLE_NONE : (kw == 16 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
		CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	return r == CUDA_SUCCESS;
}

TcPlan* tc_plan_create(const Shape& s, const TcPoints& tp, const TcMeans& tm, int device, const char** err)
{
	static const char* e_sup = "shape not supported by the tensor-core assignment";
	static const char* e_map = "cuTensorMapEncodeTiled failed or is unavailable";
	static const char* e_attr = "cannot set the shared-memory size of the tensor-core kernel";
	if (!assign_tc_supported(s) || tp.d_pad != tm.d_pad || tp.d_pad % 16 != 0) { if (err) *err = e_sup; return nullptr; }
	TcPlan* p = new (std::nothrow) TcPlan();
	if (!p) return nullptr;
	p->s = s; p->tp = tp; p->tm = tm;
	p->nt_cols = tc_nt_cols(s.k);
	// c_format = f32 (bit 4), a/b format = fp16 (0 at bits 7.., 10..), K-major both, N>>3 at bit 17, M>>4 at bit 24
	p->idesc = (1u << 4) | ((p->nt_cols >> 3) << 17) | ((TC_MTILE >> 4) << 24);
	if (cudaDeviceGetAttribute(&p->sm_count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || p->sm_count < 1) { cudaGetLastError(); if (err) *err = e_attr; delete p; return nullptr; }
	if (!encode_plane(&p->a_hi, tp.a_hi, tp.n_pad, tp.d_pad, TC_MTILE) ||
		!encode_plane(&p->a_lo, tp.a_lo, tp.n_pad, tp.d_pad, TC_MTILE) ||
		!encode_plane(&p->b_hi, tm.b_hi, tm.k_pad, tm.d_pad, p->nt_cols) ||
		!encode_plane(&p->b_lo, tm.b_lo, tm.k_pad, tm.d_pad, p->nt_cols)) {
		if (err) *err = e_map;
		delete p;
		return nullptr;
	}
	auto allow = [](auto kern) { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM_ALLOC) == cudaSuccess; };
	if (!allow(assign_tc_kernel<true, false, false>) || !allow(assign_tc_kernel<false, false, false>) || !allow(assign_tc_kernel<true, true, false>) ||
		!allow(assign_tc_kernel<false, true, false>) || !allow(assign_tc_kernel<true, false, true>) || !allow(assign_tc_kernel<true, true, true>)) {
		cudaGetLastError();
		if (err) *err = e_attr;
		delete p;
		return nullptr;
	}
	p->pair_allowed = true;
	p->pair_ok = assign_tc_pair_supported(s.k, tm.k_pad, s.dim, tp.d_pad, p->nt_cols, p->sm_count) &&
		encode_plane(&p->bh_hi, tm.b_hi, tm.k_pad, tm.d_pad, TC_NT_MAX / 2) &&
		encode_plane(&p->bh_lo, tm.b_lo, tm.k_pad, tm.d_pad, TC_NT_MAX / 2);
	p->max_pairs = 0;
	if (p->pair_ok && (assign_tc_pair_prepare(p->sm_count, &p->max_pairs) != cudaSuccess || p->max_pairs < 1)) {
		cudaGetLastError();
		p->pair_ok = false;
	}
	// (a screening pass that cannot be set up is left out: the pass with all three products serves every shape)
	p->screen_mode = 1;
	p->screen_ok = tp.xlow != nullptr && tp.screen_list != nullptr &&
		encode_plane(&p->as_hi, tp.a_hi, tp.n_pad, tp.d_pad, TC_MTILE, TC_KCHUNK) &&
		encode_plane(&p->bs_hi, tm.b_hi, tm.k_pad, tm.d_pad, TC_NT_MAX / 2, TC_KCHUNK) &&
		encode_plane(&p->bs_aug, tm.b_aug, tm.k_pad / 4, 32, TC_NT_MAX / 8, 32, false);
	p->screen_pairs = 0;
	if (p->screen_ok && (assign_tc_screen_prepare(p->sm_count, &p->screen_pairs) != cudaSuccess || p->screen_pairs < 1)) {
		cudaGetLastError();
		p->screen_ok = false;
	}
	return p;
}

void tc_plan_allow_pair(TcPlan* plan, bool allow) { if (plan) plan->pair_allowed = allow; }
void tc_plan_screen(TcPlan* plan, int mode) { if (plan) plan->screen_mode = mode; }
bool tc_plan_uses_pair(const TcPlan* plan) { return plan && plan->pair_ok && plan->pair_allowed; }

// Where CTA pairs can run they serve what they are better at: the fused update sums, a range of the
// points, operand rows of 32 words (dim 33..64: 517 against 648 us for 2^21 points and 1024 means), and three
// or four mean tiles that are not full (iterations with
// 2^21 points, pair / one CTA: k = 900 d = 24 556 / 571, k = 700 d = 32 464 / 469; k = 300, two tiles, 360 / 351).
// With 16-word rows and full tiles the one-CTA kernel is the faster one (k = 512: 227 against 243 us, k = 1024:
// 427 against 440 us, 2^21 points of 32 dimensions).
static bool launch_uses_pair(const TcPlan* p, bool fused, bool ranged)
{
	return tc_plan_uses_pair(p) && (fused || ranged || p->tp.d_pad == TC_KCHUNK || (p->s.k > 2 * TC_NT_MAX && p->s.k < p->tm.k_pad));
}

void tc_plan_destroy(TcPlan* plan) { delete plan; }

// The pair kernel can accumulate the update sums when a point's row can go out as 128-bit vector
// reductions: dim a multiple of 4 and 16-byte aligned accumulators.  The reductions take as long however
// few the means are, while the pass itself gets shorter with them, so up to three mean tiles the fused form pays
// for the launches it saves only, and the sooner the shorter the rows.  Iterations in us, fused / one-CTA pass
// and update apart: four tiles (k = 900) 2^21 points d = 20 537 / 565, d = 32 551 / 579, 2^17 points 81 / 87;
// three tiles (k = 768) 2^21 points d = 24 447 / 443, d = 32 497 / 454, 2^17 points d = 32 77 / 79; two tiles (k = 512)
// 2^17 / 2^18 / 2^19 / 2^21 points d = 20 66 / 71, 86 / 87, 128 / 127, 362 / 340, d = 24 68 / 71, 89 / 87, 136 / 127,
// 390 / 344, d = 32 72 / 71, 97 / 87, 149 / 129, 442 / 351.  (After an upload in chunks the sums of the first
// iteration are hidden behind it, which is why the bound for d = 20 serves for d = 24 as well.)
static bool pair_fuse_pays(const Shape& s)
{
	if (s.k > 3 * TC_NT_MAX) return true;
	if (s.k > 2 * TC_NT_MAX) return s.dim <= 28 || s.n <= 1u << 17;
	return s.n <= (s.dim <= 24 ? 3u << 17 : 1u << 17);
}

bool tc_plan_can_fuse(const TcPlan* p, const FusedAcc& f)
{
	return tc_plan_uses_pair(p) && pair_fuse_pays(p->s) && assign_tc_pair_can_fuse(p->tm.k_pad, p->s.dim, p->tp.d_pad) && f.acc != nullptr && f.counts != nullptr && f.points != nullptr &&
		(reinterpret_cast<uintptr_t>(f.acc) & 15u) == 0 && (f.rep_stride * sizeof(float)) % 16 == 0;
}

// K loop with several mean tiles: pairs of neighbouring CTAs share a point block (see the kernel)
static uint32_t plan_jsplit(const TcPlan* p)
{
	return p->tp.partial != nullptr && p->sm_count >= (int)TC_JSPLIT ? TC_JSPLIT : 1u;
}

bool tc_plan_collects_pairs(const TcPlan* p) { return plan_jsplit(p) > 1 && p->tp.pairs != nullptr; }

void tc_plan_describe(const TcPlan* p, bool fused, uint32_t out[4])
{
	out[1] = p->tm.k_pad / p->nt_cols;
	out[2] = 1;
	if (launch_uses_pair(p, fused, false)) { out[0] = BKM_PLAN_TC_PAIR; return; }
	out[0] = p->tp.d_pad > TC_KCHUNK ? BKM_PLAN_TC_KLOOP : BKM_PLAN_TC_RESIDENT;
	out[2] = plan_jsplit(p);
}

cudaError_t launch_assign_tc(TcPlan* p, uint32_t* asg, Control* ctl, int slot, uint32_t* flag_list,
	float margin_scale, cudaStream_t stream, const FusedAcc* fused, uint64_t p_begin, uint64_t p_end)
{
	if (!p) return cudaErrorInvalidValue;
	if (fused && !tc_plan_can_fuse(p, *fused)) return cudaErrorInvalidValue;
	// a range of the points: CTA pairs only, in whole steps of two point tiles
	const bool ranged = p_begin != 0 || p_end != 0;
	if (ranged && (!tc_plan_uses_pair(p) || p_begin % (2 * TC_MTILE) != 0 || (p_end % (2 * TC_MTILE) != 0 && p_end < p->s.n))) return cudaErrorInvalidValue;
	const uint32_t n_tiles = (uint32_t)(p->tp.n_pad / TC_MTILE);
	const uint32_t nblocks = (n_tiles + TC_MA - 1) / TC_MA;
	const uint32_t grid = std::min<uint32_t>(nblocks, (uint32_t)p->sm_count);
	// error band of the split GEMM form relative to |x|^2 + max|c|^2
	const uint32_t dim_band = p->s.dim <= 16 ? 16u : round_up(p->s.dim, 32);
	const float margin_coef = margin_scale * (48.0f + 0.5f * (float)dim_band) * 1.1920929e-07f;
	const float sqrt_dim = sqrtf((float)p->s.dim);
	// rows of 16 or 32 words stay resident whole; longer rows stream in slices of 16 words
	const bool kloop = p->tp.d_pad > TC_KCHUNK;
	const uint32_t kw = (p->tp.d_pad == 16 || kloop) ? 16u : TC_KCHUNK;
	const uint32_t kchunks = kloop ? p->tp.d_pad / kw : 1u;
	const uint32_t ksteps_last = (p->s.dim - (kchunks - 1) * 2 * kw + 15) / 16;    // K steps (16 dimensions) of the last slice
	const uint32_t idesc = p->idesc;
	if (launch_uses_pair(p, fused != nullptr, ranged))
		return launch_assign_tc_pair(p->a_hi, p->a_lo, p->bh_hi, p->bh_lo, p->tm.b_aug, p->tp.xnorm, asg, p->s.n, n_tiles,
			p->s.k, p->tm.k_pad, p->tp.d_pad, ksteps_last, p->max_pairs, ctl, slot, flag_list, margin_coef, sqrt_dim, stream, fused, p->s.dim,
			ranged ? (uint32_t)(p_begin / (2 * TC_MTILE)) : 0u,
			ranged ? (uint32_t)((std::min<uint64_t>(p_end, p->tp.n_pad) + 2 * TC_MTILE - 1) / (2 * TC_MTILE)) : 0u);
	const uint32_t jsplit = plan_jsplit(p);
	const uint32_t grid_j = jsplit * std::min<uint32_t>(nblocks, (uint32_t)p->sm_count / jsplit);
	const bool even = p->nt_cols % 128 == 0, three = tc_plan_collects_pairs(p);
	const bool screens = p->screen_ok && (p->screen_mode == 2 || (p->screen_mode == 1 && tc_screen_pays(p->s)));
	const uint32_t* list = screens ? p->tp.screen_list : nullptr;
	if (screens) {
		// the high parts alone first; what they leave open goes through the pass with all three products
		const cudaError_t e = launch_assign_tc_screen(p->as_hi, p->bs_hi, p->bs_aug, p->tp, asg, p->s.n, p->s.k, p->tm.k_pad, p->s.dim, p->screen_pairs,
			ctl, slot, margin_coef, margin_scale, sqrt_dim, stream);
		if (e != cudaSuccess) return e;
	}
#define BKM_LAUNCH_TC(LIST) do { \
		/* (a list has mean tiles of 256) */ \
		auto kern = three ? (even || LIST ? assign_tc_kernel<true, true, LIST> : assign_tc_kernel<LIST, true, LIST>) : (even || LIST ? assign_tc_kernel<true, false, LIST> : assign_tc_kernel<LIST, false, LIST>); \
		kern<<<jsplit > 1 ? grid_j : grid, TC_THREADS, SM_ALLOC, stream>>>(p->a_hi, p->a_lo, p->b_hi, p->b_lo, \
			p->tm.b_aug, p->tp.xnorm, asg, p->s.n, n_tiles, p->s.k, p->tm.k_pad, p->nt_cols, kw, kchunks, ksteps_last, idesc, \
			ctl, slot, flag_list, margin_coef, sqrt_dim, jsplit, jsplit > 1 ? p->tp.partial : nullptr, p->tp.n_pad, list, p->tp.a_hi, p->tp.a_lo, p->tp.d_pad); \
		if (jsplit > 1) { \
			const uint32_t mgrid = (uint32_t)std::min<uint64_t>((p->s.n + 255) / 256, (uint64_t)p->sm_count * 8); \
			auto merge = three ? merge_partials_kernel<true, LIST> : merge_partials_kernel<false, LIST>; \
			merge<<<mgrid, 256, 0, stream>>>(p->tp.partial, p->tp.n_pad, jsplit, p->tp.xnorm, asg, p->s.n, p->s.k, ctl, slot, \
				flag_list, margin_coef, sqrt_dim, p->tp.pairs, list); \
		} \
	} while (0)
	if (screens) BKM_LAUNCH_TC(true);
	else BKM_LAUNCH_TC(false);
#undef BKM_LAUNCH_TC
	return cudaGetLastError();
}

} // namespace bkm
