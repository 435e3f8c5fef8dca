// Assignment on CUDA cores.
//
//  * assign_exact_kernel: tiles of points and means, the reference's arithmetic
//    (sequential subtract / multiply / add without fusing, square root, strictly-smaller
//    comparison in ascending index order).  Used for every point by the EXACT variant and
//    for the queued near-ties of the fast passes.  Replaces baseAssignmentKernel
//    (kernels/kernels.cu:182-199 of the reference) and follows serial.hpp:21-35.
//
//  * assign_simt_kernel<D, SOA, P>: small-d fast pass (see the comment above the kernel): the
//    means in shared memory, P points per thread in registers, |c|^2 - 2 x.c on the FMA pipe, arg-min on integer keys, near-ties queued for the exact
//    kernel.  Covers the shape range of cachedFixedAssignmentKernel (kernels/kernels.cu:218-273)
//    and cachedAllMeansAssignmentKernel (:330-374).
#include "kernels.cuh"
#include "ptx.cuh"
#include "keys.cuh"

#include <cmath>
#include <atomic>
#include <type_traits>

namespace bkm {

// ------------------------------------------------------------------------------------------
// exact kernel
// ------------------------------------------------------------------------------------------
//
// The reference's arithmetic for a list of queued points, or for all points (list == null): subtract,
// multiply, add in dimension order with one rounding each, square root, strictly smaller in ascending
// index order.  A block takes 64 points and 128 means at a time, a thread four points and eight means of them; the
// operands lie dimension-major in shared memory, and additions work on two neighbouring means at a time
// (add.rn.f32x2: each half is rounded like the scalar operation), so a dimension costs a thread 64 arithmetic
// instructions and four 128-bit loads.  Lists too short to fill the machine in that way go through tiles of 32
// means, as many blocks to a group of points as there are.  The kernel before (one mean and 4 or 16 points per
// thread, scalar) spent more instructions on loads and barriers than on arithmetic: list of 58 800 points of 50
// dimensions against 1000 means 818 us, now 427 (its 9.0e9 dimension pairs are 176 us of issue slots at 68
// instructions for 32); 51 900 of 200 against 300 1261 -> 553 us; 22 900 of 32 against 512 106 -> 70 us; 44
// points of 512 against 4096 46 -> 43 us.
constexpr int EX_THREADS = 256;
constexpr uint32_t EX_POINTS = 64, EX_DIMS = 32;                       // of a block: points, dimensions per slab
constexpr uint32_t EX_PSTRIDE = 2 * EX_POINTS + 8;                     // floats per dimension: every coordinate twice (the two halves of an operand)
constexpr uint32_t EX_MSTRIDE = 128 + 4;                               // floats per dimension: up to 128 negated means
constexpr uint32_t EX_RESIDENT_DIMS = 2 * EX_DIMS;                     // up to here a block's points stay in shared memory for all means
constexpr uint32_t EX_MAX_BLOCKS = 512;                                // for lists whose groups of points are shared between blocks

// The nearest of the mean tiles [t_begin, t_end), PAIRS * 32 means each, for the block's 64 points: the thread's
// four points (4 ty ..) against its means of every tile, as (distance, index) of the nearest it has seen.
// Strides of both arrays put the 8 dimensions x 4 items that a warp stores at a time (row-major sources: 32-byte pieces of
// four rows) into different banks.
template<bool SOA, bool SOAM, bool RESIDENT, int PAIRS>
__device__ __forceinline__ void exact_scan(const float* __restrict__ pts, const float* __restrict__ means, uint64_t n, uint32_t k, uint32_t d,
	const uint32_t* s_index, float* s_points, float* s_means, uint32_t t_begin, uint32_t t_end, unsigned long long (&key)[4])
{
	static_assert(PAIRS == 1 || PAIRS == 4, "pairs of means per thread");
	constexpr uint32_t TILE = PAIRS * 32;               // means of a tile
	constexpr uint32_t LOADS = TILE * EX_DIMS / EX_THREADS;
	const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, tx = tid & 15u, ty = tid >> 4;
	const uint32_t slabs = (d + EX_DIMS - 1) / EX_DIMS;

	// slab of the points / of a mean tile -> registers; registers -> shared memory
	auto fetch_points = [&](uint32_t j0, float (&r)[8]) {
		#pragma unroll
		for (uint32_t e = 0; e < 8; ++e) {
			const uint32_t j = j0 + (SOA ? e * 4 + (tid >> 6) : (e & 3u) * 8 + (lane >> 2));
			const uint32_t p = SOA ? tid & 63u : (e >> 2) * 32 + warp * 4 + (lane & 3u);
			r[e] = j < d ? pts[at<SOA>((uint64_t)s_index[p], j, n, d)] : 0.0f;
		}
	};
	auto store_points = [&](float* dst, const float (&r)[8]) {
		#pragma unroll
		for (uint32_t e = 0; e < 8; ++e) {
			const uint32_t j = SOA ? e * 4 + (tid >> 6) : (e & 3u) * 8 + (lane >> 2);
			const uint32_t p = SOA ? tid & 63u : (e >> 2) * 32 + warp * 4 + (lane & 3u);
			*reinterpret_cast<float2*>(dst + j * EX_PSTRIDE + 2 * p) = make_float2(r[e], r[e]);
		}
	};
	auto fetch_means = [&](uint32_t m0, uint32_t j0, float (&r)[LOADS]) {
		#pragma unroll
		for (uint32_t e = 0; e < LOADS; ++e) {
			const uint32_t j = j0 + (SOAM ? (e * EX_THREADS + tid) / TILE : (e & 3u) * 8 + (lane >> 2));
			const uint32_t m = m0 + (SOAM ? tid % TILE : (e >> 2) * 32 + warp * 4 + (lane & 3u));
			// (a distance to what lies behind the last mean is infinite, or not a number: it never wins)
			r[e] = m < k ? (j < d ? -means[at<SOAM>(m, j, k, d)] : 0.0f) : -INFINITY;
		}
	};
	auto store_means = [&](float* dst, const float (&r)[LOADS]) {
		#pragma unroll
		for (uint32_t e = 0; e < LOADS; ++e) {
			const uint32_t j = SOAM ? (e * EX_THREADS + tid) / TILE : (e & 3u) * 8 + (lane >> 2);
			const uint32_t m = SOAM ? tid % TILE : (e >> 2) * 32 + warp * 4 + (lane & 3u);
			dst[j * EX_MSTRIDE + m] = r[e];
		}
	};

	float rp[8], rm[LOADS];
	fetch_means(t_begin * TILE, 0, rm);
	if (RESIDENT) {
		for (uint32_t sl = 0; sl < slabs; ++sl) {
			fetch_points(sl * EX_DIMS, rp);
			store_points(s_points + sl * EX_DIMS * EX_PSTRIDE, rp);
		}
	} else {
		fetch_points(0, rp);
	}

	float best[4], best_sum[4];
	uint32_t bidx[4];
	#pragma unroll
	for (int p = 0; p < 4; ++p) { best[p] = best_sum[p] = INFINITY; bidx[p] = 0xffffffffu; }
	uint32_t buf = 0;
	for (uint32_t t = t_begin; t < t_end; ++t) {
		uint64_t sum[4][PAIRS];                         // means 4 tx + 0..3 and 64 + 4 tx + 0..3, or 2 tx + 0..1
		#pragma unroll
		for (int p = 0; p < 4; ++p)
			#pragma unroll
			for (int q = 0; q < PAIRS; ++q) sum[p][q] = 0;
		for (uint32_t sl = 0; sl < slabs; ++sl) {
			float* mslab = s_means + buf * EX_DIMS * EX_MSTRIDE;
			float* pslab = s_points + (RESIDENT ? sl : buf) * EX_DIMS * EX_PSTRIDE;
			store_means(mslab, rm);
			if (!RESIDENT) store_points(pslab, rp);
			// (one barrier per slab: the slab before the previous one has been read by all when this one is written)
			__syncthreads();
			const bool same = sl + 1 < slabs;
			if (same || t + 1 < t_end) {
				fetch_means((same ? t : t + 1) * TILE, same ? (sl + 1) * EX_DIMS : 0u, rm);
				if (!RESIDENT) fetch_points(same ? (sl + 1) * EX_DIMS : 0u, rp);
			}
			const uint32_t jn = min(EX_DIMS, d - sl * EX_DIMS);
			const float* mrow = mslab + (PAIRS == 4 ? 4 : 2) * tx;
			const float* prow = pslab + 8 * ty;
			#pragma unroll 4
			for (uint32_t j = 0; j < jn; ++j) {
				uint64_t mm[PAIRS];
				if (PAIRS == 4) {
					const ulonglong2 m0 = *reinterpret_cast<const ulonglong2*>(mrow + j * EX_MSTRIDE);
					const ulonglong2 m1 = *reinterpret_cast<const ulonglong2*>(mrow + j * EX_MSTRIDE + 64);
					mm[0] = m0.x; mm[PAIRS / 4] = m0.y; mm[PAIRS / 2] = m1.x; mm[PAIRS - 1] = m1.y;
				} else {
					mm[0] = *reinterpret_cast<const unsigned long long*>(mrow + j * EX_MSTRIDE);
				}
				const ulonglong2 p0 = *reinterpret_cast<const ulonglong2*>(prow + j * EX_PSTRIDE);
				const ulonglong2 p1 = *reinterpret_cast<const ulonglong2*>(prow + j * EX_PSTRIDE + 4);
				const uint64_t pp[4] = {p0.x, p0.y, p1.x, p1.y};
				#pragma unroll
				for (int p = 0; p < 4; ++p)
					#pragma unroll
					for (int q = 0; q < PAIRS; ++q) sum[p][q] = ptx::add2(sum[p][q], ptx::square2(ptx::add2(pp[p], mm[q])));
			}
			buf ^= 1u;
		}
		// The reference compares square roots.  The correctly rounded square root never decreases with its
		// argument, so only a sum below the best sum can give a smaller root (equal roots of different sums keep
		// the earlier mean, as the reference's strict comparison does).
		const uint32_t m_first = t * TILE + (PAIRS == 4 ? 4 : 2) * tx;
		#pragma unroll
		for (int p = 0; p < 4; ++p) {
			float v[2 * PAIRS];
			#pragma unroll
			for (int q = 0; q < PAIRS; ++q) {
				uint32_t lo, hi;
				ptx::unpack2(sum[p][q], lo, hi);
				v[2 * q] = __uint_as_float(lo);
				v[2 * q + 1] = __uint_as_float(hi);
			}
			if (m_first == 0 && !(v[0] < INFINITY)) {
				// the first mean is taken whatever its distance; nothing replaces what is not a number
				bidx[p] = 0;
				if (v[0] != v[0]) best[p] = best_sum[p] = 0.0f;
			}
			#pragma unroll
			for (int q = 0; q < 2 * PAIRS; ++q) {
				if (v[q] < best_sum[p]) {
					const float dist = __fsqrt_rn(v[q]);
					if (dist < best[p]) { best[p] = dist; best_sum[p] = v[q]; bidx[p] = m_first + (q < 4 ? q : 60 + q); }
				}
			}
		}
	}
	// distances are >= +0, so their bit patterns order like the values
	#pragma unroll
	for (int p = 0; p < 4; ++p) key[p] = ((unsigned long long)__float_as_uint(best[p]) << 32) | bidx[p];
}

template<bool SOA, bool SOAM, bool RESIDENT>
__global__ void __launch_bounds__(EX_THREADS, 2) assign_exact_kernel(const float* __restrict__ pts,
	const float* __restrict__ means, uint32_t* __restrict__ asg, uint64_t n, uint32_t k, uint32_t d,
	const uint32_t* __restrict__ list, const uint32_t* __restrict__ list_count,
	float* __restrict__ fix_acc, uint32_t* __restrict__ fix_counts,
	unsigned long long* __restrict__ split_keys, uint32_t* __restrict__ split_arrive)
{
	extern __shared__ __align__(16) float sx[];         // points: all dimensions, or two slabs of them; then two slabs of means
	__shared__ uint32_t s_index[EX_POINTS];
	__shared__ uint32_t s_moved[EX_POINTS][2];          // (old, new) cluster of a point that changed, else old == new
	__shared__ uint32_t s_last;                         // this block is the last of its group's blocks to finish
	const uint32_t tid = threadIdx.x, tx = tid & 15u, ty = tid >> 4;
	uint64_t total = n;
	if (list != nullptr) {
		const uint64_t c = *list_count;
		total = c < n ? c : n;
	}
	float* s_means = sx + (RESIDENT ? (d + EX_DIMS - 1) / EX_DIMS : 2u) * EX_DIMS * EX_PSTRIDE;
	const uint64_t groups = (total + EX_POINTS - 1) / EX_POINTS;
	// Few points would leave most of the machine idle while a few blocks walk all means.  The blocks then share
	// the groups: `splits` blocks take one group, each a contiguous range of the means in narrow tiles, and
	// combine their results in global memory; every block has at most one piece of work.
	// Wide or narrow tiles by what the busiest block has to do, a wide one at 2.8 times a narrow one: 43 400 points of 40 dimensions
	// against 10 means 50 us with a wide tile, 37 with a narrow one; 51 900 of 200 against 300 553 / 559 us.
	const bool share = split_keys != nullptr && gridDim.x <= EX_MAX_BLOCKS && groups > 0 && groups < gridDim.x;
	const uint32_t most = share ? gridDim.x / (uint32_t)groups : 1u;
	const uint32_t wide_tiles = (k + 127) / 128, narrow_tiles = (k + 31) / 32;
	const uint32_t wide_splits = min(most, wide_tiles), narrow_splits = min(most, narrow_tiles);
	const bool narrow = 5 * ((narrow_tiles + narrow_splits - 1) / narrow_splits) < 14 * ((wide_tiles + wide_splits - 1) / wide_splits);
	const uint32_t mtiles = narrow ? narrow_tiles : wide_tiles, splits = narrow ? narrow_splits : wide_splits;
	const uint32_t part = blockIdx.x % splits;
	const uint32_t t_begin = part * mtiles / splits, t_end = (part + 1) * mtiles / splits;
	const uint64_t stride = splits > 1 ? groups : gridDim.x;   // (shared groups: one piece of work per block)

	for (uint64_t grp = blockIdx.x / splits; grp < groups; grp += stride) {
		const uint64_t w0 = grp * EX_POINTS;
		const uint32_t np = total - w0 < EX_POINTS ? (uint32_t)(total - w0) : EX_POINTS;
		__syncthreads();                                // the previous group is done with the shared arrays
		if (tid < EX_POINTS) {
			const uint64_t e = tid < np ? w0 + tid : w0;  // unused slots repeat the first point
			s_index[tid] = list ? list[e] : (uint32_t)e;
		}
		__syncthreads();
		unsigned long long key[4], mine = 0;
		if (narrow) exact_scan<SOA, SOAM, RESIDENT, 1>(pts, means, n, k, d, s_index, sx, s_means, t_begin, t_end, key);
		else exact_scan<SOA, SOAM, RESIDENT, 4>(pts, means, n, k, d, s_index, sx, s_means, t_begin, t_end, key);

		// lowest (distance, index) over the sixteen threads of a point
		#pragma unroll
		for (int p = 0; p < 4; ++p) {
			#pragma unroll
			for (int off = 8; off > 0; off >>= 1) {
				const unsigned long long o = __shfl_xor_sync(0xffffffffu, key[p], off);
				key[p] = o < key[p] ? o : key[p];
			}
			if ((uint32_t)p == tx) mine = key[p];
		}
		const uint32_t q = ty * 4 + tx;                 // the point that this thread (tx < 4) reports
		const bool reports = tx < 4 && q < np;
		if (splits > 1) {
			// stored inverted, so that zero means "nothing yet"
			if (reports) atomicMax(&split_keys[w0 + q], ~mine);
			// The block that arrives last for its group finds all partial results in place; it
			// writes the assignment and leaves keys and counter zeroed for the next launch.
			__threadfence();
			__syncthreads();
			if (tid == 0) s_last = atomicAdd(&split_arrive[grp], 1u) == splits - 1 ? 1u : 0u;
			__syncthreads();
			if (s_last == 0) break;
			__threadfence();
			if (reports) mine = ~atomicExch(&split_keys[w0 + q], 0ull);
			if (tid == 0) split_arrive[grp] = 0;
		}
		if (reports) {
			const uint32_t to = (uint32_t)mine, i = s_index[q];
			s_moved[q][0] = fix_acc ? asg[i] : to;
			s_moved[q][1] = to;
			asg[i] = to;
		}
		if (fix_acc) {
			// the fast pass has already added these points to the sums of the clusters it picked
			__syncthreads();
			for (uint32_t p = 0; p < np; ++p) {
				const uint32_t from = s_moved[p][0], to = s_moved[p][1];
				if (from == to) continue;
				// (no previous cluster: the fast pass could not hold the point and has not added it)
				for (uint32_t j = tid; j < d; j += EX_THREADS) {
					const float x = pts[at<SOA>((uint64_t)s_index[p], j, n, d)];
					if (from < k) atomicAdd(&fix_acc[(size_t)from * d + j], -x);
					atomicAdd(&fix_acc[(size_t)to * d + j], x);
				}
				if (tid == 0) { if (from < k) atomicSub(&fix_counts[from], 1u); atomicAdd(&fix_counts[to], 1u); }
			}
		}
	}
}

// Points with exactly two candidate means: a warp per point.  The lanes square the differences of 128
// dimensions to both candidates (coalesced reads), lanes 0 and 1 add them up in dimension order, one
// rounding per operation - two rows of means instead of all of them (a list of 4400 points of 512
// dimensions against 4096 means took 1.5 ms in the list kernel above).
template<bool SOA, bool SOAM>
__global__ void __launch_bounds__(256) assign_exact_pairs_kernel(const float* __restrict__ pts, const float* __restrict__ means,
	uint32_t* __restrict__ asg, uint64_t n, uint32_t k, uint32_t d, const uint32_t* __restrict__ pairs, const uint32_t* __restrict__ pair_count)
{
	__shared__ __align__(16) float squares[8][2][128];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	uint64_t total = *pair_count;
	if (total > n) total = n;
	for (uint64_t w = (uint64_t)blockIdx.x * 8 + warp; w < total; w += (uint64_t)gridDim.x * 8) {
		const uint64_t i = pairs[w];
		const uint32_t c0 = asg[i], c1 = pairs[n + w];
		const uint32_t lo = min(c0, c1), hi = max(c0, c1);
		float sum = 0.0f;
		for (uint32_t j0 = 0; j0 < d; j0 += 128) {
			__syncwarp();
			#pragma unroll
			for (uint32_t r = 0; r < 4; ++r) {
				const uint32_t j = j0 + r * 32 + lane;
				if (j < d) {
					const float x = pts[at<SOA>(i, j, n, d)];
					const float d0 = __fsub_rn(x, means[at<SOAM>(lo, j, k, d)]), d1 = __fsub_rn(x, means[at<SOAM>(hi, j, k, d)]);
					squares[warp][0][r * 32 + lane] = __fmul_rn(d0, d0);
					squares[warp][1][r * 32 + lane] = __fmul_rn(d1, d1);
				}
			}
			__syncwarp();
			if (lane < 2) {
				const uint32_t jn = d - j0 < 128 ? d - j0 : 128;
				const float* sq = squares[warp][lane];
				uint32_t j = 0;
				for (; j + 4 <= jn; j += 4) {
					const float4 v = *reinterpret_cast<const float4*>(sq + j);
					sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, v.x), v.y), v.z), v.w);
				}
				for (; j < jn; ++j) sum = __fadd_rn(sum, sq[j]);
			}
		}
		const float dist = __fsqrt_rn(sum), other = __shfl_down_sync(0xffffffffu, dist, 1);
		if (lane == 0) asg[i] = other < dist ? hi : lo;          // strictly smaller, the lower index first
	}
}

cudaError_t launch_assign_exact_pairs(const float* pts, const float* means, uint32_t* asg, const Shape& s,
	const uint32_t* pairs, const uint32_t* pair_count, int sm_count, cudaStream_t stream)
{
	const uint32_t grid = (uint32_t)sm_count * 8;
	if (s.soa && s.soa_means) assign_exact_pairs_kernel<true, true><<<grid, 256, 0, stream>>>(pts, means, asg, s.n, s.k, s.dim, pairs, pair_count);
	else if (s.soa) assign_exact_pairs_kernel<true, false><<<grid, 256, 0, stream>>>(pts, means, asg, s.n, s.k, s.dim, pairs, pair_count);
	else if (s.soa_means) assign_exact_pairs_kernel<false, true><<<grid, 256, 0, stream>>>(pts, means, asg, s.n, s.k, s.dim, pairs, pair_count);
	else assign_exact_pairs_kernel<false, false><<<grid, 256, 0, stream>>>(pts, means, asg, s.n, s.k, s.dim, pairs, pair_count);
	return cudaGetLastError();
}

// The same arithmetic with all means in shared memory and the lanes of a warp shared out over points:
// for mean sets of a few thousand floats and at most 16 dimensions, where a block per four points
// spends its time in barriers and reductions.  A long list gives every point one thread and fills the
// machine by itself; a short one gives a point 2 to 32 lanes, each of which walks every 2nd to 32nd
// mean.  A thread is bound by the latency of its D dependent additions, so it keeps four sums going at
// a time (encode of 250 000 8-dimensional vectors against 256 means, a few thousand of them queued:
// 31 us with one thread per point and one sum at a time).
constexpr uint32_t LIST_SMALL_MAX_FLOATS = 4096;
constexpr uint32_t LIST_SMALL_MAX_DIM = 16;
constexpr uint32_t LIST_SMALL_SUMS = 4;

// Exact distances of one point to the means sub, sub + lanes, ... in shared memory (rows of RS floats,
// LIST_SMALL_SUMS - 1 rows of infinities behind the last), four at a time.
// The reference compares square roots.  The correctly rounded square root never decreases with its
// argument, so a sum that is not below the best sum cannot give a smaller root: only the few
// candidates that are below it need the root itself (equal roots of different sums keep the earlier
// mean, as the reference's strict comparison does).
template<int D, uint32_t RS>
__device__ __forceinline__ void scan_means(const float* sm, const float (&x)[D], uint32_t k, uint32_t sub, uint32_t lanes,
	float& best, float& best_sum, uint32_t& bidx)
{
	for (uint32_t m0 = sub; m0 < k; m0 += lanes * LIST_SMALL_SUMS) {
		float sum[LIST_SMALL_SUMS];
		#pragma unroll
		for (uint32_t u = 0; u < LIST_SMALL_SUMS; ++u) {
			const float* row = sm + (lanes == 1 ? m0 + u : min(m0 + u * lanes, k - 1u)) * RS;
			float c[D];
			if (D % 4 == 0) {
				#pragma unroll
				for (int q = 0; q < D / 4; ++q) {
					const float4 v = *reinterpret_cast<const float4*>(row + 4 * q);
					c[4 * q] = v.x; c[4 * q + 1] = v.y; c[4 * q + 2] = v.z; c[4 * q + 3] = v.w;
				}
			} else if (D % 2 == 0) {
				#pragma unroll
				for (int q = 0; q < D / 2; ++q) {
					const float2 v = *reinterpret_cast<const float2*>(row + 2 * q);
					c[2 * q] = v.x; c[2 * q + 1] = v.y;
				}
			} else {
				#pragma unroll
				for (int j = 0; j < D; ++j) c[j] = row[j];
			}
			sum[u] = 0.0f;
			#pragma unroll
			for (int j = 0; j < D; ++j) {
				const float diff = __fsub_rn(x[j], c[j]);
				sum[u] = __fadd_rn(sum[u], __fmul_rn(diff, diff));
			}
		}
		// the first mean is taken whatever its distance, as in the sequential scan
		if (m0 == 0) { best_sum = sum[0]; best = __fsqrt_rn(sum[0]); bidx = 0; }
		// (a row of infinities is not below the best, nor is anything below what is not a number; behind the last
		// mean of a lane the very last mean is looked at again)
		if (fminf(fminf(sum[0], sum[1]), fminf(sum[2], sum[3])) < best_sum) {
			#pragma unroll
			for (uint32_t u = 0; u < LIST_SMALL_SUMS; ++u) {
				if (sum[u] < best_sum) {
					const float dist = __fsqrt_rn(sum[u]);
					if (dist < best) { best = dist; best_sum = sum[u]; bidx = min(m0 + u * lanes, k - 1u); }
				}
			}
		}
	}
}

// Lowest (distance, index) over the `lanes` lanes of a point, for the first of them, which has seen mean 0.
__device__ __forceinline__ void lowest_of_lanes(float& best, uint32_t& bidx, uint32_t lanes)
{
	for (uint32_t off = lanes >> 1; off > 0; off >>= 1) {
		const float ob = __shfl_down_sync(0xffffffffu, best, off, lanes);
		const uint32_t oi = __shfl_down_sync(0xffffffffu, bidx, off, lanes);
		if (oi != 0xffffffffu && (ob < best || (ob == best && oi < bidx))) { best = ob; bidx = oi; }
	}
}

// Floats of a mean's row for scan_means, which reads it as vectors of 4, 2 or 1: an odd number of vectors, so
// that lanes on neighbouring means meet different banks.
__host__ __device__ constexpr uint32_t scan_row_floats(uint32_t dim) { return dim % 8 == 0 ? dim + 4 : dim; }

template<int D, bool SOA, bool SOAM>
__global__ void __launch_bounds__(256) assign_exact_list_small_kernel(const float* __restrict__ pts, const float* __restrict__ means,
	uint32_t* __restrict__ asg, uint64_t n, uint32_t k, const uint32_t* __restrict__ list, const uint32_t* __restrict__ list_count)
{
	constexpr uint32_t RS = scan_row_floats(D);
	__shared__ __align__(16) float sm[(LIST_SMALL_MAX_FLOATS / D + LIST_SMALL_SUMS - 1) * RS];
	uint64_t total = *list_count;
	if (total > n) total = n;
	const uint64_t threads = (uint64_t)gridDim.x * blockDim.x;
	// 2^shift lanes per point, as far as about half of the grid is resident at a time (as far as the grid
	// goes: 227 000 points, d = 3, 100 means 34 instead of 29 us; 61 000, d = 8, 256 means 34 instead of 31)
	uint32_t shift = 0;
	while (shift < 5 && (total << (shift + 1)) <= threads / 2 && (2u << shift) * LIST_SMALL_SUMS <= k) ++shift;
	if ((((uint64_t)blockIdx.x * blockDim.x) >> shift) >= total) return;  // the grid is sized for long lists: most blocks of a short one have nothing to do
	for (uint32_t e = threadIdx.x; e < k * D; e += blockDim.x) {
		const uint32_t m = e / D, j = e - m * D;
		sm[m * RS + j] = means[at<SOAM>(m, j, k, D)];
	}
	for (uint32_t e = threadIdx.x; e < (LIST_SMALL_SUMS - 1) * RS; e += blockDim.x) sm[k * RS + e] = INFINITY;
	__syncthreads();
	const uint32_t lanes = 1u << shift, sub = threadIdx.x & (lanes - 1u);
	const uint64_t step = threads >> shift;
	uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> shift, w_warp = ((uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) >> shift;
	// whole warps, as the lanes of a point meet in shuffles, as long as one of the lanes has a point (warps without
	// any that walk the means all the same: 69 instead of 64 us for 1.1 million points, d = 2, 64 means)
	for (; w_warp < total; w += step, w_warp += step) {
		const uint64_t i = list[w < total ? w : 0];
		float x[D];
		#pragma unroll
		for (int j = 0; j < D; ++j) x[j] = pts[at<SOA>(i, j, n, D)];
		float best = INFINITY, best_sum = INFINITY;
		uint32_t bidx = 0xffffffffu;
		// (one lane per point: the stride is a constant and the four rows are one address away from each other)
		if (lanes == 1) scan_means<D, RS>(sm, x, k, 0u, 1u, best, best_sum, bidx);
		else scan_means<D, RS>(sm, x, k, sub, lanes, best, best_sum, bidx);
		lowest_of_lanes(best, bidx, lanes);
		if (sub != 0 || w >= total) continue;
		asg[i] = bidx;
	}
}

template<int D>
static cudaError_t launch_list_small(const float* pts, const float* means, uint32_t* asg, const Shape& s,
	const uint32_t* list, const uint32_t* list_count, int sm_count, cudaStream_t stream)
{
	// a thread's point is a dependent gather behind its list entry: many threads in flight hide that,
	// so a long list gets one or two points per thread rather than a loop
	const uint32_t grid = (uint32_t)sm_count * 16;
	if (s.soa && s.soa_means) assign_exact_list_small_kernel<D, true, true><<<grid, 256, 0, stream>>>(pts, means, asg, s.n, s.k, list, list_count);
	else if (s.soa) assign_exact_list_small_kernel<D, true, false><<<grid, 256, 0, stream>>>(pts, means, asg, s.n, s.k, list, list_count);
	else if (s.soa_means) assign_exact_list_small_kernel<D, false, true><<<grid, 256, 0, stream>>>(pts, means, asg, s.n, s.k, list, list_count);
	else assign_exact_list_small_kernel<D, false, false><<<grid, 256, 0, stream>>>(pts, means, asg, s.n, s.k, list, list_count);
	return cudaGetLastError();
}

size_t list_split_scratch_bytes()
{
	return (size_t)EX_MAX_BLOCKS * EX_POINTS * sizeof(unsigned long long) + (size_t)EX_MAX_BLOCKS * sizeof(uint32_t);
}

// The permission for more than 48 KiB, once per kernel and device: asked for with every launch it cost a call that is bound by the
// host 2 us (5538 x 36 against 3 means, stateless iterations).
template<class KERNEL>
static cudaError_t exact_allow_smem(KERNEL kern)
{
	constexpr size_t most = (size_t)(2 * EX_PSTRIDE + 2 * EX_MSTRIDE) * EX_DIMS * sizeof(float);
	static std::atomic<const void*> allowed[64][8];          // per device: the kernels that have it
	int dev = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e != cudaSuccess) return e;
	const void* self = reinterpret_cast<const void*>(kern);
	for (int i = 0; dev >= 0 && dev < 64 && i < 8; ++i) if (allowed[dev][i].load(std::memory_order_acquire) == self) return cudaSuccess;
	e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
	if (e != cudaSuccess) return e;
	for (int i = 0; dev >= 0 && dev < 64 && i < 8; ++i) {
		const void* none = nullptr;
		if (allowed[dev][i].compare_exchange_strong(none, self) || none == self) break;
	}
	return cudaSuccess;
}

cudaError_t launch_assign_exact(const float* pts, const float* means, uint32_t* asg, const Shape& s,
	const uint32_t* list, const uint32_t* list_count, int sm_count, cudaStream_t stream, const FusedAcc* fix, void* split_scratch)
{
	unsigned long long* split_keys = reinterpret_cast<unsigned long long*>(split_scratch);
	uint32_t* split_arrive = split_scratch ? reinterpret_cast<uint32_t*>(split_keys + (size_t)EX_MAX_BLOCKS * EX_POINTS) : nullptr;
	if (fix != nullptr && list == nullptr) return cudaErrorInvalidValue;
	// (the passes that leave sums to be corrected, `fix`, serve longer rows or settle their near-ties themselves)
	if (list != nullptr && fix == nullptr && s.dim <= LIST_SMALL_MAX_DIM && (uint64_t)s.k * s.dim <= LIST_SMALL_MAX_FLOATS) {
		switch (s.dim) {
		case 1: return launch_list_small<1>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 2: return launch_list_small<2>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 3: return launch_list_small<3>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 4: return launch_list_small<4>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 5: return launch_list_small<5>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 6: return launch_list_small<6>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 7: return launch_list_small<7>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 8: return launch_list_small<8>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 9: return launch_list_small<9>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 10: return launch_list_small<10>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 11: return launch_list_small<11>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 12: return launch_list_small<12>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 13: return launch_list_small<13>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 14: return launch_list_small<14>(pts, means, asg, s, list, list_count, sm_count, stream);
		case 15: return launch_list_small<15>(pts, means, asg, s, list, list_count, sm_count, stream);
		default: return launch_list_small<16>(pts, means, asg, s, list, list_count, sm_count, stream);
		}
	}
	if ((size_t)s.dim * sizeof(float) > 200 * 1024) return cudaErrorInvalidValue;
	// Two blocks per SM are resident; a list's length is known on the device only.
	const uint64_t groups = (s.n + EX_POINTS - 1) / EX_POINTS;
	const uint32_t grid = (uint32_t)std::min<uint64_t>(list ? (uint64_t)sm_count * 2 : groups, (uint64_t)sm_count * 2);
	const uint32_t slabs = (s.dim + EX_DIMS - 1) / EX_DIMS;
	const bool resident = s.dim <= EX_RESIDENT_DIMS;
	const size_t smem = (size_t)((resident ? slabs : 2u) * EX_PSTRIDE + 2 * EX_MSTRIDE) * EX_DIMS * sizeof(float);
#define BKM_LAUNCH_EXACT(SOA, SOAM) do { \
		auto kern = resident ? assign_exact_kernel<SOA, SOAM, true> : assign_exact_kernel<SOA, SOAM, false>; \
		const cudaError_t e = exact_allow_smem(kern); \
		if (e != cudaSuccess) return e; \
		kern<<<grid, EX_THREADS, smem, stream>>>(pts, means, asg, s.n, s.k, s.dim, list, list_count, \
			fix ? fix->acc : nullptr, fix ? fix->counts : nullptr, list ? split_keys : nullptr, split_arrive); \
	} while (0)
	if (s.soa && s.soa_means) BKM_LAUNCH_EXACT(true, true);
	else if (s.soa) BKM_LAUNCH_EXACT(true, false);
	else if (s.soa_means) BKM_LAUNCH_EXACT(false, true);
	else BKM_LAUNCH_EXACT(false, false);
#undef BKM_LAUNCH_EXACT
	return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------
// small-d fast pass
// ------------------------------------------------------------------------------------------
//
// Every thread keeps P points in registers (shifted by the common centre vector) and walks the
// means in chunks of 32.  A mean's row is [ |c|^2 + C, -2c_0 .. -2c_{D-1} ], so a point's value
// |c|^2 - 2 x.c + C costs D fused multiply-adds per mean.  The rows of two neighbouring means are
// interleaved in shared memory, and one instruction does the multiply-add of both (fma.rn.f32x2, the
// point's coordinate in both halves): the pass is bound by instruction issue, and this halves the D
// instructions per mean and point.  The constant C (from the
// largest |x|^2 and |c|^2, see make_key_consts) puts all values into one binade, where their bit
// patterns order like the values.  The values go into minima over two partitions of the means (RowMin):
// about one integer instruction per point and mean where keys with a pass each for the smallest and the
// second smallest took 1.75 and a multiply-add (2^24 points of two dimensions against 64 means: 0.278 ->
// 0.261 ms), and D instead of 2D arithmetic instructions.  The form cancels where the
// difference form does not, so a point whose best and second-best keys are closer than the
// rounding band of the pass (and of the reference's own sum and square root) is queued for the
// exact kernel; the final assignment is the reference's for every point.

//
// The band, in spacings of the values (ulp = P * 2^-23 in the binade [P, 2P), P at least 2.5 times the largest |x|^2 plus the
// largest |c|^2; u = 2^-24), for the difference of two values:
//   D + 1     roundings of the D multiply-adds and of |c|^2 + C, half an ulp each, for two values;
//   1.6       |c|^2 itself: four roundings of at most 0.4 P, for two values;
//   and, with r the distance to the mean in question, relative to what is small for a point near its mean:
//   the centring of both operands, 2 r u (|x| + |c|) for each, |c| <= |x| + r, and the reference's own sum (D + 2) u r^2
//   for each and the collapse of its square root, 4 u r^2: together (2 D + 12) u r^2 + 8 u |x| r.
// A flat band of 4 D + 16 spacings, which covers all of that at any distance, queued 6.3 % of 2^24 points in tight two-dimensional
// clusters, and the list took 60 us; 1.5 % and 24 us now.  The flat band stays where near-ties are few, with more
// dimensions (batches of 250 000 x 8 against 256: 298.8 us with it, 310.3 with the other, whose sums of squares cost registers), and
// in the fused form, which settles its near-ties on the spot (66.3 / 66.8 us per iteration).

constexpr int SIMT_THREADS = 256;
constexpr int SIMT_EVAL_POINTS = 2;  // points that a thread evaluates at a time
constexpr int SIMT_TILE_ROWS = 1024; // means per shared-memory tile (a multiple of the 32-mean chunk)

// Fused update sums (FUSE): every WARP sorts the 32 * P points it has just assigned by cluster, in
// shared memory of its own (counters whose atomic also yields the rank, prefix sum over the counters,
// scatter of the centred coordinates to the sorted position).  A lane then walks P neighbouring
// sorted positions, adds rows while the cluster stays the same and sends one row of reductions when
// it changes (with the centre added back, once per point of the run); the sizes are counted per
// block and sent at the end.  Nothing here waits for another warp, and no separate update pass reads
// the points again.  (Measured alternatives on 2^24 two-dimensional points, 64 clusters, where the
// plain pass takes 0.32 ms and a separate sorted update 0.10 ms: this form 0.43 ms; the same sort per
// block with five block-wide barriers 0.48 ms; match.any groups added by the warp's integer
// reduction 1.53 ms - both instructions are replayed once per distinct cluster in the warp.)
constexpr uint32_t SIMT_FUSE_MAX_K = 1024;

// sum[0..D) + len * cen[0..D) onto the row `dst` of the accumulators, as vector reductions where the row allows
template<int D>
__device__ __forceinline__ void send_row(float* dst, const float (&sum)[D], float len, const float (&cen)[D])
{
	float v[D];
	#pragma unroll
	for (int j = 0; j < D; ++j) v[j] = fmaf(len, cen[j], sum[j]);
	if (D % 4 == 0) {
		#pragma unroll
		for (int q = 0; q < D / 4; ++q)
			asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" :: "l"(dst + 4 * q), "f"(v[4 * q]), "f"(v[4 * q + 1]), "f"(v[4 * q + 2]), "f"(v[4 * q + 3]) : "memory");
	} else if (D % 2 == 0) {
		#pragma unroll
		for (int q = 0; q < D / 2; ++q)
			asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" :: "l"(dst + 2 * q), "f"(v[2 * q]), "f"(v[2 * q + 1]) : "memory");
	} else {
		#pragma unroll
		for (int j = 0; j < D; ++j) atomicAdd(dst + j, v[j]);
	}
}

// The near-ties of a warp, `count` (1 to 32 * P) point indices in `buf`, settled by the reference's arithmetic
// against all means in shared memory (`rows`, see scan_means); every index is replaced by its cluster.  A few
// points get many lanes each, so that the warp is soon done with them; many points get one or two lanes
// each, which costs what the list kernel costs.  (A whole warp per point, one after another, over means in
// global memory made the pass up to 4.2 times as long where many points are near-ties.)
template<int D, bool SOA, uint32_t RS>
__device__ __forceinline__ void settle(const float* __restrict__ pts, uint64_t n, const float* rows, uint32_t k, uint32_t* buf, uint32_t count)
{
	const uint32_t lane = threadIdx.x & 31u;
	uint32_t lanes = 1;
	while (lanes < 32 && 2 * lanes * LIST_SMALL_SUMS <= k && 2 * lanes * count <= 64) lanes *= 2;
	const uint32_t sub = lane & (lanes - 1u), per_round = 32 / lanes;
	for (uint32_t e0 = 0; e0 < count; e0 += per_round) {
		const uint32_t e = e0 + lane / lanes;
		const uint64_t i = buf[e < count ? e : e0];
		__syncwarp();                      // (entry e0 is read by the lanes without a point as well)
		float x[D];
		#pragma unroll
		for (int j = 0; j < D; ++j) x[j] = pts[at<SOA>(i, j, n, D)];
		float best = INFINITY, best_sum = INFINITY;
		uint32_t bidx = 0xffffffffu;
		if (lanes == 1) scan_means<D, RS>(rows, x, k, 0u, 1u, best, best_sum, bidx);
		else scan_means<D, RS>(rows, x, k, sub, lanes, best, best_sum, bidx);
		lowest_of_lanes(best, bidx, lanes);
		if (sub == 0 && e < count) buf[e] = bidx;
	}
}

template<int D, bool SOA, int P, bool FUSE>
__global__ void __launch_bounds__(SIMT_THREADS, 2) assign_simt_kernel(const float* __restrict__ pts,
	const float* __restrict__ cprep, const float* __restrict__ center, uint32_t* __restrict__ asg, uint64_t n, uint32_t rows,
	Control* __restrict__ ctl, int slot, uint32_t* __restrict__ flag_list, float margin_scale, int vec_ok,
	uint32_t k, float* __restrict__ fuse_acc, uint32_t* __restrict__ fuse_counts, const float* __restrict__ means, int soa_means)
{
	constexpr int Q = SIMT_EVAL_POINTS;          // points evaluated at a time
	constexpr bool TIGHT = !FUSE && D <= 4;      // the band follows a point's distance to its mean (see above)
	static_assert(P % Q == 0 && (FUSE || P == Q), "points per thread");
	constexpr int RS = (D + 1 + 3) / 4 * 4;      // floats of a prepared row in global memory
	extern __shared__ __align__(128) float tile[];  // rows of two means interleaved: (D + 1) pairs
	// fused update sums: see above
	__shared__ uint32_t s_hist[FUSE ? SIMT_THREADS / 32 : 1][FUSE ? (SIMT_FUSE_MAX_K + 2) / 2 : 1];   // per warp: points per cluster, 16 bits each
	__shared__ uint32_t s_cnt[FUSE ? SIMT_FUSE_MAX_K : 1];                  // sizes counted by this block
	__shared__ __align__(16) float s_x[FUSE ? SIMT_THREADS * P * D : 1];    // per warp: sorted position -> centred coordinates
	__shared__ __align__(8) uint16_t s_cl[FUSE ? SIMT_THREADS * P : 4];     // per warp: sorted position -> cluster
	float* fuse_acc_rep = fuse_acc;
	if (FUSE) {
		fuse_acc_rep += (blockIdx.x % acc_replicas(k, D)) * acc_replica_stride(k, D);
		for (uint32_t c = threadIdx.x; c < SIMT_FUSE_MAX_K; c += SIMT_THREADS) s_cnt[c] = 0;
	}
	__shared__ uint32_t flag_bufs[SIMT_THREADS / 32][FUSE ? 32 * P : FLAG_BUFFER];  // per warp: near-ties to be settled, or on their way to the list
	uint32_t* flag_buf = flag_bufs[threadIdx.x >> 5];
	uint32_t flag_cnt = 0;

	const uint32_t tid = threadIdx.x;
	const uint32_t ntiles = (rows + SIMT_TILE_ROWS - 1) / SIMT_TILE_ROWS;
	const uint64_t per_block = (uint64_t)SIMT_THREADS * P;
	const uint64_t nblocks = (n + per_block - 1) / per_block;
	const float x2max = ctl->xmax2, c2max = ctl->mean_max[slot].c2;
	const KeyConsts kc = make_key_consts(x2max, c2max);
	const uint32_t key_mult = kc.key_mult, key_base = kc.key_base, key_magic = kc.key_magic;
	// Up to 2^125 the binade of the values and the reference's squared distances (at most 2 * (|x|^2 + |c|^2))
	// are inside the range of 32-bit floats; beyond, or with means that are not finite, the keys mean nothing
	// and every point is settled by the exact arithmetic.
	const float margin_floor = x2max + c2max < 4.2535296e37f ? margin_scale * (float)(TIGHT ? D + 3 : 4 * D + 16) : INFINITY;
	const float value_ulp = kc.pow2 * 1.1920929e-07f, per_value = margin_scale * 0.5f / kc.pow2;
	const float pad_value = kc.pow2 * (2.0f - 1.0f / 32.0f);     // padding rows: above every real value, inside [P, 2P)
	float cen[D];
	#pragma unroll
	for (int j = 0; j < D; ++j) cen[j] = center[j];

	// Brings tile t of the prepared means into shared memory, interleaved by pairs, and adds the offset
	// constant to its |c|^2 column (padding rows, marked by +inf there, get the top of the value band).
	// Fused (a single tile, see assign_simt_can_fuse): beside it the means as they are, for the near-ties, and the
	// rows of infinities that scan_means wants behind them.
	constexpr uint32_t MS = scan_row_floats(D);
	float* s_means = tile + rows * (D + 1);
	auto load_tile = [&](uint32_t t) -> uint32_t {
		uint32_t trows = rows - t * SIMT_TILE_ROWS;
		if (trows > SIMT_TILE_ROWS) trows = SIMT_TILE_ROWS;
		for (uint32_t r = tid; r < trows; r += SIMT_THREADS) {
			const float4* src = reinterpret_cast<const float4*>(cprep + ((size_t)t * SIMT_TILE_ROWS + r) * RS);
			float* dst = tile + (r >> 1) * (2 * (D + 1)) + (r & 1u);
			float v[RS], mean[FUSE ? D : 1];
			#pragma unroll
			for (int q = 0; q < RS / 4; ++q) {
				const float4 w = src[q];
				v[4 * q + 0] = w.x; v[4 * q + 1] = w.y; v[4 * q + 2] = w.z; v[4 * q + 3] = w.w;
			}
			if (FUSE) {
				#pragma unroll
				for (int j = 0; j < D; ++j) if (r < k) mean[j] = means[at_rt(soa_means, r, j, k, D)];
			}
			v[0] = v[0] > 3.0e38f ? pad_value : v[0] + kc.offset_c;
			#pragma unroll
			for (int j = 0; j <= D; ++j) dst[2 * j] = v[j];
			if (FUSE && r < k) {
				#pragma unroll
				for (int j = 0; j < D; ++j) s_means[r * MS + j] = mean[j];
			}
		}
		if (FUSE) for (uint32_t e = tid; e < (LIST_SMALL_SUMS - 1) * MS; e += SIMT_THREADS) s_means[k * MS + e] = INFINITY;
		__syncthreads();
		return trows;
	};

	// Values of the means m .. m + 3 of a chunk (two interleaved pairs, D + 1 128-bit loads) for Q points.
	auto four_means = [&](const float* chunk, int m, const uint64_t (&xx)[Q][D], auto&& put) {
		const float4* rowp = reinterpret_cast<const float4*>(chunk) + (m / 4) * (D + 1);
		float f[4 * (D + 1)];
		#pragma unroll
		for (int q = 0; q <= D; ++q) {
			const float4 w = rowp[q];
			f[4 * q + 0] = w.x; f[4 * q + 1] = w.y; f[4 * q + 2] = w.z; f[4 * q + 3] = w.w;
		}
		#pragma unroll
		for (int h = 0; h < 2; ++h) {
			const float* mean2 = f + h * 2 * (D + 1);
			#pragma unroll
			for (int p = 0; p < Q; ++p) {
				uint64_t val = ptx::pack2(mean2[0], mean2[1]);
				#pragma unroll
				for (int j = 0; j < D; ++j) val = ptx::fma2(xx[p][j], ptx::pack2(mean2[2 * j + 2], mean2[2 * j + 3]), val);
				uint32_t lo, hi;
				ptx::unpack2(val, lo, hi);
				put(p, 2 * h, lo);
				put(p, 2 * h + 1, hi);
			}
		}
	};

	// The points of a block of work, as they lie in memory (slots behind the last point read as the
	// centre).  The next block's points are fetched while the current block is being evaluated.
	float raw[P][D];
	auto load_points = [&](uint64_t blk) {
		const uint64_t base = blk * per_block;
		if (SOA) {
			#pragma unroll
			for (int p = 0; p < P; ++p) {
				const uint64_t i = base + (uint64_t)p * SIMT_THREADS + tid;
				#pragma unroll
				for (int j = 0; j < D; ++j) raw[p][j] = i < n ? pts[(size_t)j * n + i] : cen[j];
			}
		} else {
			const uint64_t i0 = base + (uint64_t)tid * P;
			if ((P * D) % 4 == 0 && vec_ok && i0 + P - 1 < n) {
				// 128-bit loads: the thread's P points are P*D consecutive floats
				const float4* src = reinterpret_cast<const float4*>(pts + (size_t)i0 * D);
				float buf[P * D];
				#pragma unroll
				for (int q = 0; q < (P * D) / 4; ++q) {
					float4 v = src[q];
					buf[4 * q + 0] = v.x; buf[4 * q + 1] = v.y; buf[4 * q + 2] = v.z; buf[4 * q + 3] = v.w;
				}
				#pragma unroll
				for (int p = 0; p < P; ++p)
					#pragma unroll
					for (int j = 0; j < D; ++j) raw[p][j] = buf[p * D + j];
			} else {
				#pragma unroll
				for (int p = 0; p < P; ++p)
					#pragma unroll
					for (int j = 0; j < D; ++j) raw[p][j] = i0 + p < n ? pts[(size_t)(i0 + p) * D + j] : cen[j];
			}
		}
	};
	if (blockIdx.x < nblocks) load_points(blockIdx.x);     // (on their way while the means are brought in)
	uint32_t trows0 = 0;
	if (ntiles == 1) trows0 = load_tile(0);

	for (uint64_t blk = blockIdx.x; blk < nblocks; blk += gridDim.x) {
		float x[P][D];
		uint64_t idx[P];
		const uint64_t base = blk * per_block;
		#pragma unroll
		for (int p = 0; p < P; ++p) {
			idx[p] = SOA ? base + (uint64_t)p * SIMT_THREADS + tid : base + (uint64_t)tid * P + p;
			#pragma unroll
			for (int j = 0; j < D; ++j) x[p][j] = raw[p][j] - cen[j];
		}
		uint32_t near = 0;             // bit p: point p is a near-tie
		#pragma unroll
		for (int p = 0; p < P; ++p) {
			// an infinity or what is not a number in the point: its keys mean nothing
			float zero = 0.0f;
			#pragma unroll
			for (int j = 0; j < D; ++j) zero = fmaf(x[p][j], 0.0f, zero);
			if (zero != 0.0f) near |= 1u << p;
		}
		if (blk + gridDim.x < nblocks) load_points(blk + gridDim.x);

		uint32_t cl[P];
		#pragma unroll
		for (int g = 0; g < P; g += Q) {
			uint64_t xx[Q][D];
			#pragma unroll
			for (int p = 0; p < Q; ++p)
				#pragma unroll
				for (int j = 0; j < D; ++j) xx[p][j] = ptx::pack2(x[g + p][j], x[g + p][j]);

			uint32_t best[Q], second[Q], bchunk[Q];
			// Means 0 .. N - 1 at once, straight to keys: for up to 16 or 32 means that is shorter than minima over two partitions
			// and their ranking (ten iterations of 65 536 x 4 against 16 means, 2 % less).
			auto few_means = [&](auto count) {
				constexpr int N = decltype(count)::value;
				uint32_t v[Q][N];
				#pragma unroll
				for (int m = 0; m < N; m += 4) four_means(tile, m, xx, [&](int p, int u, uint32_t bits) { v[p][m + u] = bits; });
				#pragma unroll
				for (int p = 0; p < Q; ++p) {
					#pragma unroll
					for (int t = 0; t < N; ++t) v[p][t] = v[p][t] * key_mult + (uint32_t)t;
					two_smallest(v[p], best[p], second[p]);
					bchunk[p] = 0;
				}
			};
			if (rows == 32) {
				if (k <= 16) few_means(std::integral_constant<int, 16>());
				else few_means(std::integral_constant<int, 32>());
			} else {
			RowMin row[Q];
			#pragma unroll
			for (int p = 0; p < Q; ++p) row[p].reset();

			for (uint32_t t = 0; t < ntiles; ++t) {
				uint32_t trows = trows0;
				if (ntiles > 1) {
					__syncthreads();   // everyone is done reading the previous tile
					trows = load_tile(t);
				}
				const uint32_t chunk_base = t * (SIMT_TILE_ROWS / 32);
				#pragma unroll 1
				for (uint32_t ch = 0; ch < trows / 32; ++ch) {
					// Columns m .. m + 3 and m + 16 .. m + 19 together: they meet in the same position minima.
					uint32_t group[Q][2];
					#pragma unroll
					for (int p = 0; p < Q; ++p) group[p][0] = group[p][1] = 0xFFFFFFFFu;
					#pragma unroll
					for (int m = 0; m < 16; m += 4) {
						uint32_t v[Q][2][4];
						#pragma unroll
						for (int half = 0; half < 2; ++half)
							four_means(tile + (size_t)ch * 32 * (D + 1), m + half * 16, xx, [&](int p, int u, uint32_t bits) { v[p][half][u] = bits; });
						#pragma unroll
						for (int p = 0; p < Q; ++p) {
							#pragma unroll
							for (int u = 0; u < 4; ++u) row[p].position[m + u] = umin3(row[p].position[m + u], v[p][0][u], v[p][1][u]);
							#pragma unroll
							for (int half = 0; half < 2; ++half)
								group[p][half] = umin3(umin3(group[p][half], v[p][half][0], v[p][half][1]), v[p][half][2], v[p][half][3]);
						}
					}
					#pragma unroll
					for (int p = 0; p < Q; ++p) row[p].take_groups(group[p][0], group[p][1], key_mult, chunk_base + ch);
				}
			}

			#pragma unroll
			for (int p = 0; p < Q; ++p) row[p].finish(key_base, key_mult, key_magic, best[p], second[p], bchunk[p]);
			}

			#pragma unroll
			for (int p = 0; p < Q; ++p) {
				cl[g + p] = k;                 // rows behind the last point sort behind every cluster
				bool flag = false;
				if (idx[g + p] < n) {
					// key - key_base = M * mantissa + column
					const uint32_t bm = div_key(best[p] - key_base, key_magic);
					cl[g + p] = bchunk[p] * 32u + ((best[p] - key_base) - bm * key_mult);
					if (!FUSE) asg[idx[g + p]] = cl[g + p];
					const float gap = second[p] == 0xFFFFFFFFu ? INFINITY : (float)(div_key(second[p] - key_base, key_magic) - bm);
					float margin = margin_floor;
					if (TIGHT) {
						float x2 = 0.0f;
						#pragma unroll
						for (int j = 0; j < D; ++j) x2 = fmaf(x[g + p][j], x[g + p][j], x2);
						// the squared distance to the winner, a little more than that
						const float dist2 = fmaxf(__uint_as_float(__float_as_uint(kc.pow2) + bm) - kc.offset_c + x2, 0.0f) + 32.0f * value_ulp;
						margin += per_value * ((float)(2 * D + 12) * dist2 + 8.0f * sqrtf(x2 * dist2));
					}
					flag = !(gap > margin) || (near >> (g + p) & 1u) != 0;
				}
				if (FUSE) near = flag ? near | 1u << (g + p) : near & ~(1u << (g + p));
				else buffered_append(flag, (uint32_t)idx[g + p], flag_buf, flag_cnt, ctl, flag_list, n);
			}
		}

		if (FUSE) {
			// near-ties are settled on the spot, before the points are added anywhere: no list, no launch
			// for it, and nothing to move from one sum to another
			const uint32_t before = (1u << (tid & 31u)) - 1u;
			uint32_t count = 0;
			#pragma unroll
			for (int p = 0; p < P; ++p) {
				const uint32_t mask = __ballot_sync(0xffffffffu, (near >> p & 1u) != 0);
				if (near >> p & 1u) flag_buf[count + (uint32_t)__popc(mask & before)] = (uint32_t)idx[p];
				count += (uint32_t)__popc(mask);
			}
			if (count != 0) {
				__syncwarp();
				settle<D, SOA, MS>(pts, n, s_means, k, flag_buf, count);
				__syncwarp();
				flag_cnt += count;
				count = 0;
				#pragma unroll
				for (int p = 0; p < P; ++p) {
					const uint32_t mask = __ballot_sync(0xffffffffu, (near >> p & 1u) != 0);
					if (near >> p & 1u) cl[p] = flag_buf[count + (uint32_t)__popc(mask & before)];
					count += (uint32_t)__popc(mask);
				}
			}
			#pragma unroll
			for (int p = 0; p < P; ++p) if (idx[p] < n) asg[idx[p]] = cl[p];
		}

		if (FUSE) {
			// everything below is private to the warp: its 32 * P points, its counters, its sorted rows
			const uint32_t lane = tid & 31u, warp = tid >> 5;
			uint32_t* hist32 = s_hist[warp];
			uint16_t* hist = reinterpret_cast<uint16_t*>(hist32);      // k + 1 counters, two to a word; the start positions later
			uint16_t* w_cl = s_cl + warp * (32 * P);
			float* w_x = s_x + warp * (32 * P * D);
			const uint32_t nb = k + 1;
			__syncwarp();                  // the walk over the previous block's rows is over
			for (uint32_t w = lane; w < (nb + 1) / 2; w += 32) hist32[w] = 0;
			__syncwarp();
			uint32_t rank[P];
			#pragma unroll
			for (int p = 0; p < P; ++p) {
				if (cl[p] > k) cl[p] = k;  // (cannot happen: padding columns never win)
				const uint32_t sh = (cl[p] & 1u) * 16u;
				rank[p] = (atomicAdd(&hist32[cl[p] >> 1], 1u << sh) >> sh) & 0xffffu;   // the count also hands out the place within the cluster
			}
			__syncwarp();
			// exclusive prefix sum over the counters: a run of them per lane, warp scan of the run totals
			const uint32_t per = (nb + 31) / 32, b0 = min(nb, lane * per), b1 = min(nb, b0 + per);
			uint32_t local = 0;
			for (uint32_t b = b0; b < b1; ++b) {
				const uint32_t v = hist[b];
				local += v;
				if (v != 0 && b < k) atomicAdd(&s_cnt[b], v);          // the sizes, sent once at the end of the kernel
			}
			uint32_t incl = local;
			#pragma unroll
			for (uint32_t off = 1; off < 32; off <<= 1) { const uint32_t o = __shfl_up_sync(0xffffffffu, incl, off); if (lane >= off) incl += o; }
			uint32_t run = incl - local;
			for (uint32_t b = b0; b < b1; ++b) {
				const uint32_t v = hist[b];
				hist[b] = (uint16_t)run;
				run += v;
			}
			__syncwarp();
			#pragma unroll
			for (int p = 0; p < P; ++p) {
				const uint32_t pos = hist[cl[p]] + rank[p];
				w_cl[pos] = (uint16_t)cl[p];
				#pragma unroll
				for (int j = 0; j < D; ++j) w_x[pos * D + j] = x[p][j];
			}
			__syncwarp();
			const uint32_t total = hist[k];    // rows of real points
			float sum[D];
			#pragma unroll
			for (int j = 0; j < D; ++j) sum[j] = 0.0f;
			float len = 0.0f;
			uint32_t cur = 0;
			#pragma unroll
			for (int u = 0; u < P; ++u) {
				const uint32_t sp = lane * P + u;
				if (sp < total) {
					const uint32_t c = w_cl[sp];
					if (u == 0) cur = c;
					if (c != cur) {
						send_row<D>(fuse_acc_rep + (size_t)cur * D, sum, len, cen);
						#pragma unroll
						for (int j = 0; j < D; ++j) sum[j] = 0.0f;
						len = 0.0f;
						cur = c;
					}
					#pragma unroll
					for (int j = 0; j < D; ++j) sum[j] += w_x[sp * D + j];
					len += 1.0f;
				}
			}
			if (len > 0.0f) send_row<D>(fuse_acc_rep + (size_t)cur * D, sum, len, cen);
		}
	}
	if (FUSE) {
		__syncthreads();
		uint32_t* cnt = fuse_counts + (blockIdx.x % acc_replicas(k, D)) * acc_replica_stride(k, D);
		for (uint32_t c = tid; c < k; c += SIMT_THREADS) {
			const uint32_t v = s_cnt[c];
			if (v) atomicAdd(&cnt[c], v);
		}
	}
	if (!FUSE) flush_flag_buffer(flag_buf, flag_cnt, ctl, flag_list, n);
	else if ((tid & 31u) == 0 && flag_cnt != 0) atomicAdd(&ctl->flag_count, flag_cnt);      // (for the report only)
}

bool assign_simt_supported(const Shape& s)
{
	return s.dim >= 1 && s.dim <= 8 && s.n < (1ull << 32);
}

bool assign_simt_can_fuse(const Shape& s, const FusedAcc& f)
{
	// one tile of means (so that a block meets its points once), vector reductions need aligned rows
	return assign_simt_supported(s) && s.k <= SIMT_FUSE_MAX_K && simt_rows(s.k) <= (uint32_t)SIMT_TILE_ROWS && f.acc != nullptr && f.counts != nullptr &&
		(reinterpret_cast<uintptr_t>(f.acc) & 15u) == 0 && (f.rep_stride * sizeof(float)) % 16 == 0;
}

template<int D>
static cudaError_t launch_simt_d(const float* pts, const float* means, const float* cprep, const float* center, uint32_t* asg, const Shape& s,
	Control* ctl, int slot, uint32_t* flag_list, float margin_scale, int sm_count, cudaStream_t stream, const FusedAcc* fused)
{
	// The fused sums are sent per warp and run of sorted points, and with few clusters all of them meet on a few
	// rows: where the coordinates fit, a warp sorts 128 points instead of 64 (2^21 points in 5 clusters, per
	// iteration: 81 -> 55 us for d = 1, 80 -> 50 us for d = 2), unless that leaves SMs without a block (20 000
	// points, d = 2: 18 instead of 16 us).
	constexpr int MANY_P = D <= 2 ? 4 : 2;
	const bool many = MANY_P != SIMT_EVAL_POINTS && s.n >= (uint64_t)sm_count * SIMT_THREADS * MANY_P;
	const int points = fused && many ? MANY_P : SIMT_EVAL_POINTS;
	const uint32_t rows = simt_rows(s.k);
	const uint32_t trows = rows < (uint32_t)SIMT_TILE_ROWS ? rows : (uint32_t)SIMT_TILE_ROWS;
	const size_t smem = ((size_t)trows * (D + 1) + (fused ? (size_t)(s.k + LIST_SMALL_SUMS - 1) * scan_row_floats(D) : 0)) * sizeof(float);
	const uint64_t per_block = (uint64_t)SIMT_THREADS * points;
	const uint64_t nblocks = (s.n + per_block - 1) / per_block;
	// persistent grid: a whole number of resident blocks per SM
	int per_sm = 1;
	const int vec_ok = ((reinterpret_cast<uintptr_t>(pts) & 15u) == 0) ? 1 : 0;
#define BKM_LAUNCH_SIMT(SOA, FUSE) do { \
		auto kern = FUSE && many ? assign_simt_kernel<D, SOA, FUSE ? MANY_P : SIMT_EVAL_POINTS, FUSE> : assign_simt_kernel<D, SOA, SIMT_EVAL_POINTS, FUSE>; \
		cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
		if (e != cudaSuccess) return e; \
		e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, SIMT_THREADS, smem); \
		if (e != cudaSuccess) return e; \
		if (per_sm < 1) per_sm = 1; \
		uint32_t grid = (uint32_t)std::min<uint64_t>(nblocks, (uint64_t)sm_count * per_sm); \
		if (grid < 1) grid = 1; \
		kern<<<grid, SIMT_THREADS, smem, stream>>>(pts, cprep, center, asg, s.n, rows, ctl, slot, flag_list, margin_scale, vec_ok, \
			s.k, fused ? fused->acc : nullptr, fused ? fused->counts : nullptr, means, s.soa_means); \
	} while (0)
	if (fused && !assign_simt_can_fuse(s, *fused)) return cudaErrorInvalidValue;
	if (fused) { if (s.soa) BKM_LAUNCH_SIMT(true, true); else BKM_LAUNCH_SIMT(false, true); }
	else { if (s.soa) BKM_LAUNCH_SIMT(true, false); else BKM_LAUNCH_SIMT(false, false); }
#undef BKM_LAUNCH_SIMT
	return cudaGetLastError();
}

cudaError_t launch_assign_simt(const float* pts, const float* means, const SimtMeans& sm, uint32_t* asg, const Shape& s,
	Control* ctl, int slot, uint32_t* flag_list, float margin_scale, int sm_count, cudaStream_t stream, const FusedAcc* fused)
{
	switch (s.dim) {
	case 1: return launch_simt_d<1>(pts, means, sm.rows, sm.center, asg, s, ctl, slot, flag_list, margin_scale, sm_count, stream, fused);
	case 2: return launch_simt_d<2>(pts, means, sm.rows, sm.center, asg, s, ctl, slot, flag_list, margin_scale, sm_count, stream, fused);
	case 3: return launch_simt_d<3>(pts, means, sm.rows, sm.center, asg, s, ctl, slot, flag_list, margin_scale, sm_count, stream, fused);
	case 4: return launch_simt_d<4>(pts, means, sm.rows, sm.center, asg, s, ctl, slot, flag_list, margin_scale, sm_count, stream, fused);
	case 5: return launch_simt_d<5>(pts, means, sm.rows, sm.center, asg, s, ctl, slot, flag_list, margin_scale, sm_count, stream, fused);
	case 6: return launch_simt_d<6>(pts, means, sm.rows, sm.center, asg, s, ctl, slot, flag_list, margin_scale, sm_count, stream, fused);
	case 7: return launch_simt_d<7>(pts, means, sm.rows, sm.center, asg, s, ctl, slot, flag_list, margin_scale, sm_count, stream, fused);
	case 8: return launch_simt_d<8>(pts, means, sm.rows, sm.center, asg, s, ctl, slot, flag_list, margin_scale, sm_count, stream, fused);
	default: return cudaErrorInvalidValue;
	}
}

// max over the points of |x - center|^2 -> ctl->xmax2 (which must start at zero): one pass over
// the points, done once per data set (the key constants of the fast pass need the bound).
template<bool SOA>
__global__ void __launch_bounds__(256) points_norm_max_kernel(const float* __restrict__ pts, const float* __restrict__ center,
	uint64_t n, uint32_t d, Control* __restrict__ ctl, const uint32_t* __restrict__ skip_if)
{
	if (skip_if && *skip_if) return;
	float local = 0.0f;
	for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		float s = 0.0f;
		for (uint32_t j = 0; j < d; ++j) {
			const float v = pts[at<SOA>(i, j, n, d)] - center[j];
			s = fmaf(v, v, s);
		}
		local = fmaxf(local, s);
	}
	#pragma unroll
	for (int off = 16; off > 0; off >>= 1) local = fmaxf(local, __shfl_xor_sync(0xffffffffu, local, off));
	// non-negative floats order like their bit patterns
	if ((threadIdx.x & 31u) == 0) atomicMax(reinterpret_cast<int*>(&ctl->xmax2), __float_as_int(local));
}

cudaError_t launch_points_norm_max(const float* pts, const Shape& s, const float* center, Control* ctl, int sm_count, cudaStream_t stream,
	const uint32_t* skip_if)
{
	const uint32_t grid = (uint32_t)std::min<uint64_t>((s.n + 255) / 256, (uint64_t)sm_count * 8);
	if (s.soa) points_norm_max_kernel<true><<<grid, 256, 0, stream>>>(pts, center, s.n, s.dim, ctl, skip_if);
	else points_norm_max_kernel<false><<<grid, 256, 0, stream>>>(pts, center, s.n, s.dim, ctl, skip_if);
	return cudaGetLastError();
}

} // namespace bkm
