// The fp64 counterpart of the iteration, for the reference executable's --double mode
// (k-means.cpp:313-315, 340-345 of krulis-martin/cuda-kmeans instantiate every algorithm for
// double as well).  The reference's arithmetic in double - sequential subtract / multiply / add in
// dimension order without fusing, correctly rounded square root, strictly-smaller comparison in
// ascending index order (headers/serial.hpp:21-35, headers/metric_policies.hpp:50-64) - so the
// assignment is the serial algorithm's bit for bit for the same means; the sums are accumulated with
// double atomics (order differs from the serial loop: means agree to rounding, ~1e-15 relative).
#include "../../include/bkm.h"
#include "common.cuh"

#include <algorithm>
#include <cmath>

int bkm_internal_fail(int code, const char* fmt, ...);

namespace bkm {

// One warp per point, lanes over the means; the point's coordinates in shared memory.
template<bool SOA, bool SOAM>
__global__ void __launch_bounds__(256) assign_exact_f64_kernel(const double* __restrict__ pts, const double* __restrict__ means,
	uint32_t* __restrict__ asg, uint64_t n, uint32_t k, uint32_t d)
{
	extern __shared__ double sx64[];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
	double* x = sx64 + (size_t)warp * d;
	for (uint64_t i = (uint64_t)blockIdx.x * wpb + warp; i < n; i += (uint64_t)gridDim.x * wpb) {
		__syncwarp();
		for (uint32_t j = lane; j < d; j += 32) x[j] = pts[at<SOA>(i, j, n, d)];
		__syncwarp();
		double best = INFINITY;
		uint32_t bidx = 0xffffffffu;
		for (uint32_t m = lane; m < k; m += 32) {
			double sum = 0.0;
			for (uint32_t j = 0; j < d; ++j) {
				const double diff = __dsub_rn(x[j], means[at<SOAM>(m, j, k, d)]);
				sum = __dadd_rn(sum, __dmul_rn(diff, diff));
			}
			const double dist = __dsqrt_rn(sum);
			if (dist < best || (dist == best && m < bidx)) { best = dist; bidx = m; }
			// what is not a number never wins, but nothing replaces it as the first distance of the sequential scan
			if (m == 0 && dist != dist) { best = 0.0; bidx = 0; }
		}
		// lowest (distance, index) pair over the warp = what the sequential scan keeps
		#pragma unroll
		for (int off = 16; off > 0; off >>= 1) {
			const double ob = __shfl_xor_sync(0xffffffffu, best, off);
			const uint32_t oi = __shfl_xor_sync(0xffffffffu, bidx, off);
			if (ob < best || (ob == best && oi < bidx)) { best = ob; bidx = oi; }
		}
		if (lane == 0) asg[i] = bidx;
	}
}

// Up to 32 dimensions: a THREAD per point, its coordinates in registers, the means in shared memory (a tile
// of them at a time), rows padded with zeros to DP dimensions - a zero difference adds +0 and changes no
// bit.  The square root is taken only of sums below the best sum: the correctly rounded root never decreases
// with its argument, so no other candidate can be strictly smaller (equal roots of different sums keep the
// earlier mean, as the reference's comparison does).  Bound by the fp64 pipe (three operations per
// coordinate) where there are enough points.  Few points give too few threads, each in a chain of dependent
// additions through all means: a point then gets 2 to 32 `lanes`, each of which walks every 2nd to 32nd mean
// (see f64_lanes; iterations with 2000 points,
// d = 2, k = 256: 48 us with one lane, 14 us now; 500 points, d = 32: 107 and 25 us).  The form with a warp per point that serves longer rows
// spends its time on loading the means again for every point.
constexpr uint32_t F64_TILE_DOUBLES = 4096;

template<int DP, bool SOA>
__global__ void __launch_bounds__(256) assign_f64_kernel(const double* __restrict__ pts, const double* __restrict__ means,
	uint32_t* __restrict__ asg, uint64_t n, uint32_t k, uint32_t d, int soa_means, uint32_t lanes)
{
	// a row is an odd number of 16-byte vectors, so that lanes on neighbouring means meet different banks
	constexpr uint32_t RS = (DP / 2) % 2 == 0 ? DP + 2 : DP, TILE = F64_TILE_DOUBLES / RS;
	__shared__ __align__(16) double sm[F64_TILE_DOUBLES];
	const uint32_t sub = threadIdx.x & (lanes - 1u), per_block = 256 / lanes;
	for (uint64_t i0 = (uint64_t)blockIdx.x * per_block; i0 < n; i0 += (uint64_t)gridDim.x * per_block) {
		const uint64_t i = i0 + threadIdx.x / lanes;
		double x[DP];
		#pragma unroll
		for (uint32_t j = 0; j < DP; ++j) x[j] = (i < n && j < d) ? pts[at<SOA>(i, j, n, d)] : 0.0;
		double best = INFINITY, best_sum = INFINITY;
		uint32_t bidx = 0xffffffffu;
		for (uint32_t m0 = 0; m0 < k; m0 += TILE) {
			const uint32_t rows = k - m0 < TILE ? k - m0 : TILE;
			if (k > TILE || i0 == (uint64_t)blockIdx.x * per_block) {          // a single tile stays
				__syncthreads();
				for (uint32_t e = threadIdx.x; e < rows * DP; e += 256) {
					const uint32_t m = e / DP, j = e % DP;
					sm[m * RS + j] = j < d ? means[at_rt(soa_means, m0 + m, j, k, d)] : 0.0;
				}
				__syncthreads();
			}
			for (uint32_t m = sub; m < rows; m += lanes) {
				double sum = 0.0;
				#pragma unroll
				for (uint32_t j = 0; j < DP; j += 2) {
					const double2 c = *reinterpret_cast<const double2*>(&sm[m * RS + j]);
					const double d0 = __dsub_rn(x[j], c.x), d1 = __dsub_rn(x[j + 1], c.y);
					sum = __dadd_rn(sum, __dmul_rn(d0, d0));
					sum = __dadd_rn(sum, __dmul_rn(d1, d1));
				}
				if (m0 + m == 0) {                      // taken whatever its distance, as in the sequential scan
					best_sum = sum;
					best = __dsqrt_rn(sum);
					bidx = 0;
				} else if (sum < best_sum) {
					const double dist = __dsqrt_rn(sum);
					if (dist < best) { best = dist; best_sum = sum; bidx = m0 + m; }
				}
			}
		}
		// lowest (distance, index) over the lanes of the point, for the first of them, which has seen mean 0
		for (uint32_t off = lanes >> 1; off > 0; off >>= 1) {
			const double ob = __shfl_down_sync(0xffffffffu, best, off, lanes);
			const uint32_t oi = __shfl_down_sync(0xffffffffu, bidx, off, lanes);
			if (oi != 0xffffffffu && (ob < best || (ob == best && oi < bidx))) { best = ob; bidx = oi; }
		}
		if (sub == 0 && i < n) asg[i] = bidx;
	}
}

// Lanes per point: as many as fill the machine with 1024 threads per SM, and at least two means for each.
static uint32_t f64_lanes(uint64_t n, uint32_t k, int sms)
{
	uint32_t lanes = 1;
	while (lanes < 32 && 4 * lanes <= k && n * lanes * 2 <= (uint64_t)sms * 1024) lanes *= 2;
	return lanes;
}

// sums[c][:] += x_i, sizes[c] += 1 (row-major sums, zero on entry); one thread per coordinate.  The
// accumulators exist in `replicas` copies (16, or 1 when they are large) that the blocks share out, so
// that fewer atomics wait for one another on a line.
constexpr uint32_t F64_REPLICAS = 16;

template<bool SOA>
__global__ void __launch_bounds__(256) update_f64_kernel(const double* __restrict__ pts, const uint32_t* __restrict__ asg,
	double* __restrict__ sums, uint32_t* __restrict__ sizes, uint64_t n, uint32_t k, uint32_t d, uint32_t replicas)
{
	sums += (size_t)(blockIdx.x % replicas) * k * d;
	sizes += (size_t)(blockIdx.x % replicas) * k;
	const uint64_t total = n * d;
	for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (uint64_t)gridDim.x * blockDim.x) {
		// walk the points array in memory order
		const uint64_t i = SOA ? e % n : e / d;
		const uint32_t j = (uint32_t)(SOA ? e / n : e % d);
		const uint32_t c = asg[i];
		if (c >= k) continue;
		atomicAdd(&sums[(size_t)c * d + j], pts[e]);
		if (j == 0) atomicAdd(&sizes[c], 1u);
	}
}

// Adds the copies up, divides (an empty cluster gets zeros) and clears what it has read.
__global__ void __launch_bounds__(256) divide_f64_kernel(double* __restrict__ sums, uint32_t* __restrict__ sizes, double* __restrict__ means,
	uint32_t k, uint32_t d, int soa_means, uint32_t replicas)
{
	// one warp per cluster
	const uint32_t lane = threadIdx.x & 31u;
	for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < k; c += (gridDim.x * blockDim.x) >> 5) {
		uint32_t count = lane < replicas ? sizes[(size_t)lane * k + c] : 0u;
		count = __reduce_add_sync(0xffffffffu, count);
		if (lane < replicas) sizes[(size_t)lane * k + c] = 0u;
		for (uint32_t j = lane; j < d; j += 32) {
			// all copies on their way together, cleared only after that (one after another: 14 us for 256 x 2)
			double part[F64_REPLICAS], sum = 0.0;
			double* src = sums + (size_t)c * d + j;
			#pragma unroll
			for (uint32_t r = 0; r < F64_REPLICAS; ++r) part[r] = r < replicas ? src[(size_t)r * k * d] : 0.0;
			#pragma unroll
			for (uint32_t r = 0; r < F64_REPLICAS; ++r) {
				sum += part[r];
				if (r < replicas) src[(size_t)r * k * d] = 0.0;
			}
			means[at_rt(soa_means, c, j, k, d)] = count ? __ddiv_rn(sum, (double)count) : 0.0;
		}
	}
}

} // namespace bkm

#define F64_TRY(expr) do { cudaError_t e_ = (expr); if (e_ != cudaSuccess) { rc = bkm_internal_fail(BKM_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e_)); goto done; } } while (0)

extern "C" int bkm_kmeans_host_f64(const double* host_points, double* means, uint32_t* assignment,
	uint64_t n, uint32_t k, uint32_t dim, uint32_t iters, int layout, int layout_means, int device)
{
	if (!host_points || !means || !assignment) return bkm_internal_fail(BKM_ERR_INVALID, "null argument");
	if (n == 0 || k == 0 || dim == 0 || iters == 0) return bkm_internal_fail(BKM_ERR_INVALID, "n, k, dim and iters must be positive");
	if (n >= (1ull << 32)) return bkm_internal_fail(BKM_ERR_UNSUPPORTED, "at most 2^32-1 points");
	if ((layout != BKM_LAYOUT_AOS && layout != BKM_LAYOUT_SOA) || (layout_means != BKM_LAYOUT_AOS && layout_means != BKM_LAYOUT_SOA))
		return bkm_internal_fail(BKM_ERR_INVALID, "unknown layout code");
	if ((size_t)dim * sizeof(double) * 8 > 96 * 1024) return bkm_internal_fail(BKM_ERR_UNSUPPORTED, "dim too large for the fp64 path (%u)", dim);
	int rc = BKM_OK, sms = 0;
	char* mem = nullptr;
	const size_t kd = (size_t)k * dim, nd = (size_t)n * dim;
	const bool soa = layout == BKM_LAYOUT_SOA;
	const int soam = layout_means == BKM_LAYOUT_SOA;
	const uint32_t replicas = kd <= 65536 ? bkm::F64_REPLICAS : 1u;
	// one allocation: points, two sets of means, accumulator copies (sums, sizes), assignment
	auto up = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
	const size_t off_means = up(nd * sizeof(double)), off_sums = off_means + 2 * up(kd * sizeof(double));
	const size_t off_sizes = off_sums + up(replicas * kd * sizeof(double)), off_asg = off_sizes + up(replicas * (size_t)k * sizeof(uint32_t));
	{
		F64_TRY(cudaSetDevice(device));
		F64_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
		F64_TRY(cudaMalloc(&mem, off_asg + n * sizeof(uint32_t)));
		double* d_pts = reinterpret_cast<double*>(mem);
		double* d_means[2] = {reinterpret_cast<double*>(mem + off_means), reinterpret_cast<double*>(mem + off_means + up(kd * sizeof(double)))};
		double* d_sums = reinterpret_cast<double*>(mem + off_sums);
		uint32_t* d_sizes = reinterpret_cast<uint32_t*>(mem + off_sizes);
		uint32_t* d_asg = reinterpret_cast<uint32_t*>(mem + off_asg);
		F64_TRY(cudaMemcpy(d_pts, host_points, nd * sizeof(double), cudaMemcpyHostToDevice));
		F64_TRY(cudaMemcpy(d_means[0], means, kd * sizeof(double), cudaMemcpyHostToDevice));
		F64_TRY(cudaMemsetAsync(d_sums, 0, off_asg - off_sums));
		const size_t smem = (size_t)8 * dim * sizeof(double);
		const uint32_t grid_a = (uint32_t)std::min<uint64_t>((n + 7) / 8, (uint64_t)sms * 16);
		const uint32_t lanes = bkm::f64_lanes(n, k, sms);
		const uint32_t grid_t = (uint32_t)std::min<uint64_t>((n * lanes + 255) / 256, (uint64_t)sms * 16);
		const uint32_t grid_u = (uint32_t)std::min<uint64_t>((nd + 255) / 256, (uint64_t)sms * 16);
		const uint32_t grid_d = (uint32_t)std::min<uint64_t>(((uint64_t)k + 7) / 8, (uint64_t)sms * 8);
		int cur = 0;
		for (uint32_t it = 0; it < iters; ++it) {
			const int next = cur ^ 1;
#define F64_ASSIGN(DP) do { \
				if (soa) bkm::assign_f64_kernel<DP, true><<<grid_t, 256>>>(d_pts, d_means[cur], d_asg, n, k, dim, soam, lanes); \
				else bkm::assign_f64_kernel<DP, false><<<grid_t, 256>>>(d_pts, d_means[cur], d_asg, n, k, dim, soam, lanes); \
			} while (0)
#define F64_ASSIGN_LONG(SOA, SOAM) do { \
				auto ka = bkm::assign_exact_f64_kernel<SOA, SOAM>; \
				if (smem > 48 * 1024) F64_TRY(cudaFuncSetAttribute(ka, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
				ka<<<grid_a, 256, smem>>>(d_pts, d_means[cur], d_asg, n, k, dim); \
			} while (0)
			if (dim <= 2) F64_ASSIGN(2);
			else if (dim <= 4) F64_ASSIGN(4);
			else if (dim <= 8) F64_ASSIGN(8);
			else if (dim <= 16) F64_ASSIGN(16);
			else if (dim <= 32) F64_ASSIGN(32);
			else if (soa && soam) F64_ASSIGN_LONG(true, true);
			else if (soa) F64_ASSIGN_LONG(true, false);
			else if (soam) F64_ASSIGN_LONG(false, true);
			else F64_ASSIGN_LONG(false, false);
#undef F64_ASSIGN
#undef F64_ASSIGN_LONG
			if (soa) bkm::update_f64_kernel<true><<<grid_u, 256>>>(d_pts, d_asg, d_sums, d_sizes, n, k, dim, replicas);
			else bkm::update_f64_kernel<false><<<grid_u, 256>>>(d_pts, d_asg, d_sums, d_sizes, n, k, dim, replicas);
			bkm::divide_f64_kernel<<<grid_d, 256>>>(d_sums, d_sizes, d_means[next], k, dim, soam, replicas);
			F64_TRY(cudaGetLastError());
			cur = next;
		}
		F64_TRY(cudaDeviceSynchronize());
		F64_TRY(cudaMemcpy(means, d_means[cur], kd * sizeof(double), cudaMemcpyDeviceToHost));
		F64_TRY(cudaMemcpy(assignment, d_asg, n * sizeof(uint32_t), cudaMemcpyDeviceToHost));
	}
done:
	cudaFree(mem);
	return rc;
}
