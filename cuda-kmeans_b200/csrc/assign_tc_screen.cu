// Screening pass of the tensor-core assignment for rows longer than 64 dimensions: x.c from the fp16 HIGH parts
// alone, one product instead of three.
//
// With x = xh + xl and b = -2c = bh + bl the value |c|^2 + x.b that the arg-min needs differs from |c|^2 + xh.bh by
//     |xl.b + xh.bl| <= |xl| |b| + |xh| |bl|,
// and the lengths of what the high parts leave over are known: |xl| of every point from the split, the largest
// |bl| from the preparation of the means.  Where the two smallest values of a point's row are further apart than
// twice that bound (and the band of the pass with all three products) the smallest is the nearest mean, as the exact
// arithmetic would find it.  The other points (2 to 10 % of them, more where clusters lie close
// together against their distance from the centre of all points) go to a list and through the pass with all
// three products, K loop of assign_tc.cu, and from there to the exact kernel as ever: the labels are the same.
// Long rows are bound by the tensor pipe, and at three products by the power limit as well: 2^20 x 512
// against 4096 means 9.06 ms per iteration in one pass, 3.10 with screening and list.
//
// One CTA pair (cta_group::2) multiplies 256 points by 256 means at a time: each CTA holds its 128 points and half of
// the means, and gets the 128 x 256 block of its points in tensor memory, twice over, so that one block
// is reduced while the next is multiplied.  Operands come in slices of 64 dimensions (16 KiB: one 128-byte swizzle
// row per point or mean).  Up to 512 dimensions the points' slices stay in shared memory for all
// mean tiles and only the means stream, 64 bytes per clock and pair where points and means together would
// need 128; a point slice is handed back with its last use, so that the next points arrive during the last
// mean tile.  Longer rows stream both.  Roles as in assign_tc_pair.cu: warp 0 loads, warp 1 of the pair's
// first CTA issues, warps 2..17 reduce (a lane quarter and 64 columns each).  All waits are bounded.
#include <cuda.h>

#include "kernels.cuh"
#include "ptx.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <cmath>

namespace bkm {

constexpr uint32_t SC_PLANE_BYTES = TC_MTILE * TC_KCHUNK * 4;     // 16 KiB: 128 rows of one slice
constexpr uint32_t SC_SLOTS = 12;                                 // slices of points and means in shared memory
constexpr uint32_t SC_RESIDENT_SLICES = 8;                        // the most that a point's row may have to stay there
constexpr uint32_t SC_AUG_BYTES = (TC_NT_MAX / 2) * 8 * 4;        // 4 KiB: |c|^2 step of half a mean tile
constexpr uint32_t SC_AUG_SLOTS = 4;                              // as many of them: the loader must not wait for a mean tile's end with the next ones
constexpr uint32_t SC_AUG_OFF = SC_SLOTS * SC_PLANE_BYTES;
constexpr uint32_t SC_AAUG_OFF = SC_AUG_OFF + SC_AUG_SLOTS * SC_AUG_BYTES;
constexpr uint32_t SC_MERGE_OFF = SC_AAUG_OFF + TC_MTILE * 8 * 4;
constexpr uint32_t SC_BAR_OFF = SC_MERGE_OFF + 2 * 3 * 3 * TC_MTILE * 4;   // two slots x column parts 0..2 x (best, second, chunk)

struct ScreenBars {
	uint64_t a_full[SC_SLOTS], b_full[SC_SLOTS], aug_full[SC_AUG_SLOTS];      // first CTA: what both CTAs load has landed
	uint64_t a_empty[SC_SLOTS], b_empty[SC_SLOTS], aug_empty[SC_AUG_SLOTS];   // every CTA: the MMAs that read it are done
	uint64_t acc_full[2];                                          // every CTA: accumulator complete
	uint64_t acc_empty[2];                                         // first CTA: the epilogue warps of both CTAs have read it
	uint32_t tmem_slot;
	uint32_t abort_flag;
};
constexpr uint32_t SC_ALLOC = SC_BAR_OFF + sizeof(ScreenBars) + 1024;      // slack for 1024-byte alignment
static_assert(SC_ALLOC <= 227 * 1024, "shared memory budget exceeded");

// Slots of the points' ring: their slices twice over where there is room for it.
static uint32_t screen_a_slots(uint32_t slices) { return slices <= 4 ? 2 * slices : (slices <= SC_RESIDENT_SLICES ? slices : SC_SLOTS / 2); }

// (The hand-over between epilogue warps relies on two mean tiles at least.)
bool tc_screen_fits(uint32_t k, uint32_t dim) { return tc_dpad(dim) > TC_KCHUNK && k > TC_NT_MAX; }

// The pass costs two or three launches more, and the few points that it leaves open take as long as a block of them
// takes: us per call with / without, by n x k x d: 6.3e9 (262 144 x 300 x 80) 112 / 107, 6.4e9 (131 072 x 512 x 96) 95 / 82,
// 8.6e9 (65 536 x 512 x 256) 105 / 95, 1.0e10 (65 536 x 300 x 512) 159 / 161, 1.3e10 (100 003 x 1024 x 128) 110 / 156,
// 1.8e10 (131 072 x 2000 x 70) 158 / 170, 3.1e10 (100 000 x 512 x 600) 234 / 254, 1.0e11 (10^6 x 1000 x 100, 28 % open) 955 / 1019;
// 30 000 points x 1024 x 128 83 / 77.  Where the first wave leaves most points open: 3141 / 3056 (99.5 % of 10^6 x 1000 x 100).
bool tc_screen_pays(const Shape& s) { return s.n >= 1u << 15 && (double)s.n * s.k * s.dim >= 1.2e10; }

// Waits for the last fill of every buffer that has been filled (a lap at most); `pos` is the next one to be filled.
__device__ __forceinline__ void drain_ring(uint64_t* full, RingPos pos, uint32_t slots, uint32_t fills)
{
	for (uint32_t back = 0; back < slots && back < fills; ++back) {
		if (pos.slot == 0) { pos.slot = slots; pos.phase ^= 1u; }
		--pos.slot;
		ptx::mbar_wait(&full[pos.slot], pos.phase);
	}
}

// Appends the points whose `flag` is set to the list of open points, one atomic per warp.
__device__ __forceinline__ uint32_t append_open(bool flag, uint32_t point, Control* __restrict__ ctl, uint32_t* __restrict__ list, uint64_t n)
{
	const uint32_t mask = __ballot_sync(0xffffffffu, flag);
	if (mask == 0) return 0;
	const uint32_t lane = threadIdx.x & 31u, count = (uint32_t)__popc(mask);
	uint32_t base = 0;
	if (lane == 0) base = atomicAdd(&ctl->screen_count, count);
	base = __shfl_sync(0xffffffffu, base, 0);
	if (flag) {
		const uint32_t pos = base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
		if ((uint64_t)pos < n) list[pos] = point;
		else atomicOr(&ctl->status, (uint32_t)STATUS_LIST_OVERFLOW);
	}
	return count;
}

// A launch takes the steps (256 points each) [step_begin, step_end).  `probe_points` > 0: an earlier launch has screened that
// many points; where it has left most of them open this one does not multiply but leaves all of its points open.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1) assign_tc_screen_kernel(
	const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_aug,
	const float* __restrict__ xnorm, const float* __restrict__ xlow, uint32_t* __restrict__ asg, uint32_t* __restrict__ list,
	uint64_t n, uint32_t k, uint32_t n_ctiles, uint32_t slices, uint32_t a_slots, uint32_t ksteps_last, uint32_t idesc,
	Control* __restrict__ ctl, int slot, float margin_coef, float margin_scale, float sqrt_dim, uint32_t step_begin, uint32_t step_end, uint32_t probe_points)
{
	extern __shared__ uint8_t smem_raw[];
	// (an offset from the array, so that the compiler still knows it for shared memory: 32-bit addresses in the epilogue)
	uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
	ScreenBars* bars = reinterpret_cast<ScreenBars*>(smem + SC_BAR_OFF);
	uint32_t* mg_state = reinterpret_cast<uint32_t*>(smem + SC_MERGE_OFF);
	volatile uint32_t* abort_flag = &bars->abort_flag;

	const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
	const uint32_t rank = ptx::cluster_ctarank();
	const uint32_t pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
	if (probe_points != 0 && 2u * ctl->probe_count > probe_points) {
		// (the same decision in all blocks: nothing writes the count any more)
		for (uint32_t step = step_begin + pair; step < step_end; step += n_pairs)
			if (warp < TC_MTILE / 32) {
				const uint64_t p = (uint64_t)(2 * step + rank) * TC_MTILE + threadIdx.x;
				append_open(p < n, (uint32_t)p, ctl, list, n);
			}
		return;
	}
	const uint32_t peer_abort_addr = ptx::map_to_cta(ptx::smem_u32(&bars->abort_flag), rank ^ 1u);
	const bool resident = slices <= SC_RESIDENT_SLICES;
	const uint32_t b_slots = SC_SLOTS - a_slots;
	uint8_t* b_ring = smem + a_slots * SC_PLANE_BYTES;

	if (threadIdx.x == 0) {
		for (uint32_t i = 0; i < SC_SLOTS; ++i) {
			ptx::mbar_init(&bars->a_full[i], 1);
			ptx::mbar_init(&bars->b_full[i], 1);
			ptx::mbar_init(&bars->a_empty[i], 1);
			ptx::mbar_init(&bars->b_empty[i], 1);
		}
		for (uint32_t i = 0; i < SC_AUG_SLOTS; ++i) {
			ptx::mbar_init(&bars->aug_full[i], 1);
			ptx::mbar_init(&bars->aug_empty[i], 1);
		}
		for (uint32_t i = 0; i < 2; ++i) {
			ptx::mbar_init(&bars->acc_full[i], 1);
			ptx::mbar_init(&bars->acc_empty[i], 2 * TC_EPI_WARPS);
		}
		bars->abort_flag = 0;
		ptx::fence_mbar_init();
	}
	if (warp == 1) {
		ptx::tmem_alloc_pair(&bars->tmem_slot, TC_TMEM_COLS);
		ptx::tmem_relinquish_pair();
	}
	const float x2max = ctl->xmax2, c2max = ctl->mean_max[slot].c2, bl2max = ctl->mean_max[slot].bl2;
	const KeyConsts kc = tc_key_consts(x2max, c2max);
	const uint32_t key_mult = kc.key_mult, key_base = kc.key_base, key_magic = kc.key_magic;
	fill_a_aug(smem + SC_AAUG_OFF, kc, x2max, threadIdx.x, TC_THREADS);
	ptx::fence_proxy_async();
	ptx::tc_fence_before();
	ptx::cluster_sync();            // barriers of both CTAs initialised, tensor memory allocated, constant tiles written
	ptx::tc_fence_after();
	const uint32_t tmem_base = bars->tmem_slot;

	if (warp == 0) {
		// ---------------- TMA producer (both CTAs) ----------------
		if (lane == 0) {
			ptx::prefetch_tmap(&tm_a); ptx::prefetch_tmap(&tm_b); ptx::prefetch_tmap(&tm_aug);
			RingPos a_pos, b_pos, aug_pos;
			uint32_t a_fills = 0, b_fills = 0, aug_fills = 0;
			const uint32_t a_full0 = ptx::leader_cta_addr(ptx::smem_u32(bars->a_full)), b_full0 = ptx::leader_cta_addr(ptx::smem_u32(bars->b_full));
			const uint32_t aug_full0 = ptx::leader_cta_addr(ptx::smem_u32(bars->aug_full));
			bool ok = true;
			for (uint32_t step = step_begin + pair; step < step_end && ok; step += n_pairs) {
				for (uint32_t j = 0; j < n_ctiles && ok; ++j) {
					const uint32_t mean = j * TC_NT_MAX + rank * (TC_NT_MAX / 2);
					ok = pair_wait<20>(&bars->aug_empty[aug_pos.slot], aug_pos.phase ^ 1u, abort_flag, peer_abort_addr);
					if (!ok) break;
					if (rank == 0) ptx::mbar_arrive_expect_tx(&bars->aug_full[aug_pos.slot], 2 * SC_AUG_BYTES);
					ptx::tma_load_2d_pair(smem + SC_AUG_OFF + aug_pos.slot * SC_AUG_BYTES, &tm_aug, 0, (int32_t)(mean / 4), aug_full0 + aug_pos.slot * 8u);
					aug_pos.next(SC_AUG_SLOTS);
					++aug_fills;
					for (uint32_t sl = 0; sl < slices; ++sl) {
						if (!resident || j == 0) {
							ok = pair_wait<20>(&bars->a_empty[a_pos.slot], a_pos.phase ^ 1u, abort_flag, peer_abort_addr);
							if (!ok) break;
							if (rank == 0) ptx::mbar_arrive_expect_tx(&bars->a_full[a_pos.slot], 2 * SC_PLANE_BYTES);
							// (rows behind the last tile read as zeros)
							ptx::tma_load_2d_pair(smem + a_pos.slot * SC_PLANE_BYTES, &tm_a, (int32_t)(sl * TC_KCHUNK), (int32_t)((2 * step + rank) * TC_MTILE), a_full0 + a_pos.slot * 8u);
							a_pos.next(a_slots);
							++a_fills;
						}
						ok = pair_wait<20>(&bars->b_empty[b_pos.slot], b_pos.phase ^ 1u, abort_flag, peer_abort_addr);
						if (!ok) break;
						if (rank == 0) ptx::mbar_arrive_expect_tx(&bars->b_full[b_pos.slot], 2 * SC_PLANE_BYTES);
						ptx::tma_load_2d_pair(b_ring + b_pos.slot * SC_PLANE_BYTES, &tm_b, (int32_t)(sl * TC_KCHUNK), (int32_t)mean, b_full0 + b_pos.slot * 8u);
						b_pos.next(b_slots);
						++b_fills;
					}
				}
			}
			if (rank == 0) {
				// Nobody leaves while a copy may still be in flight: the first CTA's barriers count
				// the bytes of both CTAs, and the second CTA stays until the final cluster barrier.
				drain_ring(bars->a_full, a_pos, a_slots, a_fills);
				drain_ring(bars->b_full, b_pos, b_slots, b_fills);
				drain_ring(bars->aug_full, aug_pos, SC_AUG_SLOTS, aug_fills);
			}
		}
	} else if (warp == 1) {
		// ---------------- MMA issuer (first CTA of the pair) ----------------
		if (rank == 0) {
			const uint32_t a_aug_lo = desc_lo_aug(ptx::smem_u32(smem + SC_AAUG_OFF));
			auto commit_both = [](uint64_t* bar) {
				const uint32_t own = ptx::smem_u32(bar);
				ptx::mma_commit_pair(own);
				ptx::mma_commit_pair(ptx::map_to_cta(own, 1u));
			};
			RingPos a_pos, b_pos, aug_pos, acc_pos;      // a_pos: resident, the first slice of the step's points
			bool ok = true;
			for (uint32_t step = step_begin + pair; step < step_end && ok; step += n_pairs) {
				RingPos next_points = a_pos;
				for (uint32_t j = 0; j < n_ctiles && ok; ++j) {
					const uint32_t d_tmem = tmem_base + acc_pos.slot * TC_NT_MAX;
					ok = pair_wait<20>(&bars->acc_empty[acc_pos.slot], acc_pos.phase ^ 1u, abort_flag, peer_abort_addr);
					if (!ok) break;
					RingPos points = a_pos;
					for (uint32_t sl = 0; sl < slices; ++sl) {
						if (!resident || j == 0) ok = pair_wait<20>(&bars->a_full[points.slot], points.phase, abort_flag, peer_abort_addr);
						if (ok) ok = pair_wait<20>(&bars->b_full[b_pos.slot], b_pos.phase, abort_flag, peer_abort_addr);
						if (!ok) break;
						ptx::tc_fence_after();
						const uint32_t a_lo = desc_lo_sw128(ptx::smem_u32(smem + points.slot * SC_PLANE_BYTES)), b_lo = desc_lo_sw128(ptx::smem_u32(b_ring + b_pos.slot * SC_PLANE_BYTES));
						const uint32_t steps = sl + 1 == slices ? ksteps_last : 4u;
						if (ptx::elect_one()) {
							if (sl == 0) ptx::mma_f16_pair_halves<false>(d_tmem, a_lo, DESC_HI_SW128, b_lo, DESC_HI_SW128, idesc);
							else ptx::mma_f16_pair_halves<true>(d_tmem, a_lo, DESC_HI_SW128, b_lo, DESC_HI_SW128, idesc);
							#pragma unroll
							for (uint32_t ks = 1; ks < 4; ++ks)
								if (ks < steps) ptx::mma_f16_pair_halves<true>(d_tmem, a_lo + 2 * ks, DESC_HI_SW128, b_lo + 2 * ks, DESC_HI_SW128, idesc);
							commit_both(&bars->b_empty[b_pos.slot]);
							if (!resident || j + 1 == n_ctiles) commit_both(&bars->a_empty[points.slot]);
						}
						__syncwarp();
						b_pos.next(b_slots);
						points.next(a_slots);
					}
					if (!ok) break;
					if (!resident) a_pos = points;
					next_points = points;
					ok = pair_wait<20>(&bars->aug_full[aug_pos.slot], aug_pos.phase, abort_flag, peer_abort_addr);
					if (!ok) break;
					ptx::tc_fence_after();
					if (ptx::elect_one()) {
						ptx::mma_f16_pair_halves<true>(d_tmem, a_aug_lo, DESC_HI_AUG, desc_lo_aug(ptx::smem_u32(smem + SC_AUG_OFF + aug_pos.slot * SC_AUG_BYTES)), DESC_HI_AUG, idesc);
						commit_both(&bars->acc_full[acc_pos.slot]);
						commit_both(&bars->aug_empty[aug_pos.slot]);
					}
					__syncwarp();
					aug_pos.next(SC_AUG_SLOTS);
					acc_pos.next(2);
				}
				a_pos = next_points;
			}
		}
	} else {
		// ---------------- epilogue (both CTAs, own accumulator rows) ----------------
		// Warp (q, g): TMEM lane quarter q, columns 64 g .. 64 g + 63 of every fill.
		const uint32_t q = warp & 3u, g = (warp - 2) >> 2, row = q * 32 + lane;
		constexpr uint32_t merger = 3;
		const float ulp = kc.pow2 * 1.1920929e-07f;   // spacing of the values inside [P, 2P)
		const float margin_floor = tc_margin_floor(ulp, x2max, c2max, sqrt_dim, tc_scale(ctl->xdev));
		// twice the bound above, a little more for its own roundings
		const float low_coef = 2.002f * margin_scale * 2.0f * sqrtf(c2max), rest_coef = 2.002f * margin_scale * sqrtf(bl2max);
		const uint32_t acc_empty_base = ptx::map_to_cta(ptx::smem_u32(&bars->acc_empty[0]), 0);
		uint32_t it = 0, c = 0, open_count = 0;
		bool ok = true;
		for (uint32_t step = step_begin + pair; step < step_end; step += n_pairs, ++it) {
			RowMin rows;
			rows.reset();
			const uint64_t p = (uint64_t)(2 * step + rank) * TC_MTILE + row;
			float xn = 0.0f, xl = 0.0f;
			if (g == merger && p < n) { xn = xnorm[p]; xl = xlow[p]; }      // needed at the end of the step only: fetch early
			#pragma unroll 1
			for (uint32_t j = 0; j < n_ctiles; ++j, ++c) {
				const uint32_t acc = c & 1u;
				if (ok) ok = __all_sync(0xffffffffu, pair_wait(&bars->acc_full[acc], (c >> 1) & 1u, abort_flag, peer_abort_addr)) != 0;
				ptx::tc_fence_after();
				uint32_t v0[32], v1[32];
				const uint32_t taddr = tmem_base + ((q * 32u) << 16) + acc * TC_NT_MAX + g * 64u;
				const uint32_t chunk0 = j * 8u + g * 2u;
				// the second half of the columns travels while the first is reduced
				ptx::tmem_ld32(taddr, v0);
				ptx::tmem_ld_wait();
				ptx::tmem_ld32(taddr + 32, v1);
				rows.take_chunk(v0, key_mult, chunk0);
				ptx::tmem_ld_wait();
				ptx::tc_fence_before();
				__syncwarp();
				if (lane == 0) ptx::mbar_arrive_cluster(acc_empty_base + acc * 8u);
				rows.take_chunk(v1, key_mult, chunk0 + 1);
			}
			// Three warps of a quarter hand their state to the fourth and go on (see assign_tc_pair.cu).  Slots and barrier
			// numbers alternate with the step count: a step has two fills at least, and a fill needs all
			// warps to have released the one two before it.
			uint32_t best, second, bchunk;
			rows.finish(key_base, key_mult, key_magic, best, second, bchunk);
			uint32_t* mg = mg_state + (it & 1u) * (3 * 3 * TC_MTILE);
			const uint32_t merge_bar = 1u + (it & 1u) * 4u + q;
			if (g != merger) {
				uint32_t* dst = mg + g * (3 * TC_MTILE);
				dst[row] = best; dst[TC_MTILE + row] = second; dst[2 * TC_MTILE + row] = bchunk;
				asm volatile("bar.arrive %0, 128;" :: "r"(merge_bar) : "memory");
			} else {
				asm volatile("bar.sync %0, 128;" :: "r"(merge_bar) : "memory");
				bool open = false;
				if (p < n && ok) {
					#pragma unroll
					for (uint32_t o = 0; o < 3; ++o) {
						const uint32_t* src = mg + o * (3 * TC_MTILE);
						const uint32_t ob = src[row], os = src[TC_MTILE + row], oc = src[2 * TC_MTILE + row];
						second = umin3(second, os, max(best, ob));
						bchunk = ob < best ? oc : bchunk;
						best = min(best, ob);
					}
					const float margin = margin_coef * (xn + c2max) + margin_floor + low_coef * xl + rest_coef * sqrtf(xn);
					open = finish_point(best, second, bchunk, key_base, key_mult, key_magic, ulp, margin, k, p, asg);
				}
				open_count += append_open(open, (uint32_t)p, ctl, list, n);
			}
		}
		if (probe_points == 0 && lane == 0 && open_count != 0) atomicAdd(&ctl->probe_count, open_count);
	}

	// Both CTAs stay until neither can touch the other's shared memory or barriers any more.
	__syncwarp();
	ptx::tc_fence_before();
	ptx::cluster_sync();
	if (warp == 1) {
		ptx::tc_fence_after();
		ptx::tmem_dealloc_pair(tmem_base, TC_TMEM_COLS);
	}
	if (threadIdx.x == 0 && bars->abort_flag) atomicOr(&ctl->status, (uint32_t)STATUS_WAIT_TIMEOUT);
}

cudaError_t assign_tc_screen_prepare(int sm_count, int* max_pairs)
{
	cudaError_t e = cudaFuncSetAttribute(assign_tc_screen_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SC_ALLOC);
	if (e != cudaSuccess) return e;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(2 * (uint32_t)(sm_count / 2), 1, 1);
	cfg.blockDim = dim3(TC_THREADS, 1, 1);
	cfg.dynamicSmemBytes = SC_ALLOC;
	cudaLaunchAttribute attr;
	attr.id = cudaLaunchAttributeClusterDimension;
	attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
	cfg.attrs = &attr;
	cfg.numAttrs = 1;
	return cudaOccupancyMaxActiveClusters(max_pairs, assign_tc_screen_kernel, &cfg);
}

// Where the points make several waves the first one is a launch of its own, whose result decides about the rest.
constexpr uint32_t SC_PROBE_WAVES = 6;

cudaError_t launch_assign_tc_screen(const CUtensorMap& a_hi, const CUtensorMap& b_hi, const CUtensorMap& b_aug, const TcPoints& tp, uint32_t* asg,
	uint64_t n, uint32_t k, uint32_t k_pad, uint32_t dim, int max_pairs, Control* ctl, int slot, float margin_coef, float margin_scale, float sqrt_dim,
	cudaStream_t stream)
{
	const uint32_t steps = (uint32_t)((n + 2 * TC_MTILE - 1) / (2 * TC_MTILE)), pairs = (uint32_t)max_pairs;
	const uint32_t slices = (tp.d_pad + TC_KCHUNK - 1) / TC_KCHUNK;
	const uint32_t ksteps_last = (dim - (slices - 1) * 2 * TC_KCHUNK + 15) / 16;     // K steps (16 dimensions) of the last slice
	// c_format = f32 (bit 4), a/b format = fp16 (0 at bits 7.., 10..), K-major both, N>>3 at bit 17, M>>4 at bit 24: M = 256 over the pair, N = 256
	const uint32_t idesc = (1u << 4) | ((TC_NT_MAX >> 3) << 17) | (((2 * TC_MTILE) >> 4) << 24);
	auto go = [&](uint32_t begin, uint32_t end, uint32_t probe_points) {
		assign_tc_screen_kernel<<<2 * std::min<uint32_t>(end - begin, pairs), TC_THREADS, SC_ALLOC, stream>>>(a_hi, b_hi, b_aug, tp.xnorm, tp.xlow, asg, tp.screen_list,
			n, k, k_pad / TC_NT_MAX, slices, screen_a_slots(slices), ksteps_last, idesc, ctl, slot, margin_coef, margin_scale, sqrt_dim, begin, end, probe_points);
	};
	const uint32_t first = steps >= SC_PROBE_WAVES * pairs ? pairs : steps;
	go(0, first, 0);
	if (first < steps) go(first, steps, first * 2 * TC_MTILE);
	return cudaGetLastError();
}

} // namespace bkm
