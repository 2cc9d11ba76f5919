// lg_coop.cuh - building blocks of the one-launch traversals and iterations
// (lg_bfs_levels.cu, lg_sssp_flat.cu, lg_sssp_levels.cu, lg_scc_flat.cu,
// lg_flat_run.cuh): cooperative launches, a grid barrier for them whose waits
// are bounded by the global timer, and CTA-wide sums and scans.
#ifndef LG_COOP_CUH_
#define LG_COOP_CUH_

#include <cuda_runtime.h>
#include <stdint.h>

#include "lg_internal.h"

namespace lg {

// Barrier state in device memory; count must be 0 before the launch.
struct alignas(16) CoopBar {
	unsigned long long count;   // arrivals so far
	unsigned int err;           // bit 0: a barrier wait ran out; higher bits: the caller's
	unsigned int pad;
};

constexpr uint64_t kCoopWaitNs = 1000000000ull;   // a barrier wait gives up after 1 s
// A kernel whose steps depend on the graph (a chain takes as many as it has
// vertices, or their square) returns with its state after so long, and the
// host launches it again: neither the host nor other streams wait longer.  In
// cycles of the SM that looks (50 ms at 2 GHz), a register read.
constexpr long long kCoopRunCycles = 100000000;
// That the time is up is a bit of one of the step's counters, which every CTA
// reads after the barrier anyway.
constexpr unsigned long long kCoopTimeUp = 1ull << 63;

__device__ __forceinline__ uint64_t global_ns() {
	uint64_t t;
	asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
	return t;
}

// Barrier over all CTAs of a cooperative grid (all co-resident).  Thread 0
// of each CTA publishes the CTA's writes (fence), arrives, and waits until the
// arrivals reach the next multiple of the grid's size; false once any CTA gave
// up waiting or set an error.  The count only grows, so the last arrival needs
// no reset, and a poll reads count and error in one load: some 1 us less per
// barrier than a counter that is reset beside a generation word.
__device__ inline bool grid_barrier(CoopBar* b) {
	__shared__ int s_ok;
	__syncthreads();
	if (threadIdx.x == 0) {
		__threadfence();
		const unsigned long long old = atomicAdd(&b->count, 1ull);
		const unsigned long long target = (old / gridDim.x + 1ull) * gridDim.x;
		uint64_t t0 = 0;
		int ok = 1;
		for (uint32_t polls = 0;; polls++) {
			unsigned long long seen, err;
			asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];"
				: "=l"(seen), "=l"(err) : "l"(b) : "memory");
			if ((unsigned int)err) {         // a CTA left on an error: it will not arrive
				ok = 0;
				break;
			}
			if (seen >= target) break;
			if (polls < 64) continue;
			if (!t0) t0 = global_ns();
			if (global_ns() - t0 > kCoopWaitNs) {
				atomicOr(&b->err, 1u);
				ok = 0;
				break;
			}
			__nanosleep(64);
		}
		__threadfence();
		s_ok = ok;
	}
	__syncthreads();
	return s_ok != 0;
}

// Sum of x over a CTA of kWarps warps, returned to every thread (all
// threads call it).
template <int kWarps>
__device__ __forceinline__ unsigned long long block_sum(unsigned long long x) {
	__shared__ unsigned long long s_part[kWarps];
	const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
	__syncthreads();                     // s_part free from a previous call
	if (lane == 0) s_part[wid] = x;
	__syncthreads();
	unsigned long long t = 0;
#pragma unroll
	for (int w = 0; w < kWarps; w++) t += s_part[w];
	return t;
}

// Exclusive scan of x over a CTA of kWarps warps in thread order; *total =
// the CTA's sum (all threads call it).
template <int kWarps>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t x, uint32_t* total) {
	__shared__ uint32_t s_warp[kWarps];
	const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
	uint32_t inc = x;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
		if (lane >= (uint32_t)o) inc += y;
	}
	__syncthreads();
	if (lane == 31u) s_warp[wid] = inc;
	__syncthreads();
	uint32_t before = 0, all = 0;
#pragma unroll
	for (int w = 0; w < kWarps; w++) {
		const uint32_t s = s_warp[w];
		if (w < (int)wid) before += s;
		all += s;
	}
	*total = all;
	return before + inc - x;
}

// Co-resident CTAs of `kernel` at `threads` and `smem` bytes of dynamic shared
// memory per CTA on `device` (SMs x CTAs per SM), 0 when the device has no
// cooperative launch.
inline int coop_grid_size(const void* kernel, int threads, int device, size_t smem = 0) {
	int coop = 0, sms = 0, per_sm = 0;
	if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess ||
			cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
			cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) !=
					cudaSuccess) {
		cudaGetLastError();
		return 0;
	}
	return coop && sms > 0 && per_sm > 0 ? sms * per_sm : 0;
}

// Launches `kernel` on *grid CTAs (a grid of any size gives its result), or,
// where the caller's share of the GPU holds fewer at once than the device's
// properties say, on half, a quarter ... as many, which *grid becomes.  bar:
// the kernel's barrier, whose count is a multiple of the grid's size.
inline cudaError_t coop_launch(const void* kernel, unsigned* grid, int threads, void** args,
		size_t smem, cudaStream_t st, CoopBar* bar) {
	for (;; *grid /= 2u) {
		const cudaError_t e = *grid > test_limits().ctas ? cudaErrorCooperativeLaunchTooLarge
				: cudaLaunchCooperativeKernel(kernel, dim3(*grid), dim3((unsigned)threads), args,
						smem, st);
		if (e != cudaErrorCooperativeLaunchTooLarge || *grid <= 1u) return e;
		(void)cudaGetLastError();
		const cudaError_t me = cudaMemsetAsync(&bar->count, 0, sizeof(bar->count), st);
		if (me != cudaSuccess) return me;
	}
}

// Cycles after which a launch's time is up (kCoopRunCycles; a test's: none).
inline long long coop_run_cycles() { return test_limits().one_step ? -1 : kCoopRunCycles; }

// The CTAs that coop_grid_size found, 0 where a test wants no cooperative launch.
inline int coop_allowed(int grid) { return test_limits().ctas > 0 ? grid : 0; }

} // namespace lg

#endif // LG_COOP_CUH_
