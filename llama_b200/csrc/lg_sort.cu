// lg_sort.cu - device LSD radix sort of 64-bit keys (optional 32-bit
// payload), used to flatten, orient and build snapshots.
//
// One pass per 8-bit digit that may vary (the caller says which bits, or they
// are found with an OR/AND reduction; 48-bit keys cost 6 passes):
//   rs_hist     per-tile digit counts, stored digit-major
//   scan        exclusive scan of the counts -> scatter bases
//   rs_scatter  stable scatter: a warp ranks its 512 consecutive keys of the
//               tile 32 at a time (the lanes that share a digit are found with
//               one match or nine votes, the warp's own counters carry the
//               ranks forward), one block-wide scan adds the other warps'
//               counts, and the tile goes through shared memory in digit order,
//               so a digit's keys leave as one contiguous run.
// What bounds rs_scatter is finding those lanes: matches alone keep their unit
// 74 % busy, votes alone the ALU 85 %.  A third of the rounds by match and the
// rest by votes uses both: 21.6 M keys take 115 us a pass (153 by match, 126 by
// votes, 120 half and half; the traffic of 16 bytes per key is worth 53).  Keys
// are read twice instead of held, which makes three CTAs resident of two (160
// us); four would spill (136).
#include "lg_device.cuh"
#include "lg_sort.cuh"

namespace lg {

constexpr int kRsThreads = 256;
constexpr int kRsItems = 16;
constexpr uint64_t kRsTile = (uint64_t)kRsThreads * kRsItems;
constexpr int kRsWarps = kRsThreads / 32;

__global__ void rs_bits(const unsigned long long* k, uint64_t n,
		unsigned long long* or_and) {
	unsigned long long o = 0, a = ~0ull;
	for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
			i += (uint64_t)gridDim.x * blockDim.x) {
		o |= k[i];
		a &= k[i];
	}
	for (int s = 16; s > 0; s >>= 1) {
		o |= __shfl_down_sync(0xffffffffu, o, s);
		a &= __shfl_down_sync(0xffffffffu, a, s);
	}
	if ((threadIdx.x & 31) == 0) { atomicOr(or_and, o); atomicAnd(or_and + 1, a); }
}

__global__ void __launch_bounds__(kRsThreads)
rs_hist(const unsigned long long* k, uint64_t n, int shift, uint32_t* counts,
		uint32_t tiles) {
	__shared__ uint32_t h[256];
	h[threadIdx.x] = 0;
	const uint64_t base = (uint64_t)blockIdx.x * kRsTile + threadIdx.x;
	uint32_t dig[kRsItems];              // all loads before the first count
#pragma unroll
	for (int r = 0; r < kRsItems; r++) {
		const uint64_t i = base + (uint64_t)r * kRsThreads;
		dig[r] = i < n ? (uint32_t)(k[i] >> shift) & 0xffu : 256u;
	}
	__syncthreads();
#pragma unroll
	for (int r = 0; r < kRsItems; r++)
		if (dig[r] < 256u) atomicAdd(&h[dig[r]], 1u);
	__syncthreads();
	counts[(uint64_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// Shared memory of rs_scatter: the tile in digit order (keys, then payloads).
constexpr size_t rs_smem(bool pay) { return kRsTile * (pay ? 12 : 8); }

// Lanes of the warp that hold the same digit (0 .. 255); a lane past the end
// (valid false) meets none of the others.
__device__ __forceinline__ unsigned rs_peers(uint32_t dig, bool valid) {
	const unsigned in = __ballot_sync(0xffffffffu, valid);
	unsigned peers = valid ? in : ~in;
#pragma unroll
	for (int b = 0; b < 8; b++) {
		const unsigned m = __ballot_sync(0xffffffffu, (dig >> b) & 1u);
		peers &= (dig >> b) & 1u ? m : ~m;
	}
	return peers;
}

template <bool kPay>
__global__ void __launch_bounds__(kRsThreads, 3)
rs_scatter(const unsigned long long* k, const uint32_t* pin, uint64_t n, int shift,
		const uint32_t* offsets, uint32_t tiles, unsigned long long* kout,
		uint32_t* pout) {
	extern __shared__ unsigned long long skey[];
	uint32_t* spay = reinterpret_cast<uint32_t*>(skey + kRsTile);
	__shared__ uint32_t wcnt[kRsWarps][256];   // per warp: keys of a digit so far
	__shared__ uint32_t dbase[256];            // digit -> output base - tile position
	__shared__ uint32_t wsum[kRsWarps];
	const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
	const uint64_t tile0 = (uint64_t)blockIdx.x * kRsTile;
	const uint64_t first = tile0 + w * (32u * kRsItems) + lane;
	uint32_t dig[kRsItems];                    // the digit; then digit << 16 | rank in the warp
#pragma unroll
	for (int r = 0; r < kRsItems; r++) {
		const uint64_t i = first + (uint64_t)r * 32u;
		dig[r] = i < n ? (uint32_t)(k[i] >> shift) & 0xffu : 0u;
	}
#pragma unroll
	for (int x = 0; x < kRsWarps; x++) wcnt[x][tid] = 0;
	const uint32_t goff = offsets[(uint64_t)tid * tiles + blockIdx.x];
	__syncthreads();
	const uint32_t below = (1u << lane) - 1u;
#pragma unroll
	for (int r = 0; r < kRsItems; r++) {
		const bool valid = first + (uint64_t)r * 32u < n;
		const uint32_t d = dig[r];
		const unsigned peers = r % 3 == 0 ? __match_any_sync(0xffffffffu, valid ? d : 256u)
				: rs_peers(d, valid);
		const uint32_t before = valid ? wcnt[w][d] : 0u;
		__syncwarp();
		dig[r] = d << 16 | (before + __popc(peers & below));
		if (valid && 31 - __clz(peers) == (int)lane) wcnt[w][d] = before + __popc(peers);
		__syncwarp();
	}
	__syncthreads();
	// thread d: digit d's keys per warp -> exclusive over the warps, then the
	// digits' starts within the tile
	{
		uint32_t run = 0;
#pragma unroll
		for (int x = 0; x < kRsWarps; x++) {
			const uint32_t c = wcnt[x][tid];
			wcnt[x][tid] = run;
			run += c;
		}
		uint32_t inc = run;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
			if (lane >= (uint32_t)o) inc += y;
		}
		if (lane == 31u) wsum[w] = inc;
		__syncthreads();
		uint32_t start = inc - run;
		for (uint32_t x = 0; x < w; x++) start += wsum[x];
#pragma unroll
		for (int x = 0; x < kRsWarps; x++) wcnt[x][tid] += start;
		dbase[tid] = goff - start;
	}
	__syncthreads();
	// the keys again (from L2): held since the first read they were 32 registers
	constexpr int kHalf = kRsItems / 2;
#pragma unroll
	for (int h = 0; h < kRsItems; h += kHalf) {
		unsigned long long key[kHalf];
#pragma unroll
		for (int r = 0; r < kHalf; r++) {
			const uint64_t i = first + (uint64_t)(h + r) * 32u;
			key[r] = i < n ? k[i] : 0ull;
		}
#pragma unroll
		for (int r = 0; r < kHalf; r++) {
			const uint64_t i = first + (uint64_t)(h + r) * 32u;
			if (i < n) {
				const uint32_t pos = wcnt[w][dig[h + r] >> 16] + (dig[h + r] & 0xffffu);
				skey[pos] = key[r];
				if (kPay) spay[pos] = pin[i];
			}
		}
	}
	__syncthreads();
	const uint32_t m = (uint32_t)(n - tile0 < kRsTile ? n - tile0 : kRsTile);
	for (uint32_t j = tid; j < m; j += kRsThreads) {
		const unsigned long long x = skey[j];
		const uint32_t p = dbase[(x >> shift) & 0xff] + j;
		kout[p] = x;
		if (kPay) pout[p] = spay[j];
	}
}

lg_status radix_sort_u64(lg_store* s, unsigned long long* keys, uint32_t* payload,
		uint64_t n, DevBuf& tmp_keys, DevBuf& tmp_pay, DevBuf& counts, DevBuf& scan_tmp,
		unsigned long long** sorted_keys, uint32_t** sorted_pay, unsigned long long vary) {
	cudaStream_t st = s->stream;
	*sorted_keys = keys;
	if (sorted_pay) *sorted_pay = payload;
	if (n < 2) return LG_OK;
	if (n >= 0xffffffffull) return set_error(LG_ENOTSUP, "sort of more than 2^32-1 keys");
	const uint32_t tiles = (uint32_t)((n + kRsTile - 1) / kRsTile);
	LG_TRY(tmp_keys.reserve(n * 8));
	if (payload) LG_TRY(tmp_pay.reserve(n * 4));
	LG_TRY(counts.reserve(((uint64_t)256 * tiles + 1) * 8 + 16));
	uint32_t* cnt = counts.as<uint32_t>();
	uint32_t* off = cnt + (uint64_t)256 * tiles + 1;
	if (vary == 0) {
		// which bits vary
		unsigned long long oa[2] = {0, ~0ull};
		unsigned long long* d_oa = (unsigned long long*)(counts.as<char>()
				+ ((uint64_t)256 * tiles + 1) * 8);
		LG_CUDA(cudaMemcpyAsync(d_oa, oa, 16, cudaMemcpyHostToDevice, st), "h2d");
		rs_bits<<<592, 256, 0, st>>>(keys, n, d_oa);
		LG_CUDA(cudaMemcpyAsync(oa, d_oa, 16, cudaMemcpyDeviceToHost, st), "d2h");
		LG_CUDA(cudaStreamSynchronize(st), "sort bits");
		s->launches++;
		vary = oa[0] ^ oa[1];
	}
	const size_t smem = rs_smem(payload != nullptr);
	if (payload)
		LG_CUDA(cudaFuncSetAttribute(rs_scatter<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
				(int)smem), "rs_scatter");
	unsigned long long* src = keys;
	unsigned long long* dst = tmp_keys.as<unsigned long long>();
	uint32_t* psrc = payload;
	uint32_t* pdst = payload ? tmp_pay.as<uint32_t>() : nullptr;
	for (int shift = 0; shift < 64; shift += 8) {
		if (((vary >> shift) & 0xff) == 0) continue;
		rs_hist<<<tiles, kRsThreads, 0, st>>>(src, n, shift, cnt, tiles);
		LG_TRY(exclusive_scan_u32(cnt, off, (uint64_t)256 * tiles, scan_tmp, st, nullptr));
		if (payload)
			rs_scatter<true><<<tiles, kRsThreads, smem, st>>>(src, psrc, n, shift, off, tiles, dst,
					pdst);
		else
			rs_scatter<false><<<tiles, kRsThreads, smem, st>>>(src, nullptr, n, shift, off, tiles,
					dst, nullptr);
		LG_CUDA(cudaGetLastError(), "radix sort pass");
		s->launches += 2 + scan_launches((uint64_t)256 * tiles);
		std::swap(src, dst);
		std::swap(psrc, pdst);
	}
	*sorted_keys = src;
	if (sorted_pay) *sorted_pay = psrc;
	return LG_OK;
}

} // namespace lg
