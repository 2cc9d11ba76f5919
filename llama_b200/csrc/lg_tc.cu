// lg_tc.cu - triangle counting on the symmetrised snapshot.
//
// Reference: ll_b_triangle_counting_LU (benchmark/benchmarks/
// triangle_counting.h:343-470), run on a graph loaded with -U (both arcs of
// every edge) and flattened to one level: it counts triangles u < v < w with
// all three undirected edges present, each once.  The reference requires a
// single level with sorted adjacency (triangle_counting.h:422-425); here the
// multiversion snapshot is flattened on the device:
//   1. every vertex gets a label, 0 for the highest degree (out + in), equal
//      degree classes in any order (a class: 1/64 of an octave);
//   2. every live arc u->v (u != v) becomes the undirected edge oriented from
//      the larger to the smaller label, a total order that keeps the forward
//      lists of hubs short and makes their labels small;
//   3. the keys (a << bits | b) are radix sorted and de-duplicated, giving
//      the forward lists N+(a), sorted by label;
//   4. every triangle c < b < a is found at its largest label a: for b in
//      N+(a), |N+(b) & N+(a)|.  A group of warps holds N+(a) in shared memory
//      (a bitmap over the labels below a, or a hash table) and reads the N+(b)
//      against it: as rows of bits for the hubs, as ids otherwise.
//
// What bounds step 4: the visits.  At 700 k vertices and 10.6 M undirected edges
// there are some 9 M pairs (a, b) and 1.8 G ids in their lists; a form with a
// binary search per element of the shorter list took 7.3 G search steps and
// 5950 us, streaming every id against N+(a) 1430 us (one shared-memory probe
// per id, its bank conflicts, and one list in flight per warp).  Rows of bits
// for b < 8 Ki leave 218 M ids and 290 M words, and half a warp per row and a
// quarter per list some 300 M instructions: 600 us.  Because labels follow the
// degrees, a vertex whose list is long has a small label, so bitmaps stay
// short: 64 Ki labels (8 KB, two warps') hold nearly all of the work of
// that graph.
// The count is an exact integer sum (atomicAdd of per-warp partials), so the
// order inside a degree class does not matter.
#include "lg_flat.cuh"
#include "lg_queue.cuh"
#include "lg_sort.cuh"

#include <algorithm>

namespace lg {

typedef unsigned long long u64;

// ---------------------------------------------------------------------------
// Labels: a counting sort of the vertices by degree class, descending.
// ---------------------------------------------------------------------------

constexpr int kTcThreads = 256;
constexpr uint32_t kTcBins = 33u * 64u;     // classes: exponent and 6 mantissa bits
constexpr uint32_t kTcLabelChunk = 4096;    // vertices per CTA

__device__ __forceinline__ uint32_t tc_bin(uint32_t deg) {
	// the float's exponent and top mantissa bits grow with the degree
	return deg ? (__float_as_uint((float)deg) >> 17) - (127u << 6) : 0u;
}

__device__ __forceinline__ uint32_t tc_degree(const uint32_t* out_deg, const uint32_t* in_deg,
		uint64_t v) {
	return __ldg(out_deg + v) + (in_deg ? __ldg(in_deg + v) : 0u);
}

__global__ void __launch_bounds__(kTcThreads)
tc_bins(const uint32_t* out_deg, const uint32_t* in_deg, uint64_t V, uint32_t* hist) {
	__shared__ uint32_t h[kTcBins];
	for (uint32_t b = threadIdx.x; b < kTcBins; b += kTcThreads) h[b] = 0;
	__syncthreads();
	for (uint64_t v = (uint64_t)blockIdx.x * kTcThreads + threadIdx.x; v < V;
			v += (uint64_t)gridDim.x * kTcThreads)
		atomicAdd(h + tc_bin(tc_degree(out_deg, in_deg, v)), 1u);
	__syncthreads();
	for (uint32_t b = threadIdx.x; b < kTcBins; b += kTcThreads)
		if (h[b]) atomicAdd(hist + b, h[b]);
}

// hist[b] <- number of vertices in the classes above b (one CTA).
__global__ void __launch_bounds__(1024)
tc_bin_starts(uint32_t* hist) {
	__shared__ uint32_t wsum[32];
	const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
	uint32_t carry = 0;
	for (uint32_t b0 = 0; b0 < kTcBins; b0 += 1024) {
		const uint32_t i = b0 + threadIdx.x;
		const uint32_t b = kTcBins - 1u - i;         // highest class first
		const uint32_t x = i < kTcBins ? hist[b] : 0u;
		uint32_t inc = x;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
			if (lane >= (uint32_t)o) inc += y;
		}
		if (lane == 31u) wsum[wid] = inc;
		__syncthreads();
		uint32_t before = carry, all = 0;
		for (uint32_t w = 0; w < 32; w++) {
			if (w < wid) before += wsum[w];
			all += wsum[w];
		}
		if (i < kTcBins) hist[b] = before + inc - x;
		carry += all;
		__syncthreads();
	}
}

// label[v] from the class's next free place; a CTA takes the places of its
// vertices with one atomic per class.
__global__ void __launch_bounds__(kTcThreads)
tc_labels(const uint32_t* out_deg, const uint32_t* in_deg, uint64_t V, uint32_t* cursor,
		uint32_t* label) {
	constexpr int kPer = kTcLabelChunk / kTcThreads;
	__shared__ uint32_t cnt[kTcBins];
	for (uint32_t b = threadIdx.x; b < kTcBins; b += kTcThreads) cnt[b] = 0;
	__syncthreads();
	uint32_t bin[kPer], at[kPer];
#pragma unroll
	for (int j = 0; j < kPer; j++) {
		const uint64_t v = (uint64_t)blockIdx.x * kTcLabelChunk + j * kTcThreads + threadIdx.x;
		bin[j] = kTcBins;
		at[j] = 0;
		if (v < V) {
			bin[j] = tc_bin(tc_degree(out_deg, in_deg, v));
			at[j] = atomicAdd(cnt + bin[j], 1u);
		}
	}
	__syncthreads();
	for (uint32_t b = threadIdx.x; b < kTcBins; b += kTcThreads)
		if (cnt[b]) cnt[b] = atomicAdd(cursor + b, cnt[b]);
	__syncthreads();
#pragma unroll
	for (int j = 0; j < kPer; j++) {
		const uint64_t v = (uint64_t)blockIdx.x * kTcLabelChunk + j * kTcThreads + threadIdx.x;
		if (v < V) label[v] = cnt[bin[j]] + at[j];
	}
}

// ---------------------------------------------------------------------------
// Forward lists
// ---------------------------------------------------------------------------

// Key of every edge of the flat out-CSR, in edge order (lane j of the warp
// owning tile t takes edges 256 t + 8 j .. + 7): a << bits | b with a > b the
// labels of its ends.  Self-loops get the key V << bits, which sorts last,
// and are counted in *loops.
constexpr int kTcEmitWarps = 8;
__global__ void __launch_bounds__(kTcEmitWarps * 32)
tc_emit(const uint32_t* ids, const uint32_t* heads, const uint32_t* nz_rows,
		const uint32_t* tile_seg, uint32_t E, uint32_t ntiles, const uint32_t* label, int bits,
		u64 loop_key, u64* keys, u64* loops) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t t = blockIdx.x * kTcEmitWarps + (threadIdx.x >> 5);
	if (t >= ntiles) return;
	const uint32_t eb = t * kFlatTile + lane * kFlatPerLane;
	const uint32_t hb = __ldg(reinterpret_cast<const unsigned char*>(heads)
			+ (size_t)t * (kFlatTile / 8) + lane);
	uint32_t id[kFlatPerLane];
#pragma unroll
	for (int i = 0; i < kFlatPerLane; i++) id[i] = kNoId;
	if (eb + kFlatPerLane <= E) {
		const uint4 x = __ldcs(reinterpret_cast<const uint4*>(ids + eb));
		const uint4 y = __ldcs(reinterpret_cast<const uint4*>(ids + eb + 4));
		id[0] = x.x; id[1] = x.y; id[2] = x.z; id[3] = x.w;
		id[4] = y.x; id[5] = y.y; id[6] = y.z; id[7] = y.w;
	} else {
#pragma unroll
		for (int i = 0; i < kFlatPerLane; i++)
			if (eb + i < E) id[i] = __ldcs(ids + eb + i);
	}
	uint32_t ln[kFlatPerLane];
#pragma unroll
	for (int i = 0; i < kFlatPerLane; i++) ln[i] = id[i] != kNoId ? __ldg(label + id[i]) : 0u;
	uint32_t before = __popc(hb);               // heads in the lanes to the left
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t q = __shfl_up_sync(0xffffffffu, before, o);
		if (lane >= (uint32_t)o) before += q;
	}
	before -= __popc(hb);
	uint32_t row = __ldg(tile_seg + t) + before - 1u;   // of the lane's first edge, unless a head
	uint32_t ls = 0;
	if (eb < E && !(hb & 1u)) ls = __ldg(label + __ldg(nz_rows + row));
	uint32_t nl = 0;
	u64 k[kFlatPerLane];
#pragma unroll
	for (int i = 0; i < kFlatPerLane; i++) {
		if ((hb >> i) & 1u) {
			row++;
			ls = __ldg(label + __ldg(nz_rows + row));
		}
		const bool loop = ls == ln[i];
		nl += (id[i] != kNoId && loop) ? 1u : 0u;
		k[i] = loop ? loop_key : ((u64)max(ls, ln[i]) << bits) | min(ls, ln[i]);
	}
	if (eb + kFlatPerLane <= E) {
#pragma unroll
		for (int i = 0; i < kFlatPerLane; i += 2)
			*reinterpret_cast<ulonglong2*>(keys + eb + i) = make_ulonglong2(k[i], k[i + 1]);
	} else {
#pragma unroll
		for (int i = 0; i < kFlatPerLane; i++)
			if (eb + i < E) keys[eb + i] = k[i];
	}
	nl = __reduce_add_sync(0xffffffffu, nl);
	if (lane == 0 && nl) atomicAdd(loops, (u64)nl);
}

// The distinct keys in two passes over tiles of kUqTile sorted keys: the
// number of first occurrences per tile, then (after a scan of those) the
// lists themselves.  Keys at or above `end` (the self-loops) are left out.
constexpr int kUqPer = 8;
constexpr uint32_t kUqTile = (uint32_t)kTcThreads * kUqPer;

__global__ void __launch_bounds__(kTcThreads)
tc_uniq_count(const u64* keys, uint64_t n, u64 end, uint32_t* tile_cnt) {
	__shared__ uint32_t s_sum;
	if (threadIdx.x == 0) s_sum = 0;
	__syncthreads();
	const uint64_t base = (uint64_t)blockIdx.x * kUqTile;
	uint32_t c = 0;
#pragma unroll
	for (int j = 0; j < kUqPer; j++) {
		const uint64_t i = base + (uint64_t)j * kTcThreads + threadIdx.x;
		if (i < n) {
			const u64 k = keys[i];
			c += k < end && (i == 0 || keys[i - 1] != k);
		}
	}
	c = __reduce_add_sync(0xffffffffu, c);
	if ((threadIdx.x & 31u) == 0 && c) atomicAdd(&s_sum, c);
	__syncthreads();
	if (threadIdx.x == 0) tile_cnt[blockIdx.x] = s_sum;
}

// adj = the targets of the distinct keys; cnt[a] = length of N+(a) (formed as
// end - start of a's run, each added where the run begins or ends).
__global__ void __launch_bounds__(kTcThreads)
tc_uniq_write(const u64* keys, uint64_t n, u64 end, int bits, const uint32_t* tile_pos,
		uint32_t* adj, uint32_t* cnt) {
	__shared__ uint32_t wsum[kTcThreads / 32];
	const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
	const uint64_t base = (uint64_t)blockIdx.x * kUqTile;
	const u64 low = (1ull << bits) - 1ull;
	uint32_t run = __ldg(tile_pos + blockIdx.x);
	for (int j = 0; j < kUqPer; j++) {
		const uint64_t i = base + (uint64_t)j * kTcThreads + threadIdx.x;
		u64 k = end, p = end;
		if (i < n) {
			k = keys[i];
			if (i > 0) p = keys[i - 1];
		}
		const bool first = k < end && (i == 0 || p != k);
		const unsigned m = __ballot_sync(0xffffffffu, first);
		if (lane == 0) wsum[wid] = __popc(m);
		__syncthreads();
		uint32_t pos = run, all = 0;
		for (uint32_t w = 0; w < kTcThreads / 32; w++) {
			if (w < wid) pos += wsum[w];
			all += wsum[w];
		}
		pos += __popc(m & ((1u << lane) - 1u));
		if (first) adj[pos] = (uint32_t)(k & low);
		if (i < n) {
			// a run of equal a begins at key i (and the run before it ends)
			const bool begin = k < end && (i == 0 || (p >> bits) != (k >> bits));
			if (begin) atomicSub(cnt + (k >> bits), pos);
			if (i > 0 && p < end && (begin || k >= end)) atomicAdd(cnt + (p >> bits), pos);
			if (i == n - 1 && k < end) atomicAdd(cnt + (k >> bits), pos + (first ? 1u : 0u));
		}
		run += all;
		__syncthreads();
	}
}

// ---------------------------------------------------------------------------
// Counting
// ---------------------------------------------------------------------------

__device__ __forceinline__ bool bsearch_u32(const uint32_t* base, uint32_t n, uint32_t x) {
	uint32_t lo = 0, hi = n;
	while (lo < hi) {
		const uint32_t mid = (lo + hi) >> 1;
		const uint32_t y = __ldg(base + mid);
		if (y < x) lo = mid + 1; else hi = mid;
	}
	return lo < n && __ldg(base + lo) == x;
}

// Vertices by the length la of N+(a) and the label a:
//   la <= kTcPairs         one thread looks up every pair of the list
//   a < kTcDomain0         list 0: two warps with a bitmap of kTcDomain0 labels
//   la <= kTcHashMost      list 1: a warp with a hash table of N+(a)
//   a < kTcDomain1, 2      list 2, 3: a CTA with a bitmap of so many labels
//   else                   list 4: a warp looks up every pair
// A pair (c, b) is looked up by a binary search of c in N+(b): up to eight
// ids that is 28 searches at most, against eight lists of some 200 ids to
// stream (the same holds for the first eight ids of a longer list, whose
// pairs one warp looks up at once).  The hash table costs twice a bitmap's
// instructions per id, but no barriers between the four warps that would share
// a larger bitmap: 99 k vertices with 9 to 64 ids took them 842 us against
// 240.  Two warps per 8 KB bitmap keep 48 resident on an SM (one: 24, 610 us
// against 476; four: 477, and slower with two rows in flight, 516 against 417).
constexpr uint32_t kTcPairs = 8;
constexpr int kTcLists = 5;
constexpr uint32_t kTcDomain0 = 1u << 16;     //   8 KB per bitmap: two warps
constexpr uint32_t kTcDomain1 = 1u << 18;     //  32 KB: four warps
constexpr uint32_t kTcDomain2 = 7u << 18;     // 224 KB: a CTA of 32 warps, one per SM
constexpr uint32_t kTcHashMost = 64;          // a quarter of the table's slots
constexpr uint32_t kTcHashBits = 8;

__global__ void __launch_bounds__(kTcThreads)
tc_classify(uint32_t V, const uint32_t* off, const uint32_t* adj, uint32_t* lists, u64* ctr,
		u64* total) {
	const uint32_t a = blockIdx.x * kTcThreads + threadIdx.x;
	uint32_t sa = 0, la = 0;
	if (a < V) {
		sa = __ldg(off + a);
		la = __ldg(off + a + 1) - sa;
	}
	uint32_t c = 0;
	if (la >= 2 && la <= kTcPairs) {
		for (uint32_t j = 1; j < la; j++) {
			const uint32_t b = __ldg(adj + sa + j);
			const uint32_t sb = __ldg(off + b), lb = __ldg(off + b + 1) - sb;
			if (lb == 0) continue;
			for (uint32_t i = 0; i < j; i++) c += bsearch_u32(adj + sb, lb, __ldg(adj + sa + i));
		}
	}
	c = __reduce_add_sync(0xffffffffu, c);
	if ((threadIdx.x & 31u) == 0 && c) atomicAdd(total, (u64)c);
	const int cls = la <= kTcPairs ? -1 : a < kTcDomain0 ? 0 : la <= kTcHashMost ? 1
			: a < kTcDomain1 ? 2 : a < kTcDomain2 ? 3 : 4;
	// (a CTA's labels do not straddle a bound between the bitmaps)
	const uint64_t a0 = (uint64_t)blockIdx.x * kTcThreads;
	const int wide = a0 < kTcDomain1 ? 2 : a0 < kTcDomain2 ? 3 : 4;
	if (a0 < kTcDomain0) {
		block_push<kTcThreads>(cls == 0, a, lists, ctr);
		return;
	}
	block_push<kTcThreads>(cls == 1, a, lists + V, ctr + 1);
	__syncthreads();
	block_push<kTcThreads>(cls == wide, a, lists + (size_t)wide * V, ctr + wide);
}

// Pairs (i, j), i < j, of the first eight ids of N+(a) = adj[sa ...): lane =
// pair; returns whether the lane's two are adjacent.
__device__ __forceinline__ uint32_t tc_first_pairs(const uint32_t* off, const uint32_t* adj,
		uint32_t sa) {
	const uint32_t lane = threadIdx.x & 31u;
	if (lane >= kTcPairs * (kTcPairs - 1) / 2) return 0;
	uint32_t j = 1, i = lane;
	while (i >= j) { i -= j; j++; }
	const uint32_t b = __ldg(adj + sa + j), x = __ldg(adj + sa + i);
	const uint32_t sb = __ldg(off + b), lb = __ldg(off + b + 1) - sb;
	return bsearch_u32(adj + sb, lb, x);
}

// N+(b) of b < kTcRows as a row of bits, where that is the cheaper form: half
// a warp takes 2048 labels of a row at a time and a quarter 32 ids of a list,
// with bank conflicts (so from an eighth of an id per word on; a quarter: 418
// against 410 us).
constexpr uint32_t kTcRows = 8192;
constexpr uint32_t kTcRowWords = kTcRows / 32;

__device__ __forceinline__ bool tc_has_row(uint32_t b, uint32_t lb) {
	return b < kTcRows && 4u * lb > (b >> 5) + 32u;
}

// rows[b] <- the bits of N+(b), for every b that has a row: a warp each.
__global__ void __launch_bounds__(kTcThreads)
tc_rows(uint32_t n, const uint32_t* off, const uint32_t* adj, uint32_t* rows) {
	__shared__ uint32_t bits[kTcThreads / 32][kTcRowWords];
	uint32_t* w = bits[threadIdx.x >> 5];
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t b = blockIdx.x * (kTcThreads / 32) + (threadIdx.x >> 5);
	if (b >= n) return;
	const uint32_t sb = __ldg(off + b), lb = __ldg(off + b + 1) - sb;
	if (!tc_has_row(b, lb)) return;
	const uint32_t nw = (b + 127u) >> 7 << 2;             // whole 16-byte words
	for (uint32_t i = lane; i < nw; i += 32) w[i] = 0;
	__syncwarp();
	for (uint32_t i = lane; i < lb; i += 32) {
		const uint32_t x = __ldg(adj + sb + i);
		atomicOr(w + (x >> 5), 1u << (x & 31u));
	}
	__syncwarp();
	uint32_t* row = rows + (size_t)b * kTcRowWords;
	for (uint32_t i = lane; i < nw; i += 32) row[i] = w[i];
}

// sum of |N+(b) & N+(a)| over the nb <= 32 ids b of adj[first ...): bm holds the
// labels below kTcRows of N+(a) as bits, in(x) = 1 if x is in N+(a).  Half a warp
// takes a row (2048 labels a step), a quarter a list (32 ids a step): most visits
// end within a step, so it is the instructions per visit and the loads in flight
// that count (whole warps: 676 us against 610, a row at a time 476 against 417).
// Neighbouring ids b, alike in their lengths, go to different parts of the warp.
template <class In>
__device__ __forceinline__ uint32_t tc_lists(const uint32_t* off, const uint32_t* adj,
		const uint4* rows, uint32_t first, uint32_t nb, const uint32_t* bm, In&& in) {
	const uint32_t lane = threadIdx.x & 31u;
	uint32_t b = 0, s = 0, n = 0, c = 0;
	if (lane < nb) {
		b = __ldg(adj + first + lane);
		s = __ldg(off + b);
		n = __ldg(off + b + 1) - s;
	}
	const bool row = tc_has_row(b, n);
	uint32_t m = __ballot_sync(0xffffffffu, row) & (0x55555555u << (lane >> 4));
	while (__any_sync(0xffffffffu, m != 0)) {
		const uint4* w = (const uint4*)bm;
		const uint4* p[2];
		uint32_t len[2];
#pragma unroll
		for (int i = 0; i < 2; i++) {
			const uint32_t q = __shfl_sync(0xffffffffu, b, m ? __ffs(m) - 1 : 0);
			len[i] = m ? (q + 127u) >> 7 : 0u;
			p[i] = rows + (size_t)q * (kTcRowWords / 4);
			m &= m - 1u;
		}
		for (uint32_t k = lane & 15u; k < max(len[0], len[1]); k += 16) {
			uint4 x[2];
#pragma unroll
			for (int i = 0; i < 2; i++)
				x[i] = k < len[i] ? __ldg(p[i] + k) : make_uint4(0, 0, 0, 0);
			const uint4 u = w[k];
#pragma unroll
			for (int i = 0; i < 2; i++)
				c += __popc(x[i].x & u.x) + __popc(x[i].y & u.y) + __popc(x[i].z & u.z)
						+ __popc(x[i].w & u.w);
		}
	}
	m = __ballot_sync(0xffffffffu, n != 0 && !row) & (0x11111111u << (lane >> 3));
	while (__any_sync(0xffffffffu, m != 0)) {
		constexpr int kAhead = 4;
		const uint32_t q = m ? __ffs(m) - 1 : 0;
		const uint32_t* p = adj + __shfl_sync(0xffffffffu, s, q);
		const uint32_t l = __shfl_sync(0xffffffffu, n, q);
		const uint32_t len = m ? l : 0u;
		m &= m - 1u;
		for (uint32_t k = lane & 7u; k < len; k += 8u * kAhead) {
			uint32_t x[kAhead];
#pragma unroll
			for (int u = 0; u < kAhead; u++) x[u] = k + 8u * u < len ? __ldg(p + k + 8u * u) : kNoId;
#pragma unroll
			for (int u = 0; u < kAhead; u++)
				if (x[u] != kNoId) c += in(x[u]);
		}
	}
	return c;
}

// A warp per vertex of its list (taken from a ticket counter): N+(a), at most
// kTcHashMost ids, in a hash table of 2^kTcHashBits slots (open addressing).
__global__ void __launch_bounds__(kTcThreads)
tc_hash(const uint32_t* list, const u64* n_list, u64* ticket, const uint32_t* off,
		const uint32_t* adj, const uint4* rows, u64* total) {
	constexpr uint32_t kSlots = 1u << kTcHashBits;
	__shared__ uint32_t tab[kTcThreads / 32][kSlots];
	__shared__ __align__(16) uint32_t bits[kTcThreads / 32][kTcRowWords];
	uint32_t* t = tab[threadIdx.x >> 5];
	uint32_t* bm = bits[threadIdx.x >> 5];
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t n = (uint32_t)__ldg(n_list);
	auto slot = [](uint32_t x) { return (x * 2654435769u) >> (32u - kTcHashBits); };
	u64 sum = 0;
	for (uint32_t i = lane; i < kTcRowWords; i += 32) bm[i] = 0;
	for (;;) {
		uint32_t k = 0;
		if (lane == 0) k = (uint32_t)atomicAdd(ticket, 1ull);
		k = __shfl_sync(0xffffffffu, k, 0);
		if (k >= n) break;
		const uint32_t a = __ldg(list + k);
		const uint32_t sa = __ldg(off + a), la = __ldg(off + a + 1) - sa;
		for (uint32_t i = lane; i < kSlots; i += 32) t[i] = kNoId;
		__syncwarp();
		for (uint32_t i = lane; i < la; i += 32) {
			const uint32_t x = __ldg(adj + sa + i);
			uint32_t h = slot(x);
			while (atomicCAS(t + h, kNoId, x) != kNoId) h = (h + 1u) & (kSlots - 1u);
			if (x < kTcRows) atomicOr(bm + (x >> 5), 1u << (x & 31u));
		}
		__syncwarp();
		uint32_t c = tc_first_pairs(off, adj, sa);
		for (uint32_t j = kTcPairs; j < la; j += 32)
			c += tc_lists(off, adj, rows, sa + j, min(32u, la - j), bm, [&](uint32_t x) {
				uint32_t h = slot(x), y = t[h];
				while (y != x && y != kNoId) {
					h = (h + 1u) & (kSlots - 1u);
					y = t[h];
				}
				return y == x ? 1u : 0u;
			});
		sum += c;
		__syncwarp();
		for (uint32_t i = lane; i < la; i += 32) {
			const uint32_t x = __ldg(adj + sa + i);
			if (x < kTcRows) bm[x >> 5] = 0;
		}
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
	if (lane == 0 && sum) atomicAdd(total, sum);
}

// A CTA of kWarps warps takes the vertices of its list one after the other
// (from a ticket counter), marks N+(a) in the bitmap and streams N+(b) of
// every b but the first eight, a list per warp.
template <int kWarps>
__global__ void __launch_bounds__(kWarps * 32)
tc_bitmap(const uint32_t* list, const u64* n_list, u64* ticket, const uint32_t* off,
		const uint32_t* adj, const uint4* rows, uint32_t words, u64* total) {
	extern __shared__ __align__(16) uint32_t bm[];
	__shared__ uint32_t s_next;
	constexpr uint32_t kBatch = kWarps < 32 ? 16u : 8u;   // lists a warp takes at a time
	const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
	const uint32_t n = (uint32_t)__ldg(n_list);
	if (n == 0) return;
	for (uint32_t w = tid; w < words; w += kWarps * 32) bm[w] = 0;
	u64 sum = 0;
	for (;;) {
		if (tid == 0) s_next = (uint32_t)atomicAdd(ticket, 1ull);
		__syncthreads();
		const uint32_t t = s_next;
		if (t >= n) break;
		const uint32_t a = __ldg(list + t);
		const uint32_t sa = __ldg(off + a), la = __ldg(off + a + 1) - sa;
		for (uint32_t i = tid; i < la; i += kWarps * 32) {
			const uint32_t x = __ldg(adj + sa + i);
			atomicOr(bm + (x >> 5), 1u << (x & 31u));
		}
		__syncthreads();
		uint32_t c = wid == kWarps - 1 ? tc_first_pairs(off, adj, sa) : 0u;
		for (uint32_t j = kTcPairs + wid * kBatch; j < la; j += kWarps * kBatch)
			c += tc_lists(off, adj, rows, sa + j, min(kBatch, la - j), bm, [&](uint32_t x) {
				return (bm[x >> 5] >> (x & 31u)) & 1u;
			});
		sum += c;
		__syncthreads();
		for (uint32_t i = tid; i < la; i += kWarps * 32) bm[__ldg(adj + sa + i) >> 5] = 0;
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
	if (lane == 0 && sum) atomicAdd(total, sum);
}

// The vertices whose label no bitmap holds: a warp each, the searches of one
// b's pairs 32 at a time.
__global__ void __launch_bounds__(kTcThreads)
tc_search(const uint32_t* list, const u64* n_list, const uint32_t* off, const uint32_t* adj,
		u64* total) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t nwarps = gridDim.x * (kTcThreads / 32);
	const uint32_t n = (uint32_t)__ldg(n_list);
	u64 c = 0;
	for (uint32_t t = blockIdx.x * (kTcThreads / 32) + (threadIdx.x >> 5); t < n; t += nwarps) {
		const uint32_t a = __ldg(list + t);
		const uint32_t sa = __ldg(off + a), la = __ldg(off + a + 1) - sa;
		for (uint32_t j = 1; j < la; j++) {
			const uint32_t b = __ldg(adj + sa + j);
			const uint32_t sb = __ldg(off + b), lb = __ldg(off + b + 1) - sb;
			if (lb == 0) continue;
			for (uint32_t i = lane; i < j; i += 32)
				c += bsearch_u32(adj + sb, lb, __ldg(adj + sa + i));
		}
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
	if (lane == 0 && c) atomicAdd(total, c);
}

} // namespace lg

using namespace lg;

namespace {

// One bitmap class: kWarps warps per CTA, as many CTAs as are resident.
template <int kWarps>
lg_status launch_bitmap(lg_store* s, int sms, uint32_t domain, const uint32_t* list, u64* n_list,
		u64* ticket, const uint32_t* off, const uint32_t* adj, const uint4* rows, u64* total) {
	const uint32_t words = (domain + 127u) / 128u * 4u;   // rows are read by 16 bytes
	const size_t smem = (size_t)words * 4;
	LG_CUDA(cudaFuncSetAttribute(tc_bitmap<kWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize,
			(int)smem), "tc_bitmap");
	int per_sm = 0;
	LG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tc_bitmap<kWarps>, kWarps * 32,
			smem), "tc_bitmap");
	if (per_sm < 1) return set_error(LG_ECUDA, "tc_bitmap does not fit an SM");
	tc_bitmap<kWarps><<<(unsigned)(sms * per_sm), kWarps * 32, smem, s->stream>>>(list, n_list,
			ticket, off, adj, rows, words, total);
	LG_CUDA(cudaGetLastError(), "tc_bitmap");
	s->launches++;
	return LG_OK;
}

} // namespace

extern "C" lg_status lg_triangle_count(lg_snapshot* sn, lg_tc_result* result) {
	clear_error();
	if (!sn || !result) return set_error(LG_EINVAL, "null argument");
	lg_store* s = sn->store;
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	cudaStream_t st = s->stream;
	const uint64_t V = sn->V;
	if (sn->out.n_edges >= 0xffffffffull)
		return set_error(LG_ENOTSUP, "more than 2^32-1 live edges");
	result->triangles = 0;
	result->undirected_edges = 0;
	result->arcs = 0;
	// the live arcs: the snapshot's flat out-CSR, or one built for the call
	const FlatCsr* f = sn->flat[0];
	if (!f) {
		if (!s->flat_scratch) s->flat_scratch = new FlatCsr;
		LG_TRY(build_flat(sn, 0, *s->flat_scratch, false, false, false));
		f = s->flat_scratch;
	}
	const uint64_t E = f->E;
	if (E == 0) return LG_OK;
	DevBuf label(s->pool), hist(s->pool), keys(s->pool), tmpk(s->pool), tmpp(s->pool),
			counts(s->pool), scan_tmp(s->pool), tiles(s->pool), off(s->pool), ctr(s->pool),
			adj(s->pool), lists(s->pool), rows(s->pool);
	int sms = 148;
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
	// ctr: [0..4] list sizes, [5..8] tickets, [9] self-loops, [10] triangles
	LG_TRY(ctr.reserve(11 * sizeof(u64)));
	u64* cd = ctr.as<u64>();
	LG_CUDA(cudaMemsetAsync(cd, 0, 11 * sizeof(u64), st), "memset");
	const uint32_t* odeg = sn->out.deg.as<uint32_t>();
	const uint32_t* ideg = sn->in.present ? sn->in.deg.as<uint32_t>() : nullptr;
	LG_TRY(label.reserve(V * 4));
	LG_TRY(hist.reserve(kTcBins * 4));
	LG_CUDA(cudaMemsetAsync(hist.p, 0, kTcBins * 4, st), "memset");
	tc_bins<<<std::min(grid_for(V, kTcLabelChunk), (unsigned)sms * 4u), kTcThreads, 0, st>>>(odeg,
			ideg, V, hist.as<uint32_t>());
	tc_bin_starts<<<1, 1024, 0, st>>>(hist.as<uint32_t>());
	tc_labels<<<grid_for(V, kTcLabelChunk), kTcThreads, 0, st>>>(odeg, ideg, V,
			hist.as<uint32_t>(), label.as<uint32_t>());
	// keys a << bits | b; V itself (the self-loops' a) fits the bits too
	int bits = 1;
	while ((V >> bits) != 0) bits++;
	const u64 loop_key = (u64)V << bits;
	LG_TRY(keys.reserve(E * 8));
	tc_emit<<<grid_for(f->ntiles, kTcEmitWarps), kTcEmitWarps * 32, 0, st>>>(f->ids.as<uint32_t>(),
			f->heads(), f->nz_rows(), f->tile_seg(), (uint32_t)E, f->ntiles, label.as<uint32_t>(),
			bits, loop_key, keys.as<u64>(), cd + 9);
	LG_CUDA(cudaGetLastError(), "tc_emit");
	s->launches += 4;
	u64* sorted = nullptr;
	auto sort = [&]() {
		return radix_sort_u64(s, keys.as<u64>(), nullptr, E, tmpk, tmpp, counts, scan_tmp, &sorted,
				nullptr, bits < 32 ? (1ull << (2 * bits)) - 1ull : ~0ull);
	};
	lg_status sorted_ok = sort();
	if (sorted_ok == LG_ENOMEM && f == s->flat_scratch) {
		// with what the flat copy took: the keys hold the edges now
		clear_error();
		LG_CUDA(cudaStreamSynchronize(st), "triangles");
		f = nullptr;
		delete s->flat_scratch;
		s->flat_scratch = nullptr;
		sorted_ok = sort();
	}
	LG_TRY(sorted_ok);
	const unsigned uq_tiles = grid_for(E, kUqTile);
	LG_TRY(tiles.reserve((2ull * uq_tiles + 1) * 4));
	uint32_t* tile_cnt = tiles.as<uint32_t>();
	uint32_t* tile_pos = tile_cnt + uq_tiles;
	tc_uniq_count<<<uq_tiles, kTcThreads, 0, st>>>(sorted, E, loop_key, tile_cnt);
	LG_CUDA(cudaGetLastError(), "tc_uniq_count");
	uint64_t m = 0;
	LG_TRY(exclusive_scan_u32(tile_cnt, tile_pos, uq_tiles, scan_tmp, st, &m));
	LG_TRY(adj.reserve(std::max<uint64_t>(m, 1) * 4));
	LG_TRY(off.reserve((2 * V + 1) * 4));
	uint32_t* fcnt = off.as<uint32_t>();
	uint32_t* foff = fcnt + V;
	LG_CUDA(cudaMemsetAsync(fcnt, 0, V * 4, st), "memset");
	tc_uniq_write<<<uq_tiles, kTcThreads, 0, st>>>(sorted, E, loop_key, bits, tile_pos,
			adj.as<uint32_t>(), fcnt);
	LG_CUDA(cudaGetLastError(), "tc_uniq_write");
	LG_TRY(exclusive_scan_u32(fcnt, foff, V, scan_tmp, st, nullptr));
	LG_TRY(lists.reserve(kTcLists * V * 4));
	uint32_t* ls = lists.as<uint32_t>();
	const uint32_t* ad = adj.as<uint32_t>();
	u64* found = cd + 10;
	tc_classify<<<grid_for(V, kTcThreads), kTcThreads, 0, st>>>((uint32_t)V, foff, ad, ls, cd,
			found);
	LG_CUDA(cudaGetLastError(), "tc_classify");
	const uint32_t nr = (uint32_t)std::min<uint64_t>(V, kTcRows);
	LG_TRY(rows.reserve((size_t)nr * kTcRowWords * 4));
	tc_rows<<<grid_for(nr, kTcThreads / 32), kTcThreads, 0, st>>>(nr, foff, ad,
			rows.as<uint32_t>());
	LG_CUDA(cudaGetLastError(), "tc_rows");
	s->launches += 4 + scan_launches(uq_tiles) + scan_launches(V);
	LG_TRY(launch_bitmap<2>(s, sms, (uint32_t)std::min<uint64_t>(V, kTcDomain0), ls, cd, cd + 5,
			foff, ad, rows.as<uint4>(), found));
	if (V > kTcDomain0) {
		tc_hash<<<(unsigned)sms * 8u, kTcThreads, 0, st>>>(ls + V, cd + 1, cd + 6, foff, ad,
				rows.as<uint4>(), found);
		LG_CUDA(cudaGetLastError(), "tc_hash");
		s->launches++;
		LG_TRY(launch_bitmap<4>(s, sms, (uint32_t)std::min<uint64_t>(V, kTcDomain1), ls + 2 * V,
				cd + 2, cd + 7, foff, ad, rows.as<uint4>(), found));
	}
	if (V > kTcDomain1)
		LG_TRY(launch_bitmap<32>(s, sms, (uint32_t)std::min<uint64_t>(V, kTcDomain2), ls + 3 * V,
				cd + 3, cd + 8, foff, ad, rows.as<uint4>(), found));
	if (V > kTcDomain2) {
		tc_search<<<(unsigned)sms * 8u, kTcThreads, 0, st>>>(ls + 4 * V, cd + 4, foff, ad, found);
		LG_CUDA(cudaGetLastError(), "tc_search");
		s->launches++;
	}
	u64 h[2] = {0, 0};
	LG_TRY(read_words(s, cd + 9, 2, h));
	result->triangles = (int64_t)h[1];
	result->undirected_edges = m;
	result->arcs = E - h[0];
	return LG_OK;
}
