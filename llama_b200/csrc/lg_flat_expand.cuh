// lg_flat_expand.cuh - a warp's walk over the rows of a few vertices of a
// flat CSR (one array of ids, row starts in `off`).
//
// Every lane brings one row (start and length, 0 for none).  The rows' edges,
// one after the other, are taken 32 at a time: the rows that begin inside a
// chunk are bits of one word (a reduction over the lanes), so an edge's row is
// a population count away, and the row's values come from shared memory.  The
// loads of kFeAhead chunks are issued before any of them is used.  Compared
// with the walk over fragments (lg_expand.cuh) an edge costs no search for its
// owner (5 shuffles), no fragment record and no deletion word.
#ifndef LG_FLAT_EXPAND_CUH_
#define LG_FLAT_EXPAND_CUH_

#include <cuda_runtime.h>
#include <stdint.h>

namespace lg {

constexpr int kFeAhead = 4;

// A warp's shared memory: per non-empty row, its edges' array position minus
// their position in the walk, and a value of the caller's.
struct RowWindow {
	uint2 row[32];
};

// Walks the rows of the calling warp's lanes, kFeAhead chunks of 32 edges at a
// time: load(u, active, edge, value) for every chunk u (edge: its position in
// the flat arrays, value: the one the edge's lane brought), then use() for the
// loaded chunks; the next chunks' loads are issued between take(), which sets
// the loaded ones aside, and use().  All run on all lanes, so they may use
// warp collectives.
template <class Load, class Take, class Use>
__device__ __forceinline__ void flat_expand(RowWindow* sw, uint32_t start, uint32_t len,
		uint32_t value, Load&& load, Take&& take, Use&& use) {
	const uint32_t lane = threadIdx.x & 31u;
	uint32_t inc = len;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
		if (lane >= (uint32_t)o) inc += y;
	}
	const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
	const uint32_t at = inc - len;
	// empty rows drop out: lane i keeps the i-th non-empty row's position
	const unsigned ne = __ballot_sync(0xffffffffu, len != 0);
	const uint32_t rank = __popc(ne & ((1u << lane) - 1u));
	__syncwarp();
	if (len != 0) sw->row[rank] = make_uint2(at, 0u);
	__syncwarp();
	const uint32_t first = lane < (uint32_t)__popc(ne) ? sw->row[lane].x : 0xffffffffu;
	__syncwarp();
	if (len != 0) sw->row[rank] = make_uint2(start - at, value);
	__syncwarp();
	const uint32_t upto = (2u << lane) - 1u;
	auto fetch = [&](uint32_t base) {
#pragma unroll
		for (int u = 0; u < kFeAhead; u++) {
			const uint32_t c = base + u * 32u;
			const uint32_t rel = first - c;
			const uint32_t begun = __popc(__ballot_sync(0xffffffffu, first <= c));
			const uint32_t mask = __reduce_or_sync(0xffffffffu,
					first > c && rel < 32u ? 1u << rel : 0u);
			const uint2 r = sw->row[begun - 1u + __popc(mask & upto)];
			load(u, c + lane < total, c + lane + r.x, r.y);
		}
	};
	if (total == 0) return;
	fetch(0);
	for (uint32_t base = 0; base < total;) {
		take();
		base += 32u * kFeAhead;
		if (base < total) fetch(base);
		use();
	}
}

} // namespace lg

#endif // LG_FLAT_EXPAND_CUH_
