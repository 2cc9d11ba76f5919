// lg_ppr_walk.cu - personalized PageRank over the levels' fragments, for where
// there is no memory for the flat in-CSR that lg_ppr.cu reads, or more live
// edges than it can hold.
//
// Warps take fixed ranges of the in-CSR's slot space (lg_expand.cuh); the 32
// edges of a chunk are handled one after another by the whole warp, whose lane j
// owns columns j, j + 32, ...  One row load per lane is in flight, so it takes
// some five times as long as the flat form.  Rows of vertices that straddle
// ranges are combined in range order by ppr_walk_fixup.
#include "lg_expand.cuh"
#include "lg_ppr.h"
#include "lg_tune.h"

#include <algorithm>

namespace lg {

namespace {

constexpr int kWalkThreads = 256;

struct WalkArgs {
	SnapCsr in;
	const uint32_t* pos;
	uint32_t total;
	uint32_t nranges;
	const uint32_t* outdeg;
	const double* y;          // x / out_degree of the previous iteration
	double* y_next;
	double* x_out;            // written on the last iteration (or null)
	double d;
	double tele;              // 1 - d
	const uint32_t* seed_first;   // V: first index into seed_col, or kNoSeed
	const uint2* seed_col;        // (vertex, column) sorted by vertex
	uint32_t n_seeds;
	double* carry_first;      // nranges x K
	double* carry_last;       // nranges x K
	uint32_t K;               // row length of y / x / carries
	uint32_t col0;            // first column of this pass (a K-tile of CPL * 32 columns)
	uint32_t range;           // virtual slots per warp range
};

template <int CPL>
__device__ __forceinline__ void walk_finish(const WalkArgs& a, uint32_t v, const double* s) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t dg = __ldg(a.outdeg + v);
	const uint32_t sf = __ldg(a.seed_first + v);
#pragma unroll
	for (int i = 0; i < CPL; i++) {
		const uint32_t c = a.col0 + lane + 32 * i;
		double t = 0.0;
		if (sf != kNoSeed)
			for (uint32_t q = sf; q < a.n_seeds && a.seed_col[q].x == v; q++)
				if (a.seed_col[q].y == c) t = a.tele;
		const double x = __dadd_rn(t, __dmul_rn(a.d, s[i]));
		a.y_next[(uint64_t)v * a.K + c] = dg ? x / (double)dg : 0.0;
		if (a.x_out) a.x_out[(uint64_t)v * a.K + c] = x;
	}
}

template <int CPL>
__global__ void __launch_bounds__(kWalkThreads)
ppr_walk_step(WalkArgs a) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint64_t r64 = (uint64_t)blockIdx.x * (kWalkThreads / 32) + (threadIdx.x >> 5);
	if (r64 >= a.nranges) return;
	const uint32_t r = (uint32_t)r64;
	const bool last_range = r == a.nranges - 1;
	const uint32_t ra = r * a.range;
	const uint32_t rb = last_range ? a.total : ra + a.range;
	uint32_t e_begin, e_end;
	range_entries(a.pos, (uint32_t)a.in.V, ra, rb, last_range, &e_begin, &e_end);
	const LevelTab* lt = a.in.lt;
	for (uint32_t ew = e_begin; ew < e_end; ew += 32) {
		const Window w = load_window(a.in, nullptr, a.pos, ew, e_end, ra, rb);
		const uint32_t my_end = w.valid ? __ldg(a.pos + w.e + 1) : 0;
		double acc[CPL];
#pragma unroll
		for (int i = 0; i < CPL; i++) acc[i] = 0.0;
		int cur = -1;
		auto flush = [&](int o) {
			const uint32_t st = __shfl_sync(0xffffffffu, w.start, o);
			const uint32_t en = __shfl_sync(0xffffffffu, my_end, o);
			const uint32_t v = __shfl_sync(0xffffffffu, w.v, o);
			if (st < ra) {
#pragma unroll
				for (int i = 0; i < CPL; i++) a.carry_first[(uint64_t)r * a.K + a.col0 + lane + 32 * i] = acc[i];
			} else if (en > rb) {
#pragma unroll
				for (int i = 0; i < CPL; i++) a.carry_last[(uint64_t)r * a.K + a.col0 + lane + 32 * i] = acc[i];
			} else {
				walk_finish<CPL>(a, v, acc);
			}
#pragma unroll
			for (int i = 0; i < CPL; i++) acc[i] = 0.0;
		};
		for (uint32_t base = w.lo; base < w.hi; base += 32) {
			const uint32_t k = base + lane;
			uint32_t own, lv, idx, nb = 0;
			locate_slot(a.in, w, k, &own, &lv, &idx);
			bool act = k < w.hi;
			if (act) {
				const uint32_t word = __ldg(lt->del[lv] + (idx >> 5));
				nb = __ldg(lt->ids[lv] + idx);
				act = !((word >> (idx & 31)) & 1u);
			}
			const unsigned inside = __ballot_sync(0xffffffffu, k < w.hi);
			for (unsigned m = inside; m; m &= m - 1) {
				const int t = __ffs(m) - 1;
				const int o = (int)__shfl_sync(0xffffffffu, own, t);
				const uint32_t src = __shfl_sync(0xffffffffu, nb, t);
				const bool live = __shfl_sync(0xffffffffu, act, t);
				if (o != cur) {
					if (cur >= 0) flush(cur);
					cur = o;
				}
				if (live) {
					const double* row = a.y + (uint64_t)src * a.K + a.col0;
#pragma unroll
					for (int i = 0; i < CPL; i++) acc[i] += __ldg(row + lane + 32 * i);
				}
			}
		}
		if (cur >= 0) flush(cur);
		// entries without slots in the snapshot: teleport term only
		unsigned empty = __ballot_sync(0xffffffffu, w.valid && w.s0 == w.s1);
		for (; empty; empty &= empty - 1) {
			const int o = __ffs(empty) - 1;
			const uint32_t v = __shfl_sync(0xffffffffu, w.v, o);
			double z[CPL];
#pragma unroll
			for (int i = 0; i < CPL; i++) z[i] = 0.0;
			walk_finish<CPL>(a, v, z);
		}
	}
}

// One warp per range boundary: the vertex that starts in range q-1 and
// crosses q * range sums its carried rows in range order.
template <int CPL>
__global__ void ppr_walk_fixup(WalkArgs a) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint64_t q = (uint64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5) + 1;
	if (q >= a.nranges) return;
	const uint32_t s = (uint32_t)q * a.range;
	uint32_t lo = 0, hi = (uint32_t)a.in.V;
	while (lo < hi) {
		const uint32_t mid = (lo + hi + 1) >> 1;
		if (__ldg(a.pos + mid) <= s) lo = mid; else hi = mid - 1;
	}
	const uint32_t e = lo;
	if (e >= a.in.V) return;
	const uint32_t start = __ldg(a.pos + e), end = __ldg(a.pos + e + 1);
	if (!(start < s && start >= s - a.range && end > s)) return;
	const uint32_t r2 = (end - 1) / a.range;
	const uint32_t c0 = a.col0 + lane;
	double t[CPL];
#pragma unroll
	for (int i = 0; i < CPL; i++) t[i] = __ldcg(a.carry_last + (uint64_t)(q - 1) * a.K + c0 + 32 * i);
	for (uint32_t x = (uint32_t)q; x <= r2; x++)
#pragma unroll
		for (int i = 0; i < CPL; i++) t[i] += __ldcg(a.carry_first + (uint64_t)x * a.K + c0 + 32 * i);
	walk_finish<CPL>(a, e, t);
}

template <int CPL>
void launch_walk(const WalkArgs& a, cudaStream_t st) {
	ppr_walk_step<CPL><<<grid_for(a.nranges, kWalkThreads / 32), kWalkThreads, 0, st>>>(a);
	if (a.nranges > 1) ppr_walk_fixup<CPL><<<grid_for(a.nranges, 8), 256, 0, st>>>(a);
}

} // namespace

lg_status ppr_walk(lg_snapshot* sn, const PprSeeds& seeds, uint32_t K, int ktile, int iterations,
		double damping, double* y0, double* y1, DevBuf& carry, double* x) {
	lg_store* s = sn->store;
	cudaStream_t st = s->stream;
	WalkArgs a;
	a.in = sn->view(1);
	a.pos = sn->in.slot_off.as<uint32_t>();
	a.total = (uint32_t)sn->in.n_frag_slots;
	a.range = (uint32_t)tune_value(s->device, LG_TUNE_PPR_RANGE);
	a.nranges = (uint32_t)std::max<uint64_t>(1, ((uint64_t)a.total + a.range - 1) / a.range);
	LG_TRY(carry.reserve(2ull * a.nranges * K * sizeof(double)));
	a.outdeg = sn->out.deg.as<uint32_t>();
	a.d = damping;
	a.tele = 1.0 - damping;
	a.seed_first = seeds.first;
	a.seed_col = seeds.cols;
	a.n_seeds = seeds.n;
	a.carry_first = carry.as<double>();
	a.carry_last = carry.as<double>() + (uint64_t)a.nranges * K;
	a.K = K;
	// column tiles are independent: each runs all iterations on its columns
	for (uint32_t c0 = 0; c0 < K; c0 += (uint32_t)ktile) {
		a.col0 = c0;
		for (int it = 0; it < iterations; it++) {
			a.y = it & 1 ? y1 : y0;
			a.y_next = it & 1 ? y0 : y1;
			a.x_out = it == iterations - 1 ? x : nullptr;
			switch (ktile / 32) {
			case 1: launch_walk<1>(a, st); break;
			case 2: launch_walk<2>(a, st); break;
			case 3: launch_walk<3>(a, st); break;
			case 4: launch_walk<4>(a, st); break;
			case 5: launch_walk<5>(a, st); break;
			case 6: launch_walk<6>(a, st); break;
			case 7: launch_walk<7>(a, st); break;
			default: launch_walk<8>(a, st); break;
			}
			s->launches += a.nranges > 1 ? 2 : 1;
		}
	}
	LG_CUDA(cudaGetLastError(), "ppr_walk_step");
	return LG_OK;
}

} // namespace lg
