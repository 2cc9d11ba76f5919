// lg_flat_run.cuh - repeated sweeps over a flat CSR inside one cooperative
// launch (PageRank over small graphs, lg_pagerank.cu; the weighted fixed-point
// solves, lg_adjoint.cu).
//
// The launch-per-iteration form (lg_flat_sweep.cuh) pays two launches per sweep
// and, for rows that cross tiles, a second kernel whose chain of loads takes 5
// to 10 us: as long as the sweep itself below some 10^6 edges.  Here every warp
// owns a run of consecutive tiles and keeps the open row's sum in registers
// from tile to tile; the warps of a CTA join their ends in shared memory, and
// only the row open at each CTA's end crosses the grid: the CTAs publish two
// partial sums each, meet at one bounded barrier per iteration, and then every
// CTA finishes all those rows itself, so that its next sweep needs no second
// barrier.  All sums are formed in a fixed order (edge order within a lane, a
// segmented warp scan, tiles, warps, CTAs), so results are deterministic.
//
// Vectors the iterations rewrite are read by plain loads: the barrier's fence
// makes them current, which the read-only path does not promise.
//
// An Op supplies
//   Row                                      what a row's end needs that no
//                                            iteration changes
//   Row    row(k) const                      of row k
//   void   values(eb, id[8], x[8]) const     the 8 edge values of a lane
//   double old(row) const                    the row's last value, if finish
//                                            wants it
//   double finish(row, s, old) const         the row has sum s; its residual
//                                            term
//   static constexpr bool kResidual          finish() returns something
// Rows' constants are loaded beside the edges' values, so that no chain of
// loads follows the sums; a CTA keeps those of the rows that cross CTAs.
#ifndef LG_FLAT_RUN_CUH_
#define LG_FLAT_RUN_CUH_

#include "lg_coop.cuh"
#include "lg_flat_sweep.cuh"

namespace lg {

constexpr int kRunThreads = 1024;      // one CTA per SM, 64 registers a thread
constexpr int kRunWarps = kRunThreads / 32;
constexpr int kRunRows = 4;
constexpr int kRunMaxCtas = 256;       // more SMs than any device of this architecture has

// What a CTA publishes of its edges, twice: iterations alternate.
struct RunEnds {
	double first[kRunMaxCtas];         // sum of the row begun before, up to its end here
	double last[kRunMaxCtas];          // sum of the row open at the end, if it began here
	double resid[kRunMaxCtas];         // residual of the rows that ended here
	uint32_t row[kRunMaxCtas];         // that row, kNoId if no row begins here
};

struct RunCtl {
	RunEnds ends[2];
	CoopBar bar;
	double resid;                      // last residual
	uint32_t iters, pad;
};

struct RunShared {
	double rs[kRunWarps][kFlatTile];   // rows finished in a warp's tile
	double first[kRunWarps], last[kRunWarps];
	uint32_t row[kRunWarps];
	double cfirst[kRunMaxCtas], clast[kRunMaxCtas];
	uint32_t crow[kRunMaxCtas];
	double part[kRunWarps];
};

// Sum of x over the CTA, the same bits in every thread.
__device__ __forceinline__ double run_block_sum(RunShared& sh, double x) {
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
	__syncthreads();
	if ((threadIdx.x & 31u) == 0) sh.part[threadIdx.x >> 5] = x;
	__syncthreads();
	double t = 0.0;
#pragma unroll
	for (int w = 0; w < kRunWarps; w++) t += sh.part[w];
	return t;
}

// One sweep over the calling warp's tiles [t0, t1), whose first one begins with
// `seg` rows begun before it; returns the lane's residual terms and leaves the
// run's ends in sh.first / last / row of the warp.
template <class Op>
__device__ __forceinline__ double run_tiles(const FlatTiles& a, const Op& op, RunShared& sh,
		uint32_t t0, uint32_t t1, uint32_t seg) {
	const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
	double* rs = sh.rs[wid];
	const unsigned char* hbytes = reinterpret_cast<const unsigned char*>(a.heads);
	uint32_t id[kFlatPerLane], hb = 0;
	auto fetch = [&](uint32_t t) {
		const uint32_t eb = t * kFlatTile + lane * kFlatPerLane;
		hb = __ldg(hbytes + (size_t)t * (kFlatTile / 8) + lane);
		if (eb + kFlatPerLane <= a.E) {
			asm("ld.global.cs.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
				: "=r"(id[0]), "=r"(id[1]), "=r"(id[2]), "=r"(id[3]),
				  "=r"(id[4]), "=r"(id[5]), "=r"(id[6]), "=r"(id[7])
				: "l"(a.ids + eb));
		} else {
#pragma unroll
			for (int i = 0; i < kFlatPerLane; i++)
				id[i] = eb + i < a.E ? __ldcs(a.ids + eb + i) : kNoId;
		}
	};
	double open = 0.0, res = 0.0;              // the open row's sum so far
	bool before = true;                        // it began before the run
	double first = 0.0;
	if (t0 < t1) fetch(t0);
	for (uint32_t t = t0; t < t1; t++) {
		const uint32_t eb = t * kFlatTile + lane * kFlatPerLane;
		double x[kFlatPerLane];
		op.values(eb, id, x);
		// the row that head `lane` of the tile ends (more heads: loaded later)
		typename Op::Row row = op.row(min(seg + lane - 1u, a.R - 1u));
		double was = op.old(row);
		const uint32_t h = hb;
		if (t + 1 < t1) fetch(t + 1);
		// heads in the lanes to the left; H of them in the tile
		const uint32_t nh = __popc(h);
		uint32_t left = nh;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t q = __shfl_up_sync(0xffffffffu, left, o);
			if (lane >= (uint32_t)o) left += q;
		}
		const uint32_t H = __shfl_sync(0xffffffffu, left, 31);
		left -= nh;
		// head j of the tile ends row seg + j - 1, whose sum goes to rs[j]
		double acc = 0.0, lead = 0.0;
		uint32_t seen = 0;
#pragma unroll
		for (int i = 0; i < kFlatPerLane; i++) {
			if ((h >> i) & 1u) {
				if (seen == 0) lead = acc;
				else rs[left + seen] = acc;            // a row inside the lane
				seen++;
				acc = 0.0;
			}
			acc += x[i];
		}
		if (seen == 0) lead = acc;
		const uint32_t hm = __ballot_sync(0xffffffffu, nh != 0);
		const uint32_t with_head = hm & ((2u << lane) - 1u);
		const int start = with_head ? 31 - __clz(with_head) : -1;
		double v = nh != 0 ? acc : lead;
		if (lane == 0 && nh == 0) v = open + v;        // the row open from the last tile
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const double pv = __shfl_up_sync(0xffffffffu, v, o);
			if (lane >= (uint32_t)o && (int)lane - o >= start) v = pv + v;
		}
		double open_in = __shfl_up_sync(0xffffffffu, v, 1);
		if (lane == 0) open_in = open;
		if (nh != 0) rs[left] = open_in + lead;
		open = __shfl_sync(0xffffffffu, v, 31);
		__syncwarp();
		const bool lead_row = H > 0 && before;   // row 0 began before the run
		if (lead_row) {
			if (lane == 0) first = rs[0];
			before = false;
		}
		if (lane < H && (lane > 0 || !lead_row)) res += op.finish(row, rs[lane], was);
		// the rows behind the first 32 (short rows: up to 256 in a tile), the loads
		// of some of a lane's before the first of them is finished
		for (uint32_t r0 = 32u; r0 < H; r0 += 32u * kRunRows) {
			typename Op::Row rw[kRunRows];
			double old[kRunRows];
#pragma unroll
			for (int u = 0; u < kRunRows; u++)
				rw[u] = op.row(min(seg + r0 + u * 32u + lane - 1u, a.R - 1u));
#pragma unroll
			for (int u = 0; u < kRunRows; u++) old[u] = op.old(rw[u]);
#pragma unroll
			for (int u = 0; u < kRunRows; u++) {
				const uint32_t r = r0 + u * 32u + lane;
				if (r < H) res += op.finish(rw[u], rs[r], old[u]);
			}
		}
		seg += H;
		__syncwarp();                          // rs is reused by the next tile
	}
	if (lane == 0) {
		sh.first[wid] = before ? open : first;
		sh.last[wid] = open;
		sh.row[wid] = before ? kNoId : seg - 1u;
	}
	return res;
}

// Rows open from warp i of n into later warps (or from CTA i into later CTAs):
// the sum of row[i], which began in i, over i's last part and the first parts
// up to the next entry in which a row begins; *closed = false if there is none.
__device__ __forceinline__ double run_join(const double* first, const double* last,
		const uint32_t* row, uint32_t i, uint32_t n, bool* closed) {
	double s = last[i];
	*closed = false;
	for (uint32_t j = i + 1; j < n && !*closed; j++) {
		s += first[j];
		*closed = row[j] != kNoId;
	}
	return s;
}

// One iteration by the whole grid: sweep, join, barrier, and the rows that
// cross CTAs, finished by every CTA alike.  *resid = the iteration's residual
// (the same in every thread of the grid: the CTAs' terms in CTA order);
// first_time: the launch's first iteration, which fills `cross`, the constants
// of the row the thread finishes.  False once a barrier wait gave up.
template <class Op>
__device__ __forceinline__ bool run_iteration(const FlatTiles& a, const Op& op, RunCtl* c,
		RunShared& sh, uint32_t t0, uint32_t t1, uint32_t seg, double extra, int parity,
		bool first_time, typename Op::Row& cross, double* resid) {
	const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
	double res = extra + run_tiles(a, op, sh, t0, t1, seg);
	__syncthreads();
	RunEnds& e = c->ends[parity];
	if (wid == 0) {
		bool closed;
		const uint32_t row = sh.row[lane];
		const double s = run_join(sh.first, sh.last, sh.row, lane, kRunWarps, &closed);
		if (row != kNoId && closed) {
			const typename Op::Row r = op.row(row);
			res += op.finish(r, s, op.old(r));
		}
		// the CTA's own ends
		const unsigned begins = __ballot_sync(0xffffffffu, row != kNoId);
		if (lane == 0) {
			double f = 0.0;
			const int upto = begins ? __ffs(begins) - 1 : kRunWarps - 1;
			for (int j = 0; j <= upto; j++) f += sh.first[j];
			e.first[blockIdx.x] = f;
			if (!begins) {
				e.last[blockIdx.x] = 0.0;
				e.row[blockIdx.x] = kNoId;
			}
		}
		if (begins && (int)lane == 31 - __clz(begins)) {
			e.last[blockIdx.x] = s;
			e.row[blockIdx.x] = row;
		}
	}
	if (Op::kResidual) {
		res = run_block_sum(sh, res);
		if (tid == 0) e.resid[blockIdx.x] = res;
	}
	// (no CTA writes the last vector before it has passed the barrier)
	double was = first_time ? 0.0 : op.old(cross);
	if (!grid_barrier(&c->bar)) return false;
	static_assert(kRunMaxCtas <= kRunThreads, "a thread per CTA");
	res = 0.0;
	if (tid < gridDim.x) {
		sh.cfirst[tid] = __ldcg(e.first + tid);
		sh.clast[tid] = __ldcg(e.last + tid);
		if (first_time) sh.crow[tid] = __ldcg(e.row + tid);
		if (Op::kResidual) res = __ldcg(e.resid + tid);
	}
	__syncthreads();
	if (tid < gridDim.x && sh.crow[tid] != kNoId) {
		if (first_time) {
			cross = op.row(sh.crow[tid]);
			was = op.old(cross);
		}
		bool closed;                             // (the last one ends with the edges)
		res += op.finish(cross, run_join(sh.cfirst, sh.clast, sh.crow, tid, gridDim.x, &closed), was);
	}
	if (Op::kResidual) *resid = run_block_sum(sh, res);
	__syncthreads();
	return true;
}

// CTAs for ntiles tiles: one for every four, at most one per SM.
inline unsigned run_ctas(uint32_t ntiles, int resident) {
	const unsigned need = (ntiles + 3u) / 4u;
	const unsigned most = (unsigned)(resident < kRunMaxCtas ? resident : kRunMaxCtas);
	return need < 1u ? 1u : need < most ? need : most;
}

// Iterations of one launch, so that it ends within some 50 ms: neither the host
// nor other streams wait longer (7 us an iteration and 6 ps an edge, measured
// at 30 k and 15 M edges; as much for a vertex).
inline int run_iterations(uint64_t E, uint64_t V) {
	const double n = 50000.0 / (7.0 + 6e-6 * ((double)E + (double)V));
	return n < 1.0 || test_limits().one_step ? 1 : (int)n;
}

// The calling warp's tiles (warps in CTA order).
__device__ __forceinline__ void run_share(uint32_t ntiles, uint32_t* t0, uint32_t* t1) {
	const uint64_t w = (uint64_t)blockIdx.x * kRunWarps + (threadIdx.x >> 5);
	const uint64_t n = (uint64_t)gridDim.x * kRunWarps;
	*t0 = (uint32_t)(w * ntiles / n);
	*t1 = (uint32_t)((w + 1) * ntiles / n);
}

} // namespace lg

#endif // LG_FLAT_RUN_CUH_
