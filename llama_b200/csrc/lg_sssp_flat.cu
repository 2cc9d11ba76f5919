// lg_sssp_flat.cu - delta-stepping SSSP over the flat out-CSR, every step in
// one cooperative launch (of very many steps in several: one returns after
// kCoopRunCycles, with the traversal's state in the control block).
//
// Buckets and bounds are those of lg_sssp.cu's host loop: the near queue holds
// vertices whose distance fell below the bucket's bound, the far pile every
// other reached one; when the queue has drained, the pile is split at the next
// bound, or at the bucket of the smallest distance left.  What differs:
//   - the rows are read from the flat out-CSR (lg_flat_expand.cuh) and a warp
//     takes a few queue entries at a time, so no step needs the queue's slot
//     offsets; longer rows are cut into pieces that all warps take after a
//     grid barrier;
//   - the counters of a step are read on the device: one or two grid barriers
//     per step where the host loop had three to five launches, two copies and
//     a wait;
//   - while the queue and the pile are short, one CTA takes the steps alone,
//     with block barriers, and the others wait at one grid barrier;
//   - a vertex is in the far pile exactly when its distance is finite and at or
//     above the bound, so an edge appends its target to the pile only where it
//     is the first to reach it: the pile needs no stamps;
//   - from a bucket's second round on, a long queue relaxes only edges lighter
//     than delta (a vertex of the first bucket of an R-MAT graph is improved
//     three times on average), and the heavier edges of the vertices whose
//     distance ended up in the bucket are relaxed once when it has drained (with
//     no heavier edge anywhere all rounds relax all edges, and that pass over the
//     rows falls away: delta 1000 with weights below 100 at 16 M edges and 4 M
//     vertices 1320 -> 1100 us);
//   - edges that would improve their target are collected per warp and relaxed
//     32 at a time: few edges of a step do, and waiting for the atomics of each
//     128 edges doubled the time of the large steps; the next edges' loads are
//     issued before the distances of the last ones are looked at;
//   - counters and state are read by one warp per CTA and passed on in shared
//     memory (read by every thread of the grid, one L2 sector took 5 to 20 us
//     a step).
//
// Bound at 3 M vertices by the distance gathers and atomics of the first
// bucket's rounds, and by the chain of dependent loads and a barrier in each of
// some 60 short steps.
//
// Buffers the kernel rewrites are read through L2 or by plain loads after a
// barrier.  Barrier waits are bounded (lg_coop.cuh).  The grid's counters rotate
// over three slots: step s fills slot s % 3 and clears slot (s + 1) % 3, which
// every CTA read before the barrier that ended step s - 1.
#include "lg_coop.cuh"
#include "lg_flat.cuh"
#include "lg_flat_expand.cuh"
#include "lg_sssp.cuh"
#include "lg_sssp_flat.h"
#include "lg_tune.h"

#include <algorithm>
#include <cstddef>
#include <mutex>

namespace lg {

namespace {

constexpr int kSfThreads = 1024;
constexpr int kSfWarps = kSfThreads / 32;
// Steps one CTA takes alone: at most so many queue entries, out-edges of
// theirs and far entries (about what it does in the time of a grid barrier
// and the other CTAs' start).
constexpr uint32_t kSoloQueue = 64, kSoloEdges = 8192, kSoloFar = 4096;
// ... and so many steps in a row, well within the other CTAs' bounded wait.
constexpr uint32_t kSoloSteps = 4096;

// The traversal's state, the same in every CTA.
struct SfState {
	unsigned long long qlen, flen;
	uint32_t lo, hi;               // the bucket: distances in [lo, hi)
	uint32_t step;                 // grid steps taken (counter slot)
	uint32_t round, buckets;
	uint32_t in_bucket;            // relaxation rounds of this bucket
	uint32_t mind;                 // smallest distance the last split kept
	uint32_t qsel, fsel;           // which of the two queues / piles is current
	uint32_t light;                // rounds relax light edges only
	uint32_t heavy;                // whether there are other edges (SfHeavy)
	uint32_t jump;                 // the next split goes to mind's bucket
	uint32_t grid;                 // the next step is for the whole grid
};

struct SfCtl {
	unsigned long long ctr[3][4];   // per step: [0] near appends, [1] far appends,
	                                // [2] split: max of ~kept distance, [3] row pieces
	                                // (and kCoopTimeUp)
	SfState st;                     // handed over by the CTA that worked alone, and to
	                                // the next launch
	uint32_t up;                    // by that CTA: the launch's time is up
	alignas(16) unsigned long long out[8];   // rounds, buckets, relaxations, reached,
	                                // out-edges of the reached, largest distance, done,
	                                // an edge of at least delta was found
	CoopBar bar;                    // err bit 2: a count out of range, bit 3: step cap
};

struct SfArgs {
	const uint32_t* off;
	const uint32_t* ids;
	const uint32_t* w;
	const uint32_t* outdeg;
	uint32_t V, E, root, delta, piece;
	uint32_t max_pieces, light_min;
	uint32_t* q[2];
	uint32_t* far[2];
	uint32_t *dist, *stamp;
	uint2* pieces;                  // {vertex, first edge} of long rows' pieces
	long long cycles;               // the launch's time
};

constexpr uint32_t kSfCand = 64;

struct SfShared {                   // dynamic shared memory
	uint32_t sbuf[kSfWarps][2][kPushBuf];
	uint2 cand[kSfWarps][kSfCand];  // {target, offered distance}
	RowWindow win[kSfWarps];
	unsigned long long ctr[3][4];   // the lone CTA's counters
	unsigned long long got[4];      // the last step's counters
	long long t0;                   // the launch's start (CTA 0)
	uint32_t up;                    // its time is up
	uint32_t heavy;
	SfState st;
};

enum SfHeavy : uint32_t { kNotLooked, kSomeHeavy, kNoHeavy };

enum SfEdges : uint32_t { kAllEdges, kLightEdges, kHeavyEdges };

// What a relaxation step needs besides the edges.
struct SfStep {
	uint32_t round, hi, edges;
	uint32_t *near_next, *far_end;
	unsigned long long* cnt;        // the step's counters
	uint32_t *sbuf_near, *sbuf_far; // the warp's staging buffers
	uint2* cand;
	RowWindow* win;
};

// What every edge reads, in registers: the functions below are kept out of
// line, so their argument structs are in local memory, and a field read from
// there after an atomic is loaded again.
struct SfHot {
	const uint32_t *ids, *w;
	uint32_t *dist, *stamp;
	uint32_t delta, edges, hi, round;
	__device__ __forceinline__ SfHot(const SfArgs& a, const SfStep& s)
		: ids(a.ids), w(a.w), dist(a.dist), stamp(a.stamp), delta(a.delta), edges(s.edges),
		  hi(s.hi), round(s.round) {}
};

// kFeAhead edges of every lane, as loaded (id kNoId past the end).
struct SfBatch {
	uint32_t id[kFeAhead], w[kFeAhead], d[kFeAhead];
};

// A warp's relaxations of one step.
struct SfRelax {
	const SfHot h;
	const SfStep& s;
	uint32_t nn = 0, nf = 0, nc = 0;     // staged near, far and candidates
	unsigned long long relax = 0;
	SfBatch next, cur;
	__device__ __forceinline__ SfRelax(const SfArgs& a, const SfStep& st) : h(a, st), s(st) {}
	// The candidates' minima, and the queue entries these make.
	__device__ __forceinline__ void flush() {
		const uint32_t lane = threadIdx.x & 31u;
		__syncwarp();
		for (uint32_t b = 0; b < nc; b += 32u) {
			uint32_t id = 0, nd = 0, old = 0;
			if (b + lane < nc) {
				const uint2 x = s.cand[b + lane];
				id = x.x;
				nd = x.y;
				old = atomicMin(h.dist + id, nd);
				relax++;
			}
			const bool better = nd < old;
			const bool near = better && nd < h.hi && atomicExch(h.stamp + id, h.round) != h.round;
			wq_add(near, id, s.sbuf_near, nn, s.near_next, s.cnt);
			wq_add(better && nd >= h.hi && old == kInf, id, s.sbuf_far, nf, s.far_end, s.cnt + 1);
		}
		__syncwarp();
		nc = 0;
	}
	__device__ __forceinline__ void rows(uint32_t start, uint32_t len, uint32_t dv) {
		const uint32_t lane = threadIdx.x & 31u;
		flat_expand(s.win, start, len, dv,
			[&](int u, bool act, uint32_t e, uint32_t d) {
				next.id[u] = kNoId;
				next.w[u] = 0;
				next.d[u] = d;
				if (act) {
					next.id[u] = __ldg(h.ids + e);
					next.w[u] = __ldg(h.w + e);
				}
			},
			[&]() { cur = next; },
			[&]() {
				uint32_t dc[kFeAhead];
#pragma unroll
				for (int u = 0; u < kFeAhead; u++) {
					dc[u] = 0;                   // nothing to improve
					if (cur.id[u] != kNoId && (h.edges == kAllEdges
							|| (cur.w[u] < h.delta) == (h.edges == kLightEdges)))
						dc[u] = __ldcg(h.dist + cur.id[u]);
				}
#pragma unroll
				for (int u = 0; u < kFeAhead; u++) {
					const uint32_t nd = cur.d[u] + cur.w[u];
					const bool take = nd < dc[u];
					const unsigned m = __ballot_sync(0xffffffffu, take);
					if (!m) continue;
					if (nc + (uint32_t)__popc(m) > kSfCand) flush();
					if (take)
						s.cand[nc + __popc(m & ((1u << lane) - 1u))] = make_uint2(cur.id[u], nd);
					nc += __popc(m);
				}
			});
	}
	__device__ __forceinline__ void finish() {
		flush();
		wq_flush(s.sbuf_near, nn, s.near_next, s.cnt);
		wq_flush(s.sbuf_far, nf, s.far_end, s.cnt + 1);
	}
};

// The queue entries q[0, n), or (q null) the n vertices whose distance lies in
// [lo, hi): a warp takes up to 32 at a time, fewer when there are not enough
// to give every warp some.
__device__ __noinline__ unsigned long long sf_rows(const SfArgs& a, const SfStep& s,
		const uint32_t* q, uint32_t n, uint32_t lo, uint32_t gwarp, uint32_t nwarps) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t per = n ? min(32u, (n - 1u) / nwarps + 1u) : 1u;
	SfRelax r(a, s);
	for (uint64_t b = (uint64_t)gwarp * per; b < n; b += (uint64_t)nwarps * per) {
		uint32_t v = 0, start = 0, len = 0, dv = 0;
		if (lane < per && b + lane < n) {
			v = q ? __ldcg(q + b + lane) : (uint32_t)b + lane;
			dv = __ldcg(a.dist + v);
			if (q || (dv >= lo && dv < s.hi)) {
				start = __ldg(a.off + v);
				len = __ldg(a.off + v + 1) - start;
			}
		}
		// long rows become pieces
		const uint32_t k = len > a.piece ? (len - 1u) / a.piece + 1u : 0u;
		if (__any_sync(0xffffffffu, k != 0)) {
			uint32_t inc = k;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
				if (lane >= (uint32_t)o) inc += y;
			}
			unsigned long long p = 0;
			if (lane == 31u) p = atomicAdd(s.cnt + 3, (unsigned long long)inc);
			p = (__shfl_sync(0xffffffffu, p, 31) & ~kCoopTimeUp) + inc - k;
			if (k <= 32u)
				for (uint32_t i = 0; i < k; i++)
					if (p + i < a.max_pieces) a.pieces[p + i] = make_uint2(v, start + i * a.piece);
			unsigned big = __ballot_sync(0xffffffffu, k > 32u);
			while (big) {
				const int t = __ffs(big) - 1;
				big &= big - 1u;
				const uint32_t bv = __shfl_sync(0xffffffffu, v, t);
				const uint32_t bs = __shfl_sync(0xffffffffu, start, t);
				const uint32_t bk = __shfl_sync(0xffffffffu, k, t);
				const unsigned long long bp = __shfl_sync(0xffffffffu, p, t);
				for (uint32_t i = lane; i < bk; i += 32u)
					if (bp + i < a.max_pieces)
						a.pieces[bp + i] = make_uint2(bv, bs + i * a.piece);
			}
		}
		if (len > a.piece) len = 0;
		r.rows(start, len, dv);
	}
	r.finish();
	return r.relax;
}

// The pieces of the step's long rows, walked like rows.
__device__ __noinline__ unsigned long long sf_pieces(const SfArgs& a, const SfStep& s, uint32_t n,
		uint32_t gwarp, uint32_t nwarps) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t per = min(32u, (n - 1u) / nwarps + 1u);
	SfRelax r(a, s);
	for (uint64_t b = (uint64_t)gwarp * per; b < n; b += (uint64_t)nwarps * per) {
		uint32_t start = 0, len = 0, dv = 0;
		if (lane < per && b + lane < n) {
			const uint2 pc = __ldcg(a.pieces + b + lane);
			start = pc.y;
			len = min(__ldg(a.off + pc.x + 1) - start, a.piece);
			dv = __ldcg(a.dist + pc.x);
		}
		r.rows(start, len, dv);
	}
	r.finish();
	return r.relax;
}

// Split of the pile far[0, n) at [lo, hi): closer entries were settled from a
// near queue, those in the bucket become the near queue, the others are kept;
// returns the lane's smallest kept distance (~0 if none).
__device__ __noinline__ uint32_t sf_split(const SfArgs& a, const uint32_t* far, uint32_t n,
		uint32_t lo, uint32_t hi, uint32_t* near, uint32_t* keep, unsigned long long* cnt,
		uint32_t* sbuf_near, uint32_t* sbuf_keep, uint32_t gwarp, uint32_t nwarps) {
	const uint32_t lane = threadIdx.x & 31u;
	uint32_t nn = 0, nk = 0, m = 0xffffffffu;
	for (uint64_t b = (uint64_t)gwarp * (32u * kFeAhead); b < n;
			b += (uint64_t)nwarps * (32u * kFeAhead)) {
		uint32_t v[kFeAhead], d[kFeAhead];
#pragma unroll
		for (int u = 0; u < kFeAhead; u++) {
			const uint64_t i = b + u * 32u + lane;
			v[u] = i < n ? __ldcg(far + i) : kNoId;
		}
#pragma unroll
		for (int u = 0; u < kFeAhead; u++) d[u] = v[u] != kNoId ? __ldcg(a.dist + v[u]) : 0u;
#pragma unroll
		for (int u = 0; u < kFeAhead; u++) {
			const bool in = v[u] != kNoId;
			wq_add(in && d[u] >= lo && d[u] < hi, v[u], sbuf_near, nn, near, cnt);
			wq_add(in && d[u] >= hi, v[u], sbuf_keep, nk, keep, cnt + 1);
			if (in && d[u] >= hi) m = min(m, d[u]);
		}
	}
	wq_flush(sbuf_near, nn, near, cnt);
	wq_flush(sbuf_keep, nk, keep, cnt + 1);
	return m;
}

// One step of the traversal by the whole grid, or (kSolo) by the calling CTA
// alone; false when a barrier failed or a count is out of range (err set).
template <bool kSolo>
__device__ __forceinline__ bool sf_step(const SfArgs& a, SfCtl* c, SfShared& sh, SfState& t,
		uint32_t& slot, unsigned long long& relaxations) {
	const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
	// consecutive windows of a list go to different SMs
	const uint32_t gwarp = kSolo ? wid : wid * gridDim.x + blockIdx.x;
	const uint32_t nwarps = kSolo ? kSfWarps : kSfWarps * gridDim.x;
	unsigned long long* cnt = kSolo ? sh.ctr[slot] : c->ctr[slot];
	slot = slot == 2u ? 0u : slot + 1u;
	if (tid < 4 && (kSolo || blockIdx.x == 0)) (kSolo ? sh.ctr[slot] : c->ctr[slot])[tid] = 0;
	// (by a warp that has the fewest rows, beside the others' work)
	if (tid == kSfThreads - 1 && blockIdx.x == 0 && clock64() - sh.t0 > a.cycles)
		atomicOr(cnt + 3, kCoopTimeUp);
	// after a barrier every thread finds the step's counters in sh.got
	auto barrier = [&]() {
		if (!kSolo && !grid_barrier(&c->bar)) return false;
		if (kSolo) __syncthreads();
		if (tid < 4) {
			const unsigned long long x = kSolo ? *(volatile unsigned long long*)(cnt + tid)
					: __ldcg(cnt + tid);
			sh.got[tid] = x & ~kCoopTimeUp;
			if (tid == 3) sh.up = x >= kCoopTimeUp;
		}
		__syncthreads();
		return true;
	};
	auto count = [&](int k) { return sh.got[k]; };
	t.round++;
	if (t.qlen > 0 || t.light) {
		const bool heavy = t.qlen == 0;          // the bucket has drained
		if (!heavy && t.in_bucket > 0 && t.qlen >= a.light_min && t.heavy == kSomeHeavy)
			t.light = 1;
		SfStep s;
		s.round = t.round;
		s.hi = t.hi;
		s.edges = heavy ? kHeavyEdges : t.light ? kLightEdges : kAllEdges;
		s.near_next = a.q[t.qsel ^ 1u];
		s.far_end = a.far[t.fsel] + t.flen;
		s.cnt = cnt;
		s.sbuf_near = sh.sbuf[wid][0];
		s.sbuf_far = sh.sbuf[wid][1];
		s.cand = sh.cand[wid];
		s.win = sh.win + wid;
		relaxations += sf_rows(a, s, heavy ? nullptr : a.q[t.qsel],
				heavy ? a.V : (uint32_t)t.qlen, t.lo, gwarp, nwarps);
		if (!barrier()) return false;
		const unsigned long long np = count(3);
		if (np > a.max_pieces) {
			if (tid == 0) atomicOr(&c->bar.err, 4u);
			return false;
		}
		if (np) {
			relaxations += sf_pieces(a, s, (uint32_t)np, gwarp, nwarps);
			if (!barrier()) return false;
		}
		const unsigned long long nq = count(0), nf = count(1);
		if (nq > a.V || t.flen + nf > a.V || (heavy && nq)) {
			if (tid == 0) atomicOr(&c->bar.err, 4u);
			return false;
		}
		t.flen += nf;
		if (heavy) {
			t.light = 0;
		} else {
			t.qlen = nq;
			t.qsel ^= 1u;
			t.in_bucket++;
		}
	} else {
		// split the far pile at the next bound (or, where that gave nothing, at
		// the bucket of the smallest distance left)
		t.lo = t.jump ? (t.mind / a.delta) * a.delta : t.hi;
		t.hi = t.lo > kInf - a.delta ? kInf : t.lo + a.delta;
		uint32_t m = sf_split(a, a.far[t.fsel], (uint32_t)t.flen, t.lo, t.hi, a.q[t.qsel],
				a.far[t.fsel ^ 1u], cnt, sh.sbuf[wid][0], sh.sbuf[wid][1], gwarp, nwarps);
		m = __reduce_min_sync(0xffffffffu, m);
		if (lane == 0 && m != 0xffffffffu) atomicMax(cnt + 2, (unsigned long long)~m);
		if (!barrier()) return false;
		t.qlen = count(0);
		t.flen = count(1);
		t.mind = ~(uint32_t)count(2);
		if (t.qlen > a.V || t.flen > a.V) {
			if (tid == 0) atomicOr(&c->bar.err, 4u);
			return false;
		}
		t.fsel ^= 1u;
		t.buckets++;
		t.in_bucket = 0;
		t.jump = !t.jump && t.qlen == 0 && t.flen > 0;
	}
	return true;
}

// Looks for an edge of at least delta, until a CTA has found one (one thread of
// a CTA says so and asks: all of them at one address took 100 us).  A first look,
// at a tile per CTA while the distances are filled, usually finds one.
__device__ __noinline__ void sf_look(const SfArgs& a, SfCtl* c, bool first) {
	constexpr uint32_t kLook = 8, kTile = kLook * kSfThreads;
	for (uint64_t b = (uint64_t)blockIdx.x * kTile; b < a.E; b += (uint64_t)gridDim.x * kTile) {
		uint32_t w = 0;
#pragma unroll
		for (uint32_t u = 0; u < kLook; u++) {
			const uint64_t e = b + u * kSfThreads + threadIdx.x;
			w = max(w, e < a.E ? __ldg(a.w + e) : 0u);
		}
		volatile unsigned long long* some = c->out + 7;
		const bool others = threadIdx.x == 0 && *some != 0;
		const bool found = __syncthreads_or(w >= a.delta);
		if (found && threadIdx.x == 0) *some = 1;
		if (__syncthreads_or(found || others) || first) break;
	}
}

// The state in c->st, read by a CTA behind a barrier.
__device__ __forceinline__ SfState sf_load_state(const SfCtl* c, SfShared& sh) {
	if (threadIdx.x < sizeof(SfState) / 4)
		reinterpret_cast<unsigned int*>(&sh.st)[threadIdx.x] =
				__ldcg(reinterpret_cast<const unsigned int*>(&c->st) + threadIdx.x);
	__syncthreads();
	return sh.st;
}

// One CTA of 1024 per SM: 64 registers.  resume: goes on from c->st, where the
// last launch's time was up.
__global__ void __launch_bounds__(kSfThreads, 1)
sssp_flat(SfArgs a, SfCtl* c, int resume) {
	extern __shared__ __align__(16) unsigned char sf_smem[];
	SfShared& sh = *reinterpret_cast<SfShared*>(sf_smem);
	const uint32_t tid = threadIdx.x, lane = tid & 31u;
	const uint32_t gtid = blockIdx.x * kSfThreads + tid;
	const uint32_t nthreads = gridDim.x * kSfThreads;
	SfState t = {};
	if (resume) {
		t = sf_load_state(c, sh);
	} else {
		for (uint64_t v = gtid; v < a.V; v += nthreads) {
			a.dist[v] = v == a.root ? 0u : kInf;
			a.stamp[v] = 0xffffffffu;
		}
		sf_look(a, c, true);
		if (gtid == 0) a.q[0][0] = a.root;
		t.qlen = 1;
		t.hi = a.delta;
		t.buckets = 1;
	}
	// (also: every CTA has read c->st)
	if (!grid_barrier(&c->bar)) return;
	unsigned long long relaxations = 0;              // the thread's own
	const uint64_t step_cap = 4ull * a.V + 64;
	uint32_t solo_slot = 0;
	if (tid < 4) sh.ctr[0][tid] = 0;
	if (tid == 0) {
		sh.t0 = clock64();
		sh.up = 0;
		sh.heavy = __ldcg(c->out + 7) ? kSomeHeavy : kNotLooked;
	}
	__syncthreads();
	if (!resume) t.heavy = sh.heavy;
	// (sh.up changes between barriers only)
	while ((t.qlen > 0 || t.flen > 0 || t.light) && !sh.up) {
		if (t.round >= step_cap) {
			if (tid == 0) atomicOr(&c->bar.err, 8u);
			return;
		}
		if (!t.grid && !t.light && t.qlen <= kSoloQueue && t.flen <= kSoloFar) {
			if (blockIdx.x == 0) {
				for (uint32_t n = 0; n < kSoloSteps && !sh.up && (t.qlen > 0 || t.flen > 0)
						&& t.qlen <= kSoloQueue && t.flen <= kSoloFar; n++) {
					if (t.qlen > 0) {
						uint32_t len = 0;
						if (tid < t.qlen) {
							const uint32_t v = __ldcg(a.q[t.qsel] + tid);
							len = __ldg(a.off + v + 1) - __ldg(a.off + v);
						}
						if (block_sum<kSfWarps>(len) > kSoloEdges) {
							t.grid = 1;                  // too many edges for one CTA
							break;
						}
					}
					if (!sf_step<true>(a, c, sh, t, solo_slot, relaxations)) return;
				}
				if (tid == 0) {
					c->st = t;
					c->up = sh.up;
				}
			}
			if (!grid_barrier(&c->bar)) return;
			if (blockIdx.x != 0) {
				if (tid == 0) sh.up = __ldcg(&c->up);
				t = sf_load_state(c, sh);            // (synchronises)
			}
			if (!t.grid) t.grid = t.qlen > 0 || t.flen > 0;   // past a CTA's limits
			// (nobody rewrites c->st before the grid step's barrier)
			continue;
		}
		t.grid = 0;
		if (t.heavy == kNotLooked && t.in_bucket > 0 && t.qlen >= a.light_min) {
			sf_look(a, c, false);
			if (!grid_barrier(&c->bar)) return;
			if (tid == 0) sh.heavy = __ldcg(c->out + 7) ? kSomeHeavy : kNoHeavy;
			__syncthreads();
			t.heavy = sh.heavy;
		}
		if (!sf_step<false>(a, c, sh, t, t.step, relaxations)) return;
	}
	relaxations = block_sum<kSfWarps>(relaxations);
	if (tid == 0 && relaxations) atomicAdd(c->out + 2, relaxations);
	if (t.qlen > 0 || t.flen > 0 || t.light) {       // the time is up
		// (c->st may still be read after a lone CTA's steps: the same values)
		if (gtid == 0) c->st = t;
		return;
	}
	// reached vertices, their out-edges, the largest distance
	unsigned long long cnt = 0, edges = 0, mx = 0;
	for (uint64_t v = gtid; v < a.V; v += nthreads) {
		const uint32_t d = __ldcg(a.dist + v);
		if (d < kInf) {
			cnt++;
			edges += __ldg(a.outdeg + v);
			mx = max(mx, (unsigned long long)d);
		}
	}
	cnt = block_sum<kSfWarps>(cnt);
	edges = block_sum<kSfWarps>(edges);
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
	if (lane == 0 && mx) atomicMax(c->out + 5, mx);
	if (tid == 0) {
		if (cnt) atomicAdd(c->out + 3, cnt);
		if (edges) atomicAdd(c->out + 4, edges);
		if (blockIdx.x == 0) {
			c->out[0] = t.round;
			c->out[1] = t.buckets;
			c->out[6] = 1;
		}
	}
}

std::mutex g_coop_mu;
int g_coop[LG_TUNE_MAX_DEVICES];          // co-resident CTAs + 1, 0 = not probed

int coop_grid(int device) {
	std::lock_guard<std::mutex> lk(g_coop_mu);
	if (device < 0 || device >= LG_TUNE_MAX_DEVICES) return 0;
	if (cudaFuncSetAttribute(sssp_flat, cudaFuncAttributeMaxDynamicSharedMemorySize,
			(int)sizeof(SfShared)) != cudaSuccess) {
		cudaGetLastError();
		return 0;
	}
	if (!g_coop[device])
		g_coop[device] = 1 + coop_grid_size((const void*)sssp_flat, kSfThreads, device,
				sizeof(SfShared));
	return coop_allowed(g_coop[device] - 1);
}

} // namespace

lg_status sssp_flat_run(lg_snapshot* sn, const FlatCsr* f, uint32_t root, uint32_t delta,
		uint32_t* dist, lg_sssp_result* result, bool* ran) {
	*ran = false;
	lg_store* s = sn->store;
	const int grid = coop_grid(s->device);
	if (grid <= 0) return LG_OK;
	unsigned ctas = (unsigned)grid;
	cudaStream_t st = s->stream;
	const uint64_t V = sn->V;
	DevBuf* sc = s->scratch;
	SfArgs a;
	// 64 edges for the tunable's default: a window of 32 rows or pieces then
	// holds at most 2048 edges, so no warp holds up a step
	a.piece = std::max((uint32_t)tune_value(s->device, LG_TUNE_SSSP_RANGE) / 16u, 32u);
	a.max_pieces = (uint32_t)(2 * f->E / a.piece + 1);
	// a second pass over a bucket's rows pays once every warp has several
	a.light_min = (uint32_t)grid * kSfWarps * 4u;
	LG_TRY(sc[0].reserve(V * 4));          // near queue
	LG_TRY(sc[1].reserve(V * 4));          // next near queue
	LG_TRY(sc[2].reserve(V * 4));          // far pile
	LG_TRY(sc[3].reserve(V * 4));          // far pile being compacted
	LG_TRY(sc[5].reserve(2 * V * 4));      // stamps
	LG_TRY(sc[7].reserve((uint64_t)a.max_pieces * sizeof(uint2)));
	LG_TRY(sc[11].reserve(sizeof(SfCtl)));
	SfCtl* ctl = sc[11].as<SfCtl>();
	a.off = f->off.as<uint32_t>();
	a.ids = f->ids.as<uint32_t>();
	a.w = f->w.as<uint32_t>();
	a.outdeg = sn->out.deg.as<uint32_t>();
	a.V = (uint32_t)V;
	a.E = (uint32_t)f->E;
	a.root = root;
	a.delta = delta;
	a.q[0] = sc[0].as<uint32_t>();
	a.q[1] = sc[1].as<uint32_t>();
	a.far[0] = sc[2].as<uint32_t>();
	a.far[1] = sc[3].as<uint32_t>();
	a.dist = dist;
	a.stamp = sc[5].as<uint32_t>();
	a.pieces = sc[7].as<uint2>();
	LG_CUDA(cudaMemsetAsync(ctl, 0, sizeof(SfCtl), st), "clear control block");
	a.cycles = coop_run_cycles();
	int resume = 0;
	void* kargs[] = {&a, &ctl, &resume};
	unsigned long long h[10];
	static_assert(offsetof(SfCtl, bar) == offsetof(SfCtl, out) + 64 && 10 <= kReadWords,
			"two words after the results");
	for (;; resume = 1) {
		LG_CUDA(coop_launch((const void*)sssp_flat, &ctas, kSfThreads, kargs, sizeof(SfShared), st, &ctl->bar),
				"sssp_flat");
		s->launches++;
		LG_TRY(read_words(s, ctl->out, 10, h));
		const unsigned int err = (unsigned int)h[9];      // the barrier's error word
		if (err & 1u) return set_error(LG_ETIMEOUT, "sssp: a grid barrier wait ran out");
		if (err & 4u) return set_error(LG_ECUDA, "sssp: a queue count out of range");
		if (err & 8u) return set_error(LG_ECUDA, "sssp: step cap reached");
		if (h[6]) break;
	}
	if (result) {
		result->rounds = (int32_t)h[0];
		result->buckets = (int32_t)h[1];
		result->relaxations = h[2];
		result->reached = h[3];
		result->reach_edges = h[4];
		result->max_dist = (uint32_t)h[5];
	}
	*ran = true;
	return LG_OK;
}

} // namespace lg
