// lg_scc_flat.cu - strongly connected components over flat CSRs.
//
// The partition and labels of lg_scc.cu (each component labelled by its
// smallest vertex), in three parts:
//   1. trim: vertices without live in- or out-edges are their own component;
//   2. the component of the vertex with the largest product of degrees, as the
//      vertices both reached from it and reaching it: two direction-optimising
//      searches of one launch each (lg_bfs_levels.cu).  In a graph with one
//      giant component that settles nearly all vertices that have edges both
//      ways, at about a tenth of the edges read once, where colouring reads
//      them all several times;
//   3. what is left by rounds of colouring, the steps of all rounds in one
//      cooperative launch (scc_rest), or several of kCoopRunCycles each: the smallest
//      label is pushed along out-edges to a fixpoint, a backward search within a
//      colour from the vertices that kept their own collects their components.
//      (A chain whose ids ascend settles one vertex per round, with as many
//      steps as it is still long.)
// Colouring alone, over fragments and with the host reading each step's
// counts, took 2.9 ms at 3 M vertices / 39 M edges, 1.2 ms of it pushing and
// 1.0 ms searching through the giant component.
#include "lg_bfs_levels.h"
#include "lg_coop.cuh"
#include "lg_flat_expand.cuh"
#include "lg_queue.cuh"
#include "lg_scc_flat.h"
#include "lg_tune.h"

#include <cstddef>
#include <cstring>
#include <mutex>

namespace lg {

namespace {

constexpr uint32_t kOpen = 0xffffffffu;      // label of a vertex not yet settled
constexpr int kSrThreads = 1024;
constexpr int kSrWarps = kSrThreads / 32;
constexpr int kListThreads = 256;
constexpr uint32_t kSrPiece = 256;           // edges of a row a warp takes at a time

typedef unsigned long long u64;

// Vertices without live in- or out-edges are settled, the others listed;
// ctr[0] = their number, ctr[1] = the largest {product of degrees (as a
// float's bits), ~vertex}.
__global__ void __launch_bounds__(kListThreads)
scc_trim_flat(const uint32_t* outdeg, const uint32_t* indeg, uint64_t V, uint32_t* label,
		uint32_t* mark, uint32_t* stamp, uint32_t* rem, u64* ctr) {
	__shared__ u64 s_best[kListThreads / 32];
	const uint64_t v = (uint64_t)blockIdx.x * kListThreads + threadIdx.x;
	bool keep = false;
	u64 key = 0;
	if (v < V) {
		const uint32_t o = __ldg(outdeg + v), i = __ldg(indeg + v);
		keep = o != 0 && i != 0;
		label[v] = keep ? kOpen : (uint32_t)v;
		mark[v] = 0;
		stamp[v] = 0;
		if (keep) key = (u64)__float_as_uint((float)o * (float)i) << 32 | (uint32_t)~v;
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
	if ((threadIdx.x & 31u) == 0) s_best[threadIdx.x >> 5] = key;
	block_push<kListThreads>(keep, (uint32_t)v, rem, ctr);       // (synchronises)
	if (threadIdx.x == 0) {
		for (int w = 1; w < kListThreads / 32; w++) key = max(key, s_best[w]);
		if (key) atomicMax(ctr + 1, key);
	}
}

// Smallest listed vertex reached in both searches.
__global__ void __launch_bounds__(kListThreads)
scc_giant_min(const uint32_t* rem, uint32_t n, const int32_t* fwd, const int32_t* bwd,
		uint32_t* best) {
	const uint64_t i = (uint64_t)blockIdx.x * kListThreads + threadIdx.x;
	uint32_t m = kOpen;
	if (i < n) {
		const uint32_t v = rem[i];
		if (fwd[v] != LG_UNREACHED && bwd[v] != LG_UNREACHED) m = v;
	}
	m = __reduce_min_sync(0xffffffffu, m);
	if ((threadIdx.x & 31u) == 0 && m != kOpen && m < *(volatile uint32_t*)best)
		atomicMin(best, m);
}

// Their component is labelled; the others form the next list, ctr[0] of them.
__global__ void __launch_bounds__(kListThreads)
scc_giant_label(const uint32_t* rem, uint32_t n, const int32_t* fwd, const int32_t* bwd,
		const uint32_t* best, uint32_t* label, uint32_t* rem_next, u64* ctr) {
	const uint64_t i = (uint64_t)blockIdx.x * kListThreads + threadIdx.x;
	bool keep = false;
	uint32_t v = 0;
	if (i < n) {
		v = rem[i];
		keep = !(fwd[v] != LG_UNREACHED && bwd[v] != LG_UNREACHED);
		if (!keep) label[v] = *best;
	}
	block_push<kListThreads>(keep, v, rem_next, ctr);
}

// The colouring between two steps, the same in every CTA.
enum SrPhase : uint32_t { kSrColour, kSrPush, kSrRoots, kSrSearch, kSrCollect };
struct alignas(16) SrState {
	u64 n_rem;              // vertices left, listed in rem[rsel]
	u64 n;                  // a push or search step's, in list[lsel]
	uint32_t rsel, lsel;
	uint32_t phase;         // of the next step
	uint32_t slot;          // its counters
	uint32_t round, stamp, steps, pad;
};

struct SrCtl {
	u64 ctr[3][2];          // per step: [0] appends, [1] row pieces (and kCoopTimeUp)
	SrState st;             // where the last launch left off
	CoopBar bar;            // err bit 2: a count out of range, bit 3: round cap
};

struct SrArgs {
	const uint32_t *ooff, *oids, *ioff, *iids;
	uint32_t V;
	uint32_t max_pieces;
	uint32_t* rem[2];
	uint32_t* list[2];
	uint32_t *label, *color, *mark, *stamp;
	uint2* pieces;          // {vertex, first edge}
	long long cycles;       // the launch's time
};

struct SrShared {
	uint32_t sbuf[kSrWarps][kPushBuf];
	RowWindow win[kSrWarps];
	u64 got[2];
	SrState st;
};

// A warp's expansion of list vertices: colours pushed along out-edges
// (kPush), or a backward search within a colour.
template <bool kPush>
struct SrStep {
	const SrArgs& a;
	const uint32_t *off, *ids;
	uint32_t *label, *color, *mark;      // mark: the stamps of a push
	uint32_t round;
	uint32_t* sbuf;
	uint32_t* next;
	u64* cnt;
	RowWindow* win;
	uint32_t nb = 0;
	uint32_t id[kFeAhead], val[kFeAhead], cid[kFeAhead], cval[kFeAhead];
	__device__ __forceinline__ SrStep(const SrArgs& x, uint32_t r, uint32_t* sb, uint32_t* nx,
			u64* c, RowWindow* w)
		: a(x), off(kPush ? x.ooff : x.ioff), ids(kPush ? x.oids : x.iids), label(x.label),
		  color(x.color), mark(kPush ? x.stamp : x.mark), round(r), sbuf(sb), next(nx), cnt(c),
		  win(w) {}
	__device__ __forceinline__ void rows(uint32_t start, uint32_t len, uint32_t c) {
		flat_expand(win, start, len, c,
			[&](int u, bool act, uint32_t e, uint32_t x) {
				id[u] = act ? __ldg(ids + e) : kNoId;
				val[u] = x;
			},
			[&]() {
#pragma unroll
				for (int u = 0; u < kFeAhead; u++) { cid[u] = id[u]; cval[u] = val[u]; }
			},
			[&]() {
				uint32_t lb[kFeAhead], cl[kFeAhead];
#pragma unroll
				for (int u = 0; u < kFeAhead; u++)
					lb[u] = cid[u] != kNoId ? __ldcg(label + cid[u]) : 0u;
#pragma unroll
				for (int u = 0; u < kFeAhead; u++)
					cl[u] = cid[u] != kNoId && lb[u] == kOpen ? __ldcg(color + cid[u]) : kNoId;
#pragma unroll
				for (int u = 0; u < kFeAhead; u++) {
					bool push = false;
					if (cl[u] != kNoId) {
						if (kPush)
							push = cval[u] < cl[u] && cval[u] < atomicMin(color + cid[u], cval[u]);
						else
							push = cval[u] == cl[u] && __ldcg(mark + cid[u]) != round;
						if (push) push = atomicExch(mark + cid[u], round) != round;
					}
					wq_add(push, cid[u], sbuf, nb, next, cnt);
				}
			});
	}
	// The list's rows (rows longer than kSrPiece become pieces).
	__device__ __forceinline__ void lists(const uint32_t* list, uint32_t n, uint32_t gwarp,
			uint32_t nwarps) {
		const uint32_t lane = threadIdx.x & 31u;
		const uint32_t per = n ? min(32u, (n - 1u) / nwarps + 1u) : 1u;
		for (uint64_t b = (uint64_t)gwarp * per; b < n; b += (uint64_t)nwarps * per) {
			uint32_t v = 0, start = 0, len = 0, c = 0;
			if (lane < per && b + lane < n) {
				v = __ldcg(list + b + lane);
				start = __ldg(off + v);
				len = __ldg(off + v + 1) - start;
				c = __ldcg(color + v);
			}
			unsigned big = __ballot_sync(0xffffffffu, len > kSrPiece);
			while (big) {
				const int t = __ffs(big) - 1;
				big &= big - 1u;
				const uint32_t bv = __shfl_sync(0xffffffffu, v, t);
				const uint32_t bs = __shfl_sync(0xffffffffu, start, t);
				const uint32_t k = (__shfl_sync(0xffffffffu, len, t) - 1u) / kSrPiece + 1u;
				u64 p = 0;
				if (lane == 0) p = atomicAdd(cnt + 1, (u64)k);
				p = __shfl_sync(0xffffffffu, p, 0) & ~kCoopTimeUp;
				for (uint32_t i = lane; i < k; i += 32u)
					if (p + i < a.max_pieces) a.pieces[p + i] = make_uint2(bv, bs + i * kSrPiece);
			}
			rows(start, len > kSrPiece ? 0u : len, c);
		}
		wq_flush(sbuf, nb, next, cnt);
	}
	__device__ __forceinline__ void pieces(uint32_t n, uint32_t gwarp, uint32_t nwarps) {
		const uint32_t lane = threadIdx.x & 31u;
		const uint32_t per = min(32u, (n - 1u) / nwarps + 1u);
		for (uint64_t b = (uint64_t)gwarp * per; b < n; b += (uint64_t)nwarps * per) {
			uint32_t start = 0, len = 0, c = 0;
			if (lane < per && b + lane < n) {
				const uint2 pc = __ldcg(a.pieces + b + lane);
				start = pc.y;
				len = min(__ldg(off + pc.x + 1) - start, kSrPiece);
				c = __ldcg(color + pc.x);
			}
			rows(start, len, c);
		}
		wq_flush(sbuf, nb, next, cnt);
	}
};

__global__ void __launch_bounds__(kSrThreads, 1)
scc_rest(SrArgs a, SrCtl* c) {
	__shared__ SrShared sh;
	const uint32_t tid = threadIdx.x, wid = tid >> 5;
	const uint32_t gtid = blockIdx.x * kSrThreads + tid, nthreads = gridDim.x * kSrThreads;
	const uint32_t gwarp = wid * gridDim.x + blockIdx.x, nwarps = gridDim.x * kSrWarps;
	const long long t0 = clock64();
	if (tid < sizeof(SrState) / 4)
		reinterpret_cast<uint32_t*>(&sh.st)[tid] =
				__ldcg(reinterpret_cast<const uint32_t*>(&c->st) + tid);
	__syncthreads();
	SrState t = sh.st;
	// counters rotate over three slots: a step fills cnt() and clears the slot
	// the next one fills, which was read before the last barrier but one
	auto cnt = [&]() { return c->ctr[t.slot]; };
	auto barrier = [&]() {
		// (every 16th step: reading the clock on the way to
		// every barrier took 5 % of a chain's time)
		if (gtid == 0 && (t.steps & 15u) == 0 && clock64() - t0 > a.cycles)
			atomicOr(cnt() + 1, kCoopTimeUp);
		if (!grid_barrier(&c->bar)) return false;
		if (tid < 2) sh.got[tid] = __ldcg(cnt() + tid);
		__syncthreads();
		return true;
	};
	auto fail = [&](unsigned bit) { if (tid == 0) atomicOr(&c->bar.err, bit); };
	// the vertices of rem[rsel] that take(v) picks, appended to `to`
	auto pick = [&](uint32_t* to, auto&& take) {
		uint32_t nb = 0;
		for (uint64_t i0 = (uint64_t)gwarp * 32u; i0 < t.n_rem; i0 += (uint64_t)nwarps * 32u) {
			const uint64_t i = i0 + (tid & 31u);
			const uint32_t v = i < t.n_rem ? __ldcg(a.rem[t.rsel] + i) : 0u;
			wq_add(i < t.n_rem && take(v), v, sh.sbuf[wid], nb, to, cnt());
		}
		wq_flush(sh.sbuf[wid], nb, to, cnt());
	};
	// expands list[lsel][0, n) into the other list; false: leave
	auto expand = [&](auto&& s) {
		t.steps++;
		s.lists(a.list[t.lsel], (uint32_t)t.n, gwarp, nwarps);
		if (!barrier()) return false;
		const u64 np = sh.got[1] & ~kCoopTimeUp;
		if (np > a.max_pieces) {
			fail(4u);
			return false;
		}
		if (np) {
			s.pieces((uint32_t)np, gwarp, nwarps);
			if (!barrier()) return false;
		}
		t.n = sh.got[0];
		t.lsel ^= 1u;
		if (t.n <= a.V) return true;
		fail(4u);
		return false;
	};

	for (bool up = false; t.n_rem > 0 && !up;) {
		if (gtid < 2) c->ctr[t.slot == 2u ? 0u : t.slot + 1u][gtid] = 0;
		if (t.phase == kSrColour) {
			// colours: the vertices' own; the first list is all of them
			t.round++;
			if (t.round > a.V + 1u) return fail(8u);
			for (uint64_t i = gtid; i < t.n_rem; i += nthreads) {
				const uint32_t v = __ldcg(a.rem[t.rsel] + i);
				a.color[v] = v;
				a.list[0][i] = v;
			}
			if (!barrier()) return;
			t.n = t.n_rem;
			t.lsel = 0;
			t.phase = kSrPush;
		} else if (t.phase == kSrPush) {
			t.stamp++;
			if (!expand(SrStep<true>(a, t.stamp, sh.sbuf[wid], a.list[t.lsel ^ 1u], cnt(),
					sh.win + wid)))
				return;
			if (t.n == 0) t.phase = kSrRoots;
		} else if (t.phase == kSrRoots) {
			// vertices that kept their own colour begin the backward search
			pick(a.list[t.lsel], [&](uint32_t v) {
				const bool root = __ldcg(a.color + v) == v;
				if (root) a.mark[v] = t.round;
				return root;
			});
			if (!barrier()) return;
			t.n = sh.got[0];
			t.phase = kSrSearch;
		} else if (t.phase == kSrSearch) {
			if (!expand(SrStep<false>(a, t.round, sh.sbuf[wid], a.list[t.lsel ^ 1u], cnt(),
					sh.win + wid)))
				return;
			if (t.n == 0) t.phase = kSrCollect;
		} else {
			// collected vertices are settled, the others stay for the next round
			pick(a.rem[t.rsel ^ 1u], [&](uint32_t v) {
				const bool keep = __ldcg(a.mark + v) != t.round;
				if (!keep) a.label[v] = __ldcg(a.color + v);
				return keep;
			});
			if (!barrier()) return;
			if (sh.got[0] >= t.n_rem) return fail(4u);     // a round settles some
			t.n_rem = sh.got[0];
			t.rsel ^= 1u;
			t.phase = kSrColour;
		}
		up = sh.got[1] >= kCoopTimeUp;
		t.slot = t.slot == 2u ? 0u : t.slot + 1u;
	}
	if (gtid == 0) c->st = t;
}

std::mutex g_coop_mu;
int g_coop[LG_TUNE_MAX_DEVICES];          // co-resident CTAs + 1, 0 = not probed

int coop_grid(int device) {
	std::lock_guard<std::mutex> lk(g_coop_mu);
	if (device < 0 || device >= LG_TUNE_MAX_DEVICES) return 0;
	if (!g_coop[device])
		g_coop[device] = 1 + coop_grid_size((const void*)scc_rest, kSrThreads, device);
	return coop_allowed(g_coop[device] - 1);
}

} // namespace

lg_status scc_flat_run(lg_snapshot* sn, const FlatCsr* fo, const FlatCsr* fi, uint32_t* label,
		uint64_t* trimmed, uint32_t* rounds, int* steps, bool* ran) {
	*ran = false;
	lg_store* s = sn->store;
	const int grid = coop_grid(s->device);
	if (grid <= 0) return LG_OK;
	unsigned ctas = (unsigned)grid;
	cudaStream_t st = s->stream;
	const uint64_t V = sn->V;
	const unsigned B = kListThreads;
	DevBuf buf(s->pool), ctrb(s->pool), pieces(s->pool);
	// color, mark, stamp, two lists of the vertices left, two working lists
	// (first the two searches' levels)
	LG_TRY(buf.reserve(7 * V * sizeof(uint32_t)));
	LG_TRY(ctrb.reserve(sizeof(SrCtl) + 4 * sizeof(u64)));
	uint32_t* w = buf.as<uint32_t>();
	SrArgs a;
	a.ooff = fo->off.as<uint32_t>();
	a.oids = fo->ids.as<uint32_t>();
	a.ioff = fi->off.as<uint32_t>();
	a.iids = fi->ids.as<uint32_t>();
	a.V = (uint32_t)V;
	a.label = label;
	a.color = w;
	a.mark = w + V;
	a.stamp = w + 2 * V;
	a.rem[0] = w + 3 * V;
	a.rem[1] = w + 4 * V;
	a.list[0] = w + 5 * V;
	a.list[1] = w + 6 * V;
	int32_t* fwd = reinterpret_cast<int32_t*>(a.list[0]);
	int32_t* bwd = reinterpret_cast<int32_t*>(a.list[1]);
	SrCtl* ctl = ctrb.as<SrCtl>();
	u64* ctr = reinterpret_cast<u64*>(ctl + 1);      // [0], [1] trim; [3] smallest
	u64* left = &ctl->st.n_rem;                      // the lists' length after the searches
	LG_CUDA(cudaMemsetAsync(ctl, 0, sizeof(SrCtl) + 3 * sizeof(u64), st), "clear");
	LG_CUDA(cudaMemsetAsync(ctr + 3, 0xff, sizeof(u64), st), "clear");
	const uint32_t* odeg = sn->out.deg.as<uint32_t>();
	const uint32_t* ideg = sn->in.deg.as<uint32_t>();
	scc_trim_flat<<<grid_for(V, B), B, 0, st>>>(odeg, ideg, V, label, a.mark, a.stamp, a.rem[1],
			ctr);
	LG_CUDA(cudaGetLastError(), "scc_trim");
	s->launches++;
	u64 h[2];
	LG_TRY(read_words(s, ctr, 2, h));
	const uint64_t n_rem = h[0];
	*trimmed = V - n_rem;
	*rounds = 0;
	*steps = 0;
	if (n_rem == 0) {
		*ran = true;
		return LG_OK;
	}
	// forward and backward from the pivot
	const uint32_t pivot = ~(uint32_t)h[1];
	SnapCsr out = sn->view(0), in = sn->view(1);
	lg_bfs_result r;
	bool done = false;
	LG_TRY(bfs_levels_over(s, fo->has_view ? fo->view(odeg) : out, fi, odeg, fo->E, pivot, fwd, &r,
			&done));
	if (!done) return LG_OK;
	*steps += r.top_down_steps + r.bottom_up_steps;
	LG_TRY(bfs_levels_over(s, fi->has_view ? fi->view(ideg) : in, fo, ideg, fi->E, pivot, bwd, &r,
			&done));
	if (!done) return LG_OK;
	*steps += r.top_down_steps + r.bottom_up_steps;
	uint32_t* best = reinterpret_cast<uint32_t*>(ctr + 3);
	scc_giant_min<<<grid_for(n_rem, B), B, 0, st>>>(a.rem[1], (uint32_t)n_rem, fwd, bwd, best);
	scc_giant_label<<<grid_for(n_rem, B), B, 0, st>>>(a.rem[1], (uint32_t)n_rem, fwd, bwd, best,
			label, a.rem[0], left);
	LG_CUDA(cudaGetLastError(), "scc_giant");
	s->launches += 2;
	// the rest
	a.max_pieces = (uint32_t)(2 * std::max(fo->E, fi->E) / kSrPiece + 1);
	LG_TRY(pieces.reserve((uint64_t)a.max_pieces * sizeof(uint2)));
	a.pieces = pieces.as<uint2>();
	a.cycles = coop_run_cycles();
	void* kargs[] = {&a, &ctl};
	for (;;) {
		LG_CUDA(coop_launch((const void*)scc_rest, &ctas, kSrThreads, kargs, 0, st, &ctl->bar),
				"scc_rest");
		s->launches++;
		constexpr int kWords = (int)(sizeof(SrState) / sizeof(u64)) + 2;
		static_assert(offsetof(SrCtl, bar) == offsetof(SrCtl, st) + sizeof(SrState) &&
				sizeof(SrState) % sizeof(u64) == 0 && kWords <= kReadWords, "state, then the barrier");
		u64 o[kWords];
		LG_TRY(read_words(s, reinterpret_cast<const u64*>(&ctl->st), kWords, o));
		const unsigned err = (unsigned)o[kWords - 1];  // the barrier's error word
		if (err & 1u) return set_error(LG_ETIMEOUT, "scc: a grid barrier wait ran out");
		if (err & 4u) return set_error(LG_ECUDA, "scc: a list count out of range");
		if (err & 8u) return set_error(LG_ETIMEOUT, "SCC did not converge");
		SrState t;
		std::memcpy(&t, o, sizeof(t));
		if (t.n_rem > 0) continue;
		*rounds = t.round + 1u;
		*steps += (int)t.steps;
		break;
	}
	*ran = true;
	return LG_OK;
}

} // namespace lg
