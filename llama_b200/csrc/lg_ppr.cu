// lg_ppr.cu - personalized PageRank for K seeds at once, as an N x K block.
//
// The reference has no personalized variant; this is the pull iteration of
// ll_b_pagerank_pull_ext::run (benchmark/benchmarks/pagerank.h:120-169) with
// the uniform teleport (1-d)/N replaced, per column k, by (1-d) on seed_k:
//   x0[:, k] = e_seed_k,   x'[t, k] = (1-d) [t == seed_k] + d * sum_{w in in(t)} x[w, k] / out_degree(w)
// for a fixed number of iterations, dangling mass dropped as in the reference.
//
// Layout: row-major V x K doubles of y = x / out_degree, so one in-edge
// (w -> t) reads the contiguous K-wide row of w; lane j of a warp owns columns
// j, j+32, ...  The iterations run over the snapshot's flat in-CSR
// (lg_flat.cuh: ids, head bits, rows with in-edges), its own when
// lg_snapshot_flatten made one, else one built for the call (without memory for
// it lg_ppr_walk.cu walks the levels): a warp takes a
// range of consecutive edges, loads the rows of kPprAhead of them before it
// adds any, and finishes a row where the next head bit stands.  A row over
// more than one range leaves a partial per range (carry_first, carry_last)
// that ppr_fixup adds in range order.  Rows without in-edges hold a constant
// after the first iteration and are written once.
//
// Bound by the row gathers (E x K x 8 bytes per iteration, mostly from L2 at
// 100 k vertices x 96 columns) and the instructions around them: a group of edges
// in which no row begins (most groups, rows being longer) is loaded and added
// without a test per edge: 145 us an iteration at 3.1 M edges (16 TB/s of rows),
// the mean over three snapshots of 1.5 to 3.1 M edges 122 (150 with the tests).
// x0 has one non-zero per column, but a bitmap of the rows that are not zero,
// looked up before the first two iterations load them, gained in the first what
// it cost in the second (844 us for those of the three snapshots against 862),
// and the code for it cost the others 8 us of 127.
// The form before it walked fragments and added an edge's row before it loaded
// the next one: one load per lane in flight, 2.1 TB/s of rows on a 3 M-arc graph
// with 96 columns.
//
// The K columns are processed in passes of a K-tile (a multiple of 32,
// LG_TUNE_PPR_KTILE): a pass runs every iteration on its columns, so a smaller
// tile re-reads the edge ids once more per pass but keeps the gathered rows of
// a pass narrower.  LG_TUNE_PPR_RANGE bounds the edges per warp range; smaller
// graphs get shorter ranges, so that every warp slot of the GPU has a few.
#include "lg_flat.cuh"
#include "lg_ppr.h"
#include "lg_tune.h"

#include <algorithm>
#include <vector>

namespace lg {

constexpr int kPprThreads = 256;
constexpr int kPprWarps = kPprThreads / 32;
// Edges whose rows a warp loads ahead: about 8 to 32 loads per lane in
// flight.  Up to 128 columns the registers are capped for three resident CTAs
// (96 columns, 3 M edges: 252 -> 207 us an iteration; with 8 edges ahead and
// two CTAs 237).
template <int CPL>
constexpr int kPprAhead = CPL <= 2 ? 8 : 4;

struct PprArgs {
	const uint32_t* ids;      // E, the flat in-CSR
	const uint32_t* heads;
	const uint32_t* nz_rows;
	const uint32_t* nz_off;
	const uint32_t* seg;      // nranges: rows begun before each range
	uint32_t E, R;
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
	uint32_t range;           // edges per warp range, a multiple of 32
};

// Row of vertex v (out-degree dg, first seed sf) has the in-sums s.
template <int CPL>
__device__ __forceinline__ void ppr_finish(const PprArgs& a, uint32_t v, uint32_t dg, uint32_t sf,
		const double* s) {
	const uint32_t lane = threadIdx.x & 31u;
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
__device__ __forceinline__ void ppr_carry(double* to, const PprArgs& a, uint32_t r,
		const double* s) {
#pragma unroll
	for (int i = 0; i < CPL; i++)
		to[(uint64_t)r * a.K + a.col0 + (threadIdx.x & 31u) + 32 * i] = s[i];
}

template <int CPL>
__global__ void __launch_bounds__(kPprThreads, CPL <= 4 ? 3 : 2)
ppr_step(PprArgs a) {
	constexpr int U = kPprAhead<CPL>;
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t r = blockIdx.x * kPprWarps + (threadIdx.x >> 5);
	if (r >= a.nranges) return;
	const char* y0 = reinterpret_cast<const char*>(a.y + a.col0 + lane);
	const uint32_t pitch = a.K * (uint32_t)sizeof(double);
	const uint32_t e0 = r * a.range;
	const uint32_t e1 = a.E - e0 < a.range ? a.E : e0 + a.range;
	uint32_t next = __ldg(a.seg + r);        // rows begun so far; next - 1 is the open one
	bool before = true;                      // the open row began before the range
	bool open = !(__ldg(a.heads + (e0 >> 5)) & 1u);
	double acc[CPL];
#pragma unroll
	for (int i = 0; i < CPL; i++) acc[i] = 0.0;
	for (uint32_t base = e0; base < e1; base += 32) {
		const uint32_t n = min(32u, e1 - base);
		const uint32_t hw = __ldg(a.heads + (base >> 5));
		const uint32_t id = lane < n ? __ldcs(a.ids + base + lane) : 0u;
		// lane h: vertex, out-degree and seed of the row that h heads of this
		// word leave open
		const uint32_t k = next - 1u + lane;
		uint32_t mv = 0, md = 0, ms = kNoSeed;
		if (k < a.R && lane <= (uint32_t)__popc(hw)) {
			mv = __ldg(a.nz_rows + k);
			md = __ldg(a.outdeg + mv);
			ms = __ldg(a.seed_first + mv);
		}
		for (uint32_t g = 0; g < n; g += U) {
			double v[U][CPL];
			const unsigned all = (1u << U) - 1u;
			const bool whole = g + U <= n;
#pragma unroll
			for (int u = 0; u < U; u++) {
				const uint32_t src = __shfl_sync(0xffffffffu, id, g + u);
				const double* row = reinterpret_cast<const double*>(y0 + (uint64_t)src * pitch);
				if (whole) {
#pragma unroll
					for (int i = 0; i < CPL; i++) v[u][i] = __ldg(row + 32 * i);
				} else {
#pragma unroll
					for (int i = 0; i < CPL; i++)
						v[u][i] = g + u < n ? __ldg(row + 32 * i) : 0.0;
				}
			}
			if (((hw >> g) & all) == 0) {                        // no row begins here
#pragma unroll
				for (int u = 0; u < U; u++)
#pragma unroll
					for (int i = 0; i < CPL; i++) acc[i] += v[u][i];
				continue;
			}
#pragma unroll
			for (int u = 0; u < U; u++) {
				if ((hw >> (g + u)) & 1u) {              // warp-uniform
					const int h = __popc(hw & ((1u << (g + u)) - 1u));
					if (open) {
						const uint32_t fv = __shfl_sync(0xffffffffu, mv, h);
						const uint32_t fd = __shfl_sync(0xffffffffu, md, h);
						const uint32_t fs = __shfl_sync(0xffffffffu, ms, h);
						if (before) ppr_carry<CPL>(a.carry_first, a, r, acc);
						else ppr_finish<CPL>(a, fv, fd, fs, acc);
					}
					open = true;
					before = false;
#pragma unroll
					for (int i = 0; i < CPL; i++) acc[i] = 0.0;
				}
#pragma unroll
				for (int i = 0; i < CPL; i++) acc[i] += v[u][i];
			}
		}
		next += __popc(hw);
	}
	// the row open at the end of the range
	if (before) {
		ppr_carry<CPL>(a.carry_first, a, r, acc);
	} else if (e1 >= a.E || (__ldg(a.heads + (e1 >> 5)) & 1u)) {
		const uint32_t v = __ldg(a.nz_rows + next - 1u);
		ppr_finish<CPL>(a, v, __ldg(a.outdeg + v), __ldg(a.seed_first + v), acc);
	} else {
		ppr_carry<CPL>(a.carry_last, a, r, acc);
	}
}

// seg[r] = rows begun before edge r * range.
__global__ void ppr_ranges(const uint32_t* nz_off, uint32_t R, uint32_t nranges, uint32_t range,
		uint32_t* seg) {
	const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
	if (r >= nranges) return;
	const uint32_t x = r * range;
	uint32_t lo = 0, hi = R;
	while (lo < hi) {
		const uint32_t mid = (lo + hi) >> 1;
		if (__ldg(nz_off + mid) < x) lo = mid + 1; else hi = mid;
	}
	seg[r] = lo;
}

// Rows over more than one range: the warp of boundary q (edge q * range) adds
// the partials of the row that began in range q - 1 and crosses it, in range
// order; the partials of a row over more than kPprLong ranges are split
// between the CTA's warps, whose sums are added in warp order.
constexpr uint32_t kPprLong = 32;
template <int CPL>
__global__ void __launch_bounds__(kPprThreads)
ppr_fixup(PprArgs a) {
	__shared__ double part[kPprWarps][CPL * 32];
	__shared__ uint32_t s_row[kPprWarps], s_last[kPprWarps];
	const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
	const uint32_t q0 = blockIdx.x * kPprWarps + 1u;
	const uint32_t q = q0 + wid;
	const uint32_t c0 = a.col0 + lane;
	auto sum = [&](uint32_t x0, uint32_t x1, double* t) {     // ranges [x0, x1)
#pragma unroll 4
		for (uint32_t x = x0; x < x1; x++)
#pragma unroll
			for (int i = 0; i < CPL; i++)
				t[i] += __ldcg(a.carry_first + (uint64_t)x * a.K + c0 + 32 * i);
	};
	uint32_t row = kNoId, last = 0;
	if (q < a.nranges) {
		const uint32_t e = q * a.range;
		const uint32_t seg = __ldg(a.seg + q);
		if (!(__ldg(a.heads + (e >> 5)) & 1u) && seg > 0
				&& __ldg(a.nz_off + seg - 1u) >= e - a.range) {
			row = seg - 1u;
			const uint32_t end = seg < a.R ? __ldg(a.nz_off + seg) : a.E;
			last = (end - 1u) / a.range;
		}
	}
	const bool longer = row != kNoId && last - q >= kPprLong;
	if (lane == 0) {
		s_row[wid] = longer ? row : kNoId;
		s_last[wid] = last;
	}
	double t[CPL];
	if (row != kNoId && !longer) {
#pragma unroll
		for (int i = 0; i < CPL; i++)
			t[i] = __ldcg(a.carry_last + (uint64_t)(q - 1u) * a.K + c0 + 32 * i);
		sum(q, last + 1u, t);
		const uint32_t v = __ldg(a.nz_rows + row);
		ppr_finish<CPL>(a, v, __ldg(a.outdeg + v), __ldg(a.seed_first + v), t);
	}
	__syncthreads();
	for (uint32_t w = 0; w < kPprWarps; w++) {                // block-uniform
		if (s_row[w] == kNoId) continue;
		const uint32_t b = q0 + w, n = s_last[w] + 1u - b;
		const uint32_t per = (n + kPprWarps - 1u) / kPprWarps;
		const uint32_t x0 = b + min(n, wid * per), x1 = b + min(n, (wid + 1u) * per);
#pragma unroll
		for (int i = 0; i < CPL; i++)
			t[i] = wid == 0 ? __ldcg(a.carry_last + (uint64_t)(b - 1u) * a.K + c0 + 32 * i) : 0.0;
		sum(x0, x1, t);
#pragma unroll
		for (int i = 0; i < CPL; i++) part[wid][lane + 32 * i] = t[i];
		__syncthreads();
		if (wid == 0) {
			for (uint32_t o = 1; o < kPprWarps; o++)
#pragma unroll
				for (int i = 0; i < CPL; i++) t[i] += part[o][lane + 32 * i];
			const uint32_t v = __ldg(a.nz_rows + s_row[w]);
			ppr_finish<CPL>(a, v, __ldg(a.outdeg + v), __ldg(a.seed_first + v), t);
		}
		__syncthreads();
	}
}

// seed_first[v] = first index of v's seeds in the sorted list.
__global__ void ppr_seed_index(const uint2* seed_col, uint32_t n, uint32_t* seed_first) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n && (i == 0 || seed_col[i - 1].x != seed_col[i].x)) seed_first[seed_col[i].x] = i;
}

__global__ void ppr_seed_init(const uint2* seed_col, uint32_t n, const uint32_t* outdeg,
		uint32_t K, double* y) {
	const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const uint32_t v = seed_col[i].x, c = seed_col[i].y;
	const uint32_t dg = outdeg[v];
	y[(uint64_t)v * K + c] = dg ? 1.0 / (double)dg : 0.0;
}

// Seeds without in-edges, columns [col0, col1): y = (1-d) / out_degree from
// the first iteration on (other rows without in-edges stay 0).
__global__ void ppr_seed_empty(const uint2* seed_col, uint32_t n, const uint32_t* off,
		const uint32_t* outdeg, double tele, uint32_t K, uint32_t col0, uint32_t col1, double* y) {
	const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const uint32_t v = seed_col[i].x, c = seed_col[i].y;
	if (c < col0 || c >= col1 || __ldg(off + v + 1) != __ldg(off + v)) return;
	const uint32_t dg = outdeg[v];
	y[(uint64_t)v * K + c] = dg ? tele / (double)dg : 0.0;
}

// Result rows of the vertices without in-edges: (1-d) at their own seeds.
__global__ void ppr_empty_rows(const uint32_t* off, uint64_t V, const uint32_t* seed_first,
		const uint2* seed_col, uint32_t n_seeds, double tele, uint32_t K, double* x) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
	for (uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < V; v += nwarps) {
		if (__ldg(off + v + 1) != __ldg(off + v)) continue;
		for (uint32_t c = lane; c < K; c += 32) x[v * K + c] = 0.0;
		__syncwarp();
		for (uint32_t q = __ldg(seed_first + v); q < n_seeds && seed_col[q].x == v; q++)
			if (lane == 0) x[v * K + seed_col[q].y] = tele;
	}
}

__global__ void ppr_seed_x(const uint2* seed_col, uint32_t n, uint32_t K, double* x) {
	const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) x[(uint64_t)seed_col[i].x * K + seed_col[i].y] = 1.0;
}

template <int CPL>
void launch_ppr_iteration(const PprArgs& a, cudaStream_t st) {
	ppr_step<CPL><<<grid_for(a.nranges, kPprWarps), kPprThreads, 0, st>>>(a);
	if (a.nranges > 1)
		ppr_fixup<CPL><<<grid_for(a.nranges - 1, kPprWarps), kPprThreads, 0, st>>>(a);
}

} // namespace lg

using namespace lg;

extern "C" lg_status lg_ppr(lg_snapshot* const* snaps, int n_snaps, const int64_t* seeds,
		int K, int iterations, double damping, double* out) {
	clear_error();
	if (!snaps || n_snaps <= 0 || !seeds || !out) return set_error(LG_EINVAL, "null argument");
	if (K <= 0 || K > 256 || K % 32 != 0)
		return set_error(LG_ENOTSUP, "K must be a multiple of 32 in [32, 256]");
	if (!(damping > 0.0 && damping < 1.0)) return set_error(LG_EINVAL, "damping must be in (0, 1)");
	if (iterations < 0) return set_error(LG_EINVAL, "iterations must be >= 0");
	lg_store* s = snaps[0]->store;
	const uint64_t V = snaps[0]->V;
	for (int i = 0; i < n_snaps; i++) {
		if (!snaps[i] || snaps[i]->store != s || snaps[i]->V != V)
			return set_error(LG_EINVAL, "snapshots must share the store and max_nodes");
		if (!snaps[i]->in.present) return set_error(LG_ESTATE, "PPR needs the in-CSR");
	}
	for (int k = 0; k < K; k++)
		if (seeds[k] < 0 || (uint64_t)seeds[k] >= V)
			return set_error(LG_EINVAL, "seed %lld out of range", (long long)seeds[k]);
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	cudaStream_t st = s->stream;

	// seeds sorted by vertex -> (vertex, column) pairs and a per-vertex index
	std::vector<uint2> sc(K);
	for (int k = 0; k < K; k++) sc[k] = make_uint2((uint32_t)seeds[k], (uint32_t)k);
	std::sort(sc.begin(), sc.end(), [](uint2 x, uint2 y) { return x.x < y.x || (x.x == y.x && x.y < y.y); });

	const uint64_t row = (uint64_t)K * 8;
	// the store's scratch (kept for the next call, contents not preserved)
	DevBuf* yb = s->scratch;         // scratch[0], [1]: the two V x K blocks
	DevBuf& carry = s->scratch[2];
	DevBuf& seedb = s->scratch[3];
	DevBuf& firstb = s->scratch[4];
	DevBuf& resb = s->scratch[5];
	DevBuf& segb = s->scratch[6];
	LG_TRY(yb[0].reserve(V * row));
	LG_TRY(yb[1].reserve(V * row));
	LG_TRY(seedb.reserve(K * sizeof(uint2)));
	LG_TRY(firstb.reserve(V * 4));
	// launch parameters: columns per pass (a multiple of 32 dividing K) and
	// the most edges per warp range
	int ktile = (int)tune_value(s->device, LG_TUNE_PPR_KTILE);
	ktile = std::min(K, std::max(32, ktile - ktile % 32));
	while (K % ktile) ktile -= 32;
	const uint64_t max_range = (uint64_t)tune_value(s->device, LG_TUNE_PPR_RANGE) & ~31ull;
	int sms = 148;
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
	const bool dev_out = is_device_pointer(out);
	double* res = out;
	if (!dev_out) { LG_TRY(resb.reserve((uint64_t)n_snaps * V * row)); res = resb.as<double>(); }
	const uint2* seeds_d = seedb.as<uint2>();
	const unsigned kb = grid_for(K, 256);
	LG_CUDA(cudaMemcpyAsync(seedb.p, sc.data(), K * sizeof(uint2), cudaMemcpyHostToDevice, st), "h2d");
	LG_CUDA(cudaMemsetAsync(firstb.p, 0xff, V * 4, st), "memset");
	ppr_seed_index<<<kb, 256, 0, st>>>(seeds_d, (uint32_t)K, firstb.as<uint32_t>());
	s->h2d_bytes += K * sizeof(uint2);
	s->launches++;

	// largest snapshot first: the scratch of the others fits into its own
	std::vector<int> order(n_snaps);
	for (int i = 0; i < n_snaps; i++) order[i] = i;
	std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
		return snaps[x]->in.n_edges > snaps[y]->in.n_edges;
	});
	for (int i : order) {
		lg_snapshot* sn = snaps[i];
		double* xo = res + (uint64_t)i * V * K;
		const uint32_t* outdeg = sn->out.deg.as<uint32_t>();
		if (iterations == 0) {
			LG_CUDA(cudaMemsetAsync(xo, 0, V * row, st), "memset");
			ppr_seed_x<<<kb, 256, 0, st>>>(seeds_d, K, K, xo);
			s->launches++;
			continue;
		}
		const FlatCsr* f = sn->flat[1];
		if (!f) {
			if (!s->flat_scratch) s->flat_scratch = new FlatCsr;
			const lg_status fs = build_flat(sn, 1, *s->flat_scratch, false, true, false);
			if (fs == LG_ENOMEM || fs == LG_ENOTSUP) {
				// over the levels instead, with what the flat copy took
				clear_error();
				LG_CUDA(cudaStreamSynchronize(st), "ppr");
				delete s->flat_scratch;
				s->flat_scratch = nullptr;
				LG_CUDA(cudaMemsetAsync(yb[0].p, 0, V * row, st), "memset");
				ppr_seed_init<<<kb, 256, 0, st>>>(seeds_d, K, outdeg, K, yb[0].as<double>());
				s->launches++;
				LG_TRY(ppr_walk(sn, PprSeeds{firstb.as<uint32_t>(), seeds_d, (uint32_t)K},
						(uint32_t)K, ktile, iterations, damping, yb[0].as<double>(),
						yb[1].as<double>(), carry, xo));
				continue;
			}
			LG_TRY(fs);
			f = s->flat_scratch;
		}
		PprArgs a;
		a.ids = f->ids.as<uint32_t>();
		a.heads = f->heads();
		a.nz_rows = f->nz_rows();
		a.nz_off = f->nz_off();
		a.E = (uint32_t)f->E;
		a.R = (uint32_t)f->R;
		// about four ranges for each of 24 warps per SM, a multiple of 32 edges
		// (two or one: 0 to 17 % slower, five: 2 %)
		const uint64_t even = ((f->E + (uint64_t)sms * 96u - 1) / ((uint64_t)sms * 96u) + 31) & ~31ull;
		a.range = (uint32_t)std::min(max_range, std::max<uint64_t>(even, 32));
		a.nranges = (uint32_t)((f->E + a.range - 1) / a.range);
		LG_TRY(segb.reserve(std::max<uint64_t>(a.nranges, 1) * 4));
		LG_TRY(carry.reserve(2ull * std::max<uint32_t>(a.nranges, 1) * row));
		a.seg = segb.as<uint32_t>();
		a.outdeg = outdeg;
		a.d = damping;
		a.tele = 1.0 - damping;
		a.seed_first = firstb.as<uint32_t>();
		a.seed_col = seeds_d;
		a.n_seeds = (uint32_t)K;
		a.carry_first = carry.as<double>();
		a.carry_last = carry.as<double>() + (uint64_t)a.nranges * K;
		a.K = (uint32_t)K;
		const uint32_t* off = f->off.as<uint32_t>();
		LG_CUDA(cudaMemsetAsync(yb[0].p, 0, V * row, st), "memset");
		LG_CUDA(cudaMemsetAsync(yb[1].p, 0, V * row, st), "memset");
		ppr_seed_init<<<kb, 256, 0, st>>>(seeds_d, K, outdeg, K, yb[0].as<double>());
		if (a.nranges)
			ppr_ranges<<<grid_for(a.nranges, 256), 256, 0, st>>>(a.nz_off, a.R, a.nranges, a.range,
					segb.as<uint32_t>());
		ppr_empty_rows<<<(unsigned)sms * 8u, 256, 0, st>>>(off, V, firstb.as<uint32_t>(), seeds_d,
				(uint32_t)K, a.tele, (uint32_t)K, xo);
		s->launches += 2 + (a.nranges > 0);
		// column tiles are independent: each runs all iterations on its columns
		for (int c0 = 0; c0 < K; c0 += ktile) {
			a.col0 = (uint32_t)c0;
			for (int it = 0; it < iterations; it++) {
				a.y = yb[it & 1].as<double>();
				a.y_next = yb[(it + 1) & 1].as<double>();
				a.x_out = (it == iterations - 1) ? xo : nullptr;
				if (it < 2) {
					// it 0: the block written now; it 1: the first one, read by then
					ppr_seed_empty<<<kb, 256, 0, st>>>(seeds_d, (uint32_t)K, off, outdeg, a.tele,
							(uint32_t)K, (uint32_t)c0, (uint32_t)(c0 + ktile), a.y_next);
					s->launches++;
				}
				if (a.nranges == 0) continue;
				switch (ktile / 32) {
				case 1: launch_ppr_iteration<1>(a, st); break;
				case 2: launch_ppr_iteration<2>(a, st); break;
				case 3: launch_ppr_iteration<3>(a, st); break;
				case 4: launch_ppr_iteration<4>(a, st); break;
				case 5: launch_ppr_iteration<5>(a, st); break;
				case 6: launch_ppr_iteration<6>(a, st); break;
				case 7: launch_ppr_iteration<7>(a, st); break;
				default: launch_ppr_iteration<8>(a, st); break;
				}
				s->launches += a.nranges > 1 ? 2 : 1;
			}
		}
		LG_CUDA(cudaGetLastError(), "ppr_step");
	}
	if (!dev_out) LG_TRY(copy_out(s, out, res, (uint64_t)n_snaps * V * row));
	LG_CUDA(cudaStreamSynchronize(st), "ppr");
	return LG_OK;
}
