// lg_adjoint.cu - weighted PageRank to a fixed point and its adjoint.
//
// No reference counterpart: the forward is the pull iteration of
// ll_b_pagerank_pull_ext::run (benchmark/benchmarks/pagerank.h:120-169)
// with per-edge weights P(w->t) and a teleport vector v,
//     x = (1-d) v + d P^T x                                     (forward)
// iterated from x = v until sum |x' - x| < tol.  The backward differentiates
// the fixed point implicitly: with g = dL/dx,
//     lambda = g + d P lambda                                   (adjoint)
// iterated the same way over OUT-edges, then
//     dL/dv = (1-d) lambda,   dL/dP(w->t) = d lambda[t] x[w].
// Only the converged x is kept between the two calls (the "tape"), no
// iterate is stored.
//
// Edge weights and their gradients are indexed by the snapshot's
// out-adjacency order (the order lg_snapshot_adjacency(dir 0) returns).  On
// first use a snapshot gets its live adjacency flattened in both directions
// (lg_flat.cuh) and a map from every flat in-edge to its out-adjacency
// position; the flat out-CSR lists the edges in exactly that order, so the
// backward sweep reads the weights as given and the forward gathers them
// once per call into in-edge order.
//
// Both solves run every iteration inside one cooperative launch
// (lg_flat_run.cuh) with an affine op: y[v] = base[v] + d * sum over v's edges
// k of w[k] * x[nbr(k)].  The CTAs publish their parts of the residual
// sum |y - x| before the iteration's barrier and each adds them up in the same
// order, so every CTA stops at the first one below tol, with no launch or wait
// per iteration, and calls on the same input give the same bits.  Bound by the gathers of
// x and the weights' 8 bytes an edge above some 10^6 edges (15 M edges: 89 us an
// iteration against 158 us for a launch per iteration at 16.8 M), by the barrier
// and the loads around it below (30 k edges: 7 us against 14).
#include "lg_flat_run.cuh"
#include "lg_tune.h"

#include <cmath>
#include <cstddef>
#include <cstring>
#include <mutex>

namespace lg {

constexpr uint32_t kNoPos = 0xffffffffu;

// The iterations y = base + d * (weighted pull of x) over a flat CSR.
struct AffRunOp {
	static constexpr bool kResidual = true;
	const uint32_t* nz_rows;
	const double* w;
	const double* base;
	const double* x;           // rewritten between iterations: plain loads
	double* y;
	double d;
	uint32_t E;
	__device__ __forceinline__ void values(uint32_t eb, const uint32_t (&id)[kFlatPerLane],
			double (&v)[kFlatPerLane]) const {
		double wv[kFlatPerLane];
		if (eb + kFlatPerLane <= E) {
			asm("ld.global.cs.v4.f64 {%0, %1, %2, %3}, [%4];"
				: "=d"(wv[0]), "=d"(wv[1]), "=d"(wv[2]), "=d"(wv[3]) : "l"(w + eb));
			asm("ld.global.cs.v4.f64 {%0, %1, %2, %3}, [%4];"
				: "=d"(wv[4]), "=d"(wv[5]), "=d"(wv[6]), "=d"(wv[7]) : "l"(w + eb + 4));
		} else {
#pragma unroll
			for (int i = 0; i < kFlatPerLane; i++) wv[i] = eb + i < E ? __ldcs(w + eb + i) : 0.0;
		}
#pragma unroll
		for (int i = 0; i < kFlatPerLane; i++)
			v[i] = id[i] != kNoId ? __dmul_rn(wv[i], x[id[i]]) : 0.0;
	}
	struct Row { uint32_t v; double base; };
	__device__ __forceinline__ Row row(uint32_t k) const {
		const uint32_t v = __ldg(nz_rows + k);
		return Row{v, __ldg(base + v)};
	}
	__device__ __forceinline__ double old(const Row& r) const { return x[r.v]; }
	__device__ __forceinline__ double finish(const Row& r, double s, double xv) const {
		const double yv = __dadd_rn(r.base, __dmul_rn(d, s));
		y[r.v] = yv;
		return fabs(yv - xv);
	}
};

struct AffRunArgs {
	FlatTiles a;
	const uint32_t* off;
	const uint32_t* nz_rows;
	const double* w;
	const double* base;
	double* xa;                // the start; results of even iteration counts
	double* xb;
	double d, tol;
	uint32_t V;
	int first, end;            // the launch's iterations: first .. end - 1
};

__global__ void __launch_bounds__(kRunThreads, 1)
aff_run(AffRunArgs g, RunCtl* c) {
	extern __shared__ __align__(16) unsigned char run_smem[];
	RunShared& sh = *reinterpret_cast<RunShared*>(run_smem);
	const uint32_t gtid = blockIdx.x * kRunThreads + threadIdx.x;
	const uint32_t nthreads = gridDim.x * kRunThreads;
	uint32_t t0, t1;
	run_share(g.a.ntiles, &t0, &t1);
	const uint32_t seg = t0 < t1 ? __ldg(g.a.tile_seg + t0) : 0u;
	AffRunOp op;
	op.nz_rows = g.nz_rows;
	op.w = g.w;
	op.base = g.base;
	op.d = g.d;
	op.E = g.a.E;
	AffRunOp::Row cross = {};
	double resid = 0.0;
	int it = g.first;
	for (; it < g.end; it++) {
		op.x = (it & 1) ? g.xb : g.xa;
		op.y = (it & 1) ? g.xa : g.xb;
		double extra = 0.0;
		if (it < 2) {
			// rows without edges: y = base in every iteration, written into
			// both vectors; the first step's change counts
			for (uint64_t v = gtid; v < g.V; v += nthreads)
				if (__ldg(g.off + v + 1) == __ldg(g.off + v)) {
					const double b = __ldg(g.base + v);
					if (it == 0) extra += fabs(b - op.x[v]);
					op.y[v] = b;
				}
		}
		if (!run_iteration(g.a, op, c, sh, t0, t1, seg, extra, it & 1, it == g.first, cross,
				&resid))
			return;
		if (resid < g.tol) {
			it++;
			break;
		}
	}
	if (gtid == 0) {
		c->iters = (uint32_t)it;
		c->resid = resid;
	}
}

// --- per-snapshot maps ----------------------------------------------------

// row_of[k] = the vertex whose row holds edge k of a flat CSR (lane j of the
// warp owning tile t: edges 256 t + 8 j .. + 7).
constexpr int kMapWarps = 8;
__device__ __forceinline__ void edge_rows(const uint32_t* heads, const uint32_t* nz_rows,
		const uint32_t* tile_seg, uint32_t E, uint32_t t, uint32_t (&v)[kFlatPerLane]) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t eb = t * kFlatTile + lane * kFlatPerLane;
	const uint32_t hb = __ldg(reinterpret_cast<const unsigned char*>(heads)
			+ (size_t)t * (kFlatTile / 8) + lane);
	uint32_t before = __popc(hb);               // heads in the lanes to the left
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t q = __shfl_up_sync(0xffffffffu, before, o);
		if (lane >= (uint32_t)o) before += q;
	}
	before -= __popc(hb);
	uint32_t row = __ldg(tile_seg + t) + before - 1u;
	uint32_t x = eb < E && !(hb & 1u) ? __ldg(nz_rows + row) : 0u;
#pragma unroll
	for (int i = 0; i < kFlatPerLane; i++) {
		if ((hb >> i) & 1u) x = __ldg(nz_rows + ++row);
		v[i] = x;
	}
}

__global__ void __launch_bounds__(kMapWarps * 32)
adj_sources(const uint32_t* heads, const uint32_t* nz_rows, const uint32_t* tile_seg, uint32_t E,
		uint32_t ntiles, uint32_t* src) {
	const uint32_t t = blockIdx.x * kMapWarps + (threadIdx.x >> 5);
	if (t >= ntiles) return;
	uint32_t v[kFlatPerLane];
	edge_rows(heads, nz_rows, tile_seg, E, t, v);
	const uint32_t eb = t * kFlatTile + (threadIdx.x & 31u) * kFlatPerLane;
#pragma unroll
	for (int i = 0; i < kFlatPerLane; i++)
		if (eb + i < E) src[eb + i] = v[i];
}

// in_pos[k] for every edge k = (w -> t) of the flat in-CSR: its out-adjacency
// position, found by binary search of t in w's out-fragments (each sorted by
// target id) and read from out_pos, the out-CSR's virtual slots' positions.
__global__ void __launch_bounds__(kMapWarps * 32)
adj_in_map(const uint32_t* ids, const uint32_t* heads, const uint32_t* nz_rows,
		const uint32_t* tile_seg, uint32_t E, uint32_t ntiles, SnapCsr out,
		const uint32_t* frag_start, const uint32_t* out_pos, uint32_t* in_pos, uint32_t* bad) {
	const uint32_t tile = blockIdx.x * kMapWarps + (threadIdx.x >> 5);
	if (tile >= ntiles) return;
	uint32_t v[kFlatPerLane];
	edge_rows(heads, nz_rows, tile_seg, E, tile, v);
	const uint32_t eb = tile * kFlatTile + (threadIdx.x & 31u) * kFlatPerLane;
	bool miss = false;
#pragma unroll
	for (int i = 0; i < kFlatPerLane; i++) {
		if (eb + i >= E) break;
		const uint32_t t = v[i], w = __ldg(ids + eb + i);
		uint32_t found = kNoPos;
		const uint32_t f1 = __ldg(out.frag_off + w + 1);
		for (uint32_t f = __ldg(out.frag_off + w); f < f1 && found == kNoPos; f++) {
			const uint2 of = out.frags[f];
			const uint32_t* at = out.lt->ids[frag_level(of)] + of.x;
			uint32_t lo = 0, hi = frag_len(of);
			while (lo < hi) {
				const uint32_t mid = (lo + hi) >> 1;
				if (__ldg(at + mid) < t) lo = mid + 1; else hi = mid;
			}
			// the live copy of (w, t): skip deleted duplicates
			const uint32_t k = __ldg(frag_start + f);
			for (uint32_t j = lo; j < frag_len(of) && __ldg(at + j) == t; j++) {
				const uint32_t p = __ldg(out_pos + k + j);
				if (p != kNoPos) { found = p; break; }
			}
		}
		in_pos[eb + i] = found;
		miss |= found == kNoPos;
	}
	if (miss) atomicOr(bad, 1u);
}

__global__ void gather_weights(const uint32_t* map, uint64_t n, const double* w,
		double* out) {
	const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) out[i] = w[map[i]];
}

__global__ void scale_vec(const double* a, double s, uint64_t n, double* out) {
	const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) out[i] = s * a[i];
}

__global__ void edge_grad(const uint32_t* src, const uint32_t* dst, uint64_t E, double d,
		const double* lam, const double* x, double* out) {
	const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (p < E) out[p] = d * (lam[dst[p]] * x[src[p]]);
}

} // namespace lg

using namespace lg;

struct lg_adjoint_maps {
	FlatCsr fin, fout;     // the snapshot's live adjacency, flat, per direction
	DevBuf in_pos;         // E u32: out-adjacency position of each flat in-edge
	DevBuf src;            // E u32: source of each out-adjacency position
	uint64_t E = 0;
	// solve buffers, reused by every call on the snapshot
	DevBuf xa, xb, base, win, run, stage_w, stage_v, stage_g;
};

struct lg_adjoint {
	lg_snapshot* snap = nullptr;
	double d = 0.85, tol = 1e-12;
	int max_iter = 0;
	DevBuf x, w;           // converged scores; the weights, out-adjacency order
	explicit lg_adjoint(const std::shared_ptr<lg::CallPool>& pool) : x(pool), w(pool) {}
};

namespace {

lg_status build_maps(lg_snapshot* sn, lg_adjoint_maps* m) {
	lg_store* s = sn->store;
	cudaStream_t st = s->stream;
	const uint64_t E = m->E;
	// flat CSRs of both directions, the out-edges' sources, and every in-edge's
	// place among the out-edges
	LG_TRY(build_flat(sn, 1, m->fin, false));
	LG_TRY(build_flat(sn, 0, m->fout, false, false));
	if (m->fin.E != E || m->fout.E != E)
		return set_error(LG_EINVAL, "the in- and out-CSR of the snapshot differ in edge count");
	DevBuf out_pos(s->pool), badb(s->pool);
	LG_TRY(out_pos.reserve(std::max<uint64_t>(sn->out.n_frag_slots, 1) * 4));
	LG_TRY(m->src.reserve(std::max<uint64_t>(E, 1) * 4));
	LG_TRY(m->in_pos.reserve(std::max<uint64_t>(E, 1) * 4));
	LG_TRY(badb.reserve(8));
	LG_CUDA(cudaMemsetAsync(badb.p, 0, 8, st), "memset");
	LG_TRY(flat_positions(sn, 0, m->fout, out_pos.as<uint32_t>()));
	if (E > 0) {
		const FlatCsr &fi = m->fin, &fo = m->fout;
		adj_sources<<<grid_for(fo.ntiles, kMapWarps), kMapWarps * 32, 0, st>>>(fo.heads(),
				fo.nz_rows(), fo.tile_seg(), (uint32_t)E, fo.ntiles, m->src.as<uint32_t>());
		adj_in_map<<<grid_for(fi.ntiles, kMapWarps), kMapWarps * 32, 0, st>>>(
				fi.ids.as<uint32_t>(), fi.heads(), fi.nz_rows(), fi.tile_seg(), (uint32_t)E,
				fi.ntiles, sn->view(0), sn->out.frag_start(), out_pos.as<uint32_t>(),
				m->in_pos.as<uint32_t>(), badb.as<uint32_t>());
		LG_CUDA(cudaGetLastError(), "adjoint maps");
		s->launches += 2;
	}
	unsigned long long bad = 0;
	LG_TRY(read_words(s, badb.as<unsigned long long>(), 1, &bad));
	if (bad)
		return set_error(LG_EINVAL, "out- and in-CSR of the snapshot disagree, or a "
				"fragment is not sorted by neighbour id (code %u)", (unsigned)bad);
	return LG_OK;
}

lg_status ensure_maps(lg_snapshot* sn) {
	if (sn->adj_maps) return LG_OK;
	const uint64_t E = sn->out.n_edges;
	if (E > 0xffffffffull - 2 * kFlatTile)
		return set_error(LG_ENOTSUP, "more than 2^32 - %u live edges", 2 * kFlatTile);
	lg_adjoint_maps* m = new (std::nothrow) lg_adjoint_maps();
	if (!m) return set_error(LG_ENOMEM, "host allocation");
	m->E = E;
	lg_status r = build_maps(sn, m);
	if (r) { delete m; return r; }
	sn->adj_maps = m;
	return LG_OK;
}

std::mutex g_run_mu;
int g_run[LG_TUNE_MAX_DEVICES];           // co-resident CTAs of aff_run + 1, 0 = not probed

int aff_run_resident(int device) {
	std::lock_guard<std::mutex> lk(g_run_mu);
	if (device < 0 || device >= LG_TUNE_MAX_DEVICES) return 0;
	if (!g_run[device]) {
		int n = 0;
		if (cudaFuncSetAttribute(aff_run, cudaFuncAttributeMaxDynamicSharedMemorySize,
				(int)sizeof(RunShared)) == cudaSuccess)
			n = coop_grid_size((const void*)aff_run, kRunThreads, device, sizeof(RunShared));
		else
			cudaGetLastError();
		g_run[device] = n + 1;
	}
	return coop_allowed(g_run[device] - 1);
}

// Iterate y = base + d * (weighted pull of x) over the flat CSR f until
// sum |y - x| < tol (at most max_iter iterations); m->xa holds the start on
// entry.  *out points at the result (m->xa or m->xb) on return.
lg_status fixed_point(lg_snapshot* sn, const FlatCsr& f, const double* w, const double* base,
		double d, double tol, int max_iter, int* iters, double* resid_out, double** out) {
	lg_store* s = sn->store;
	lg_adjoint_maps* m = sn->adj_maps;
	cudaStream_t st = s->stream;
	const uint64_t V = sn->V;
	double* A = m->xa.as<double>();
	double* B = m->xb.as<double>();
	const int resident = aff_run_resident(s->device);
	if (resident <= 0) return set_error(LG_ENOTSUP, "the device has no cooperative launch");
	LG_TRY(m->run.reserve(sizeof(RunCtl)));
	RunCtl* ctl = m->run.as<RunCtl>();
	LG_CUDA(cudaMemsetAsync(&ctl->bar, 0, sizeof(RunCtl) - offsetof(RunCtl, bar), st), "memset");
	AffRunArgs g;
	g.a = flat_tiles(f, nullptr);
	g.off = f.off.as<uint32_t>();
	g.nz_rows = f.nz_rows();
	g.w = w;
	g.base = base;
	g.xa = A;
	g.xb = B;
	g.d = d;
	g.tol = tol;
	g.V = (uint32_t)V;
	void* args[] = {&g, &ctl};
	unsigned long long h[4];
	static_assert(sizeof(CoopBar) == 16 && sizeof(RunCtl) - offsetof(RunCtl, bar) == 32,
			"barrier, residual, iterations");
	// (a residual that stays above tol, NaN for instance, takes max_iter
	// iterations, of which a launch takes as many as run_iterations says)
	const int most = run_iterations(f.E, V);
	unsigned grid = run_ctas(f.ntiles, resident);
	for (g.first = 0;; g.first = g.end) {
		g.end = most < max_iter - g.first ? g.first + most : max_iter;
		LG_CUDA(coop_launch((const void*)aff_run, &grid, kRunThreads, args, sizeof(RunShared), st,
				&ctl->bar), "aff_run");
		s->launches++;
		LG_TRY(read_words(s, (const unsigned long long*)&ctl->bar, 4, h));
		if ((unsigned)h[1] & 1u)
			return set_error(LG_ETIMEOUT, "pagerank: a grid barrier wait ran out");
		memcpy(resid_out, &h[2], sizeof(double));
		*iters = (int)(uint32_t)h[3];
		if (*resid_out < tol || g.end == max_iter) break;
	}
	*out = (*iters & 1) ? B : A;
	return LG_OK;
}

lg_status stage_in(lg_store* s, const double* src, uint64_t n, DevBuf& buf, const double** dev) {
	if (is_device_pointer(src)) { *dev = src; return LG_OK; }
	LG_TRY(buf.reserve(std::max<uint64_t>(n, 1) * 8));
	LG_CUDA(cudaMemcpyAsync(buf.p, src, n * 8, cudaMemcpyHostToDevice, s->stream), "h2d");
	s->h2d_bytes += n * 8;
	*dev = buf.as<double>();
	return LG_OK;
}

} // namespace

void lg_free_adjoint_maps(lg_adjoint_maps* m) { delete m; }

extern "C" lg_status lg_pagerank_fwd(lg_snapshot* sn, const double* weights,
		const double* teleport, double damping, double tol, int max_iter, double* x,
		lg_adjoint** tape, lg_fixed_point_result* result) {
	clear_error();
	if (tape) *tape = nullptr;
	if (!sn || !weights || !teleport || !x) return set_error(LG_EINVAL, "null argument");
	if (!(damping > 0 && damping < 1)) return set_error(LG_EINVAL, "damping must be in (0, 1)");
	if (!(tol > 0) || max_iter <= 0) return set_error(LG_EINVAL, "tol and max_iter must be positive");
	if (!sn->in.present) return set_error(LG_ESTATE, "needs the in-CSR (reverse edges)");
	lg_store* s = sn->store;
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	cudaStream_t st = s->stream;
	const uint64_t V = sn->V;
	LG_TRY(ensure_maps(sn));
	lg_adjoint_maps* m = sn->adj_maps;
	const uint64_t E = m->E;
	const double *w, *v;
	LG_TRY(stage_in(s, weights, E, m->stage_w, &w));
	LG_TRY(stage_in(s, teleport, V, m->stage_v, &v));
	LG_TRY(m->base.reserve(V * 8));
	LG_TRY(m->win.reserve(std::max<uint64_t>(E, 1) * 8));
	LG_TRY(m->xa.reserve(V * 8));
	LG_TRY(m->xb.reserve(V * 8));
	scale_vec<<<grid_for(V, 256), 256, 0, st>>>(v, 1.0 - damping, V, m->base.as<double>());
	gather_weights<<<grid_for(E, 256), 256, 0, st>>>(m->in_pos.as<uint32_t>(), E, w,
			m->win.as<double>());
	LG_CUDA(cudaMemcpyAsync(m->xa.p, v, V * 8, cudaMemcpyDeviceToDevice, st), "d2d");
	LG_CUDA(cudaGetLastError(), "pagerank fwd");
	s->launches += 2;
	int it = 0;
	double r = 0;
	double* res = nullptr;
	LG_TRY(fixed_point(sn, m->fin, m->win.as<double>(), m->base.as<double>(), damping, tol,
			max_iter, &it, &r, &res));
	if (tape) {
		lg_adjoint* t = new (std::nothrow) lg_adjoint(s->pool);
		if (!t) return set_error(LG_ENOMEM, "host allocation");
		t->snap = sn;
		t->d = damping;
		t->tol = tol;
		t->max_iter = max_iter;
		lg_status rs = t->x.reserve(V * 8);
		if (!rs) rs = t->w.reserve(std::max<uint64_t>(E, 1) * 8);
		if (rs) { delete t; return rs; }
		cudaError_t ce = cudaMemcpyAsync(t->x.p, res, V * 8, cudaMemcpyDeviceToDevice, st);
		if (ce == cudaSuccess)
			ce = cudaMemcpyAsync(t->w.p, w, E * 8, cudaMemcpyDeviceToDevice, st);
		if (ce != cudaSuccess) { delete t; return cuda_status(ce, "d2d"); }
		*tape = t;
	}
	LG_TRY(copy_out(s, x, res, V * 8));
	LG_CUDA(cudaStreamSynchronize(st), "pagerank fwd");
	if (result) { result->iterations = it; result->residual = r; }
	return LG_OK;
}

extern "C" lg_status lg_pagerank_bwd(lg_adjoint* t, const double* dldx, double* dldw,
		double* dlde, lg_fixed_point_result* result) {
	clear_error();
	if (!t || !dldx) return set_error(LG_EINVAL, "null argument");
	lg_snapshot* sn = t->snap;
	lg_store* s = sn->store;
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	cudaStream_t st = s->stream;
	const uint64_t V = sn->V;
	lg_adjoint_maps* m = sn->adj_maps;
	const uint64_t E = m->E;
	DevBuf outw(s->pool), oute(s->pool);
	const double* g;
	LG_TRY(stage_in(s, dldx, V, m->stage_g, &g));
	LG_TRY(m->xa.reserve(V * 8));
	LG_TRY(m->xb.reserve(V * 8));
	LG_CUDA(cudaMemcpyAsync(m->xa.p, g, V * 8, cudaMemcpyDeviceToDevice, st), "d2d");
	int it = 0;
	double r = 0;
	double* lam = nullptr;
	LG_TRY(fixed_point(sn, m->fout, t->w.as<double>(), g, t->d, t->tol, t->max_iter, &it, &r,
			&lam));
	if (dldw) {
		const bool dev = is_device_pointer(dldw);
		double* o = dldw;
		if (!dev) { LG_TRY(outw.reserve(std::max<uint64_t>(E, 1) * 8)); o = outw.as<double>(); }
		edge_grad<<<grid_for(E, 256), 256, 0, st>>>(m->src.as<uint32_t>(),
				m->fout.ids.as<uint32_t>(), E, t->d, lam, t->x.as<double>(), o);
		s->launches++;
		if (!dev) LG_TRY(copy_out(s, dldw, o, E * 8));
	}
	if (dlde) {
		const bool dev = is_device_pointer(dlde);
		double* o = dlde;
		if (!dev) { LG_TRY(oute.reserve(V * 8)); o = oute.as<double>(); }
		scale_vec<<<grid_for(V, 256), 256, 0, st>>>(lam, 1.0 - t->d, V, o);
		s->launches++;
		if (!dev) LG_TRY(copy_out(s, dlde, o, V * 8));
	}
	LG_CUDA(cudaGetLastError(), "pagerank bwd");
	LG_CUDA(cudaStreamSynchronize(st), "pagerank bwd");
	if (result) { result->iterations = it; result->residual = r; }
	return LG_OK;
}

extern "C" lg_status lg_adjoint_free(lg_adjoint* t) {
	delete t;
	return LG_OK;
}
