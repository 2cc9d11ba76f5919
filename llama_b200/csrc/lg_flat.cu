// lg_flat.cu - flattening a snapshot direction into one CSR on the device.
//
// Reference: ll_t_flatten (benchmark/tools/flatten.h) merges every level of
// a LLAMA graph into a single level by iterating each vertex's edges
// (newest fragment first, deleted edges skipped) on the host.  Here the
// same order is produced in one balanced pass over the virtual slot space:
// row starts are the scan of the live degrees, and each warp of flat_write
// copies the live slots of kSlotTile consecutive virtual slots to its base.
// With deletions the bases are the scan of the tiles' live slots (flat_live,
// which reads the deletion words only); without any, slot and edge positions
// are the same.  Every vertex's row start is checked against the position its
// first slot goes to, so a degree that is not the live slot count is found.
// Row bookkeeping for the tile kernels (heads, nz_rows, nz_off, tile_seg) and
// the optional fragment view follow.
//
// flat_write keeps up to 32 fragments in a warp's lanes: the fragments that
// begin in a 32-slot chunk are bits of one word, so a slot's fragment is a
// population count away.  The form before it built a slot-to-fragment table
// per 1024-slot block in shared memory behind a dozen block barriers: it was
// bound by those and by its instructions, 2.1 ms at 262 M slots.  Now it takes
// 890 us there, some 70 instructions per 32 slots against 3 GB of traffic.
// What counts is the chains of loads: the next window is under way with the
// ids of the present one, and where its rows ought to start is looked up per
// window, not per row (1055 us), and 48 warps per SM hide the rest (96
// slots a time and 40 registers; 64: 900 us, 128: 929 with 40 registers, 1155 with
// 48).
#include "lg_flat.cuh"
#include "lg_sort.cuh"

#include <algorithm>
#include <cstring>

namespace lg {

constexpr int kFwThreads = 256;
constexpr int kFwWarps = kFwThreads / 32;
constexpr int kFwAhead = 3;             // 32-slot chunks whose loads are issued together

// One direction's fragments in virtual slot order.
struct FragSpace {
	const uint2* frags;        // F
	const uint32_t* start;     // F + 1
	const uint32_t* vert;      // F
	const uint32_t* frag_off;  // V + 1
	const uint32_t* tile_frag;
	const LevelTab* lt;
	uint32_t F, total, ntiles;
};

constexpr int kFlAhead = 2;             // pieces of a lane whose loads are issued together

// live[t] = live slots of tile t.  A warp per tile, a lane per fragment piece:
// the deletion words of the piece's slots, counted.  Bound by its three
// dependent loads per piece: two pieces at a time 162 us at 262 M slots in some 40 M
// pieces (one 168, four 250: registers), 215 where a piece's fragment was read
// only after its start.
__global__ void __launch_bounds__(kFwThreads)
flat_live(FragSpace fs, uint32_t* live) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t t = blockIdx.x * kFwWarps + (threadIdx.x >> 5);
	if (t >= fs.ntiles) return;
	const uint32_t s0 = t * kSlotTile;
	const uint32_t s1 = fs.total - s0 < kSlotTile ? fs.total : s0 + kSlotTile;
	const uint32_t f0 = __ldg(fs.tile_frag + t);
	uint32_t dead = 0;
	for (uint32_t f = f0;; f += 32u * kFlAhead) {
		uint32_t a[kFlAhead], b[kFlAhead], x[kFlAhead];      // slots [a, b) of a piece
		const uint32_t* d[kFlAhead];
		bool more = true;
#pragma unroll
		for (int u = 0; u < kFlAhead; u++) {
			const uint32_t i = u * 32u + lane, k = f + i;
			const bool have = i < fs.F - f;              // (f <= F; f + i may wrap)
			const uint32_t st = have ? __ldg(fs.start + k) : 0xffffffffu;
			const uint2 fr = have ? __ldg(fs.frags + k) : make_uint2(0u, 0u);
			const bool in = st < s1;
			more = in;
			a[u] = in ? fr.x + (max(st, s0) - st) : 0u;
			b[u] = in ? fr.x + (min(st + frag_len(fr), s1) - st) : 0u;
			d[u] = fs.lt->del[frag_level(fr)];
		}
#pragma unroll
		for (int u = 0; u < kFlAhead; u++) {
			x[u] = a[u] < b[u] ? __ldg(d[u] + (a[u] >> 5)) & (~0u << (a[u] & 31u)) : 0u;
		}
#pragma unroll
		for (int u = 0; u < kFlAhead; u++) {
			if (a[u] >= b[u]) continue;
			const uint32_t last = (b[u] - 1u) >> 5;
			for (uint32_t w = a[u] >> 5; w < last; w++) {
				dead += __popc(x[u]);
				x[u] = __ldg(d[u] + w + 1u);
			}
			if (b[u] & 31u) x[u] &= (1u << (b[u] & 31u)) - 1u;
			dead += __popc(x[u]);
		}
		if (!__all_sync(0xffffffffu, more)) break;
	}
	dead = __reduce_add_sync(0xffffffffu, dead);
	if (lane == 0) live[t] = s1 - s0 - dead;
}

// The live slots of tile t to ids[base ...] in slot order (and their weights
// to w when non-null); base = tile_base[t], or the tile's first slot where
// nothing is deleted (tile_base null).  off = the row starts the degrees
// give: a vertex whose first slot goes elsewhere, and a last tile that does
// not end at off[V], set bit 2 of *err.  (With no degrees at vertices without a
// fragment, which the snapshot's open looked for, every row is then right.)
// kPositions: instead of the edges, every virtual slot's edge position goes to
// ids[slot], kNoId for a deleted slot.
template <bool kWeights, bool kPositions, bool kDels>
__global__ void __launch_bounds__(kFwThreads, 6)
flat_write(FragSpace fs, const uint32_t* tile_base, const uint32_t* off, uint64_t V, uint32_t E,
		uint32_t* ids, uint32_t* w, unsigned int* err) {
	__shared__ LevelTab lt;
	{
		const uint64_t* src = reinterpret_cast<const uint64_t*>(fs.lt);
		uint64_t* dst = reinterpret_cast<uint64_t*>(&lt);
		for (uint32_t i = threadIdx.x; i < sizeof(LevelTab) / 8; i += kFwThreads)
			dst[i] = __ldg(src + i);
	}
	__syncthreads();
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t t = blockIdx.x * kFwWarps + (threadIdx.x >> 5);
	if (t >= fs.ntiles) return;
	const uint32_t s0 = t * kSlotTile;
	const uint32_t s1 = fs.total - s0 < kSlotTile ? fs.total : s0 + kSlotTile;
	// The window: fragments f ... f + 31 (f <= F), a lane each, covering slots up
	// to wend.  Sums of slot or fragment numbers may wrap where there are close to
	// 2^32 of either: what bounds the loop is compared as distances.
	// want = where its vertex's row starts if the fragment is the vertex's
	// first, kNoId if not.
	uint32_t f = __ldg(fs.tile_frag + t);
	uint32_t start = 0xffffffffu, wend = fs.total, vert = 0, want = kNoId;
	uint2 fr = make_uint2(0u, 0u);
	auto load_window = [&]() {
		const uint32_t k = f + lane;
		start = 0xffffffffu;
		if (lane < fs.F - f) {
			start = __ldg(fs.start + k);
			fr = __ldg(fs.frags + k);
			if (!kPositions) vert = __ldg(fs.vert + k);
		}
		wend = fs.F - f >= 32u ? __ldg(fs.start + f + 32u) : fs.total;
	};
	auto load_want = [&]() {
		want = kNoId;
		if (kPositions || lane >= fs.F - f) return;
		const uint32_t first = __ldg(fs.frag_off + vert), o = __ldg(off + vert);
		if (first == f + lane) want = o;
	};
	load_window();
	load_want();
	uint32_t run = kDels ? __ldg(tile_base + t) : 0u;
	bool bad = false;
	const uint32_t upto = 2u << lane;          // bits at or below the lane, + 1
	for (uint32_t pos = s0; pos < s1;) {
		const uint32_t most = min(min(s1, wend) - pos, 32u * kFwAhead);
		const uint32_t end = pos + most;
		uint32_t id[kFwAhead], dw[kFwAhead], wt[kFwAhead], bit[kFwAhead];
		uint32_t row[kFwAhead];                // where a row that begins at the slot starts
#pragma unroll
		for (int u = 0; u < kFwAhead; u++) {
			const uint32_t base = pos + u * 32u;
			// fragments begun before the chunk, and those that begin in it
			const uint32_t rel = start - base;
			const uint32_t begun = __popc(__ballot_sync(0xffffffffu, start < base));
			const uint32_t mask = __reduce_or_sync(0xffffffffu, rel < 32u ? 1u << rel : 0u);
			const uint32_t own = begun - 1u + __popc(mask & (upto - 1u));
			const uint32_t ix = __shfl_sync(0xffffffffu, fr.x - start, own) + base + lane;
			const uint32_t lv = __shfl_sync(0xffffffffu, fr.y, own) & kLevelMask;
			const bool in = u * 32u + lane < most;
			bit[u] = ix & 31u;
			dw[u] = !in ? ~0u : kDels ? __ldg(lt.del[lv] + (ix >> 5)) : 0u;
			if (!kPositions) id[u] = in ? __ldcs(lt.ids[lv] + ix) : 0u;
			if (kWeights) wt[u] = in ? __ldcs(lt.w[lv] + ix) : 0u;
			if (!kPositions) {
				row[u] = __shfl_sync(0xffffffffu, want, own);
				if (!in || !((mask >> lane) & 1u)) row[u] = kNoId;
			}
		}
		// the next window, if the next slots run past this one: under way with
		// the ids
		const bool next = wend < s1 && wend - end < 32u * kFwAhead;
		if (next) {
			f = end == wend ? f + 32u : f + __popc(__ballot_sync(0xffffffffu, start <= end)) - 1u;
			load_window();
		}
#pragma unroll
		for (int u = 0; u < kFwAhead; u++) {
			const bool live = !((dw[u] >> bit[u]) & 1u);
			unsigned m = 0;
			uint32_t p = pos + u * 32u + lane;
			if (kDels) {
				m = __ballot_sync(0xffffffffu, live);
				p = run + __popc(m & ((1u << lane) - 1u));
			}
			if (kPositions) {
				const uint32_t slot = pos + u * 32u + lane;
				if (u * 32u + lane < most) ids[slot] = live ? p : kNoId;
				run += __popc(m);
				continue;
			}
			if (live) {
				if (p < E) {
					ids[p] = id[u];
					if (kWeights) w[p] = wt[u];
				} else {
					bad = true;               // degrees and live slots disagree
				}
			}
			if (row[u] != kNoId) bad |= row[u] != p;
			run += __popc(m);
		}
		if (next) load_want();
		pos = end;
	}
	if (!kPositions && t == fs.ntiles - 1u) bad |= (kDels ? run : fs.total) != __ldg(off + V);
	if (bad) atomicOr(err, 2u);
}

// Rows with edges (vertex, start, head bit) and, for every tile that begins
// inside or at the end of a row, the rows begun before it.
__global__ void flat_rows(const uint32_t* off, const uint32_t* kidx, uint64_t V,
		uint32_t* nz_rows, uint32_t* nz_off, uint32_t* heads, uint32_t ntiles,
		uint32_t* tile_seg) {
	const uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	uint32_t o = 0, e = 0, k = 0;
	if (v < V) {
		o = __ldg(off + v);
		e = __ldg(off + v + 1);
	}
	if (e != o) {
		k = __ldg(kidx + v);
		nz_rows[k] = (uint32_t)v;
		nz_off[k] = o;
		atomicOr(heads + (o >> 5), 1u << (o & 31u));
		if (k == 0) tile_seg[0] = 0;
	}
	mark_range(tile_seg, o / kFlatTile + 1u, e != o ? min(e / kFlatTile + 1u, ntiles) : 0u, k + 1u);
}

// Fragment view: row k of the flat CSR is fragment k, {start, len << 6 | 0};
// a row longer than a fragment can describe sets *err.
__global__ void flat_view(const uint32_t* nz_off, uint32_t R, uint32_t E,
		uint2* frags, unsigned int* err) {
	const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
	if (k >= R) return;
	const uint32_t st = __ldg(nz_off + k);
	const uint32_t en = k + 1 < R ? __ldg(nz_off + k + 1) : E;
	const uint32_t len = en - st;
	if (len > (uint32_t)LG_MAX_FRAGMENT_LEN) { atomicOr(err, 1u); return; }
	frags[k] = make_uint2(st, len << kLevelBits);
}

SlotSpace slot_space(const lg_snapshot* sn, int dir) {
	const SnapDir& d = dir == 0 ? sn->out : sn->in;
	SlotSpace sp;
	sp.g = sn->view(dir);
	sp.pos = d.slot_off.as<uint32_t>();
	sp.range_lb = d.range_lb.as<uint32_t>();
	sp.total = (uint32_t)d.n_frag_slots;
	sp.nranges = (uint32_t)std::max<uint64_t>(1, (sp.total + kMapRange - 1) / kMapRange);
	return sp;
}

lg_status flat_row_index(lg_store* s, FlatCsr& f, const uint32_t* deg) {
	cudaStream_t st = s->stream;
	const uint64_t V = f.V;
	uint64_t R = 0;
	LG_TRY(f.kidx.reserve((V + 1) * sizeof(uint32_t)));
	LG_TRY(exclusive_scan_nonzero(deg, f.kidx.as<uint32_t>(), V, f.scan_tmp, st, &R));
	f.R = R;
	const uint64_t head_words = (uint64_t)f.ntiles * kFlatTileWords + 1;
	LG_TRY(f.rows.reserve((2 * f.rcap() + f.ntiles + head_words) * sizeof(uint32_t)));
	uint32_t* heads = const_cast<uint32_t*>(f.heads());
	LG_CUDA(cudaMemsetAsync(heads, 0, head_words * sizeof(uint32_t), st), "clear heads");
	flat_rows<<<grid_for(V, 256), 256, 0, st>>>(f.off.as<uint32_t>(), f.kidx.as<uint32_t>(), V,
			const_cast<uint32_t*>(f.nz_rows()), const_cast<uint32_t*>(f.nz_off()), heads, f.ntiles,
			const_cast<uint32_t*>(f.tile_seg()));
	LG_CUDA(cudaGetLastError(), "flat_rows");
	s->launches += scan_launches(V) + 1;
	return LG_OK;
}

// ---------------------------------------------------------------------------
// Transpose: every edge as (target << 32 | row), radix sorted by target
// (stable, so a row's sources stay in order).
// ---------------------------------------------------------------------------

// Lane j of the warp owning tile t takes edges 256 t + 8 j .. + 7 of `a`.
__global__ void __launch_bounds__(kFwThreads)
flat_edge_keys(const uint32_t* ids, const uint32_t* heads, const uint32_t* nz_rows,
		const uint32_t* tile_seg, uint32_t E, uint32_t ntiles, unsigned long long* keys) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t t = blockIdx.x * kFwWarps + (threadIdx.x >> 5);
	if (t >= ntiles) return;
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
	uint32_t row = __ldg(tile_seg + t) + before - 1u;   // of the lane's first edge, unless a head
	uint32_t v = eb < E && !(hb & 1u) ? __ldg(nz_rows + row) : 0u;
#pragma unroll
	for (int i = 0; i < kFlatPerLane; i++) {
		if ((hb >> i) & 1u) v = __ldg(nz_rows + ++row);
		if (eb + i < E)
			keys[eb + i] = ((unsigned long long)__ldcs(ids + eb + i) << 32) | v;
	}
}

// ids = the sorted keys' rows; cnt[t] = keys of target t (formed as end -
// start of its run, each added where the run begins or ends).
__global__ void flat_from_keys(const unsigned long long* keys, uint32_t E, uint32_t* ids,
		uint32_t* cnt) {
	const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= E) return;
	const unsigned long long k = keys[i];
	const uint32_t t = (uint32_t)(k >> 32);
	ids[i] = (uint32_t)k;
	const uint32_t p = i > 0 ? (uint32_t)(keys[i - 1] >> 32) : kNoId;
	if (p != t) {
		atomicSub(cnt + t, (uint32_t)i);
		if (i > 0) atomicAdd(cnt + p, (uint32_t)i);
	}
	if (i == E - 1u) atomicAdd(cnt + t, E);
}

lg_status flat_transpose(lg_store* s, const FlatCsr& a, FlatCsr& f) {
	cudaStream_t st = s->stream;
	const uint64_t V = a.V, E = a.E;
	f.V = V;
	f.E = E;
	f.ntiles = a.ntiles;
	f.weighted = f.has_view = f.has_nz_outdeg = false;
	DevBuf keys(s->pool), tmpk(s->pool), tmpp(s->pool), counts(s->pool), cnt(s->pool);
	LG_TRY(keys.reserve(std::max<uint64_t>(E, 1) * 8));
	LG_TRY(cnt.reserve(V * 4));
	LG_TRY(f.ids.reserve(std::max<uint64_t>(E, 1) * 4));
	LG_TRY(f.off.reserve((V + 1) * 4));
	LG_CUDA(cudaMemsetAsync(cnt.p, 0, V * 4, st), "clear counts");
	if (E > 0) {
		flat_edge_keys<<<grid_for(a.ntiles, kFwWarps), kFwThreads, 0, st>>>(a.ids.as<uint32_t>(),
				a.heads(), a.nz_rows(), a.tile_seg(), (uint32_t)E, a.ntiles,
				keys.as<unsigned long long>());
		LG_CUDA(cudaGetLastError(), "flat_edge_keys");
		unsigned long long targets = 1;          // the bits targets < V may differ in
		while (targets < V) targets <<= 1;
		unsigned long long* sorted = nullptr;
		LG_TRY(radix_sort_u64(s, keys.as<unsigned long long>(), nullptr, E, tmpk, tmpp, counts,
				f.scan_tmp, &sorted, nullptr, ((targets - 1) << 32) | (1ull << 32)));
		flat_from_keys<<<grid_for(E, 256), 256, 0, st>>>(sorted, (uint32_t)E, f.ids.as<uint32_t>(),
				cnt.as<uint32_t>());
		LG_CUDA(cudaGetLastError(), "flat_from_keys");
		s->launches += 2;
	}
	LG_TRY(exclusive_scan_u32(cnt.as<uint32_t>(), f.off.as<uint32_t>(), V, f.scan_tmp, st,
			nullptr));
	s->launches += scan_launches(V);
	return flat_row_index(s, f, cnt.as<uint32_t>());
}

static FragSpace frag_space(const SnapDir& d) {
	FragSpace fs;
	fs.frags = d.frags.as<uint2>();
	fs.start = d.frag_start();
	fs.vert = d.frag_vert();
	fs.frag_off = d.frag_off.as<uint32_t>();
	fs.tile_frag = d.tile_frag();
	fs.lt = d.lt.as<LevelTab>();
	fs.F = (uint32_t)d.n_frags;
	fs.total = (uint32_t)d.n_frag_slots;
	fs.ntiles = (uint32_t)((d.n_frag_slots + kSlotTile - 1) / kSlotTile);
	return fs;
}

// build_flat with rows of deg[v] edges, E in all.  *mismatch (and LG_OK, f
// unfinished): the live slots are not laid out as those degrees say.
static lg_status build_rows(lg_snapshot* sn, int dir, FlatCsr& f, bool view, bool weights,
		const uint32_t* deg, uint64_t E, bool* mismatch) {
	lg_store* s = sn->store;
	cudaStream_t st = s->stream;
	const uint64_t V = sn->V;
	const unsigned B = 256;
	const DevCsr& csr = dir == 0 ? s->out : s->in;
	// edge weights are read only along out-edges (SSSP), so only the out
	// direction carries them into the flat CSR
	bool weighted = dir == 0 && weights;
	for (int l = sn->min_level; l <= sn->level && weighted; l++)
		if (csr.levels[l]->n_fragment_slots > 0 && !csr.levels[l]->w.p) weighted = false;

	f.V = V;
	f.has_view = false;
	f.has_nz_outdeg = false;
	// row starts from the degrees; flat_write checks them
	const SnapDir& d = dir == 0 ? sn->out : sn->in;
	*mismatch = false;
	if (E > 0xffffffffull - 2 * kFlatTile)
		return set_error(LG_ENOTSUP, "more than 2^32 - %u live edges in one direction",
				2 * kFlatTile);
	f.E = E;
	f.weighted = weighted;
	f.ntiles = (uint32_t)((E + kFlatTile - 1) / kFlatTile);
	LG_TRY(f.ids.reserve(std::max<uint64_t>(E, 1) * sizeof(uint32_t)));
	if (weighted) LG_TRY(f.w.reserve(std::max<uint64_t>(E, 1) * sizeof(uint32_t)));
	LG_TRY(f.off.reserve((V + 1) * sizeof(uint32_t)));
	LG_TRY(f.kidx.reserve((V + 1) * sizeof(uint32_t)));
	LG_TRY(f.err.reserve(sizeof(unsigned int)));
	uint32_t* off = f.off.as<uint32_t>();
	LG_CUDA(cudaMemsetAsync(f.err.p, 0, sizeof(unsigned int), st), "clear flag");
	LG_TRY(exclusive_scan_u32(deg, off, V, f.scan_tmp, st, nullptr));
	const FragSpace fs = frag_space(d);
	const uint32_t* tile_base = nullptr;
	if (d.n_dels > 0 && fs.ntiles > 0) {
		LG_TRY(f.flags.reserve((2ull * fs.ntiles + 1) * sizeof(uint32_t)));
		uint32_t* live = f.flags.as<uint32_t>();
		flat_live<<<grid_for(fs.ntiles, kFwWarps), kFwThreads, 0, st>>>(fs, live);
		LG_CUDA(cudaGetLastError(), "flat_live");
		LG_TRY(exclusive_scan_u32(live, live + fs.ntiles, fs.ntiles, f.scan_tmp, st, nullptr));
		tile_base = live + fs.ntiles;
		s->launches += 1 + scan_launches(fs.ntiles);
	}
	if (fs.ntiles > 0) {
		const unsigned blocks = grid_for(fs.ntiles, kFwWarps);
		unsigned int* err = f.err.as<unsigned int>();
		const auto k = weighted ? (tile_base ? flat_write<true, false, true>
						: flat_write<true, false, false>)
				: tile_base ? flat_write<false, false, true> : flat_write<false, false, false>;
		k<<<blocks, kFwThreads, 0, st>>>(fs, tile_base, off, V, (uint32_t)E, f.ids.as<uint32_t>(),
				weighted ? f.w.as<uint32_t>() : nullptr, err);
		LG_CUDA(cudaGetLastError(), "flat_write");
	}
	unsigned int err = 0;
	LG_CUDA(cudaMemcpyAsync(&err, f.err.p, sizeof(err), cudaMemcpyDeviceToHost, st), "d2h");
	s->launches += scan_launches(V) + (fs.ntiles > 0);
	LG_TRY(flat_row_index(s, f, deg));
	// (that waited for the stream, so err is in)
	if ((err & 2u) || (fs.ntiles == 0 && E > 0)) {
		*mismatch = true;
		return LG_OK;
	}
	const uint64_t R = f.R;
	if (!view) return LG_OK;

	LG_TRY(f.vfrags.reserve(f.rcap() * sizeof(uint2)));
	const uint64_t del_words = (E + 31) / 32 + 1;
	LG_TRY(f.vdel.reserve(del_words * sizeof(uint32_t)));
	LG_CUDA(cudaMemsetAsync(f.vdel.p, 0, del_words * sizeof(uint32_t), st), "clear view bits");
	LG_CUDA(cudaMemsetAsync(f.err.p, 0, sizeof(unsigned int), st), "clear flag");
	if (R > 0) {
		flat_view<<<grid_for(R, B), B, 0, st>>>(f.nz_off(), (uint32_t)R, (uint32_t)E,
				f.vfrags.as<uint2>(), f.err.as<unsigned int>());
		LG_CUDA(cudaGetLastError(), "flat_view");
		s->launches++;
	}
	LevelTab lt;
	std::memset(&lt, 0, sizeof(lt));
	lt.ids[0] = f.ids.as<uint32_t>();
	lt.del[0] = f.vdel.as<uint32_t>();
	lt.w[0] = weighted ? f.w.as<uint32_t>() : nullptr;
	LG_TRY(f.vlt.reserve(sizeof(LevelTab)));
	LG_CUDA(cudaMemcpyAsync(f.vlt.p, &lt, sizeof(lt), cudaMemcpyHostToDevice, st), "level table");
	LG_CUDA(cudaMemcpyAsync(&err, f.err.p, sizeof(err), cudaMemcpyDeviceToHost, st), "d2h");
	LG_CUDA(cudaStreamSynchronize(st), "flatten");
	if (err)
		return set_error(LG_ENOTSUP, "a vertex has more than %u live edges, the longest "
				"fragment a flat view can describe", (unsigned)LG_MAX_FRAGMENT_LEN);
	f.has_view = true;
	return LG_OK;
}

lg_status flat_positions(lg_snapshot* sn, int dir, const FlatCsr& f, uint32_t* pos) {
	const SnapDir& d = dir == 0 ? sn->out : sn->in;
	lg_store* s = sn->store;
	const FragSpace fs = frag_space(d);
	if (fs.ntiles == 0) return LG_OK;
	// (the tiles' bases are left from the flatten, behind their live counts)
	const uint32_t* tile_base = d.n_dels > 0 ? f.flags.as<uint32_t>() + fs.ntiles : nullptr;
	const auto k = tile_base ? flat_write<false, true, true> : flat_write<false, true, false>;
	k<<<grid_for(fs.ntiles, kFwWarps), kFwThreads, 0, s->stream>>>(fs, tile_base, nullptr, sn->V, 0,
			pos, nullptr, nullptr);
	LG_CUDA(cudaGetLastError(), "flat_positions");
	s->launches++;
	return LG_OK;
}

lg_status build_flat(lg_snapshot* sn, int dir, FlatCsr& f, bool view, bool weights,
		bool strict) {
	const SnapDir& d = dir == 0 ? sn->out : sn->in;
	// flat_write finds a row that does not start where the degrees say; the rows
	// of vertices without a fragment it never meets (a surplus there can make up
	// for a deficit of the vertex before), and more edges than slots need no look
	bool mismatch = d.n_bare > 0 || (!strict && d.n_edges > d.n_frag_slots);
	if (!mismatch)
		LG_TRY(build_rows(sn, dir, f, view, weights, d.deg.as<uint32_t>(), d.n_edges, &mismatch));
	if (!mismatch) return LG_OK;
	if (strict)
		return set_error(LG_EINVAL, "a vertex's degree differs from its live edge count");
	DevBuf cnt(sn->store->pool), tmp(sn->store->pool);
	LG_TRY(cnt.reserve((2 * sn->V + 1) * sizeof(uint32_t)));
	uint32_t* live = cnt.as<uint32_t>();
	LG_TRY(live_degrees(sn, dir, live));
	uint64_t E = 0;
	LG_TRY(exclusive_scan_u32(live, live + sn->V, sn->V, tmp, sn->store->stream, &E));
	LG_TRY(build_rows(sn, dir, f, view, weights, live, E, &mismatch));
	if (mismatch) return set_error(LG_ECUDA, "live slots changed while they were flattened");
	return LG_OK;
}

} // namespace lg

using namespace lg;

extern "C" lg_status lg_snapshot_flatten(lg_snapshot* sn, int dir) {
	clear_error();
	if (!sn) return set_error(LG_EINVAL, "null argument");
	if (dir != 0 && dir != 1) return set_error(LG_EINVAL, "dir must be 0 or 1");
	const SnapDir& d = dir == 0 ? sn->out : sn->in;
	if (!d.present) return set_error(LG_ESTATE, "the store has no in-CSR");
	if (sn->flat[dir]) return LG_OK;
	lg_store* s = sn->store;
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	// reuse the device memory of a flat CSR an earlier snapshot released
	FlatCsr* f = nullptr;
	for (int i = 0; i < 2 && !f; i++)
		if (s->flat_spare[i]) { f = s->flat_spare[i]; s->flat_spare[i] = nullptr; }
	if (!f) f = new FlatCsr;
	// the fragment view is read by the out-direction traversals only
	const lg_status st = build_flat(sn, dir, *f, dir == 0);
	if (st != LG_OK) {
		cudaStreamSynchronize(s->stream);
		delete f;
		return st;
	}
	sn->flat[dir] = f;
	return LG_OK;
}

void lg_flat_release(lg_store* s, FlatCsr* f) {
	if (!f) return;
	for (int i = 0; i < 2; i++)
		if (!s->flat_spare[i]) { s->flat_spare[i] = f; return; }
	delete f;
}

extern "C" lg_status lg_snapshot_unflatten(lg_snapshot* sn) {
	clear_error();
	if (!sn) return set_error(LG_EINVAL, "null argument");
	LG_CUDA(cudaSetDevice(sn->store->device), "cudaSetDevice");
	LG_CUDA(cudaStreamSynchronize(sn->store->stream), "unflatten");
	for (int d = 0; d < 2; d++) {
		lg_flat_release(sn->store, sn->flat[d]);
		sn->flat[d] = nullptr;
	}
	return LG_OK;
}

extern "C" lg_status lg_snapshot_is_flat(const lg_snapshot* sn, int dir, int* flat) {
	if (!sn || !flat) return set_error(LG_EINVAL, "null argument");
	if (dir != 0 && dir != 1) return set_error(LG_EINVAL, "dir must be 0 or 1");
	*flat = sn->flat[dir] != nullptr;
	return LG_OK;
}
