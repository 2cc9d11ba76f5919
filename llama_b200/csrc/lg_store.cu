// lg_store.cu - device mirror of the LLAMA level stack: ingest of levels in
// the reference's layout, snapshot views (fragment walk + deletion bitset),
// degree and adjacency queries, and the error plumbing of the C ABI.
#include "lg_device.cuh"
#include "lg_flat.cuh"

#include <omp.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

namespace lg {

// ---------------------------------------------------------------------------
// Errors
// ---------------------------------------------------------------------------

static thread_local char t_err[512];

lg_status set_error(lg_status st, const char* fmt, ...) {
	va_list ap;
	va_start(ap, fmt);
	vsnprintf(t_err, sizeof(t_err), fmt, ap);
	va_end(ap);
	return st;
}

void clear_error() { t_err[0] = 0; }

TestLimits& test_limits() {
	static thread_local TestLimits t;
	return t;
}

extern "C" void lg_test_barrier(int fails) { test_limits().barrier = fails != 0; }
extern "C" void lg_test_one_step(int on) { test_limits().one_step = on != 0; }

// Negative: no limit.  Returns the allocations left to succeed (negative if one
// failed or there was no limit).
extern "C" int64_t lg_test_limits(int64_t allocs, int64_t ctas) {
	const int64_t left = test_limits().allocs;
	test_limits().allocs = allocs;
	test_limits().ctas = ctas < 0 ? INT64_MAX : ctas;
	return left;
}

lg_status cuda_status(cudaError_t e, const char* what) {
	if (e == cudaErrorMemoryAllocation)
		return set_error(LG_ENOMEM, "%s: %s", what, cudaGetErrorString(e));
	return set_error(LG_ECUDA, "%s: %s", what, cudaGetErrorString(e));
}

// Pools of every live store, to give their idle memory back when an
// allocation fails.
static std::mutex g_pools_mu;
static std::vector<CallPool*> g_pools;

CallPool::~CallPool() {
	{
		std::lock_guard<std::mutex> lk(g_pools_mu);
		g_pools.erase(std::remove(g_pools.begin(), g_pools.end(), this), g_pools.end());
	}
	if (pool) cudaMemPoolDestroy(pool);
}

lg_status make_pool(int device, cudaStream_t stream, std::shared_ptr<CallPool>* out) {
	try {
		auto c = std::make_shared<CallPool>();
		c->device = device;
		c->stream = stream;
		std::lock_guard<std::mutex> lk(g_pools_mu);
		g_pools.push_back(c.get());
		*out = c;
	} catch (const std::bad_alloc&) {
		return set_error(LG_ENOMEM, "host allocation");
	}
	return LG_OK;
}

// The pool itself, made when the first buffer asks for memory.
static cudaError_t open_pool(CallPool* c) {
	if (c->pool) return cudaSuccess;
	cudaMemPoolProps props;
	std::memset(&props, 0, sizeof(props));
	props.allocType = cudaMemAllocationTypePinned;
	props.location.type = cudaMemLocationTypeDevice;
	props.location.id = c->device;
	cudaMemPool_t p = nullptr;
	cudaError_t e = cudaMemPoolCreate(&p, &props);
	if (e != cudaSuccess) return e;
	uint64_t keep = kPoolKeep;
	e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
	if (e != cudaSuccess) { cudaMemPoolDestroy(p); return e; }
	std::lock_guard<std::mutex> lk(g_pools_mu);       // trim_pools reads it
	c->pool = p;
	return cudaSuccess;
}

// Gives the memory no buffer holds back to the device.
static void trim_pools() {
	cudaDeviceSynchronize();        // frees queued on the pools' streams have happened
	std::lock_guard<std::mutex> lk(g_pools_mu);
	for (CallPool* c : g_pools) if (c->pool) cudaMemPoolTrimTo(c->pool, 0);
}

void DevBuf::release() {
	if (p) {
		if (pooled && from->stream) cudaFreeAsync(p, from->stream);
		else cudaFree(p);
		if (pooled) from->used -= bytes;
	}
	pooled = false;
	p = nullptr;
	bytes = 0;
}

lg_status DevBuf::reserve(size_t n) {
	if (n <= bytes && p) return LG_OK;
	release();
	if (n == 0) n = 16;
	if (test_limits().allocs >= 0 && test_limits().allocs-- == 0)
		return cuda_status(cudaErrorMemoryAllocation, "test limit");
	cudaError_t e = cudaSuccess;
	const bool in_pool = from && from->used + n <= kPoolKeep;
	for (int attempt = 0; attempt < 2; attempt++) {
		if (!in_pool) e = cudaMalloc(&p, n);
		else if ((e = open_pool(from.get())) == cudaSuccess)
			e = cudaMallocFromPoolAsync(&p, n, from->pool, from->stream);
		if (e != cudaErrorMemoryAllocation || attempt) break;
		(void)cudaGetLastError();
		trim_pools();
	}
	if (e != cudaSuccess) {
		p = nullptr;
		(void)cudaGetLastError();
		return cuda_status(e, in_pool ? "cudaMallocFromPoolAsync" : "cudaMalloc");
	}
	bytes = n;
	pooled = in_pool;
	if (in_pool) from->used += n;
	return LG_OK;
}

bool is_device_pointer(const void* ptr) {
	cudaPointerAttributes a;
	cudaError_t e = cudaPointerGetAttributes(&a, ptr);
	if (e != cudaSuccess) { (void)cudaGetLastError(); return false; }
	return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

static bool is_pinned_host(const void* ptr) {
	cudaPointerAttributes a;
	cudaError_t e = cudaPointerGetAttributes(&a, ptr);
	if (e != cudaSuccess) { (void)cudaGetLastError(); return false; }
	return a.type == cudaMemoryTypeHost;
}

// LG_OUTPUT_ASYNC: the result is copied into a staging slot on the store's
// stream (so the caller may reuse `src` at once) and from there to the host
// on copy_stream.  The slot is reused only after its previous copy ended.
static lg_status copy_out_async(lg_store* s, void* dst, const void* src, size_t bytes) {
	if (!s->copy_stream) {
		LG_CUDA(cudaStreamCreateWithFlags(&s->copy_stream, cudaStreamNonBlocking), "copy stream");
		for (int i = 0; i < 2; i++) {
			LG_CUDA(cudaEventCreateWithFlags(&s->stage_ready[i], cudaEventDisableTiming), "event");
			LG_CUDA(cudaEventCreateWithFlags(&s->stage_done[i], cudaEventDisableTiming), "event");
		}
	}
	const int i = s->stage_next;
	s->stage_next ^= 1;
	DevBuf& b = s->out_stage[i];
	if (bytes > b.bytes) {
		// the old buffer may still be read by the slot's previous copy
		LG_CUDA(cudaStreamSynchronize(s->copy_stream), "copy stream");
		LG_TRY(b.reserve(bytes));
	}
	LG_CUDA(cudaStreamWaitEvent(s->stream, s->stage_done[i], 0), "wait for slot");
	LG_CUDA(cudaMemcpyAsync(b.p, src, bytes, cudaMemcpyDeviceToDevice, s->stream), "stage result");
	LG_CUDA(cudaEventRecord(s->stage_ready[i], s->stream), "event");
	LG_CUDA(cudaStreamWaitEvent(s->copy_stream, s->stage_ready[i], 0), "wait for result");
	LG_CUDA(cudaMemcpyAsync(dst, b.p, bytes, cudaMemcpyDeviceToHost, s->copy_stream),
			"copy result");
	LG_CUDA(cudaEventRecord(s->stage_done[i], s->copy_stream), "event");
	s->d2h_bytes += bytes;
	return LG_OK;
}

lg_status host_words(lg_store* s, unsigned long long** words) {
	if (!s->host_words)
		LG_CUDA(cudaHostAlloc((void**)&s->host_words, kHostWords * sizeof(unsigned long long),
				cudaHostAllocDefault), "cudaHostAlloc");
	*words = s->host_words;
	return LG_OK;
}

lg_status read_words(lg_store* s, const unsigned long long* dev, int n, unsigned long long* out) {
	unsigned long long* hw = nullptr;
	LG_TRY(host_words(s, &hw));
	hw += kHostWords - kReadWords;
	LG_CUDA(cudaMemcpyAsync(hw, dev, (size_t)n * sizeof(unsigned long long),
			cudaMemcpyDeviceToHost, s->stream), "d2h");
	LG_CUDA(cudaStreamSynchronize(s->stream), "d2h");
	for (int i = 0; i < n; i++) out[i] = hw[i];
	s->d2h_bytes += (uint64_t)n * sizeof(unsigned long long);
	return LG_OK;
}

lg_status copy_out(lg_store* s, void* dst, const void* src, size_t bytes) {
	if (bytes == 0) return LG_OK;
	if (s->output_mode == LG_OUTPUT_ASYNC && bytes >= LG_ASYNC_MIN_BYTES && is_pinned_host(dst))
		return copy_out_async(s, dst, src, bytes);
	if (!is_device_pointer(dst)) s->d2h_bytes += bytes;
	LG_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, s->stream), "copy result");
	return LG_OK;
}

DevLevel* take_level(lg_store* s, int dir) {
	DevLevel* d = s->level_spare[dir];
	s->level_spare[dir] = nullptr;
	if (!d) return new (std::nothrow) DevLevel();
	d->max_nodes = d->n_slots = d->n_fragment_slots = 0;
	return d;
}

lg_status append_dels(lg_store* s, DevCsr& csr, const uint2* add, size_t n,
		cudaMemcpyKind kind) {
	const size_t old_n = csr.n_dels_dev;
	const size_t need = (old_n + n) * sizeof(uint2);
	if (need > csr.dels.bytes) {
		// a larger list keeps the marks already on the device
		DevBuf nb;
		LG_TRY(nb.reserve(need + need / 2));
		if (old_n)
			LG_CUDA(cudaMemcpyAsync(nb.p, csr.dels.p, old_n * sizeof(uint2),
					cudaMemcpyDeviceToDevice, s->stream), "deletion list");
		// the old list may still be read by queued kernels
		LG_CUDA(cudaStreamSynchronize(s->stream), "deletion list");
		csr.dels.swap(nb);
	}
	if (n) {
		// (a pageable host source is copied before cudaMemcpyAsync returns)
		LG_CUDA(cudaMemcpyAsync(csr.dels.as<uint2>() + old_n, add, n * sizeof(uint2), kind,
				s->stream), "deletion list");
		if (kind == cudaMemcpyHostToDevice) s->h2d_bytes += n * sizeof(uint2);
	}
	csr.dels_mark.push_back(old_n);
	csr.n_dels_dev = old_n + n;
	return LG_OK;
}

// ---------------------------------------------------------------------------
// Exclusive scan (u32 -> u32) of an array or of the slot counts of a vertex
// list.  Up to kScanOne values: one CTA.  Up to kScanOwnTiles tiles: per-tile
// sums (which also store the counts of a list), then per-tile scans whose CTAs
// each add up the sums before theirs.  More: a single-CTA scan of the sums
// between the two.  The traversals scan a frontier per step, so what counts up
// to some 10^5 entries is the number of launches (2 to 3 us each) and the
// chain of loads and barriers in each: a list of 10^4 takes 1 or 2 where
// counting and the three-kernel scan took 4.  Values go through shared memory,
// so a warp's global accesses are consecutive whatever the arrays' alignment,
// while every thread scans its own kItems consecutive values; one barrier
// per tile.  Figures: 40 k values 3.5 + 3.9 us (4.4 + 9.3 where a thread's values
// were loaded straight, vectors only in aligned arrays, and a tile took three
// block scans of three barriers), 3 M values 5 + 7.5 (7 + 10.4, or 22.7
// unaligned), the slot counts of 16 k vertices 6.5 us (11.5: one vertex's chain
// of loads after the other).
// ---------------------------------------------------------------------------

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
static_assert((uint64_t)kScanThreads * kScanItems == kScanTile, "values per CTA");
constexpr int kOneThreads = 1024;                // the one-CTA form and the scan of the sums
constexpr int kOneItems = 8;
static_assert((uint64_t)kOneThreads * kOneItems == kScanOne, "values of the one-CTA form");

__device__ __forceinline__ uint64_t block_excl_scan(uint64_t x, uint64_t* total) {
	__shared__ uint64_t warp_sums[32];
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	uint64_t v = x;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		uint64_t t = __shfl_up_sync(0xffffffffu, v, o);
		if (lane >= o) v += t;
	}
	if (lane == 31) warp_sums[wid] = v;
	__syncthreads();
	if (wid == 0) {
		int nw = blockDim.x >> 5;
		uint64_t s = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			uint64_t t = __shfl_up_sync(0xffffffffu, s, o);
			if (lane >= o) s += t;
		}
		if (lane < nw) warp_sums[lane] = s;
	}
	__syncthreads();
	uint64_t before = wid > 0 ? warp_sums[wid - 1] : 0;
	*total = warp_sums[(blockDim.x >> 5) - 1];
	__syncthreads();
	return before + v - x;
}

// What is scanned.  load: x[j] = value i + j * step, 0 from n on; the loads of
// all N values are issued before any is used.
struct ScanArray {
	const uint32_t* a;
	template <int N>
	__device__ __forceinline__ void load(uint64_t i, uint32_t step, uint64_t n,
			uint32_t (&x)[N]) const {
#pragma unroll
		for (int j = 0; j < N; j++)
			x[j] = i + (uint64_t)j * step < n ? a[i + (uint64_t)j * step] : 0u;
	}
};

// 1 for the positive values.
struct ScanNonzero {
	const uint32_t* a;
	template <int N>
	__device__ __forceinline__ void load(uint64_t i, uint32_t step, uint64_t n,
			uint32_t (&x)[N]) const {
		ScanArray{a}.load(i, step, n, x);
#pragma unroll
		for (int j = 0; j < N; j++) x[j] = x[j] != 0u;
	}
};

struct ScanSlots {
	SnapCsr g;
	const uint32_t* list;
	template <int N>
	__device__ __forceinline__ void load(uint64_t i, uint32_t step, uint64_t n,
			uint32_t (&x)[N]) const {
		uint32_t v[N], a[N], b[N];
#pragma unroll
		for (int j = 0; j < N; j++) {
			const uint64_t k = i + (uint64_t)j * step;
			v[j] = k >= n ? kNoId : list ? __ldg(list + k) : (uint32_t)k;
		}
		const uint32_t* off = g.slot_off ? g.slot_off : g.frag_off;
#pragma unroll
		for (int j = 0; j < N; j++) {
			a[j] = v[j] != kNoId ? __ldg(off + v[j]) : 0u;
			b[j] = v[j] != kNoId ? __ldg(off + v[j] + 1) : 0u;
		}
#pragma unroll
		for (int j = 0; j < N; j++) x[j] = g.slot_off ? b[j] - a[j] : 0u;
		if (g.slot_off) return;
		for (bool more = true; more;) {                // a fragment of each at a time
			more = false;
			uint2 f[N];
#pragma unroll
			for (int j = 0; j < N; j++) f[j] = a[j] < b[j] ? __ldg(g.frags + a[j]) : make_uint2(0u, 0u);
#pragma unroll
			for (int j = 0; j < N; j++) {
				x[j] += frag_len(f[j]);
				if (a[j] < b[j]) a[j]++;
				more |= a[j] < b[j];
			}
		}
	}
};

// One CTA's tile of kThreads * kItems values.
template <int kThreads, int kItems>
struct TileScan {
	static constexpr int kWarps = kThreads / 32;
	// a warp's values, one unused word after every kItems (no bank conflicts)
	uint32_t stage[kWarps][32 * (kItems + 1)];
	uint64_t sums[kWarps], first[kWarps];

	// x[j] = value warp * 32 * kItems + j * 32 + lane of the tile; add(): the
	// thread's share of what comes before the tile.  store(i, y) is called with
	// y = the sum before value i.  Returns (all threads) the sum up to the
	// tile's end.
	template <class Add, class Store>
	__device__ __forceinline__ uint64_t run(const uint32_t (&x)[kItems], Add&& add, Store&& store) {
		static_assert((kItems & (kItems - 1)) == 0, "stage index");
		const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
		uint32_t* st = stage[wid];
#pragma unroll
		for (int j = 0; j < kItems; j++) {
			const uint32_t i = j * 32u + lane;
			st[i + i / kItems] = x[j];
		}
		uint64_t b = add();
		__syncwarp();
		uint32_t y[kItems];
		uint64_t s = 0;
#pragma unroll
		for (int j = 0; j < kItems; j++) {
			y[j] = st[lane * (kItems + 1) + j];
			s += y[j];
		}
		uint64_t v = s;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint64_t t = __shfl_up_sync(0xffffffffu, v, o);
			if (lane >= o) v += t;
			b += __shfl_xor_sync(0xffffffffu, b, o);
		}
		if (lane == 31u) {
			sums[wid] = v;
			first[wid] = b;
		}
		__syncthreads();
		// lane w of every warp: the sums of warp w
		uint64_t at = lane < kWarps ? sums[lane] : 0, all = lane < kWarps ? first[lane] : 0;
		all += at;
		if (lane >= wid) at = 0;
		at += lane < kWarps ? first[lane] : 0;
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			at += __shfl_xor_sync(0xffffffffu, at, o);
			all += __shfl_xor_sync(0xffffffffu, all, o);
		}
		uint64_t ex = at + v - s;
#pragma unroll
		for (int j = 0; j < kItems; j++) {
			const uint32_t c = y[j];
			st[lane * (kItems + 1) + j] = (uint32_t)ex;
			ex += c;
		}
		__syncwarp();
#pragma unroll
		for (int j = 0; j < kItems; j++) {
			const uint32_t i = j * 32u + lane;
			store(wid * (32u * kItems) + i, st[i + i / kItems]);
		}
		return all;
	}
};

// n <= kScanOne: out[0 .. n] and the total in one CTA; cnt, if not null,
// receives the values.
template <class In>
__global__ void __launch_bounds__(kOneThreads)
scan_one(In in, uint32_t* cnt, uint32_t* out, uint32_t n, uint64_t* grand) {
	__shared__ TileScan<kOneThreads, kOneItems> ts;
	const uint32_t first = (threadIdx.x >> 5) * (32u * kOneItems) + (threadIdx.x & 31u);
	uint32_t x[kOneItems];
	in.load(first, 32u, n, x);
	if (cnt) {
#pragma unroll
		for (int j = 0; j < kOneItems; j++)
			if (first + j * 32u < n) cnt[first + j * 32u] = x[j];
	}
	const uint64_t tot = ts.run(x, [] { return (uint64_t)0; },
			[&](uint32_t i, uint32_t y) { if (i < n) out[i] = y; });
	if (threadIdx.x == 0) {
		out[n] = (uint32_t)tot;
		*grand = tot;
	}
}

template <class In>
__global__ void __launch_bounds__(kScanThreads)
scan_tile_sums(In in, uint64_t n, uint32_t* cnt, uint64_t* sums) {
	__shared__ uint64_t wsum[kScanThreads / 32];
	const uint64_t base = (uint64_t)blockIdx.x * kScanTile + threadIdx.x;
	uint32_t x[kScanItems];
	in.load(base, kScanThreads, n, x);
	uint64_t s = 0;
#pragma unroll
	for (int i = 0; i < kScanItems; i++) {
		const uint64_t idx = base + (uint64_t)i * kScanThreads;
		if (cnt && idx < n) cnt[idx] = x[i];
		s += x[i];
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
	if ((threadIdx.x & 31u) == 0) wsum[threadIdx.x >> 5] = s;
	__syncthreads();
	if (threadIdx.x == 0) {
		uint64_t tot = 0;
		for (int w = 0; w < kScanThreads / 32; w++) tot += wsum[w];
		sums[blockIdx.x] = tot;
	}
}

__global__ void __launch_bounds__(kOneThreads)
scan_sums_single(uint64_t* sums, uint64_t n, uint64_t* grand) {
	uint64_t carry = 0;
	for (uint64_t b = 0; b < n; b += kOneThreads) {
		uint64_t i = b + threadIdx.x;
		uint64_t x = i < n ? sums[i] : 0, tot;
		uint64_t ex = block_excl_scan(x, &tot);
		if (i < n) sums[i] = carry + ex;
		carry += tot;
	}
	if (threadIdx.x == 0) *grand = carry;
}

// sums: exclusive prefix of the tiles (kOwn false, *grand the total), or the
// tiles' sums, of which every CTA adds up those before it and the last one
// writes *grand.
template <bool kOwn, bool kNonzero>
__global__ void __launch_bounds__(kScanThreads)
scan_tiles(const uint32_t* in, uint32_t* out, uint64_t n, const uint64_t* sums, uint64_t* grand) {
	__shared__ TileScan<kScanThreads, kScanItems> ts;
	const uint64_t base = (uint64_t)blockIdx.x * kScanTile;
	const uint64_t first = base + (threadIdx.x >> 5) * (32u * kScanItems) + (threadIdx.x & 31u);
	uint32_t x[kScanItems];
#pragma unroll
	for (int j = 0; j < kScanItems; j++)
		x[j] = first + j * 32u < n ? __ldcs(in + first + j * 32u) : 0u;
	if (kNonzero) {
#pragma unroll
		for (int j = 0; j < kScanItems; j++) x[j] = x[j] != 0u;
	}
	const uint64_t end = ts.run(x, [&] {
		uint64_t b = 0;
		if (kOwn) {
			for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kScanThreads) b += __ldg(sums + t);
		} else if (threadIdx.x == 0) {
			b = __ldg(sums + blockIdx.x);
		}
		return b;
	}, [&](uint32_t i, uint32_t y) { if (base + i < n) out[base + i] = y; });
	if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
		if (kOwn) *grand = end;
		out[n] = (uint32_t)end;
	}
}

// Scan of in(0 .. n); vals: where the second pass reads the values again
// (cnt, if not null; kNonzero: they count as 1 where positive).
template <bool kNonzero, class In>
static lg_status exclusive_scan(const In& in, const uint32_t* vals, uint32_t* cnt, uint32_t* out,
		uint64_t n, DevBuf& tmp, cudaStream_t stream, uint64_t* total,
		const uint64_t** dev_total = nullptr) {
	const uint64_t tiles = n <= kScanOne ? 1 : (n + kScanTile - 1) / kScanTile;
	LG_TRY(tmp.reserve((tiles + 1) * sizeof(uint64_t)));
	uint64_t* sums = tmp.as<uint64_t>();
	if (tiles == 1) {
		scan_one<<<1, kOneThreads, 0, stream>>>(in, cnt, out, (uint32_t)n, sums + 1);
	} else {
		scan_tile_sums<<<(unsigned)tiles, kScanThreads, 0, stream>>>(in, n, cnt, sums);
		if (tiles <= kScanOwnTiles) {
			scan_tiles<true, kNonzero><<<(unsigned)tiles, kScanThreads, 0, stream>>>(vals, out, n,
					sums, sums + tiles);
		} else {
			scan_sums_single<<<1, kOneThreads, 0, stream>>>(sums, tiles, sums + tiles);
			scan_tiles<false, kNonzero><<<(unsigned)tiles, kScanThreads, 0, stream>>>(vals, out, n,
					sums, sums + tiles);
		}
	}
	LG_CUDA(cudaGetLastError(), "scan launch");
	if (dev_total) *dev_total = sums + tiles;
	if (total) {
		// read through one pinned word per host thread (kept for the
		// thread's life): per-level loops read a total every step
		static thread_local uint64_t* pinned_total = nullptr;
		if (!pinned_total)
			LG_CUDA(cudaHostAlloc((void**)&pinned_total, sizeof(uint64_t),
					cudaHostAllocPortable), "cudaHostAlloc");
		LG_CUDA(cudaMemcpyAsync(pinned_total, sums + tiles, sizeof(uint64_t),
				cudaMemcpyDeviceToHost, stream), "scan total");
		LG_CUDA(cudaStreamSynchronize(stream), "scan total");
		const uint64_t t = *pinned_total;
		*total = t;
		if (t > 0xffffffffull)
			return set_error(LG_ENOTSUP, "more than 2^32-1 fragments in a snapshot");
	}
	return LG_OK;
}

lg_status exclusive_scan_u32(const uint32_t* in, uint32_t* out, uint64_t n,
		DevBuf& tmp, cudaStream_t stream, uint64_t* total) {
	return exclusive_scan<false>(ScanArray{in}, in, nullptr, out, n, tmp, stream, total);
}

// The total is left at *dev_total (in tmp).
static lg_status exclusive_scan_u32_dev(const uint32_t* in, uint32_t* out, uint64_t n, DevBuf& tmp,
		cudaStream_t stream, const uint64_t** dev_total) {
	return exclusive_scan<false>(ScanArray{in}, in, nullptr, out, n, tmp, stream, nullptr, dev_total);
}

lg_status exclusive_scan_nonzero(const uint32_t* in, uint32_t* out, uint64_t n, DevBuf& tmp,
		cudaStream_t stream, uint64_t* total) {
	return exclusive_scan<true>(ScanNonzero{in}, in, nullptr, out, n, tmp, stream, total);
}

lg_status exclusive_scan_slots(const SnapCsr& g, const uint32_t* list, uint64_t n, uint32_t* cnt,
		uint32_t* out, DevBuf& tmp, cudaStream_t stream, uint64_t* total) {
	return exclusive_scan<false>(ScanSlots{g, list}, cnt, cnt, out, n, tmp, stream, total);
}

// ---------------------------------------------------------------------------
// Ingest
// ---------------------------------------------------------------------------

static constexpr size_t kStageHalf = 64ull << 20;   // bytes per staging half

static lg_status ensure_staging(lg_store* s) {
	if (s->pinned) return LG_OK;
	LG_CUDA(cudaHostAlloc(&s->pinned, 2 * kStageHalf, cudaHostAllocDefault),
			"pinned staging");
	s->pinned_bytes = 2 * kStageHalf;
	for (int i = 0; i < 2; i++)
		LG_CUDA(cudaEventCreateWithFlags(&s->staged[i], cudaEventDisableTiming),
				"staging event");
	return LG_OK;
}

// Stream `bytes` to device memory `dst` through the pinned halves; `fill`
// writes bytes [off, off + n) of the source image into the staging buffer.
template <class Fill>
static lg_status staged_copy(lg_store* s, void* dst, size_t bytes, Fill&& fill) {
	LG_TRY(ensure_staging(s));
	size_t off = 0;
	int half = 0;
	while (off < bytes) {
		size_t n = std::min(kStageHalf, bytes - off);
		char* st = (char*)s->pinned + half * kStageHalf;
		LG_CUDA(cudaEventSynchronize(s->staged[half]), "staging wait");
		lg_status fs = fill(st, off, n);
		if (fs) return fs;
		LG_CUDA(cudaMemcpyAsync((char*)dst + off, st, n,
				cudaMemcpyHostToDevice, s->stream), "ingest copy");
		LG_CUDA(cudaEventRecord(s->staged[half], s->stream), "staging event");
		s->h2d_bytes += n;
		off += n;
		half ^= 1;
	}
	return LG_OK;
}

static inline const lg_vt_entry& vt_at(const lg_csr_level& c, uint64_t v) {
	if (c.vt) return c.vt[v];
	return c.vt_pages[v >> 9][v & 511];
}

static lg_status ingest_csr(lg_store* s, DevCsr& csr, int l,
		const lg_csr_level& c, const lg_deletion* dels, uint64_t n_dels,
		const char* name) {
	const uint64_t V = c.max_nodes;
	const uint64_t S = c.n_slots;
	if (V == 0 || V >= 0xffffffffull)
		return set_error(LG_EINVAL, "%s: max_nodes must be in [1, 2^32-1)", name);
	if (S >= 0xffffffffull)
		return set_error(LG_ENOTSUP, "%s: more than 2^32-1 slots in one level", name);
	if ((c.vt == nullptr) == (c.vt_pages == nullptr))
		return set_error(LG_EINVAL, "%s: exactly one of vt / vt_pages must be set", name);
	if (S > 0 && !c.slots)
		return set_error(LG_EINVAL, "%s: slots missing", name);

	// Validate the vertex table and mark the slots that belong to fragments
	// of this level.
	std::vector<uint8_t> mask(S, 0);
	int bad = 0;
	uint64_t frag_slots = 0;
	const auto& lv = csr.levels;
#pragma omp parallel for schedule(dynamic, 65536) reduction(|:bad) reduction(+:frag_slots)
	for (uint64_t v = 0; v < V; v++) {
		const lg_vt_entry& e = vt_at(c, v);
		if (e.adj_list_start == LG_NIL_EDGE || e.level_length == 0) continue;
		uint32_t el = LG_EDGE_LEVEL(e.adj_list_start);
		uint64_t ix = LG_EDGE_INDEX(e.adj_list_start);
		if (e.level_length > LG_MAX_FRAGMENT_LEN) { bad |= 4; continue; }
		if ((int)el > l) { bad |= 1; continue; }
		uint64_t lim = (int)el == l ? S : lv[el]->n_slots;
		if (ix + e.level_length > lim) { bad |= 2; continue; }
		if ((int)el == l) {
			for (uint64_t k = 0; k < e.level_length; k++) mask[ix + k] = 1;
			frag_slots += e.level_length;
		}
	}
	if (bad & 4) return set_error(LG_ENOTSUP, "%s: fragment longer than %u slots", name, LG_MAX_FRAGMENT_LEN);
	if (bad & 1) return set_error(LG_EINVAL, "%s: vertex table points to a future level", name);
	if (bad & 2) return set_error(LG_EINVAL, "%s: fragment exceeds its edge table", name);

	DevLevel* d = take_level(s, &csr == &s->out ? 0 : 1);
	if (!d) return set_error(LG_ENOMEM, "host allocation");
	d->max_nodes = V;
	d->n_slots = S;
	d->n_fragment_slots = frag_slots;
	if (!c.weights) d->w.release();
	lg_status st = d->vt.reserve((V + 1) * sizeof(lg_vt_entry));
	if (!st) st = d->ids.reserve(std::max<uint64_t>(S, 1) * sizeof(uint32_t));
	if (!st && c.weights) st = d->w.reserve(std::max<uint64_t>(S, 1) * sizeof(uint32_t));
	if (st) { delete d; return st; }

	// vertex table
	st = staged_copy(s, d->vt.p, (V + 1) * sizeof(lg_vt_entry),
		[&](char* dst, size_t off, size_t n) -> lg_status {
			uint64_t e0 = off / sizeof(lg_vt_entry), ne = n / sizeof(lg_vt_entry);
			lg_vt_entry* o = (lg_vt_entry*)dst;
#pragma omp parallel for schedule(static)
			for (uint64_t i = 0; i < ne; i++) o[i] = vt_at(c, e0 + i);
			return LG_OK;
		});
	// neighbour ids; slots already carrying a lowered max_visible_level
	// become deletion entries
	std::vector<std::vector<uint2>> found(omp_get_max_threads());
	int bad_id = 0;
	if (!st) st = staged_copy(s, d->ids.p, S * sizeof(uint32_t),
		[&](char* dst, size_t off, size_t n) -> lg_status {
			uint64_t i0 = off / 4, ni = n / 4;
			uint32_t* o = (uint32_t*)dst;
			int b = 0;
#pragma omp parallel reduction(|:b)
			{
				std::vector<uint2>& f = found[omp_get_thread_num()];
#pragma omp for schedule(static)
				for (uint64_t i = 0; i < ni; i++) {
					uint64_t k = i0 + i;
					if (!mask[k]) { o[i] = kNoId; continue; }
					uint64_t slot = c.slots[k];
					uint64_t pay = LG_SLOT_PAYLOAD(slot);
					if (pay >= V) { b |= 1; o[i] = kNoId; continue; }
					o[i] = (uint32_t)pay;
					uint32_t ml = LG_SLOT_MAX_LEVEL(slot);
					if (ml != LG_FRESH_MAX_LEVEL)
						f.push_back(make_uint2((uint32_t)k,
								((uint32_t)l << LG_BITS_LEVEL) | ml));
				}
			}
			bad_id |= b;
			return LG_OK;
		});
	if (!st && bad_id) st = set_error(LG_EINVAL, "%s: neighbour id >= max_nodes", name);
	if (!st && c.weights) st = staged_copy(s, d->w.p, S * sizeof(uint32_t),
		[&](char* dst, size_t off, size_t n) -> lg_status {
			std::memcpy(dst, (const char*)c.weights + off, n);
			return LG_OK;
		});
	if (st) {
		cudaStreamSynchronize(s->stream);
		delete d;
		return st;
	}
	// deletion marks in older levels
	std::vector<uint2> add;
	for (auto& f : found) add.insert(add.end(), f.begin(), f.end());
	for (uint64_t i = 0; i < n_dels; i++) {
		const lg_deletion& x = dels[i];
		uint32_t el = LG_EDGE_LEVEL(x.edge);
		uint64_t ix = LG_EDGE_INDEX(x.edge);
		if (x.edge < 0 || (int)el >= l || ix >= lv[el]->n_slots
				|| x.max_visible_level >= LG_FRESH_MAX_LEVEL) {
			cudaStreamSynchronize(s->stream);
			delete d;
			return set_error(LG_EINVAL, "%s: deletion %llu does not name an older slot",
					name, (unsigned long long)i);
		}
		add.push_back(make_uint2((uint32_t)ix, (el << LG_BITS_LEVEL) | x.max_visible_level));
	}
	csr.levels.push_back(d);
	return append_dels(s, csr, add.data(), add.size(), cudaMemcpyHostToDevice);
}

// ---------------------------------------------------------------------------
// Snapshot construction
// ---------------------------------------------------------------------------

struct VtTab {
	const lg_vt_entry* vt[LG_MAX_LEVELS];
	uint64_t max_nodes[LG_MAX_LEVELS];
};

// Fragment chain of v in snapshot L: iter_begin + iter_descend
// (llama/include/llama/ll_mlcsr_sp.h:1994-2134).  The continuation record read
// by iter_descend is the element VT[level-1][v] copied when `level` was built
// (ll_mlcsr_sp.h:1474-1497) and older levels never change afterwards, so the
// walk reads that element directly.
//
// With a minimum level minL (the sliding window), the chain ends at the first
// fragment of a level below minL, as iter_begin / iter_descend end it under
// LL_MIN_LEVEL (ll_mlcsr_sp.h:2021-2026, 2107-2110); vertex tables of levels
// below minL are never read.
//
// The filling walk also writes every fragment's first virtual slot and vertex,
// the fragment that holds the first slot of each kSlotTile-slot tile, and the
// entry bounds of every kBlockSlots-slot block.
struct FragOut {
	const uint32_t* frag_off;
	const uint32_t* slot_off;
	uint2* frags;
	uint32_t* start;
	uint32_t* vert;
	uint32_t* tile_frag;
	uint32_t* range_lb;          // lb[r] = first vertex with slot_off >= r * kBlockSlots
	uint32_t nb;                 // r = 0 .. nb
	unsigned long long* bare;    // += vertices without a fragment but with a degree
	                             // (null: not a window's, whose degrees are counted)
};
// Tiles that begin before slot s.
__device__ __forceinline__ uint32_t frag_tiles(uint32_t s) {
	return s / kSlotTile + (s % kSlotTile != 0);
}
template <bool kFill>
__global__ void walk_fragments(VtTab tab, int L, int minL, uint64_t V, uint32_t* count,
		uint32_t* deg, uint32_t* slots_per_vertex, FragOut fo) {
	uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	lg_vt_entry e;
	e.adj_list_start = LG_NIL_EDGE;
	uint32_t n = 0, slots = 0, out = 0, at = 0, degree = 0;
	if (v < V) {
		e = tab.vt[L][v];
		degree = e.degree;
		if (!kFill) deg[v] = degree;
		if (kFill) out = fo.frag_off[v];
		if (kFill) at = fo.slot_off[v];
	}
	bool lengthy = false;                        // one of the fragments spans many tiles
	while (e.adj_list_start != LG_NIL_EDGE && e.level_length != 0) {
		uint32_t lv = LG_EDGE_LEVEL(e.adj_list_start);
		if ((int)lv < minL) break;
		uint32_t ix = (uint32_t)LG_EDGE_INDEX(e.adj_list_start);
		if (kFill) {
			fo.frags[out + n] = make_uint2(ix, (e.level_length << kLevelBits) | lv);
			fo.start[out + n] = at + slots;
			fo.vert[out + n] = (uint32_t)v;
			const uint32_t t0 = frag_tiles(at + slots), t1 = frag_tiles(at + slots + e.level_length);
			if (t1 - t0 > kLaneMarks) lengthy = true;
			else
				for (uint32_t t = t0; t < t1; t++) fo.tile_frag[t] = out + n;
		}
		n++;
		slots += e.level_length;
		if ((int)lv <= minL || v >= tab.max_nodes[lv - 1]) break;
		e = tab.vt[lv - 1][v];
	}
	if (!kFill) {
		if (v < V) {
			count[v] = n;
			slots_per_vertex[v] = slots;
		}
		return;
	}
	if (n == 0 && degree != 0 && fo.bare) atomicAdd(fo.bare, 1ull);
	const uint32_t last = (uint32_t)(((uint64_t)at + slots) / kBlockSlots);
	if (v == 0) fo.range_lb[0] = 0;
	mark_range(fo.range_lb, at / kBlockSlots + 1u, min(last, fo.nb) + 1u, (uint32_t)v + 1u);
	if (v == V - 1)
		for (uint32_t r = last + 1u; r <= fo.nb; r++) fo.range_lb[r] = (uint32_t)V;
	// what the lanes left of the tiles' marks, a fragment of 32 vertices at a time
	for (uint32_t i = 0; __any_sync(0xffffffffu, lengthy && i < n); i++) {
		uint32_t t0 = 0, t1 = 0;
		if (lengthy && i < n) {
			const uint32_t st = fo.start[out + i];   // (its own store)
			t0 = frag_tiles(st);
			t1 = frag_tiles(i + 1 < n ? fo.start[out + i + 1] : at + slots);
			if (t1 - t0 <= kLaneMarks) t1 = t0;
		}
		mark_range(fo.tile_frag, t0, t1, out + i);
	}
}

__global__ void live_counts(SnapCsr g, uint32_t* out);

// Sets the bit of every slot deleted at or before L and counts them in *count.
// Slots of levels below minL are outside the window and have no bitset.  A
// grid-stride loop: each warp adds its count once at the end (one atomic per
// warp of a one-pass grid on the same counter serialised in L2).
__global__ void mark_deletions(const uint2* dels, uint64_t n, int L, int minL,
		uint32_t* const* del_words, unsigned long long* count) {
	unsigned long long c = 0;
	for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
			i += (uint64_t)gridDim.x * blockDim.x) {
		const uint2 d = dels[i];
		const uint32_t lv = d.y >> LG_BITS_LEVEL;
		const uint32_t ml = d.y & ((1u << LG_BITS_LEVEL) - 1u);
		if ((int)lv <= L && (int)lv >= minL && (int)ml <= L) {
			atomicOr(del_words[lv] + (d.x >> 5), 1u << (d.x & 31));
			c++;
		}
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
	if ((threadIdx.x & 31u) == 0 && c) atomicAdd(count, c);
}

// *sum += the degrees, *most = the largest.
__global__ void sum_degrees(const uint32_t* x, uint64_t n, unsigned long long* sum,
		unsigned long long* most) {
	unsigned long long s = 0;
	uint32_t m = 0;
	for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
			i += (uint64_t)gridDim.x * blockDim.x) {
		s += x[i];
		m = max(m, x[i]);
	}
	__shared__ uint32_t warp_most[32];
	m = __reduce_max_sync(0xffffffffu, m);
	if ((threadIdx.x & 31u) == 0) warp_most[threadIdx.x >> 5] = m;
	uint64_t tot;
	block_excl_scan(s, &tot);                // (synchronises)
	if (threadIdx.x != 0 || tot == 0) return;
	for (uint32_t w = 1; w < blockDim.x / 32u; w++) m = max(m, warp_most[w]);
	atomicAdd(sum, (unsigned long long)tot);
	atomicMax(most, (unsigned long long)m);
}

// Opening a direction takes three parts, with one wait for both directions
// after each of the first two; `w` are six of the store's pinned words.

static VtTab vt_tab(const lg_snapshot* sn, const DevCsr& csr) {
	VtTab tab;
	std::memset(&tab, 0, sizeof(tab));
	for (int l = sn->min_level; l <= sn->level; l++) {
		tab.vt[l] = csr.levels[l]->vt.as<lg_vt_entry>();
		tab.max_nodes[l] = csr.levels[l]->max_nodes;
	}
	return tab;
}

// Fragment and slot counts per vertex and their prefixes; w[0], w[1] = totals.
static lg_status open_count(lg_snapshot* sn, DevCsr& csr, SnapDir& d, unsigned long long* w) {
	lg_store* s = sn->store;
	SnapDir*& spare = s->snap_spare[&csr == &s->out ? 0 : 1];
	if (spare) d.swap_buffers(*spare);       // a closed snapshot's device buffers
	const uint64_t V = sn->V;
	cudaStream_t st = s->stream;
	LG_TRY(d.tmp_cnt.reserve(V * sizeof(uint32_t)));
	LG_TRY(d.tmp_slots.reserve(V * sizeof(uint32_t)));
	LG_TRY(d.deg.reserve(V * sizeof(uint32_t)));
	LG_TRY(d.frag_off.reserve((V + 1) * sizeof(uint32_t)));
	LG_TRY(d.slot_off.reserve((V + 1) * sizeof(uint32_t)));
	uint32_t* cnt = d.tmp_cnt.as<uint32_t>();
	uint32_t* slots = d.tmp_slots.as<uint32_t>();
	walk_fragments<false><<<grid_for(V, 256), 256, 0, st>>>(vt_tab(sn, csr), sn->level,
			sn->min_level, V, cnt, d.deg.as<uint32_t>(), slots, FragOut{});
	LG_CUDA(cudaGetLastError(), "walk_fragments");
	// fragment prefix, and the per-vertex slot prefix (the virtual slot space
	// the balanced kernels cut into ranges)
	const uint64_t *f = nullptr, *n = nullptr;
	LG_TRY(exclusive_scan_u32_dev(cnt, d.frag_off.as<uint32_t>(), V, d.tmp_scan, st, &f));
	LG_TRY(exclusive_scan_u32_dev(slots, d.slot_off.as<uint32_t>(), V, d.tmp_scan2, st, &n));
	LG_CUDA(cudaMemcpyAsync(w, f, 8, cudaMemcpyDeviceToHost, st), "scan total");
	LG_CUDA(cudaMemcpyAsync(w + 1, n, 8, cudaMemcpyDeviceToHost, st), "scan total");
	s->launches += 1 + 2 * scan_launches(V);
	s->d2h_bytes += 16;
	return LG_OK;
}

// Fragments, deletion bitsets and degrees; w[2] = live edges, w[3] = deletion
// marks visible, w[4] = vertices without a fragment but with a degree, w[5] = the
// largest degree.
static lg_status open_fill(lg_snapshot* sn, DevCsr& csr, SnapDir& d, unsigned long long* w) {
	lg_store* s = sn->store;
	const int L = sn->level, minL = sn->min_level;
	const uint64_t V = sn->V;
	cudaStream_t st = s->stream;
	const unsigned B = 256;
	const uint64_t F = w[0], total_slots = w[1];
	if (F > 0xffffffffull || total_slots > 0xffffffffull)
		return set_error(LG_ENOTSUP, "more than 2^32-1 fragments in a snapshot");
	d.n_frags = F;
	d.n_frag_slots = total_slots;
	const uint64_t nb = std::max<uint64_t>(1, (total_slots + kBlockSlots - 1) / kBlockSlots);
	const uint64_t tiles = total_slots / kSlotTile + 1;
	// fragments' starts (F + 1) and vertices (F), tiles' fragments
	LG_TRY(d.frags.reserve(std::max<uint64_t>(F, 1) * sizeof(uint2)));
	LG_TRY(d.frag_aux.reserve((2 * F + 1 + tiles) * sizeof(uint32_t)));
	LG_TRY(d.range_lb.reserve((nb + 1) * sizeof(uint32_t)));
	DevBuf& counters = d.tmp_sum;     // [0] live degree sum, [1] deletions visible at L,
	                                  // [2] vertices without a fragment but with a degree,
	                                  // [3] largest degree
	LG_TRY(counters.reserve(4 * sizeof(unsigned long long)));
	LG_CUDA(cudaMemsetAsync(counters.p, 0, 4 * sizeof(unsigned long long), st), "memset");
	walk_fragments<true><<<grid_for(V, B), B, 0, st>>>(vt_tab(sn, csr), L, minL, V, nullptr,
			nullptr, nullptr, FragOut{d.frag_off.as<uint32_t>(), d.slot_off.as<uint32_t>(),
				d.frags.as<uint2>(), d.frag_start(), d.frag_vert(), d.tile_frag(),
				d.range_lb.as<uint32_t>(), (uint32_t)nb,
				minL > 0 ? nullptr : counters.as<unsigned long long>() + 2});
	LG_CUDA(cudaGetLastError(), "walk_fragments fill");
	LG_CUDA(cudaMemcpyAsync(d.frag_start() + F, d.slot_off.as<uint32_t>() + V, sizeof(uint32_t),
			cudaMemcpyDeviceToDevice, st), "slot total");
	s->launches++;

	// deletion bitsets of levels minL..L
	std::vector<uint64_t> word_off(L + 2, 0);
	for (int l = 0; l <= L; l++)
		word_off[l + 1] = word_off[l]
			+ (l < minL ? 0 : (csr.levels[l]->n_slots + 31) / 32 + 1);
	LG_TRY(d.delbits.reserve(word_off[L + 1] * sizeof(uint32_t)));
	LG_CUDA(cudaMemsetAsync(d.delbits.p, 0, word_off[L + 1] * sizeof(uint32_t), st),
			"clear deletion bits");
	LevelTab lt;
	std::memset(&lt, 0, sizeof(lt));
	for (int l = minL; l <= L; l++) {
		lt.ids[l] = csr.levels[l]->ids.as<uint32_t>();
		lt.del[l] = d.delbits.as<uint32_t>() + word_off[l];
		lt.w[l] = csr.levels[l]->w.p ? csr.levels[l]->w.as<uint32_t>() : nullptr;
	}
	LG_TRY(d.lt.reserve(sizeof(LevelTab)));
	LG_CUDA(cudaMemcpyAsync(d.lt.p, &lt, sizeof(lt), cudaMemcpyHostToDevice, st),
			"level table");
	if (csr.n_dels_dev > 0) {
		int sms = 148;
		cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
		const unsigned mark_blocks = std::min<unsigned>(grid_for(csr.n_dels_dev, B),
				(unsigned)sms * 8u);
		mark_deletions<<<mark_blocks, B, 0, st>>>(
				csr.dels.as<uint2>(), csr.n_dels_dev, L, minL,
				const_cast<uint32_t* const*>(d.lt.as<LevelTab>()->del),
				counters.as<unsigned long long>() + 1);
		LG_CUDA(cudaGetLastError(), "mark_deletions");
		s->launches++;
	}
	if (minL > 0) {
		// the vertex table's degree counts edges of every level: in a window
		// the degree is the number of live slots the chain covers
		SnapCsr g = d.view();
		g.V = V;
		live_counts<<<grid_for(V, B), B, 0, st>>>(g, d.deg.as<uint32_t>());
		LG_CUDA(cudaGetLastError(), "window degrees");
		s->launches++;
	}
	sum_degrees<<<std::min<unsigned>(grid_for(V, B), 592u), B, 0, st>>>(d.deg.as<uint32_t>(), V,
			counters.as<unsigned long long>(), counters.as<unsigned long long>() + 3);
	LG_CUDA(cudaGetLastError(), "degree sum");
	s->launches++;
	LG_CUDA(cudaMemcpyAsync(w + 2, counters.p, 32, cudaMemcpyDeviceToHost, st), "d2h");
	s->d2h_bytes += 32;
	return LG_OK;
}

static void open_done(lg_snapshot* sn, DevCsr& csr, SnapDir& d, const unsigned long long* w) {
	d.n_edges = w[2];
	d.n_slots = 0;
	for (int l = sn->min_level; l <= sn->level; l++) d.n_slots += csr.levels[l]->n_slots;
	d.n_dels = w[3];
	d.n_bare = w[4];
	d.max_degree = w[5];
	d.present = true;
}

static lg_status open_dirs(lg_snapshot* sn) {
	lg_store* s = sn->store;
	unsigned long long* w = nullptr;
	LG_TRY(host_words(s, &w));
	LG_TRY(open_count(sn, s->out, sn->out, w));
	if (s->reverse) LG_TRY(open_count(sn, s->in, sn->in, w + 6));
	LG_CUDA(cudaStreamSynchronize(s->stream), "snapshot sizes");
	LG_TRY(open_fill(sn, s->out, sn->out, w));
	if (s->reverse) LG_TRY(open_fill(sn, s->in, sn->in, w + 6));
	LG_CUDA(cudaStreamSynchronize(s->stream), "snapshot sizes");
	open_done(sn, s->out, sn->out, w);
	if (s->reverse) open_done(sn, s->in, sn->in, w + 6);
	return LG_OK;
}

// ---------------------------------------------------------------------------
// Adjacency materialisation (iteration order)
// ---------------------------------------------------------------------------

__global__ void live_counts(SnapCsr g, uint32_t* out) {
	uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (v >= g.V) return;
	uint32_t f0 = g.frag_off[v], f1 = g.frag_off[v + 1], c = 0;
	for (uint32_t f = f0; f < f1; f++) {
		uint2 fr = g.frags[f];
		uint32_t lv = frag_level(fr);
		for (uint32_t k = 0; k < frag_len(fr); k++)
			c += !slot_deleted(g.lt, lv, fr.x + k);
	}
	out[v] = c;
}

lg_status live_degrees(const lg_snapshot* sn, int dir, uint32_t* out) {
	live_counts<<<grid_for(sn->V, 256), 256, 0, sn->store->stream>>>(sn->view(dir), out);
	LG_CUDA(cudaGetLastError(), "live_counts");
	sn->store->launches++;
	return LG_OK;
}

__global__ void write_adjacency(SnapCsr g, const uint32_t* off32,
		const unsigned long long* off64, uint32_t* nbr, long long* eid) {
	uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (v >= g.V) return;
	uint64_t o = off64 ? off64[v] : off32[v];
	uint32_t f0 = g.frag_off[v], f1 = g.frag_off[v + 1];
	for (uint32_t f = f0; f < f1; f++) {
		uint2 fr = g.frags[f];
		uint32_t lv = frag_level(fr);
		for (uint32_t k = 0; k < frag_len(fr); k++) {
			uint32_t ix = fr.x + k;
			if (slot_deleted(g.lt, lv, ix)) continue;
			nbr[o] = g.lt->ids[lv][ix];
			if (eid) eid[o] = (long long)LG_EDGE_CREATE(lv, ix);
			o++;
		}
	}
}

__global__ void widen_offsets(const uint32_t* cnt, uint64_t n,
		unsigned long long* out) {
	// single-CTA exclusive scan into 64-bit offsets
	unsigned long long carry = 0;
	for (uint64_t b = 0; b < n; b += blockDim.x) {
		uint64_t i = b + threadIdx.x;
		uint64_t x = i < n ? cnt[i] : 0, tot;
		uint64_t ex = block_excl_scan(x, &tot);
		if (i < n) out[i] = carry + ex;
		carry += tot;
	}
	if (threadIdx.x == 0) out[n] = carry;
}

} // namespace lg

using namespace lg;

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------

extern "C" {

size_t lg_last_error(char* buf, size_t len) {
	size_t n = strlen(t_err);
	if (buf && len) {
		size_t c = std::min(n, len - 1);
		std::memcpy(buf, t_err, c);
		buf[c] = 0;
	}
	return n;
}

const char* lg_status_string(lg_status st) {
	switch (st) {
	case LG_OK: return "ok";
	case LG_EINVAL: return "invalid argument";
	case LG_ENOMEM: return "out of memory";
	case LG_ECUDA: return "CUDA error";
	case LG_ETIMEOUT: return "timeout";
	case LG_ESTATE: return "invalid state";
	case LG_ENOTSUP: return "not supported";
	default: return "unknown status";
	}
}

const char* lg_version(void) { return "0.1.0"; }

lg_status lg_store_create(lg_store** out, const lg_store_opts* opts) {
	clear_error();
	if (!out) return set_error(LG_EINVAL, "null output pointer");
	*out = nullptr;
	int dev = opts ? opts->device : 0;
	int n = 0;
	cudaError_t e = cudaGetDeviceCount(&n);
	if (e != cudaSuccess || n == 0) {
		(void)cudaGetLastError();
		return set_error(LG_ECUDA, "no CUDA device available: %s",
				e == cudaSuccess ? "device count is 0" : cudaGetErrorString(e));
	}
	if (dev < 0 || dev >= n) return set_error(LG_EINVAL, "bad device ordinal %d", dev);
	LG_CUDA(cudaSetDevice(dev), "cudaSetDevice");
	lg_store* s = new (std::nothrow) lg_store();
	if (!s) return set_error(LG_ENOMEM, "host allocation");
	s->device = dev;
	s->reverse = opts ? opts->reverse_edges != 0 : true;
	if (opts && opts->stream) {
		s->stream = (cudaStream_t)opts->stream;
	} else {
		e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
		if (e != cudaSuccess) { delete s; return cuda_status(e, "stream"); }
		s->own_stream = true;
	}
	const lg_status ps = make_pool(dev, s->stream, &s->pool);
	if (ps) {
		if (s->own_stream) cudaStreamDestroy(s->stream);
		delete s;
		return ps;
	}
	*out = s;
	return LG_OK;
}

lg_status lg_store_destroy(lg_store* s) {
	clear_error();
	if (!s) return LG_OK;
	if (s->open_snapshots > 0)
		return set_error(LG_ESTATE, "close all snapshots before destroying the store");
	cudaSetDevice(s->device);
	cudaStreamSynchronize(s->stream);
	if (s->copy_stream) {
		cudaStreamSynchronize(s->copy_stream);
		cudaStreamDestroy(s->copy_stream);
	}
	for (int i = 0; i < 2; i++) {
		if (s->staged[i]) cudaEventDestroy(s->staged[i]);
		if (s->stage_ready[i]) cudaEventDestroy(s->stage_ready[i]);
		if (s->stage_done[i]) cudaEventDestroy(s->stage_done[i]);
	}
	if (s->pinned) cudaFreeHost(s->pinned);
	if (s->host_words) cudaFreeHost(s->host_words);
	delete s->flat_scratch;
	for (int d = 0; d < 2; d++) {
		delete s->flat_spare[d];
		delete s->snap_spare[d];
		delete s->level_spare[d];
	}
	// buffers that outlive the store (a tape) are freed without its stream
	s->pool->stream = nullptr;
	if (s->own_stream) cudaStreamDestroy(s->stream);
	delete s;
	return LG_OK;
}

lg_status lg_store_ingest_level(lg_store* s, const lg_level_desc* d) {
	clear_error();
	if (!s || !d) return set_error(LG_EINVAL, "null argument");
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	int l = (int)s->out.levels.size();
	if (l >= LG_MAX_LEVELS) return set_error(LG_ENOTSUP, "more than %d levels", LG_MAX_LEVELS);
	bool has_in = d->in.vt || d->in.vt_pages;
	if (s->reverse && !has_in)
		return set_error(LG_EINVAL, "store keeps reverse edges but the level has no in-CSR");
	if (s->reverse && d->in.max_nodes != d->out.max_nodes)
		return set_error(LG_EINVAL, "out and in CSR disagree on max_nodes");
	if (l > 0 && d->out.max_nodes < s->out.levels[l - 1]->max_nodes)
		return set_error(LG_EINVAL, "max_nodes cannot shrink");
	try {
		LG_TRY(ingest_csr(s, s->out, l, d->out, d->out_deletions,
				d->n_out_deletions, "out"));
		if (s->reverse) {
			lg_status st = ingest_csr(s, s->in, l, d->in, d->in_deletions,
					d->n_in_deletions, "in");
			if (st) {   // keep both directions at the same number of levels
				cudaStreamSynchronize(s->stream);
				delete s->out.levels.back();
				s->out.levels.pop_back();
				return st;
			}
		}
	} catch (const std::bad_alloc&) {
		return set_error(LG_ENOMEM, "host allocation during ingest");
	}
	LG_CUDA(cudaStreamSynchronize(s->stream), "ingest");
	return LG_OK;
}

int lg_store_num_levels(const lg_store* s) {
	return s ? (int)s->out.levels.size() : 0;
}

lg_status lg_store_max_nodes(const lg_store* s, int level, uint64_t* mn) {
	clear_error();
	if (!s || !mn) return set_error(LG_EINVAL, "null argument");
	if (level < 0) level = (int)s->out.levels.size() - 1;
	if (level < 0 || level >= (int)s->out.levels.size())
		return set_error(LG_EINVAL, "no such level");
	*mn = s->out.levels[level]->max_nodes;
	return LG_OK;
}

lg_status lg_store_sync(lg_store* s) {
	clear_error();
	if (!s) return set_error(LG_EINVAL, "null store");
	if (s->copy_stream) {
		// the store's stream waits for the result copies, so that work
		// queued on it after this call (an event, say) comes after them too
		for (int i = 0; i < 2; i++)
			LG_CUDA(cudaStreamWaitEvent(s->stream, s->stage_done[i], 0), "join copies");
		LG_CUDA(cudaStreamSynchronize(s->copy_stream), "sync copies");
	}
	return finish_run(s);
}

lg_status lg_store_set_output_mode(lg_store* s, int mode) {
	clear_error();
	if (!s) return set_error(LG_EINVAL, "null store");
	if (mode != LG_OUTPUT_SYNC && mode != LG_OUTPUT_ASYNC)
		return set_error(LG_EINVAL, "unknown output mode %d", mode);
	if (mode == LG_OUTPUT_SYNC && s->copy_stream)
		LG_CUDA(cudaStreamSynchronize(s->copy_stream), "sync copies");
	s->output_mode = mode;
	return LG_OK;
}

void* lg_store_stream(const lg_store* s) { return s ? (void*)s->stream : nullptr; }

uint64_t lg_store_device_bytes(const lg_store* s) {
	if (!s) return 0;
	uint64_t b = 0;
	for (const DevCsr* c : {&s->out, &s->in}) {
		for (const DevLevel* l : c->levels) b += l->vt.bytes + l->ids.bytes + l->w.bytes;
		b += c->dels.bytes;
	}
	for (const DevBuf& x : s->scratch) b += x.bytes;
	uint64_t kept = 0;
	if (s->pool->pool && cudaMemPoolGetAttribute(s->pool->pool, cudaMemPoolAttrReservedMemCurrent,
			&kept) == cudaSuccess)
		b += kept;
	return b;
}

uint64_t lg_store_launch_count(const lg_store* s) { return s ? s->launches : 0; }

lg_status lg_store_transfer_bytes(const lg_store* s, uint64_t* h2d, uint64_t* d2h) {
	clear_error();
	if (!s) return set_error(LG_EINVAL, "null store");
	if (h2d) *h2d = s->h2d_bytes;
	if (d2h) *d2h = s->d2h_bytes;
	return LG_OK;
}

lg_status lg_store_drop_level(lg_store* s) {
	clear_error();
	if (!s) return set_error(LG_EINVAL, "null store");
	if (s->out.levels.empty()) return set_error(LG_ESTATE, "the store holds no level");
	if (s->open_snapshots > 0)
		return set_error(LG_ESTATE, "close all snapshots before dropping a level");
	if ((int)s->out.levels.size() - 1 <= s->min_level && s->min_level > 0)
		return set_error(LG_ESTATE, "the newest level is the only one not aged out");
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	LG_CUDA(cudaStreamSynchronize(s->stream), "drop level");
	for (int dir = 0; dir < 2; dir++) {
		DevCsr* c = dir == 0 ? &s->out : &s->in;
		if (c->levels.empty()) continue;
		delete s->level_spare[dir];               // keep the newest dropped level's buffers
		s->level_spare[dir] = c->levels.back();
		c->levels.pop_back();
		// the list keeps the marks of the levels below
		c->n_dels_dev = c->dels_mark.back();
		c->dels_mark.pop_back();
	}
	return LG_OK;
}

lg_status lg_snapshot_get_stats(const lg_snapshot* sn, int dir, lg_snapshot_stats* st) {
	clear_error();
	if (!sn || !st) return set_error(LG_EINVAL, "null argument");
	if (dir != 0 && dir != 1) return set_error(LG_EINVAL, "dir must be 0 or 1");
	const SnapDir& d = dir == 0 ? sn->out : sn->in;
	if (!d.present) return set_error(LG_ESTATE, "the store has no in-CSR");
	st->max_nodes = sn->V;
	st->live_edges = d.n_edges;
	st->slots = d.n_slots;
	st->fragment_slots = d.n_frag_slots;
	st->fragments = d.n_frags;
	st->ranges = (d.n_frag_slots + kBlockSlots - 1) / kBlockSlots;
	st->deletions = d.n_dels;
	return LG_OK;
}

lg_status lg_snapshot_open_window(lg_store* s, int level, int min_level,
		lg_snapshot** out) {
	clear_error();
	if (!s || !out) return set_error(LG_EINVAL, "null argument");
	*out = nullptr;
	int n = (int)s->out.levels.size();
	if (level < 0) level = n - 1;
	if (level < 0 || level >= n) return set_error(LG_EINVAL, "no such level %d", level);
	if (min_level < s->min_level || min_level > level)
		return set_error(LG_EINVAL, "min_level %d outside [%d, %d] (levels below %d are "
				"aged out)", min_level, s->min_level, level, s->min_level);
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	lg_snapshot* sn = new (std::nothrow) lg_snapshot();
	if (!sn) return set_error(LG_ENOMEM, "host allocation");
	sn->store = s;
	sn->level = level;
	sn->min_level = min_level;
	sn->V = s->out.levels[level]->max_nodes;
	const lg_status st = open_dirs(sn);
	if (st) { cudaStreamSynchronize(s->stream); delete sn; return st; }
	s->open_snapshots++;
	*out = sn;
	return LG_OK;
}

lg_status lg_snapshot_open(lg_store* s, int level, lg_snapshot** out) {
	if (!s) { clear_error(); return set_error(LG_EINVAL, "null argument"); }
	int lv = level < 0 ? (int)s->out.levels.size() - 1 : level;
	if (lv >= 0 && lv < s->min_level) {
		clear_error();
		return set_error(LG_EINVAL, "level %d is aged out (min level %d)", lv, s->min_level);
	}
	return lg_snapshot_open_window(s, level, s->min_level, out);
}

lg_status lg_snapshot_min_level(const lg_snapshot* sn, int* min_level) {
	if (!sn || !min_level) return set_error(LG_EINVAL, "null argument");
	*min_level = sn->min_level;
	return LG_OK;
}

lg_status lg_store_set_min_level(lg_store* s, int m) {
	clear_error();
	if (!s) return set_error(LG_EINVAL, "null store");
	const int n = (int)s->out.levels.size();
	if (m < s->min_level) return set_error(LG_EINVAL, "the min level cannot decrease");
	if (m > n - 1) return set_error(LG_EINVAL, "min level %d would age out every level", m);
	if (s->open_snapshots > 0)
		return set_error(LG_ESTATE, "close all snapshots before aging levels out");
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	LG_CUDA(cudaStreamSynchronize(s->stream), "set min level");
	for (int l = s->min_level; l < m; l++) {
		for (DevCsr* c : {&s->out, &s->in}) {
			if (l >= (int)c->levels.size()) continue;
			DevLevel* d = c->levels[l];
			d->vt.release();       // sizes (max_nodes, n_slots) stay for validation
			d->ids.release();
			d->w.release();
		}
	}
	s->min_level = m;
	return LG_OK;
}

int lg_store_min_level(const lg_store* s) { return s ? s->min_level : 0; }

lg_status lg_snapshot_close(lg_snapshot* sn) {
	clear_error();
	if (!sn) return LG_OK;
	cudaSetDevice(sn->store->device);
	cudaStreamSynchronize(sn->store->stream);
	sn->store->open_snapshots--;
	if (sn->adj_maps) lg_free_adjoint_maps(sn->adj_maps);
	if (sn->sssp_split) lg_free_sssp_split(sn->sssp_split);
	for (int d = 0; d < 2; d++) lg_flat_release(sn->store, sn->flat[d]);
	// keep this snapshot's device buffers for the next open
	lg_store* s = sn->store;
	for (int d = 0; d < 2; d++) {
		SnapDir& sd = d == 0 ? sn->out : sn->in;
		if (!sd.present) continue;
		if (!s->snap_spare[d]) s->snap_spare[d] = new (std::nothrow) SnapDir();
		if (s->snap_spare[d]) s->snap_spare[d]->swap_buffers(sd);
	}
	delete sn;
	return LG_OK;
}

lg_status lg_snapshot_level(const lg_snapshot* sn, int* level) {
	if (!sn || !level) return set_error(LG_EINVAL, "null argument");
	*level = sn->level;
	return LG_OK;
}

lg_status lg_snapshot_max_nodes(const lg_snapshot* sn, uint64_t* mn) {
	if (!sn || !mn) return set_error(LG_EINVAL, "null argument");
	*mn = sn->V;
	return LG_OK;
}

lg_status lg_snapshot_num_edges(const lg_snapshot* sn, uint64_t* ne) {
	if (!sn || !ne) return set_error(LG_EINVAL, "null argument");
	*ne = sn->out.n_edges;
	return LG_OK;
}

static lg_status degrees(lg_snapshot* sn, int dir, uint32_t* out) {
	clear_error();
	if (!sn || !out) return set_error(LG_EINVAL, "null argument");
	const SnapDir& d = dir == 0 ? sn->out : sn->in;
	if (!d.present) return set_error(LG_ESTATE, "the store has no in-CSR");
	lg_store* s = sn->store;
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	LG_TRY(copy_out(s, out, d.deg.p, sn->V * sizeof(uint32_t)));
	LG_CUDA(cudaStreamSynchronize(s->stream), "degrees");
	return LG_OK;
}

lg_status lg_out_degrees(lg_snapshot* sn, uint32_t* out) { return degrees(sn, 0, out); }
lg_status lg_in_degrees(lg_snapshot* sn, uint32_t* out) { return degrees(sn, 1, out); }

lg_status lg_snapshot_adjacency(lg_snapshot* sn, int dir, uint64_t* offsets,
		uint32_t* neighbors, int64_t* edge_ids) {
	clear_error();
	if (!sn || !offsets) return set_error(LG_EINVAL, "null argument");
	if (dir != 0 && dir != 1) return set_error(LG_EINVAL, "dir must be 0 or 1");
	const SnapDir& d = dir == 0 ? sn->out : sn->in;
	if (!d.present) return set_error(LG_ESTATE, "the store has no in-CSR");
	lg_store* s = sn->store;
	LG_CUDA(cudaSetDevice(s->device), "cudaSetDevice");
	cudaStream_t st = s->stream;
	SnapCsr g = sn->view(dir);
	const uint64_t V = sn->V;
	DevBuf cnt(s->pool), off(s->pool), nb(s->pool), ei(s->pool);
	LG_TRY(cnt.reserve(V * 4));
	LG_TRY(off.reserve((V + 1) * 8));
	live_counts<<<grid_for(V, 256), 256, 0, st>>>(g, cnt.as<uint32_t>());
	widen_offsets<<<1, 1024, 0, st>>>(cnt.as<uint32_t>(), V,
			off.as<unsigned long long>());
	LG_CUDA(cudaGetLastError(), "adjacency offsets");
	s->launches += 3;
	uint64_t E = 0;
	LG_CUDA(cudaMemcpyAsync(&E, off.as<unsigned long long>() + V, 8,
			cudaMemcpyDeviceToHost, st), "d2h");
	LG_CUDA(cudaStreamSynchronize(st), "adjacency");
	LG_TRY(nb.reserve(std::max<uint64_t>(E, 1) * 4));
	if (edge_ids) LG_TRY(ei.reserve(std::max<uint64_t>(E, 1) * 8));
	write_adjacency<<<grid_for(V, 256), 256, 0, st>>>(g, nullptr,
			off.as<unsigned long long>(), nb.as<uint32_t>(),
			edge_ids ? ei.as<long long>() : nullptr);
	LG_CUDA(cudaGetLastError(), "write_adjacency");
	LG_TRY(copy_out(s, offsets, off.p, (V + 1) * 8));
	if (neighbors) LG_TRY(copy_out(s, neighbors, nb.p, E * 4));
	if (edge_ids) LG_TRY(copy_out(s, edge_ids, ei.p, E * 8));
	LG_CUDA(cudaStreamSynchronize(st), "adjacency");
	return LG_OK;
}

} // extern "C"
