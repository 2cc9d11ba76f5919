// lg_ppr.h - personalized PageRank over the levels' fragments (lg_ppr_walk.cu),
// called where there is no flat in-CSR to be had (lg_ppr.cu).
#ifndef LG_PPR_H_
#define LG_PPR_H_

#include "lg_device.cuh"

namespace lg {

constexpr uint32_t kNoSeed = 0xffffffffu;

// The seeds, (vertex, column) pairs sorted by vertex, in device memory.
struct PprSeeds {
	const uint32_t* first;     // V: a vertex's first pair, or kNoSeed
	const uint2* cols;
	uint32_t n;
};

// All iterations for the K columns in passes of ktile, from y0 = x0 / out-degree
// (V x K, zero but for the seeds); the result goes to x, y1 is scratch.
lg_status ppr_walk(lg_snapshot* sn, const PprSeeds& seeds, uint32_t K, int ktile, int iterations,
		double damping, double* y0, double* y1, DevBuf& carry, double* x);

} // namespace lg

#endif // LG_PPR_H_
