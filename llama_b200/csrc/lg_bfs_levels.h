// lg_bfs_levels.h - one-root BFS with every level in one cooperative launch
// (lg_bfs_levels.cu).
#ifndef LG_BFS_LEVELS_H_
#define LG_BFS_LEVELS_H_

#include "lg_flat.cuh"

namespace lg {

// One cooperative launch for the whole BFS from `root` into device array lvl
// (lg_bfs's contract).  *ran = false, and nothing is launched, when the
// snapshot's in-CSR is kept but not flat, LG_TUNE_BFS_LEVELS is 0, or the
// device has no cooperative launch; the caller then runs its per-level loop.
lg_status bfs_levels_run(lg_snapshot* sn, uint32_t root, int32_t* lvl, lg_bfs_result* result,
		bool* ran);

// The same along the edges of `out` (n_edges of them, outdeg per vertex);
// bottom-up levels over the rows of fi, the flat CSR of the opposite
// direction, or none without it.
lg_status bfs_levels_over(lg_store* s, SnapCsr out, const FlatCsr* fi, const uint32_t* outdeg,
		uint64_t n_edges, uint32_t root, int32_t* lvl, lg_bfs_result* result, bool* ran);

} // namespace lg

#endif // LG_BFS_LEVELS_H_
