// lg_scc_flat.h - strongly connected components over flat CSRs (lg_scc_flat.cu),
// called by lg_scc (lg_scc.cu).
#ifndef LG_SCC_FLAT_H_
#define LG_SCC_FLAT_H_

#include "lg_flat.cuh"

namespace lg {

// Labels (uint32, smallest vertex of the component) of sn's components into
// device array `label`, over fo / fi, the snapshot's live edges flat in both
// directions; *trimmed, *rounds, *steps as in lg_scc_result.  *ran = false when
// the device has no cooperative launch.
lg_status scc_flat_run(lg_snapshot* sn, const FlatCsr* fo, const FlatCsr* fi, uint32_t* label,
		uint64_t* trimmed, uint32_t* rounds, int* steps, bool* ran);

} // namespace lg

#endif // LG_SCC_FLAT_H_
