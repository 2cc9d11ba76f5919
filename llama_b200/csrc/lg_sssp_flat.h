// lg_sssp_flat.h - delta-stepping over the flat out-CSR in one cooperative
// launch (lg_sssp_flat.cu), called by lg_sssp_delta (lg_sssp.cu).
#ifndef LG_SSSP_FLAT_H_
#define LG_SSSP_FLAT_H_

#include "lg_flat.cuh"

namespace lg {

// Distances from `root` into device array dist over f, the snapshot's weighted
// flat out-CSR (lg_sssp_delta's contract).  *ran = false, and nothing is
// launched, when the device has no cooperative launch.
lg_status sssp_flat_run(lg_snapshot* sn, const FlatCsr* f, uint32_t root, uint32_t delta,
		uint32_t* dist, lg_sssp_result* result, bool* ran);

} // namespace lg

#endif // LG_SSSP_FLAT_H_
