// lg_sort.cuh - device radix sort (lg_sort.cu).
#ifndef LG_SORT_CUH_
#define LG_SORT_CUH_

#include "lg_device.cuh"

namespace lg {

// Stable LSD radix sort of n 64-bit keys (and an optional u32 payload) on the
// store's stream.  The result ends up either in the input arrays or in the
// temporaries; *sorted_keys / *sorted_pay point at it.  vary: the bits in
// which keys may differ (0: found by reading the keys, which waits for the
// stream).
lg_status radix_sort_u64(lg_store* s, unsigned long long* keys, uint32_t* payload,
		uint64_t n, DevBuf& tmp_keys, DevBuf& tmp_pay, DevBuf& counts, DevBuf& scan_tmp,
		unsigned long long** sorted_keys, uint32_t** sorted_pay, unsigned long long vary = 0);

} // namespace lg

#endif // LG_SORT_CUH_
