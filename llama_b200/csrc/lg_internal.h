// lg_internal.h - error reporting shared by the host and device translation
// units of liblg.
#ifndef LG_INTERNAL_H_
#define LG_INTERNAL_H_

#include "../../include/lg.h"

namespace lg {

// Record `msg` as the calling thread's last error and return `st`.
lg_status set_error(lg_status st, const char* fmt, ...)
#if defined(__GNUC__)
	__attribute__((format(printf, 2, 3)))
#endif
	;
void clear_error();

// Limits that a test sets for the calls of its own thread (lg_test_limits, which
// the public headers leave out), to reach what the library does where the GPU
// has less to give: the device allocations that succeed before one fails
// (negative: none does), the CTAs of a cooperative launch that fit on it at once
// (0: no cooperative launch), whether the barriers of a one-launch PageRank
// give up at once, and whether a launch's time is up after its first step.
struct TestLimits {
	int64_t allocs = -1;
	int64_t ctas = INT64_MAX;
	bool barrier = false;
	bool one_step = false;
};
TestLimits& test_limits();

} // namespace lg

#endif // LG_INTERNAL_H_
