// flag_counters.h -- the counters of a pass's flagged windows (PivParams::
// flag_count), which the second launch leaves as the next pass wants them.
#pragma once
#include <cstdint>

namespace opiv {

#ifdef __CUDACC__
#define OPIV_HD __host__ __device__
#else
#define OPIV_HD
#endif

// 32-bit words: windows flagged so far; windows flagged in the last pass; the
// 64-bit number below; what it had counted as settled after the last pass, and
// before that pass (64 bits each).  All zero before the first pass.
enum { kFlagged = 0, kLastFlagged = 1, kDone = 2, kSettled = 4, kSettledBefore = 6, kFlagCounters = 8 };

// The number: CTAs of the second launch that are done in the low 16 bits, above
// them the windows that exact sums have settled in all passes.  A CTA that is
// done adds done_add(); `before` is what it found.  The last CTA of a launch
// takes the launch's CTAs out again.  Nothing is stored and the count is taken
// modulo the CTAs, so however launches on the same counters overlap (they must
// not, but a caller may share a plan between streams), it ends at zero, and the
// passes after them are whole.  (Room for 65,535 CTAs; a launch has two an SM.)
constexpr int kDoneBits = 16;
OPIV_HD inline uint64_t done_add(uint32_t settled) { return (uint64_t)settled << kDoneBits | 1; }
OPIV_HD inline bool last_done(uint64_t before, uint32_t ctas)
{
    return (uint32_t)(before & ((1u << kDoneBits) - 1)) % ctas == ctas - 1;
}
OPIV_HD inline uint64_t all_settled(uint64_t before, uint32_t settled) { return (before >> kDoneBits) + settled; }

#undef OPIV_HD

}  // namespace opiv
