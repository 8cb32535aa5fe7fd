// Rules of the tcgen05 pipeline's rings that its roles have to agree on, apart
// from the kernel so that a model of the protocol on the CPU runs the kernel's own
// (tests/test_convert_ring.py).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define SPMM_RULE __host__ __device__ constexpr
#else
#define SPMM_RULE constexpr
#endif

namespace spmm {

constexpr int kItemRing = 4;    // entries of the item ring
constexpr int kBIssuers = 4;    // B-issuing warps

// Converted e4m3: arrivals that complete a group's full barrier. The B issuers
// write the group; the lead writes nothing, but waits for every group's slot, and
// a role that waits for a slot has to arrive in the slot's next group: otherwise
// that group can be consumed before the wait is tested, and the parity then reads
// as "not free yet" until one more round has passed, which at the end of the
// items never comes.
constexpr int kConvertFullArrivals = kBIssuers + 1;

// Converted e4m3: a B issuer copies groups ahead of those it converts, across
// items. Whether one that has converted `converted` groups may wait for an entry
// of the item ring, `first` being the first group of the entry kItemRing before
// it. The lead publishes an entry once that one has been read, and the MMA threads
// and the epilogue read it after finishing the entry before it; an issuer that
// waits with a group of that entry or an older one unconverted waits for itself
// (items without blocks bring it there: they hold no group).
SPMM_RULE bool may_wait_for_entry(uint32_t converted, uint32_t first) { return (int32_t)(converted - first) >= 0; }

}  // namespace spmm
#undef SPMM_RULE
