// Rules of the tcgen05 pipeline's rings that its roles have to agree on, apart
// from the kernel so that a model of the protocol on the CPU runs the kernel's own
// (tests/test_convert_ring.py).
#pragma once

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

}  // namespace spmm
