// Rules of the kernels' launches that need no GPU: plain functions, so that
// the tests can check them on the host over their whole range.
#pragma once

namespace cc {

// Whether `issuers` warps that take the planes of a plane-stationary
// convolution in turn may run on a ring of this many planes, with `regions`
// accumulator regions.  An issuer waits for its own planes only, by the parity
// of the slot's phase, and the parity says that plane L has landed only where
// plane L - ring, the slot's content before, is known to have: either the same
// issuer waited for it (the ring is a multiple of the issuers), or the region
// that this issuer's plane before L took over had been released behind it
// (plane L - issuers - regions; the ring is at least that much).  On 3 or 5
// planes neither holds for two issuers: a plane whose load is late would be
// taken for the one after it in the same slot, and the slot read before it is
// written.
constexpr bool issue_ring_allowed(int ring, int issuers, int regions) {
    return ring % issuers == 0 || ring >= regions + issuers;
}

}  // namespace cc
