// Rules of the kernels' launches that need no GPU: plain functions, so that
// the tests can check them on the host over their whole range.
#pragma once

#include <stddef.h>

#include <map>
#include <mutex>
#include <utility>

#ifdef __CUDACC__
#define CC_RULE __host__ __device__ __forceinline__
#else
#define CC_RULE inline
#endif

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

// A transport launch hands out its n histories in units of HIST_UNIT of one
// batch, round-robin over groups of `group` batches (cc_engine.cu says why);
// unit u of a batch goes to copy u mod 2^copy_shift of the batch's slot.
constexpr int HIST_UNIT = 32;

// Histories of a batch for counting units: units beyond the launch's histories
// are handed out too, each an empty turn of the counter, so a batch size above
// them ("never split") must not enter.  At most n / 16 + 2 n_batches units then.
CC_RULE long long unit_batch(long long batch_size, long long n) { return batch_size < n ? batch_size : n; }

CC_RULE long long units_per_batch(long long batch_size) { return (batch_size + HIST_UNIT - 1) / HIST_UNIT; }

// Unit k: histories [first, end) (empty beyond a short last batch) and their
// scratch slot; false where there are no more.
CC_RULE bool unit_at(long long k, long long n, long long batch_size, int n_batches, int group, int copy_shift,
                     long long& first, long long& end, int& slot) {
    const long long per = units_per_batch(batch_size);
    if (k >= per * n_batches) return false;
    const long long in_group = per * group;
    const int g = (int)(k / in_group) * group;                         // the group's first batch
    const long long r = k % in_group;
    const int members = group < n_batches - g ? group : n_batches - g;
    const long long unit = r / members;
    const int batch = g + (int)(r - unit * members);
    first = (long long)batch * batch_size + unit * HIST_UNIT;
    const long long batch_end = (long long)(batch + 1) * batch_size < n ? (long long)(batch + 1) * batch_size : n;
    end = first + HIST_UNIT < batch_end ? first + HIST_UNIT : batch_end;
    if (end < first) end = first;
    slot = (batch << copy_shift) | ((int)unit & ((1 << copy_shift) - 1));
    return true;
}

// Batches of n > 0 histories (no overflow at the largest batch sizes).
CC_RULE long long batches_of(long long n, long long batch_size) { return (n - 1) / batch_size + 1; }

// The dynamic shared memory that kernels are allowed. The limit belongs to a
// kernel on a device, whichever context or thread launches it, and launches
// differ in size: set to each launch's own, one thread's smaller size between
// another's setting and its launch makes that launch fail. So it only rises.
class SmemLimits {
public:
    // set(bytes): the limit of this kernel on this device to the most that any
    // call asked for; returns what it returns (0: success).
    template <typename Set>
    int raise(const void* kernel, int device, size_t bytes, Set set) {
        std::lock_guard<std::mutex> lock(mu_);
        size_t& most = most_[std::make_pair(kernel, device)];
        const size_t want = bytes > most ? bytes : most;
        const int e = set(want);
        if (e == 0) most = want;
        return e;
    }

private:
    std::mutex mu_;
    std::map<std::pair<const void*, int>, size_t> most_;
};

}  // namespace cc
