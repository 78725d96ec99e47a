// A CUDA runtime without a device, for host checks of the engine's own object
// code: "device" memory is host memory, copies are copies, kernels do nothing.
// It records what the checks ask about and fails the calls they pick.
#pragma once
#include <cstddef>

namespace fake {
// Work queued on a stream while a copy or memset of the legacy stream (plain
// cudaMemcpy from pageable memory, cudaMemset: both may return before they are
// done) is not known to have ended: streams made with cudaStreamNonBlocking
// are not ordered behind it.
extern int unordered;
extern int copies_in, copies_out;  // host-to-device and device-to-host copies
extern int events;           // events alive
extern int launches;         // kernels
extern int graphs;           // graphs instantiated
extern size_t bytes, peak;   // device memory alive, and the most there was
// The n-th call from now on fails (0: none does); counted down to 0.
extern int fail_malloc, fail_copy_in, fail_memset;
// An allocation that would make `bytes` exceed this fails (0: no limit).
extern size_t limit;
}  // namespace fake
