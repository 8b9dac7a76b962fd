/* What the fake device (fake_device.cc) tells a test program. */
#pragma once
#include <cstddef>
#include <cstdint>

namespace fake {

// Late: queued work runs only when the host waits for it (or asks).  Early: as it is queued.
extern bool late;
// The n-th call from now on that can fail does (0: none); `calls` counts them.
extern long fail_at, calls;
// Calls that ask for memory on the device fail beyond this many bytes in all (0: no limit).
extern size_t memory_limit;
extern size_t device_bytes;

// A convolution or change of layout over at least so many images takes milliseconds (0: none), so that the timing
// at load prefers to run a batch of that size in parts.
extern int slow_images;

void reset_calls(long fail);
size_t pending();         // operations queued and not yet run, over all streams
size_t live_objects();    // allocations, streams, events and graphs that exist
void host_register(void* p, size_t n);     // as cudaHostRegister() does; a copy that leaves the range fails
void host_unregister(void* p);
extern long conv_plans;   // cvmk_conv2d_tc_prepare() calls

}  // namespace fake
