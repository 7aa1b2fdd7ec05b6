// fake_cuda.h - what a test sets and reads of fake_cuda.cpp.
#pragma once
#include <cstddef>
#include <cstdint>

namespace fake {
extern uint64_t allocations, operations, launches;   // since reset()
extern uint64_t violations;                          // pooled buffers freed under queued work
extern uint64_t failed;                              // operations and allocations made to fail
extern uint64_t fail_allocations_from, fail_operations_from;
extern uint64_t pool_reserved;                       // bytes the pool holds, in use or not
extern void (*on_copy_out)(void *dst, size_t bytes); // after a device-to-host copy
uint64_t pool_used();                                 // of these
size_t live_buffers();
void reset();                                        // counts and failures; queued work is done
}
