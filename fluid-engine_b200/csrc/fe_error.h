// fe_error.h — the library's thread-local last-error message (fe_last_error),
// and the allocations that the test hook counts.
#pragma once

#include <cstddef>

#include "../../include/fluid_step.h"

// printf-style; replaces the message returned by fe_last_error() on this
// host thread.  Internal (not exported).
void fe_set_error_message(const char* fmt, ...);

// cudaMalloc, counted by fe_debug_fail_allocation.  Internal.
fe_status fe_device_alloc(void** out, size_t bytes);
