// The cache of released buffers (see mpm_alloc.cpp).
#pragma once

#include "mpm_common.cuh"

namespace mpm {

struct BufferStats {
    long long requests;           // buffers asked for since the start, from the driver or kept ones
    size_t live_device, live_host, kept_device, kept_host;   // bytes in use, bytes kept
};
BufferStats buffer_stats();
// gives every kept block back to the driver
void empty_buffer_cache();

}  // namespace mpm
