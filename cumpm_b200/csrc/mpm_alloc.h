// Reuse of buffers that an object releases (see mpm_alloc.cpp).
#pragma once

#include "mpm_common.cuh"

#include <vector>

namespace mpm {

// The streams on which a caller has had an object's work queued, so that its
// buffers can be waited for whatever happens to those streams meanwhile.
class StreamUses {
public:
    StreamUses() = default;
    ~StreamUses();
    StreamUses(const StreamUses&) = delete;
    StreamUses& operator=(const StreamUses&) = delete;
    // work has been queued on s (call after it)
    void record(cudaStream_t s);
    // work may be running, or may run later, that cannot be waited for: a call
    // that was captured into a graph or that threw
    void give_up() { unknown_ = true; }
    bool unknown() const { return unknown_; }
    // waits for the work; false if it cannot
    bool wait() const;

private:
    struct Use {
        unsigned long long stream;   // the stream's id, which no later stream has
        cudaEvent_t done;
    };
    std::vector<Use> uses_;
    bool unknown_ = false;
};

// While one lives, buffers that its thread releases were used by work on
// stream s and on those of `uses` alone, and are kept for the next request once
// that has been waited for.  Scopes nest; the innermost counts.
class ReuseScope {
public:
    explicit ReuseScope(cudaStream_t s) : ReuseScope(true, s, nullptr) {}
    explicit ReuseScope(const StreamUses& uses) : ReuseScope(false, nullptr, &uses) {}
    ReuseScope(const StreamUses& uses, cudaStream_t s) : ReuseScope(true, s, &uses) {}
    ~ReuseScope();
    ReuseScope(const ReuseScope&) = delete;
    ReuseScope& operator=(const ReuseScope&) = delete;
    // whether nothing uses the buffers any more (waits for it)
    bool idle() const;

private:
    ReuseScope(bool own, cudaStream_t s, const StreamUses* uses);
    const bool own_;
    const cudaStream_t s_;
    const StreamUses* const uses_;
    const ReuseScope* const outer_;
};

struct BufferStats {
    long long requests;           // buffers asked for since the start, from the driver or kept ones
    size_t live_device, live_host, kept_device, kept_host;   // bytes in use, bytes kept
};
BufferStats buffer_stats();
// gives every kept block back to the driver
void empty_buffer_cache();

}  // namespace mpm
