// Device and page-locked host memory of DevBuf / HostBuf (see mpm_common.cuh).
//
// A program that solves one parameter set after another builds and drops a
// solver with some eighty buffers each time; cudaMalloc, cudaFree and above
// all page-locking cost more than the solve of a small system (a spectrum of
// the N = 4000 monolayer spent 27 of its 43 ms outside the kernels; with the
// tables of mpm_tables.cpp 26 ms are left, and passes no longer wait up to a
// second for the driver's allocator when other processes use it).
// Released blocks are therefore kept for the next request of about the same
// size:
//  * a block is kept only after the work that used it has been waited for, so
//    the next owner may be any thread and any stream.  The work is known by
//    stream: a solver's and a near field's own one, and those on which a
//    caller applied a field (ReuseScope).  Waiting for the whole device would
//    break a graph capture that runs in another thread, which cudaFree does
//    not;
//  * a block whose work is not known (a field whose call was captured or has
//    thrown, the tuner's trials) goes back to the driver at once;
//  * bounded: at most 256 MB of device and 64 MB of host memory, no block
//    above a quarter of that, and a block that kMaxAge later releases did not
//    reuse is freed; empty_buffer_cache() frees them all;
//  * when the driver is out of memory the kept blocks are freed first.
#include "mpm_alloc.h"

#include <list>
#include <mutex>
#include <unordered_map>

namespace mpm {

namespace {

struct Pool {
    struct Block {
        void* p;
        size_t bytes;
        int dev;
        unsigned long long born;
    };
    std::mutex mu;
    std::list<Block> kept;                                   // oldest first
    std::unordered_map<void*, std::pair<size_t, int>> live;  // size, device
    size_t total = 0, used = 0;                              // bytes kept, bytes in use
    unsigned long long clock = 0;
    long long requests = 0;
    const bool host;
    const size_t cap;
    Pool(bool h, size_t c) : host(h), cap(c) {}

    size_t largest() const { return cap / 4; }
    void drop(const Block& b) {
        if (host) cudaFreeHost(b.p);
        else cudaFree(b.p);
    }
    // frees kept blocks: all of them, or those past the age limit and beyond the cap
    void trim(bool all) {
        while (!kept.empty() && (all || total > cap || clock - kept.front().born > kMaxAge)) {
            total -= kept.front().bytes;
            drop(kept.front());
            kept.pop_front();
        }
    }
    static constexpr unsigned long long kMaxAge = 1024;
};

// (never destroyed: buffers of static objects may outlive this file's statics)
Pool& pool(bool host) {
    static Pool* dev = new Pool(false, size_t(256) << 20);
    static Pool* hst = new Pool(true, size_t(64) << 20);
    return host ? *hst : *dev;
}

thread_local const ReuseScope* t_scope = nullptr;

// steps of an eighth to a quarter, so that a kept block fits its next request;
// blocks too large to be kept are not enlarged
size_t rounded(size_t n, size_t largest) {
    size_t unit = 512;
    while (n <= largest && unit * 8 < n) unit *= 2;
    return (n + unit - 1) / unit * unit;
}

}  // namespace

namespace {
// an error that only means that a block cannot be kept
bool ok(cudaError_t e) {
    if (e == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}
}  // namespace

StreamUses::~StreamUses() {
    for (const Use& u : uses_) cudaEventDestroy(u.done);
}

void StreamUses::record(cudaStream_t s) {
    if (unknown_) return;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    if (!ok(cudaStreamIsCapturing(s, &cap)) || cap != cudaStreamCaptureStatusNone || !ok(cudaStreamGetId(s, &id))) {
        unknown_ = true;
        return;
    }
    for (const Use& u : uses_)
        if (u.stream == id) {
            if (!ok(cudaEventRecord(u.done, s))) unknown_ = true;
            return;
        }
    Use u{id, nullptr};
    if (uses_.size() >= 16) {          // a caller that makes a stream per call: wait for the oldest
        u.done = uses_.front().done;
        uses_.erase(uses_.begin());
        if (!ok(cudaEventSynchronize(u.done))) unknown_ = true;
    } else if (!ok(cudaEventCreateWithFlags(&u.done, cudaEventDisableTiming))) {
        unknown_ = true;
        return;
    }
    uses_.push_back(u);
    if (!ok(cudaEventRecord(u.done, s))) unknown_ = true;
}

bool StreamUses::wait() const {
    if (unknown_) return false;
    for (const Use& u : uses_)
        if (!ok(cudaEventSynchronize(u.done))) return false;
    return true;
}

ReuseScope::ReuseScope(bool own, cudaStream_t s, const StreamUses* uses)
    : own_(own), s_(s), uses_(uses), outer_(t_scope) {
    t_scope = this;
}
ReuseScope::~ReuseScope() { t_scope = outer_; }
bool ReuseScope::idle() const {
    return (!own_ || ok(cudaStreamSynchronize(s_))) && (!uses_ || uses_->wait());
}

void* buf_alloc(size_t n, bool host) {
    Pool& P = pool(host);
    int dev = 0;
    MPM_CUDA(cudaGetDevice(&dev));
    const size_t want = rounded(n, P.largest());
    std::lock_guard<std::mutex> lock(P.mu);
    ++P.requests;
    auto best = P.kept.end();
    for (auto it = P.kept.begin(); it != P.kept.end(); ++it)
        if (it->bytes >= want && it->bytes <= want + want / 4 + 4096 && (host || it->dev == dev) &&
            (best == P.kept.end() || it->bytes < best->bytes))
            best = it;
    void* p = nullptr;
    size_t got = want;
    if (best != P.kept.end()) {
        p = best->p;
        got = best->bytes;
        P.total -= got;
        P.kept.erase(best);
    } else {
        auto get = [&] { return host ? cudaHostAlloc(&p, want, cudaHostAllocPortable) : cudaMalloc(&p, want); };
        cudaError_t e = get();
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            P.trim(true);
            e = get();
        }
        MPM_CUDA(e);
    }
    P.live[p] = {got, dev};
    P.used += got;
    return p;
}

void buf_free(void* p, bool host) {
    if (!p) return;
    Pool& P = pool(host);
    std::pair<size_t, int> b;
    {
        std::lock_guard<std::mutex> lock(P.mu);
        auto it = P.live.find(p);
        if (it == P.live.end()) return;
        b = it->second;
        P.live.erase(it);
        P.used -= b.first;
    }
    // (the wait is outside the lock)
    if (!t_scope || b.first > P.largest() || !t_scope->idle()) {
        if (host) cudaFreeHost(p);
        else cudaFree(p);
        return;
    }
    std::lock_guard<std::mutex> lock(P.mu);
    P.kept.push_back({p, b.first, b.second, ++P.clock});
    P.total += b.first;
    P.trim(false);
}

BufferStats buffer_stats() {
    BufferStats s{};
    for (int host = 0; host < 2; ++host) {
        Pool& P = pool(host != 0);
        std::lock_guard<std::mutex> lock(P.mu);
        s.requests += P.requests;
        (host ? s.live_host : s.live_device) = P.used;
        (host ? s.kept_host : s.kept_device) = P.total;
    }
    return s;
}

void empty_buffer_cache() {
    for (int host = 0; host < 2; ++host) {
        Pool& P = pool(host != 0);
        std::lock_guard<std::mutex> lock(P.mu);
        P.trim(true);
    }
}

}  // namespace mpm
