// Definitions shared by the translation units that implement the C ABI.
#pragma once

#include <functional>
#include <optional>

#include "mpm_alloc.h"
#include "mpm_field.h"
#include "mpm_krylov.h"

struct mpm_field {
    mpm::Field* impl;
    mpm::BatchSolver* solver;
    mpm::StreamUses uses;
};

// A call that queues a field's work on a stream: buffers that it outgrows may be
// kept, and done() records that the stream has been used.  Without done() (the
// call threw, perhaps with work left on the field's second stream) the field's
// buffers are not kept any more.
class FieldCall {
public:
    FieldCall(mpm_field* f, cudaStream_t s) : f_(f), s_(s) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) {
            cudaGetLastError();
            f->uses.give_up();
        } else if (cap != cudaStreamCaptureStatusNone) {
            f->uses.give_up();
        }
        if (!f->uses.unknown()) scope_.emplace(f->uses, s);
    }
    ~FieldCall() {
        if (!done_) f_->uses.give_up();
    }
    void done() {
        done_ = true;
        f_->uses.record(s_);
    }

private:
    mpm_field* f_;
    cudaStream_t s_;
    std::optional<mpm::ReuseScope> scope_;
    bool done_ = false;
};

namespace mpm {
// Runs f, mapping exceptions to a status code and the thread's last-error text.
int capi_guard(const std::function<void()>& f);
}  // namespace mpm
