// See phase_timers.h.
#include "phase_timers.h"

namespace skmb {

PhaseTimers::~PhaseTimers() {
    auto give_back = [&](const Pending& p) {
        release_timing_event(p.a, device_);
        release_timing_event(p.b, device_);
    };
    for (const Pending& p : pending_) give_back(p);
    for (const Pending& p : open_) give_back(p);
}

void PhaseTimers::begin(int phase, cudaStream_t s) {
    if (device_ < 0) SKM_CUDA(cudaGetDevice(&device_));   // (the owner's, always the same)
    Pending p{phase, acquire_timing_event(), acquire_timing_event()};
    SKM_CUDA(cudaEventRecord(p.a, s));
    open_.push_back(p);
}

void PhaseTimers::end(cudaStream_t s) {
    if (open_.empty()) return;
    Pending p = open_.back();
    open_.pop_back();
    cudaEventRecord(p.b, s);
    pending_.push_back(p);
}

void PhaseTimers::read_first() {
    const Pending p = pending_.front();
    pending_.pop_front();
    if (finished_ > 0) --finished_;
    float t = 0.f;
    if (cudaEventElapsedTime(&t, p.a, p.b) == cudaSuccess) {
        ms[p.phase] += t;
        calls[p.phase] += 1;
    } else {
        cudaGetLastError();   // (of a phase that an exception ended)
    }
    release_timing_event(p.a, device_);
    release_timing_event(p.b, device_);
}

void PhaseTimers::read_old() {
    while (finished_ > 0 && pending_.size() > kKept) read_first();
}

void PhaseTimers::flush() {
    while (!pending_.empty()) read_first();
}

void PhaseTimers::reset() {
    for (int i = 0; i < PH_COUNT; ++i) {
        ms[i] = 0.0;
        calls[i] = 0;
    }
}

} // namespace skmb
