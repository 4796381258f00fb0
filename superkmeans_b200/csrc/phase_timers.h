// Accumulating per-phase device timers: CUDA events around the phases of an engine's work.
#pragma once

#include <cstddef>
#include <cstdint>
#include <deque>
#include <vector>

#include "common.cuh"

namespace skmb {

// Names follow the sections of the reference's profiler (profiler.h): rotator, norms_calc, search/1st_blas, search,
// update_centroids, consolidate, shift.  Then the whole Train, and three parts of the pruned assignment: first ADSampling test on the tensor
// cores, candidate-list walk, dense chain.  Then spans that no kernel phase covers: device allocation and release (host wall clock), the
// initial centroids (Forgy shuffle on the host, row gather, their rotation), the per-iteration sum across shards (device span of
// the collective, which includes waiting for the slowest shard).  The last number is kept for callers that ask for it: nothing is booked there.
enum Phase { PH_ROTATE = 0, PH_NORMS, PH_ASSIGN_FULL, PH_ASSIGN_PRUNED, PH_UPDATE, PH_CONSOLIDATE, PH_SHIFT, PH_TRAIN_TOTAL, PH_PRUNE_FIRST_TEST, PH_PRUNE_WALK, PH_PRUNE_DENSE,
             PH_ALLOC_FREE, PH_INIT_CENTROIDS, PH_ALLREDUCE, PH_HOST_OTHER, PH_COUNT };

// Reading a pair of events takes 3 us (seven of them between two iterations were a fifth of the time that the GPU stood still there), so
// the last kKept pairs are read only for whoever asks for the times.  Older ones are read one by one, as new ones come, while the
// caller is about to wait for the GPU anyway, and their events are used again: an engine that serves calls for days holds no more
// events than after the first of them, and no call pays for many before it.
class PhaseTimers {
  public:
    static constexpr size_t kKept = 128;
    PhaseTimers() = default;
    PhaseTimers(const PhaseTimers&) = delete;
    PhaseTimers& operator=(const PhaseTimers&) = delete;
    ~PhaseTimers();
    void begin(int phase, cudaStream_t s);
    void end(cudaStream_t s);
    // Around every wait for all that is under way: read_old before it, finished after it.
    void read_old();
    void finished() { finished_ = pending_.size(); }
    void flush();  // reads all; only when all is done
    void reset();
    void add_host(int phase, double milliseconds) {
        ms[phase] += milliseconds;
        calls[phase] += 1;
    }
    size_t pending() const { return pending_.size(); }
    double ms[PH_COUNT] = {};
    uint64_t calls[PH_COUNT] = {};

  private:
    struct Pending {
        int phase;
        cudaEvent_t a, b;
    };
    void read_first();
    int device_ = -1;
    std::deque<Pending> pending_;
    size_t finished_ = 0;   // of pending_, from the front, that the GPU is known to have passed
    std::vector<Pending> open_;
};

} // namespace skmb
