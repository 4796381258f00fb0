// Phase timers over many calls (fake_cuda_runtime.h, where every pair of events is a millisecond apart).
#include "../../superkmeans_b200/csrc/phase_timers.h"
#include "fake_cuda_runtime.h"

using namespace skmb;

namespace {

void call(PhaseTimers& timers, cudaStream_t s, int phases) {
    for (int i = 0; i < phases; ++i) {
        timers.begin(PH_ASSIGN_FULL, s);
        timers.end(s);
    }
    timers.read_old();
    cudaStreamSynchronize(s);
    timers.finished();
}

void many_calls() {
    const cudaStream_t s = acquire_stream();
    {
        PhaseTimers timers;
        int most_reads = 0;
        for (int i = 0; i < 20'000; ++i) {
            const int before = fake::elapsed_reads;
            call(timers, s, 2);
            most_reads = std::max(most_reads, fake::elapsed_reads - before);
            CHECK(timers.pending() <= PhaseTimers::kKept + 2);
        }
        CHECK(most_reads <= 2);
        CHECK(fake::events_alive <= 2 * static_cast<int>(PhaseTimers::kKept + 2));
        timers.flush();
        CHECK(timers.calls[PH_ASSIGN_FULL] == 40'000 && timers.ms[PH_ASSIGN_FULL] == 40'000.0);
        timers.reset();
        CHECK(timers.calls[PH_ASSIGN_FULL] == 0);
    }
    release_stream(s, 0);
    release_cached_memory();
    CHECK(fake::events_alive == 0);
}

// Work that nothing has waited for yet is left alone, however much of it there is.
void nothing_unfinished_is_read() {
    const cudaStream_t s = acquire_stream();
    {
        PhaseTimers timers;
        char a = 0, b = 1;
        for (int i = 0; i < 1000; ++i) {
            timers.begin(PH_UPDATE, s);
            SKM_CUDA(cudaMemcpyAsync(&a, &b, 1, cudaMemcpyHostToHost, s));
            timers.end(s);
            timers.read_old();
        }
        CHECK(fake::elapsed_reads == 0 && cudaGetLastError() == cudaSuccess);
        call(timers, s, 1);
        call(timers, s, 1);
        CHECK(timers.pending() <= PhaseTimers::kKept + 2);
        timers.flush();
        CHECK(timers.calls[PH_UPDATE] == 1000 && cudaGetLastError() == cudaSuccess);
    }
    release_stream(s, 0);
}

} // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "many_calls") many_calls();
    else if (what == "nothing_unfinished_is_read") nothing_unfinished_is_read();
    else return 2;
    std::puts("OK");
    return 0;
}
