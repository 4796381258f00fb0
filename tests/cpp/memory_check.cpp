// The parked blocks of memory.cu between devices, streams and failures (fake_cuda_runtime.h).
#include <cstring>

#include "../../superkmeans_b200/csrc/engine_buffers.h"
#include "fake_cuda_runtime.h"

using namespace skmb;

namespace {

// A block given up while its thread works on a stream of `device`.
template <class B>
void use_and_park(int device, size_t count) {
    cudaSetDevice(device);
    const cudaStream_t s = acquire_stream();
    {
        WorkStream work(s);
        B b;
        b.ensure(count);
    }
    CHECK(cudaGetLastError() == cudaSuccess);
    release_stream(s, device);
}

// Pinned blocks serve all devices, their events do not.
void events_between_devices() {
    use_and_park<PinnedBuffer<char>>(0, 5000);
    use_and_park<PinnedBuffer<char>>(1, 5000);   // the block of device 0
    use_and_park<DeviceBuffer<char>>(1, 3000);
    use_and_park<DeviceBuffer<char>>(0, 3000);
    use_and_park<PinnedBuffer<char>>(0, 5000);
    use_and_park<DeviceBuffer<char>>(0, 3000);
    int fresh = 0;
    for (const std::string& what : fake::log) fresh += what == "malloc" || what == "pinned";
    CHECK(fresh == 3);   // one pinned block, one of each device: nothing was given up on the way
}

// A block whose event cannot be recorded goes back to the driver once its stream is done, and the error with it.
void record_that_fails() {
    const cudaStream_t s = acquire_stream();
    {
        WorkStream work(s);
        DeviceBuffer<char> b;
        PinnedBuffer<char> h;
        char* dst = h.ensure(4096);
        std::vector<char> src(4096, 7);
        SKM_CUDA(cudaMemcpyAsync(b.ensure(4096), src.data(), 4096, cudaMemcpyHostToDevice, s));
        SKM_CUDA(cudaMemcpyAsync(dst, b.get(), 4096, cudaMemcpyDeviceToHost, s));
        fake::failing_records = 2;
        h.release();
        CHECK(!fake::in_flight(src.data(), 4096));
        b.release();
        CHECK(cudaGetLastError() == cudaSuccess);
    }
    release_stream(s, 0);
    CHECK(fake::device_in_use == 0 && fake::pinned_in_use == 0);
}

// What is parked is given back before an allocation counts as failed, of pinned memory too, and the failure leaves no error behind.
template <class B>
void memory_that_is_short(size_t& limit, size_t& in_use) {
    limit = size_t{1} << 20;
    cudaSetDevice(0);
    const cudaStream_t s = acquire_stream();
    {
        WorkStream work(s);
        {
            B b;
            b.ensure(900'000);
        }
        CHECK(in_use >= 900'000);
        B b;
        b.ensure(300'000);   // fits only once the other is gone
        B more;
        bool failed = false;
        try {
            more.ensure(900'000);
        } catch (const OutOfMemory&) {
            failed = true;
        }
        CHECK(failed && cudaGetLastError() == cudaSuccess);
        more.ensure(100'000);
        b.ensure(200'000);
    }
    release_stream(s, 0);
}

// The mode that was set is the one that is answered, and the bound holds again from when it is brought back.
void modes() {
    CHECK(workspace_cache() == CacheMode::bounded);
    auto parked = [] {
        use_and_park<DeviceBuffer<char>>(0, 30 << 20);   // (the fake device has 160 MB: ten of them may be parked)
        use_and_park<PinnedBuffer<char>>(0, 30 << 20);
        return std::pair<size_t, size_t>(fake::device_in_use, fake::pinned_in_use);
    };
    CHECK(parked().first == 0 && parked().second >= 30 << 20);
    set_workspace_cache(CacheMode::everything);
    CHECK(workspace_cache() == CacheMode::everything && parked().first >= 30 << 20);
    set_workspace_cache(CacheMode::bounded);
    CHECK(workspace_cache() == CacheMode::bounded && fake::device_in_use == 0 && fake::pinned_in_use >= 30 << 20);
    set_workspace_cache(CacheMode::nothing);
    CHECK(workspace_cache() == CacheMode::nothing && parked().first == 0 && parked().second == 0);
}

} // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "events_between_devices") events_between_devices();
    else if (what == "record_that_fails") record_that_fails();
    else if (what == "device_memory_that_is_short") memory_that_is_short<DeviceBuffer<char>>(fake::device_limit, fake::device_in_use);
    else if (what == "pinned_memory_that_is_short") memory_that_is_short<PinnedBuffer<char>>(fake::pinned_limit, fake::pinned_in_use);
    else if (what == "modes") modes();
    else return 2;
    std::puts("OK");
    return 0;
}
