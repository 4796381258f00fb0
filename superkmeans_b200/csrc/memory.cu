// Device memory, pinned host memory and streams of this library (see common.cuh).
//
// cudaMalloc and cudaFree synchronise the device and cost from 10 microseconds to hundreds of milliseconds each
// (measured on a B200: 70 pairs per flat Train of 1M x 1024, 0.1 - 0.7 s of its 0.6 - 1.1 s of wall time), so blocks that
// a call or a handle gives up are parked here and handed to the next request of about their size.
//
//   * Bounded: by default the parked blocks of one GPU stay within a sixteenth of its memory and the pinned ones within
//     256 MB; beyond that the blocks parked longest are returned to the driver.  CacheMode::everything lifts the bound,
//     CacheMode::nothing parks nothing, release_cached_memory() returns everything that is parked, and an
//     allocation that fails does so before it is tried again.
//   * Safe between streams and threads: a block released while its thread works on a stream (WorkStream) carries an event
//     recorded there, and whoever gets the block next makes its own stream wait for that event.  A block released
//     outside such a scope must be idle (the owners synchronise first).
#include <chrono>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace skmb {

namespace {

std::atomic<unsigned long long> g_device_allocs{0};
thread_local double g_alloc_ms = 0.0;
thread_local bool t_on_stream = false;
thread_local cudaStream_t t_stream = nullptr;
thread_local int t_device = 0;   // of t_stream

struct AllocClock {
    std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
    ~AllocClock() { g_alloc_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count(); }
};

struct Parked {
    void* p;
    size_t bytes;
    int device;
    cudaEvent_t last_use = nullptr;   // null: idle
    int event_device = 0;             // of last_use: the device of a pinned block's last user, which the next one need not share
};

constexpr int kMaxDevices = 64;
constexpr int kHost = -1;                 // "device" of pinned host blocks
constexpr size_t kPinnedBound = size_t{256} << 20;
constexpr size_t kMaxIdleStreams = 16;    // per device
constexpr size_t kMaxIdleEvents = 1024;   // that measure time, per device

struct FailingSizes {
    std::atomic<size_t> least{1}, most{0};
    bool hit(size_t bytes) const { return bytes >= least.load(std::memory_order_relaxed) && bytes <= most.load(std::memory_order_relaxed); }
};
FailingSizes g_fail_device, g_fail_pinned;

std::mutex g_mu;
std::vector<Parked> g_parked;   // oldest first
CacheMode g_mode = CacheMode::bounded;
std::vector<cudaEvent_t> g_events[kMaxDevices];
std::vector<cudaEvent_t> g_timing_events[kMaxDevices];
std::vector<cudaStream_t> g_streams[kMaxDevices];

// Sizes are rounded up to one of eight steps per power of two, so that requests that differ a little from call to call
// (buffers sized by a count that the data decide) land on the same block sizes and find each other's blocks.
size_t bucket(size_t bytes) {
    size_t p2 = 512;
    while (p2 * 2 <= bytes) p2 *= 2;
    const size_t step = p2 / 8;
    return std::max<size_t>(512, (bytes + step - 1) / step * step);
}

size_t bound_of(int device) {
    if (device == kHost) return kPinnedBound;
    static size_t bounds[kMaxDevices] = {0};   // under g_mu
    if (bounds[device] == 0) {
        size_t free_bytes = 0, total = 0;
        bounds[device] = cudaMemGetInfo(&free_bytes, &total) == cudaSuccess ? total / 16 : size_t{1} << 30;
    }
    return bounds[device];
}

void give_back(const Parked& b) {
    if (b.last_use) {
        cudaEventSynchronize(b.last_use);
        cudaEventDestroy(b.last_use);
    }
    if (b.device == kHost) {
        cudaFreeHost(b.p);
        return;
    }
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != b.device) cudaSetDevice(b.device);
    cudaFree(b.p);
    if (cur != b.device) cudaSetDevice(cur);
}

void give_back_all(const std::vector<Parked>& blocks) {
    for (const Parked& b : blocks) give_back(b);
}

std::vector<Parked> take_all_parked() {
    std::lock_guard<std::mutex> lock(g_mu);
    std::vector<Parked> out;
    out.swap(g_parked);
    return out;
}

// What is parked beyond the bounds, longest first (under g_mu).
std::vector<Parked> over_the_bound() {
    size_t total[kMaxDevices + 1] = {0};   // the host's last
    auto slot = [](const Parked& q) { return q.device == kHost ? kMaxDevices : q.device; };
    for (const Parked& q : g_parked) total[slot(q)] += q.bytes;
    std::vector<Parked> out;
    for (size_t i = 0; i < g_parked.size();) {
        const Parked& q = g_parked[i];
        if (total[slot(q)] <= bound_of(q.device)) {
            ++i;
            continue;
        }
        total[slot(q)] -= q.bytes;
        out.push_back(q);
        g_parked.erase(g_parked.begin() + static_cast<long>(i));
    }
    return out;
}

// The smallest parked block of this device (or of the host) that holds `bytes` and is at most a quarter larger.
bool take_parked(size_t bytes, int device, Parked& out) {
    std::lock_guard<std::mutex> lock(g_mu);
    size_t best = g_parked.size();
    for (size_t i = 0; i < g_parked.size(); ++i) {
        const Parked& b = g_parked[i];
        if (b.device == device && b.bytes >= bytes && b.bytes <= bytes + bytes / 4 && (best == g_parked.size() || b.bytes < g_parked[best].bytes)) best = i;
    }
    if (best == g_parked.size()) return false;
    out = g_parked[best];
    g_parked.erase(g_parked.begin() + static_cast<long>(best));
    return true;
}

// Orders the new owner of a block after its last one.  (An event goes back to the pool of its own device: only streams of that
// one can record it.)
void settle(const Parked& b) {
    if (!b.last_use) return;
    const cudaError_t e = b.device == kHost || !t_on_stream ? cudaEventSynchronize(b.last_use) : cudaStreamWaitEvent(t_stream, b.last_use, 0);
    if (e != cudaSuccess) {
        give_back(b);
        cuda_check(e, "wait for the last use of a parked block", __FILE__, __LINE__);
    }
    std::lock_guard<std::mutex> lock(g_mu);
    g_events[b.event_device].push_back(b.last_use);
}

// An event recorded where t_stream stands, or null.
cudaEvent_t mark_stream() {
    cudaEvent_t event = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        auto& pool = g_events[t_device];
        if (!pool.empty()) {
            event = pool.back();
            pool.pop_back();
        }
    }
    int cur = t_device;
    cudaGetDevice(&cur);
    if (cur != t_device) cudaSetDevice(t_device);
    if (!event && cudaEventCreateWithFlags(&event, cudaEventDisableTiming) != cudaSuccess) event = nullptr;
    if (event && cudaEventRecord(event, t_stream) != cudaSuccess) {
        cudaEventDestroy(event);
        event = nullptr;
    }
    if (cur != t_device) cudaSetDevice(cur);
    return event;
}

void park(Parked b) {
    if (t_on_stream) {
        b.last_use = mark_stream();
        b.event_device = t_device;
        if (!b.last_use) {
            cudaStreamSynchronize(t_stream);
            cudaGetLastError();   // (ours; the caller's next check is about its own work)
            give_back(b);
            return;
        }
    }
    std::vector<Parked> surplus;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (g_mode == CacheMode::nothing) {
            surplus.push_back(b);
        } else {
            g_parked.push_back(b);
            if (g_mode == CacheMode::bounded) surplus = over_the_bound();
        }
    }
    give_back_all(surplus);
}

} // namespace

unsigned long long device_alloc_count() { return g_device_allocs.load(std::memory_order_relaxed); }
void note_device_alloc() { g_device_allocs.fetch_add(1, std::memory_order_relaxed); }
double alloc_free_ms() { return g_alloc_ms; }

WorkStream::WorkStream(cudaStream_t stream) : was_on_(t_on_stream), previous_(t_stream), previous_device_(t_device) {
    SKM_CUDA(cudaGetDevice(&t_device));
    t_on_stream = true;
    t_stream = stream;
}
WorkStream::~WorkStream() {
    t_on_stream = was_on_;
    t_stream = previous_;
    t_device = previous_device_;
}

namespace {

// A parked block, or a new one from ALLOC.
template <class Alloc>
MemoryBlock take_or_make(size_t bytes, bool pinned, const char* what, Alloc alloc) {
    MemoryBlock m;
    SKM_CUDA(cudaGetDevice(&m.device));
    const bool fails = (pinned ? g_fail_pinned : g_fail_device).hit(bytes);
    bytes = bucket(bytes);
    Parked b;
    if (!fails && take_parked(bytes, pinned ? kHost : m.device, b)) {
        settle(b);
        m.p = b.p;
        m.bytes = b.bytes;
        return m;
    }
    note_device_alloc();
    cudaError_t e = fails ? cudaErrorMemoryAllocation : alloc(&m.p, bytes);
    if (e == cudaErrorMemoryAllocation && !fails) {
        // what is parked may be exactly what is missing
        cudaGetLastError();
        give_back_all(take_all_parked());
        e = alloc(&m.p, bytes);
    }
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();   // (the caller may know a way that needs less)
        throw OutOfMemory(std::string(what) + ": " + cudaGetErrorString(e) + " (" + std::to_string(bytes) + " bytes)");
    }
    cuda_check(e, what, __FILE__, __LINE__);
    m.bytes = bytes;
    return m;
}

} // namespace

void set_debug_alloc_failures(size_t least, size_t most, bool pinned) {
    FailingSizes& f = pinned ? g_fail_pinned : g_fail_device;
    f.least = least;
    f.most = most;
}

MemoryBlock device_alloc(size_t bytes) {
    AllocClock clock;
    return take_or_make(bytes, false, "cudaMalloc", [](void** p, size_t n) { return cudaMalloc(p, n); });
}

void device_free(const MemoryBlock& m) {
    if (!m.p) return;
    AllocClock clock;
    park(Parked{m.p, m.bytes, m.device});
}

MemoryBlock pinned_alloc(size_t bytes) {
    return take_or_make(bytes, true, "cudaHostAlloc", [](void** p, size_t n) { return cudaHostAlloc(p, n, cudaHostAllocPortable); });
}

void pinned_free(const MemoryBlock& m) {
    if (m.p) park(Parked{m.p, m.bytes, kHost});
}

cudaStream_t acquire_stream() {
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    {
        std::lock_guard<std::mutex> lock(g_mu);
        auto& pool = g_streams[device];
        if (!pool.empty()) {
            const cudaStream_t s = pool.back();
            pool.pop_back();
            return s;
        }
    }
    cudaStream_t s = nullptr;
    SKM_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    return s;
}

void release_stream(cudaStream_t s, int device) {
    if (!s) return;
    if (cudaStreamSynchronize(s) == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_mu);
        if (g_streams[device].size() < kMaxIdleStreams) {
            g_streams[device].push_back(s);
            return;
        }
    }
    cudaStreamDestroy(s);
}

cudaEvent_t acquire_timing_event() {
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    {
        std::lock_guard<std::mutex> lock(g_mu);
        auto& pool = g_timing_events[device];
        if (!pool.empty()) {
            const cudaEvent_t e = pool.back();
            pool.pop_back();
            return e;
        }
    }
    cudaEvent_t e = nullptr;
    SKM_CUDA(cudaEventCreate(&e));
    return e;
}

void release_timing_event(cudaEvent_t e, int device) {
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (g_timing_events[device].size() < kMaxIdleEvents) {
            g_timing_events[device].push_back(e);
            return;
        }
    }
    cudaEventDestroy(e);
}

void set_workspace_cache(CacheMode mode) {
    std::vector<Parked> surplus;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        g_mode = mode;
        if (mode == CacheMode::bounded) surplus = over_the_bound();
    }
    if (mode == CacheMode::nothing) release_cached_memory();
    give_back_all(surplus);
}

CacheMode workspace_cache() {
    std::lock_guard<std::mutex> lock(g_mu);
    return g_mode;
}

void release_cached_memory() {
    give_back_all(take_all_parked());
    std::lock_guard<std::mutex> lock(g_mu);
    for (auto& pool : g_timing_events) {
        for (cudaEvent_t e : pool) cudaEventDestroy(e);
        pool.clear();
    }
}

size_t cached_memory_bytes() {
    std::lock_guard<std::mutex> lock(g_mu);
    size_t total = 0;
    for (const Parked& b : g_parked) total += b.device == kHost ? 0 : b.bytes;
    return total;
}

} // namespace skmb
