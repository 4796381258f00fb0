// See fake_cuda_runtime.h.
#include "fake_cuda_runtime.h"

#include <cstring>
#include <map>
#include <set>

// A stream is a list of operations, done one after the other when somebody waits for one of them.
struct Operation {
    std::function<void()> copy;
    fake::Copy what{nullptr, nullptr, 0};
    CUevent_st* wait = nullptr;   // the work that this event stood for when the wait was enqueued
    size_t wait_upto = 0;
    CUstream_st* wait_stream = nullptr;
};
struct CUstream_st {
    int device = 0;
    std::vector<Operation> ops;
    size_t done = 0;
};
struct CUevent_st {
    int device = 0;
    CUstream_st* stream = nullptr;
    size_t upto = 0;
};

namespace fake {

size_t device_limit = size_t{1} << 40, pinned_limit = size_t{1} << 40;
size_t device_in_use = 0, pinned_in_use = 0;
int events_alive = 0, elapsed_reads = 0, failing_records = 0;
std::vector<std::string> log;

namespace {

thread_local int current = 0;
thread_local cudaError_t last = cudaSuccess;
struct Allocation {
    size_t bytes;
    bool pinned;
};
std::map<char*, Allocation> allocations;
std::set<CUstream_st*> streams;

cudaError_t answer(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}

void run(CUstream_st* s, size_t upto) {
    while (s->done < upto) {
        Operation op = s->ops[s->done++];
        if (op.wait_stream) run(op.wait_stream, op.wait_upto);
        if (op.copy) op.copy();
    }
}

const Allocation* find(const void* p) {
    auto it = allocations.upper_bound(static_cast<char*>(const_cast<void*>(p)));
    if (it == allocations.begin()) return nullptr;
    --it;
    return static_cast<const char*>(p) < it->first + it->second.bytes ? &it->second : nullptr;
}

cudaError_t allocate(void** p, size_t bytes, bool pinned) {
    size_t& in_use = pinned ? pinned_in_use : device_in_use;
    if (in_use + bytes > (pinned ? pinned_limit : device_limit)) return answer(cudaErrorMemoryAllocation);
    *p = std::malloc(bytes);
    in_use += bytes;
    allocations[static_cast<char*>(*p)] = {bytes, pinned};
    log.push_back(pinned ? "pinned" : "malloc");
    return cudaSuccess;
}

cudaError_t release(void* p) {
    auto it = allocations.find(static_cast<char*>(p));
    if (it == allocations.end()) return answer(cudaErrorInvalidValue);
    if (!it->second.pinned)
        for (CUstream_st* s : streams) run(s, s->ops.size());   // as cudaFree does
    (it->second.pinned ? pinned_in_use : device_in_use) -= it->second.bytes;
    allocations.erase(it);
    std::free(p);
    log.push_back("free");
    return cudaSuccess;
}

} // namespace

bool in_flight(const void* p, size_t bytes) {
    const char* lo = static_cast<const char*>(p);
    auto touches = [&](const void* q, size_t n) { return static_cast<const char*>(q) < lo + bytes && lo < static_cast<const char*>(q) + n; };
    for (CUstream_st* s : streams)
        for (size_t i = s->done; i < s->ops.size(); ++i)
            if (s->ops[i].copy && (touches(s->ops[i].what.dst, s->ops[i].what.bytes) || touches(s->ops[i].what.src, s->ops[i].what.bytes))) return true;
    return false;
}

bool is_device_memory(const void* p) {
    const Allocation* a = find(p);
    return a && !a->pinned;
}

} // namespace fake

using namespace fake;

extern "C" {

cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error"; }
cudaError_t cudaGetDevice(int* d) {
    *d = current;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    current = d;
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* free_bytes, size_t* total) {
    *total = size_t{160} << 20;
    *free_bytes = *total;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t bytes) { return allocate(p, bytes, false); }
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) { return allocate(p, bytes, true); }
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaFreeHost(void* p) { return release(p); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = new CUstream_st;
    (*s)->device = current;
    streams.insert(*s);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    run(s, s->ops.size());
    streams.erase(s);
    delete s;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    run(s, s->ops.size());
    log.push_back("stream synchronise");
    return cudaSuccess;
}

cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = new CUevent_st;
    (*e)->device = current;
    ++events_alive;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete e;
    --events_alive;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (failing_records > 0) {
        --failing_records;
        return answer(cudaErrorUnknown);
    }
    if (e->device != s->device) return answer(cudaErrorInvalidResourceHandle);
    e->stream = s;
    e->upto = s->ops.size();
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) { return e->stream && e->stream->done < e->upto ? answer(cudaErrorNotReady) : cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (e->stream) run(e->stream, e->upto);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    if (!e->stream) return cudaSuccess;
    Operation op;
    op.wait = e;
    op.wait_stream = e->stream;
    op.wait_upto = e->upto;
    s->ops.push_back(op);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
    ++elapsed_reads;
    for (cudaEvent_t e : {a, b}) {
        if (!e->stream) return answer(cudaErrorInvalidResourceHandle);
        if (e->stream->done < e->upto) return answer(cudaErrorNotReady);
    }
    *ms = 1.0f;
    return cudaSuccess;
}

cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    const Allocation* m = find(p);
    *a = cudaPointerAttributes{};
    a->type = !m ? cudaMemoryTypeUnregistered : (m->pinned ? cudaMemoryTypeHost : cudaMemoryTypeDevice);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t s) {
    Operation op;
    op.what = {dst, src, bytes};
    op.copy = [=] { std::memcpy(dst, src, bytes); };
    s->ops.push_back(op);
    return cudaSuccess;
}

} // extern "C"
