// See host_copy.h.
#include "host_copy.h"

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <exception>

#ifdef __SSE2__
#include <emmintrin.h>
#endif

namespace skmb {

namespace {

cudaMemoryType type_of(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return cudaMemoryTypeUnregistered;
    }
    return a.type;
}
// Pinned or managed memory, and memory of a GPU that a caller gave in place of a host array: nothing to stage.
bool copied_directly(const void* p) { return type_of(p) != cudaMemoryTypeUnregistered; }

// A thread per quarter of a megabyte, eight at most: more do not copy faster.
int threads_for(size_t bytes) { return static_cast<int>(std::max<size_t>(1, std::min<size_t>(8, bytes >> 18))); }

// Copies to memory that the GPU reads next, past the caches: what another core has just written to its cache the link fetches at
// 30 GB/s (4 MB, eight threads: 138 us), what lies in memory at 50 (84 us).  Filling it takes 66 us in place of 44, beside the copy before.
// A cache line must not be written both ways, so that only whole lines are streamed, the ends of a contiguous part are not.
// publish() comes behind the last of a thread.  A few rows are in one core's cache, and the link is not what they wait for: a call that assigns 32 KB of
// rows takes 52.3 us with plain stores and 53.5 past the caches, 48 KB 53.2 and 54.6, 56 KB 57.2 and 54.6, 128 KB 62 and 58, 1 MB 101 and 83.  Beyond
// the last level of the caches there is little in it either way: 350 MB: 7.4 - 8.0 ms and 7.8 - 8.3 when repeated, 8.8 and 8.4 the first time.
constexpr size_t kStreamFrom = 56 << 10;
void stream_bytes(char* dst, const char* src, size_t bytes) {
#ifdef __SSE2__
    const size_t head = std::min(bytes, static_cast<size_t>(-reinterpret_cast<uintptr_t>(dst) & 63));
    std::memcpy(dst, src, head);
    size_t i = head;
    for (; i + 64 <= bytes; i += 64) {
        __m128i v[4];
        for (int q = 0; q < 4; ++q) v[q] = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i) + q);
        for (int q = 0; q < 4; ++q) _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i) + q, v[q]);
    }
    std::memcpy(dst + i, src + i, bytes - i);
#else
    std::memcpy(dst, src, bytes);
#endif
}
void publish() {
#ifdef __SSE2__
    _mm_sfence();
#endif
}

// `to_gpu`: the GPU reads dst, else the caller does.
void copy_bytes(char* dst, const char* src, size_t bytes, bool to_gpu) {
    const bool past_caches = to_gpu && bytes >= kStreamFrom;
    auto part = [&](size_t b, size_t e) {
        if (past_caches) {
            stream_bytes(dst + b, src + b, e - b);
            publish();
        } else {
            std::memcpy(dst + b, src + b, e - b);
        }
    };
    const int threads = threads_for(bytes);
    if (threads == 1) {   // (a team of one too costs a call with three copies most of a microsecond)
        part(0, bytes);
        return;
    }
#pragma omp parallel for num_threads(threads) schedule(static)
    for (int t = 0; t < threads; ++t) part(bytes * t / threads, bytes * (t + 1) / threads);
}

// Rows of whole cache lines are streamed.  Others share lines with their neighbours: a Train on 98 857 of 329 524 rows of 624 bytes took 13.3 ms
// with streaming stores and 8.8 with plain ones.
void gather_rows(char* dst, const char* src, const size_t* idx, size_t n, size_t row_bytes) {
    const int threads = threads_for(n * row_bytes);
    const bool lines = n * row_bytes >= kStreamFrom && row_bytes % 64 == 0 && reinterpret_cast<uintptr_t>(dst) % 64 == 0;
#pragma omp parallel for num_threads(threads) schedule(static) if (threads > 1)
    for (int t = 0; t < threads; ++t) {
        for (size_t i = n * t / threads; i < n * (t + 1) / threads; ++i) {
            if (lines) stream_bytes(dst + i * row_bytes, src + idx[i] * row_bytes, row_bytes);
            else std::memcpy(dst + i * row_bytes, src + idx[i] * row_bytes, row_bytes);
        }
        publish();
    }
}

} // namespace

HostStage::~HostStage() {
    for (cudaEvent_t e : copied_)
        if (e) cudaEventDestroy(e);
}

// Piece i, free for the host, at least `bytes` long.
char* HostStage::piece(int i, size_t bytes) {
    if (!copied_[i]) SKM_CUDA(cudaEventCreateWithFlags(&copied_[i], cudaEventDisableTiming));
    else SKM_CUDA(cudaEventSynchronize(copied_[i]));
    return pieces_[i].ensure(bytes);
}

void HostStage::upload(void* dst, const void* src, const size_t* idx, size_t n, size_t row_bytes, cudaStream_t stream) {
    if (n == 0 || row_bytes == 0) return;
    if (!idx && copied_directly(src)) {
        SKM_CUDA(cudaMemcpyAsync(dst, src, n * row_bytes, cudaMemcpyDefault, stream));
        return;
    }
    if (idx && type_of(src) == cudaMemoryTypeDevice) {
        for (size_t i = 0; i < n; ++i)
            SKM_CUDA(cudaMemcpyAsync(static_cast<char*>(dst) + i * row_bytes, static_cast<const char*>(src) + idx[i] * row_bytes, row_bytes, cudaMemcpyDefault, stream));
        return;
    }
    const size_t per_piece = std::max<size_t>(1, kPieceBytes / row_bytes);
    for (size_t r0 = 0; r0 < n; r0 += per_piece) {
        const size_t cnt = std::min(per_piece, n - r0);
        const int i = next_;
        next_ = (next_ + 1) % kPieces;
        char* p = piece(i, cnt * row_bytes);
        if (idx) gather_rows(p, static_cast<const char*>(src), idx + r0, cnt, row_bytes);
        else copy_bytes(p, static_cast<const char*>(src) + r0 * row_bytes, cnt * row_bytes, true);
        SKM_CUDA(cudaMemcpyAsync(static_cast<char*>(dst) + r0 * row_bytes, p, cnt * row_bytes, cudaMemcpyHostToDevice, stream));
        SKM_CUDA(cudaEventRecord(copied_[i], stream));
    }
}

void HostStage::download(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
    if (bytes == 0) return;
    if (copied_directly(dst)) {
        SKM_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, stream));
        SKM_CUDA(cudaStreamSynchronize(stream));
        return;
    }
    const size_t n = (bytes + kPieceBytes - 1) / kPieceBytes;
    int slot[kPieces];
    auto enqueue = [&](size_t q) {
        const size_t b = q * kPieceBytes, cnt = std::min(kPieceBytes, bytes - b);
        const int i = next_;
        next_ = (next_ + 1) % kPieces;
        slot[q % kPieces] = i;
        SKM_CUDA(cudaMemcpyAsync(piece(i, cnt), static_cast<const char*>(src) + b, cnt, cudaMemcpyDeviceToHost, stream));
        SKM_CUDA(cudaEventRecord(copied_[i], stream));
    };
    // one piece less than the ring in flight: the one being emptied must not be reused
    size_t sent = 0;
    for (size_t q = 0; q < n; ++q) {
        for (; sent < n && sent < q + kPieces - 1; ++sent) enqueue(sent);
        const int i = slot[q % kPieces];
        SKM_CUDA(cudaEventSynchronize(copied_[i]));
        const size_t b = q * kPieceBytes;
        copy_bytes(static_cast<char*>(dst) + b, pieces_[i].get(), std::min(kPieceBytes, bytes - b), false);
    }
}

RowPipe::RowPipe(HostStage& stage, cudaStream_t copies, cudaStream_t work) : stage_(stage), copies_(copies), work_(work), unwinding_(std::uncaught_exceptions()) {}

RowPipe::~RowPipe() {
    if (std::uncaught_exceptions() > unwinding_) cudaStreamSynchronize(copies_);
    for (cudaEvent_t e : {copied_[0], copied_[1], used_[0], used_[1]})
        if (e) cudaEventDestroy(e);
}

void RowPipe::reserve(size_t floats, int buffers) {
    for (int i = 0; i < buffers; ++i) buffers_[i].ensure(floats);
}

float* RowPipe::upload(float* to, const float* src, const size_t* idx, size_t n, size_t row_bytes) {
    const int b = static_cast<int>(pieces_ & 1);
    if (pieces_ == 0) {
        for (cudaEvent_t* e : {&copied_[0], &copied_[1], &used_[0], &used_[1]}) SKM_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
        // what the copies write may still be in use by earlier work that was enqueued on the kernels' stream
        SKM_CUDA(cudaEventRecord(used_[0], work_));
        SKM_CUDA(cudaStreamWaitEvent(copies_, used_[0], 0));
    }
    if (!to) {
        if (pieces_ >= 2) SKM_CUDA(cudaStreamWaitEvent(copies_, used_[b], 0));
        to = buffers_[b].get();
    }
    stage_.upload(to, src, idx, n, row_bytes, copies_);
    SKM_CUDA(cudaEventRecord(copied_[b], copies_));
    return to;
}

void RowPipe::arrive() { SKM_CUDA(cudaStreamWaitEvent(work_, copied_[pieces_ & 1], 0)); }

void RowPipe::used() {
    SKM_CUDA(cudaEventRecord(used_[pieces_ & 1], work_));
    ++pieces_;
}

} // namespace skmb
