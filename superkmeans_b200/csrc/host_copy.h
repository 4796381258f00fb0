// Copies between ordinary host memory and the GPU through a ring of pinned pieces that several host threads fill or empty.
#pragma once

#include <cstddef>

#include "common.cuh"
#include "engine_buffers.h"

namespace skmb {

// cudaMemcpy from or to pageable memory moves 11 GB/s (one thread fills the driver's staging buffer); eight threads fill
// pinned memory at 70 GB/s (32 GB/s when they gather rows of 3 KB) and the link moves 55 GB/s from there, so the copies
// below run at 30 - 50 GB/s.  Memory that is pinned already is copied from directly.
//
// One per engine, used by one thread at a time; whoever owns it waits for both streams before it goes away.
class HostStage {
  public:
    HostStage() = default;
    HostStage(const HostStage&) = delete;
    HostStage& operator=(const HostStage&) = delete;
    ~HostStage();

    // dst[i] = src[idx ? idx[i] : i] for n rows of row_bytes, enqueued on `stream`; src and idx may be changed or freed
    // on return, except that a pinned src without idx must stay until the stream has passed the copy.
    void upload(void* dst, const void* src, const size_t* idx, size_t n, size_t row_bytes, cudaStream_t stream);
    // dst (host) = src (device), in order on `stream`; waits for it.
    void download(void* dst, const void* src, size_t bytes, cudaStream_t stream);

  private:
    static constexpr int kPieces = 4;
    static constexpr size_t kPieceBytes = size_t{4} << 20;
    char* piece(int i, size_t bytes);
    PinnedBuffer<char> pieces_[kPieces];
    cudaEvent_t copied_[kPieces] = {};   // the last copy from or to a piece
    int next_ = 0;
};

} // namespace skmb
