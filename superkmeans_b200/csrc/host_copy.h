// Copies between ordinary host memory and the GPU through a ring of pinned pieces that several host threads fill or empty.
#pragma once

#include <cstddef>

#include "common.cuh"
#include "engine_buffers.h"

namespace skmb {

// cudaMemcpy from or to pageable memory moves 11 GB/s (one thread fills the driver's staging buffer); eight threads fill
// pinned memory at 63 GB/s (32 GB/s when they gather rows of 3 KB) and the link moves 50 - 55 GB/s from there, so the copies
// below run at 30 - 50 GB/s.  Memory that the GPU can read by itself is copied from directly.
//
// One per engine, used by one thread at a time; whoever owns it waits for both streams before it goes away.
class HostStage {
  public:
    HostStage() = default;
    HostStage(const HostStage&) = delete;
    HostStage& operator=(const HostStage&) = delete;
    ~HostStage();

    // dst[i] = src[idx ? idx[i] : i] for n rows of row_bytes, enqueued on `stream`; src and idx may be changed or freed
    // on return, except that a src that is copied directly must stay until the stream has passed the copy.
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

// Rows of a host matrix on their way through one or two device buffers, in turn: copies on one stream, the kernels that use the rows
// on another.  Per piece: upload, arrive, the kernels, used.
//
// The buffers go back with an event of the kernels' stream, which says nothing about copies that it does not wait for yet, and a
// pinned source is read until the last copy is done: when an exception ends the loop, the copies are waited for first.
class RowPipe {
  public:
    RowPipe(HostStage& stage, cudaStream_t copies, cudaStream_t work);
    ~RowPipe();
    RowPipe(const RowPipe&) = delete;
    RowPipe& operator=(const RowPipe&) = delete;

    // Buffers of `floats` each, before the first upload.
    void reserve(size_t floats, int buffers);
    DeviceBuffer<float>& buffer(int i) { return buffers_[i]; }
    // The next n rows (see HostStage::upload) to `to`, or to the next buffer if that is null; returns where they go.
    float* upload(float* to, const float* src, const size_t* idx, size_t n, size_t row_bytes);
    void arrive();   // what follows on the kernels' stream finds them there
    void used();     // what uses them is enqueued

  private:
    HostStage& stage_;
    cudaStream_t copies_, work_;
    DeviceBuffer<float> buffers_[2];
    cudaEvent_t copied_[2] = {}, used_[2] = {};
    size_t pieces_ = 0;
    int unwinding_;   // exceptions on their way when this was made
};

} // namespace skmb
