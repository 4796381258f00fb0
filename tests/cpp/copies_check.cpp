// Copies of host rows (host_copy.cu) when something goes wrong on the way (fake_cuda_runtime.h).
#include <algorithm>
#include <cstring>
#include <stdexcept>

#include "../../superkmeans_b200/csrc/host_copy.h"
#include "fake_cuda_runtime.h"

using namespace skmb;

namespace {

constexpr size_t kRow = 64, kRows = 100;

// An exception between a copy and the kernels that would have waited for it.
void exception_behind_a_copy(bool pinned) {
    const cudaStream_t copies = acquire_stream(), work = acquire_stream();
    {
        WorkStream on(work);
        HostStage stage;
        std::vector<float> rows(3 * kRows * kRow, 1.0f);
        PinnedBuffer<float> pinned_rows;
        const float* src = pinned ? pinned_rows.ensure(rows.size()) : rows.data();
        const int events = fake::events_alive;
        const float* raw = nullptr;
        try {
            RowPipe pipe(stage, copies, work);
            pipe.reserve(kRows * kRow, 2);
            for (int piece = 0; piece < 3; ++piece) {
                raw = pipe.upload(nullptr, src + piece * kRows * kRow, nullptr, kRows, kRow * sizeof(float));
                CHECK(fake::is_device_memory(raw) && fake::in_flight(raw, kRows * kRow * sizeof(float)));
                if (piece == 2) throw std::runtime_error("no matrix");
                pipe.arrive();
                pipe.used();
            }
        } catch (const std::runtime_error&) {
        }
        // the buffers are parked now: their next owner waits for `work` only
        CHECK(!fake::in_flight(raw, kRows * kRow * sizeof(float)));
        CHECK(!fake::in_flight(src, rows.size() * sizeof(float)));
        CHECK(fake::events_alive <= events + 2 + 4);   // of the two parked buffers and the stage's pieces
    }
    release_stream(copies, 0);
    release_stream(work, 0);
}

// All pieces arrive in their place, from either kind of source, by index too.
void rows_arrive() {
    const cudaStream_t copies = acquire_stream(), work = acquire_stream();
    {
        WorkStream on(work);
        HostStage stage;
        std::vector<float> rows(7 * kRows * kRow), got(rows.size());
        for (size_t i = 0; i < rows.size(); ++i) rows[i] = static_cast<float>(i);
        std::vector<size_t> idx(7 * kRows);
        for (size_t i = 0; i < idx.size(); ++i) idx[i] = idx.size() - 1 - i;
        for (const size_t* by : {static_cast<const size_t*>(nullptr), static_cast<const size_t*>(idx.data())}) {
            RowPipe pipe(stage, copies, work);
            pipe.reserve(kRows * kRow, 2);
            for (size_t r0 = 0; r0 < 7 * kRows; r0 += kRows) {
                const float* at = pipe.upload(nullptr, by ? rows.data() : rows.data() + r0 * kRow, by ? by + r0 : nullptr, kRows, kRow * sizeof(float));
                pipe.arrive();
                SKM_CUDA(cudaMemcpyAsync(got.data() + r0 * kRow, at, kRows * kRow * sizeof(float), cudaMemcpyDeviceToHost, work));
                pipe.used();
            }
            SKM_CUDA(cudaStreamSynchronize(work));
            for (size_t r = 0; r < 7 * kRows; ++r)
                for (size_t j = 0; j < kRow; ++j) CHECK(got[r * kRow + j] == rows[(by ? by[r] : r) * kRow + j]);
        }
    }
    release_stream(copies, 0);
    release_stream(work, 0);
}

// Pieces of all lengths around those from which the stores go past the caches, from rows that start anywhere.
void pieces_of_any_length() {
    const cudaStream_t s = acquire_stream();
    {
        WorkStream on(s);
        HostStage stage;
        std::vector<unsigned char> rows((3 << 20) + 128), got(rows.size());
        for (size_t i = 0; i < rows.size(); ++i) rows[i] = static_cast<unsigned char>(i * 2654435761u >> 13);
        for (const size_t row_bytes : {size_t{4}, size_t{60}, size_t{64}, size_t{256}}) {
            for (const size_t bytes : {size_t{4}, size_t{60}, size_t{64}, size_t{4096}, size_t{57'340}, size_t{57'344}, size_t{57'348}, size_t{114'688}, size_t{600'000}, size_t{3} << 20}) {
                const size_t n = bytes / row_bytes;
                std::vector<size_t> idx(n);
                for (size_t i = 0; i < n; ++i) idx[i] = n - 1 - i;
                for (const size_t from : {size_t{0}, size_t{4}, size_t{68}}) {
                    for (const bool gathered : {false, true}) {
                        std::fill(got.begin(), got.end(), 0);
                        stage.upload(got.data(), rows.data() + from, gathered ? idx.data() : nullptr, n, row_bytes, s);
                        SKM_CUDA(cudaStreamSynchronize(s));
                        for (size_t i = 0; i < n; ++i) CHECK(std::memcmp(got.data() + i * row_bytes, rows.data() + from + (gathered ? idx[i] : i) * row_bytes, row_bytes) == 0);
                        CHECK(std::count(got.begin() + n * row_bytes, got.begin() + n * row_bytes + 64, 0) == 64);
                    }
                }
            }
        }
    }
    release_stream(s, 0);
}

// Device memory where host memory is expected.
void device_memory() {
    const cudaStream_t s = acquire_stream();
    {
        WorkStream on(s);
        HostStage stage;
        std::vector<float> rows(kRows * kRow, 3.0f);
        for (size_t j = 0; j < kRow; ++j) rows[kRow + j] = 4.0f;
        DeviceBuffer<float> src, dst, out;
        SKM_CUDA(cudaMemcpyAsync(src.ensure(rows.size()), rows.data(), rows.size() * sizeof(float), cudaMemcpyHostToDevice, s));
        stage.upload(dst.ensure(rows.size()), src.get(), nullptr, kRows, kRow * sizeof(float), s);
        CHECK(fake::in_flight(src.get(), 1));   // (no host code has touched it)
        stage.download(out.ensure(rows.size()), dst.get(), rows.size() * sizeof(float), s);
        for (size_t i = 0; i < rows.size(); ++i) CHECK(out.get()[i] == rows[i]);
        const std::vector<size_t> idx(kRows, 1);
        stage.upload(dst.get(), src.get(), idx.data(), kRows, kRow * sizeof(float), s);
        stage.download(out.get(), dst.get(), rows.size() * sizeof(float), s);
        for (size_t i = 0; i < rows.size(); ++i) CHECK(out.get()[i] == 4.0f);
    }
    release_stream(s, 0);
}

} // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "exception_behind_a_copy") exception_behind_a_copy(false);
    else if (what == "exception_behind_a_pinned_copy") exception_behind_a_copy(true);
    else if (what == "rows_arrive") rows_arrive();
    else if (what == "pieces_of_any_length") pieces_of_any_length();
    else if (what == "device_memory") device_memory();
    else return 2;
    std::puts("OK");
    return 0;
}
