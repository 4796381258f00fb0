// Exact assignment by a proven fp16 filter and an fp32 decision (exact_assign.cu).
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"
#include "engine_buffers.h"

namespace skmb {

// How to assign n rows to k centroids exactly: `direct` (launch_direct_assign) for few pairs, `filter` (ExactAssign) for many
// rows and centroids, `blocks` (launch_assign_full: three products per pair) for many rows and few centroids, or when the
// tensor cores are switched off.  By estimates of what each takes, from timings of 4096 .. 100 000 rows, 32 .. 4000
// centroids, 32 .. 768 dimensions on a B200; they need to be right only to the factor that separates the ways.
enum class AssignRoute { direct, filter, blocks };
AssignRoute assign_route(size_t n, size_t k, size_t d);

// launch_direct_assign and its scratch.
class DirectAssign {
  public:
    void run(const float* x, const float* y, size_t n, size_t k, size_t d, float* norms_x, float* norms_y, uint32_t* knn, float* dist, cudaStream_t stream);

  private:
    DeviceBuffer<unsigned long long> keys_;
    DeviceBuffer<uint32_t> counters_, arrived_;
};

// Up to 256 rows and the centroids they are assigned to: rows [row0, row0 + rows) of x, rows [y0, y0 + k) of y.
struct AssignTile {
    uint32_t row0, rows, y0, k;
};

// Nearest centroid of every row, in three steps:
//   1. rows and centroids, centred on the mean of some centroids, are rounded to fp16 (scaled by powers of two) together
//      with the norms of what the rounding took away;
//   2. one fp16 tensor-core product per pair gives every distance within a bound that follows from those norms
//      (Cauchy-Schwarz) and the accumulator's truncation; the centroids of a row whose distance could be the smallest
//      are kept, up to four;
//   3. their distances are computed in fp32 from the original rows, by the formula and the tie rules of refine_top2_kernel.
// A row with more than four such centroids is listed and goes through the three-product kernel (launch_assign_full) with
// the others of its kind: settle() says how many there are, the caller provides the rows again.
class ExactAssign {
  public:
    // Once per set of centroids and batch of rows: fp16 centroids, their squared norms (also to norms_y, as
    // launch_row_sqnorms gives them), an empty list, and memory for up to piece_rows rows at a time.  False: there is not enough
    // of it (the fp16 rows take a gigabyte at most), nothing has been done and none is held.
    bool begin(const float* y, size_t k, size_t d, size_t batch_rows, size_t piece_rows, float* norms_y, cudaStream_t stream);
    // Rows [first, first + n) of the batch, one piece after the other; their squared norms go to norms_x (as launch_row_sqnorms gives them).
    void rows(const float* x, size_t first, size_t n, float* norms_x, uint32_t* out_knn, float* out_dist, cudaStream_t stream);
    // Number of listed rows (waits for the stream); their indices inside the batch are in listed().
    size_t settle(cudaStream_t stream);
    const uint32_t* listed() const { return listed_.get(); }
    // Whether most of the first `done` rows are listed (waits for the stream): the rest had better not go through the filter.
    bool in_vain(size_t done, cudaStream_t stream) { return 2 * settle(stream) > done; }
    // out_knn / out_dist (may be null) of the rows listed()[at .. at + count), given those rows.
    void finish(const float* x_listed, size_t at, size_t count, uint32_t* out_knn, float* out_dist, cudaStream_t stream);
    // Both, for a batch that is still on the device.
    size_t settle_on_device(const float* x_batch, uint32_t* out_knn, float* out_dist, cudaStream_t stream);

    // Many problems at once: every row tile has centroids of its own.  begin_groups converts the rows (which may then be
    // assigned several times; y gives the mean), assign_groups assigns the rows of the tiles, which are sorted by row; the
    // other rows' answers stay as they are.  Indices count from the beginning of y.
    void begin_groups(const float* x, size_t n, size_t d, const float* y, size_t k, float* norms_x, cudaStream_t stream);
    void assign_groups(const float* x, size_t n, const float* y, size_t k, const AssignTile* tiles, size_t n_tiles, const float* norms_x, float* norms_y, uint32_t* out_knn,
                       float* out_dist, cudaStream_t stream);
    void give_back();   // the memory for rows and centroids

  private:
    void centroids(const float* y, size_t k, float* norms_y, bool with_mean, cudaStream_t stream);
    void convert(const float* x, size_t n, size_t before, float* norms_x, cudaStream_t stream);
    void search(const float* x, size_t first, size_t n, const AssignTile* tiles, size_t n_tiles, const float* norms_x, uint32_t* out_knn, float* out_dist, cudaStream_t stream);
    size_t rows_at_once(size_t n) const;
    const float* y_ = nullptr;
    const float* norms_y_ = nullptr;
    size_t k_ = 0, d_ = 0, dp_ = 0, kp_ = 0;
    DeviceBuffer<__half> xh_, yh_;
    DeviceBuffer<float> mean_, centred_norms_;
    DeviceBuffer<uint32_t> stats_;
    DeviceBuffer<float4> row_info_;
    DeviceBuffer<uint4> cand_;
    DeviceBuffer<uint32_t> listed_, n_listed_;
    PinnedBuffer<uint32_t> n_listed_host_;
    // of the listed rows
    DeviceBuffer<float> l_rows_, l_norms_, l_dist_, l_split_;
    DirectAssign direct_;
    DeviceBuffer<uint32_t> l_knn_;
    DeviceBuffer<uint2> l_top2_;
};

} // namespace skmb
