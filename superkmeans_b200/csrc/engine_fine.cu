// Fine clustering of many mesoclusters at once (hierarchical_superkmeans.h:301-425).
//
// Every mesocluster is a k-means problem of its own: a few thousand rows, about sqrt(k) clusters, up to five exact
// iterations.  One after the other they are some twenty launches and three host round trips per iteration (0.27 ms each at
// 6000 x 768, most of it waiting).  Here a run of mesoclusters shares every launch: their rows lie one behind the other, the
// assignment takes row tiles that name their centroids (ExactAssign), the sums run over all clusters, and what is decided on
// the host - splits, early stopping - is decided for all of them between two round trips.  The random streams, the order of
// the operations inside a mesocluster and the numbers the decisions are made from are those of the sequential form.
#include "engine.h"

#include <cmath>
#include <stdexcept>

#include "device_utils.cuh"
#include "kernels_tc.cuh"

namespace skmb {

namespace {

// A mesocluster inside its run: rows [row0, row0 + rows), clusters [y0, y0 + k), split operations [op0, op0 + ops).
struct Group {
    uint32_t row0, rows, y0, k, op0, ops, active, pad;
};

// Means of the active groups' clusters from their sums; the other groups keep last iteration's centroids.
__global__ void __launch_bounds__(256) group_means_kernel(float* __restrict__ c, const float* __restrict__ prev, const uint32_t* __restrict__ counts, const uint32_t* __restrict__ group_of,
                                                          const Group* __restrict__ groups, size_t d) {
    const size_t row = blockIdx.x;
    float* p = c + row * d;
    if (!groups[group_of[row]].active) {
        for (size_t j = threadIdx.x; j < d; j += blockDim.x) p[j] = prev[row * d + j];
        return;
    }
    const uint32_t cnt = counts[row];
    if (cnt == 0) return;
    const float mult = static_cast<float>(1.0 / static_cast<double>(cnt));
    for (size_t j = threadIdx.x; j < d; j += blockDim.x) p[j] = __fmul_rn(p[j], mult);
}

// Split operations of a group in list order, a thread per dimension (see apply_split_ops_kernel).
__global__ void group_split_kernel(float* __restrict__ c, size_t d, const SplitOpDev* __restrict__ ops, const Group* __restrict__ groups) {
    const Group g = groups[blockIdx.y];
    const size_t j = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= d) return;
    for (uint32_t o = g.op0; o < g.op0 + g.ops; ++o) apply_split_op(c, d, j, ops[o]);
}

// normalize_rows_kernel for the active groups.
__global__ void __launch_bounds__(256) group_normalize_kernel(float* __restrict__ c, size_t k, size_t d, const uint32_t* __restrict__ group_of, const Group* __restrict__ groups) {
    const size_t row = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (row >= k || !groups[group_of[row]].active) return;
    normalize_row(c + row * d, d, threadIdx.x & 31);
}

// out[g] = sum of the distances of the group's rows
__global__ void __launch_bounds__(256) group_cost_kernel(const float* __restrict__ dist, const Group* __restrict__ groups, double* __restrict__ out) {
    __shared__ double part[8];
    const Group g = groups[blockIdx.x];
    double s = 0.0;
    for (uint32_t i = threadIdx.x; i < g.rows; i += 256) s += static_cast<double>(dist[g.row0 + i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += part[w];
        out[blockIdx.x] = t;
    }
}

// out[g][slice] = sum of the squared differences of every kShiftSlices-th of the group's centroids (a block alone for all of them waits for
// its loads: 50 groups of 50 x 768: 55 us)
constexpr int kShiftSlices = 8;
__global__ void __launch_bounds__(256) group_shift_kernel(const float* __restrict__ a, const float* __restrict__ b, size_t d, const Group* __restrict__ groups, double* __restrict__ out) {
    __shared__ double part[8];
    const Group g = groups[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double total = 0.0;
    for (uint32_t c = blockIdx.y * 8 + warp; c < g.k; c += 8 * kShiftSlices) {
        const float* pa = a + static_cast<size_t>(g.y0 + c) * d;
        const float* pb = b + static_cast<size_t>(g.y0 + c) * d;
        float s = 0.f;
#pragma unroll 8   // (bound by the latency of its loads)
        for (size_t j = lane; j < d; j += 32) {
            const float t = __ldg(pa + j) - __ldg(pb + j);
            s = fmaf(t, t, s);
        }
        total += static_cast<double>(warp_sum(s));
    }
    if (lane == 0) part[warp] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += part[w];
        out[blockIdx.x * kShiftSlices + blockIdx.y] = t;
    }
}

} // namespace

// Mesoclusters [first, last) of the partition (members meso_indices_dev_[offsets[m] ..), rows[m] of them, fine[m] clusters,
// Forgy rows forgy[m]): final assignments and centroids as the sequential form leaves them.  fine_offset: clusters of the
// mesoclusters before `first`.
void Engine::train_fine_run(size_t first, size_t last, const std::vector<size_t>& offsets, const std::vector<size_t>& rows, const std::vector<size_t>& fine,
                            const std::vector<std::vector<size_t>>& forgy, size_t fine_offset) {
    const size_t n_groups = last - first;
    std::vector<Group> groups(n_groups);
    std::vector<uint32_t> group_of;
    std::vector<uint64_t> seeds;
    size_t n = 0, k = 0;
    for (size_t q = 0; q < n_groups; ++q) {
        const size_t m = first + q;
        groups[q] = {static_cast<uint32_t>(n), static_cast<uint32_t>(rows[m]), static_cast<uint32_t>(k), static_cast<uint32_t>(fine[m]), 0u, 0u, fine[m] ? 1u : 0u, 0u};
        for (size_t i : forgy[m]) seeds.push_back(n + i);
        group_of.insert(group_of.end(), fine[m], static_cast<uint32_t>(q));
        n += rows[m];
        k += fine[m];
    }
    if (k == 0) return;
    const uint64_t* idx = meso_indices_dev_.get() + offsets[first];
    float* x = meso_buffer_.ensure(n * d_);
    float* norms = meso_norms_.ensure(n);
    launch_gather_rows(x_rot_.get(), idx, x, n, d_, stream_);   // CompactMesoclusterToBuffer (:685-704), all of the run
    stage_.upload(init_idx_dev_.ensure(k), seeds.data(), nullptr, k, sizeof(uint64_t), stream_);
    launch_gather_rows(x, init_idx_dev_.get(), c_prev_.get(), k, d_, stream_);
    DeviceBuffer<uint32_t> group_of_dev;
    DeviceBuffer<AssignTile> tiles_dev;
    DeviceBuffer<Group> groups_dev;
    DeviceBuffer<double> sums_dev;
    PinnedBuffer<double> sums;
    stage_.upload(group_of_dev.ensure(k), group_of.data(), nullptr, k, sizeof(uint32_t), stream_);
    groups_dev.ensure(n_groups);
    sums_dev.ensure(n_groups);
    sums.ensure(n_groups);
    // per iteration and group, in slices
    const size_t shift_words = n_groups * kShiftSlices;
    DeviceBuffer<double> all_shifts;
    PinnedBuffer<double> shifts;
    all_shifts.ensure(shift_words * cfg_.iters_fineclustering);
    shifts.ensure(shift_words * cfg_.iters_fineclustering);
    auto shifts_dev = [&](size_t iter) { return all_shifts.get() + shift_words * iter; };
    auto shift_of = [&](size_t iter, size_t q) {
        double t = 0.0;
        for (int w = 0; w < kShiftSlices; ++w) t += shifts.get()[shift_words * iter + q * kShiftSlices + w];
        return static_cast<float>(t);
    };
    exact_.begin_groups(x, n, d_, c_prev_.get(), k, norms, stream_);

    struct State {
        float cost = 0.f, prev_cost = 0.f, shift = 0.f;
        size_t n_split = 0;
        double cost_f64 = 0.0;
        std::vector<uint32_t> sizes;   // after the last split
        std::vector<skm_iter_stats> stats;
    };
    std::vector<State> state(n_groups);
    std::vector<AssignTile> tiles;
    std::vector<SplitOp> ops;
    std::vector<std::vector<SplitOp>> ops_of(n_groups);
    bool tiles_current = false;
    for (size_t iter = 0; iter < cfg_.iters_fineclustering; ++iter) {
        if (!tiles_current) {
            tiles.clear();
            for (const Group& g : groups)
                if (g.active)
                    for (uint32_t r = 0; r < g.rows; r += 256) tiles.push_back({g.row0 + r, std::min(256u, g.rows - r), g.y0, g.k});
            if (tiles.empty()) break;
            stage_.upload(tiles_dev.ensure(tiles.size()), tiles.data(), nullptr, tiles.size(), sizeof(AssignTile), stream_);
            stage_.upload(groups_dev.get(), groups.data(), nullptr, n_groups, sizeof(Group), stream_);
            tiles_current = true;
        }
        if (iter > 0) c_cur_.swap(c_prev_);
        {
            PhaseScope ps(*this, PH_ASSIGN_FULL);
            exact_.assign_groups(x, n, c_prev_.get(), k, tiles_dev.get(), tiles.size(), norms, centroid_norms_.get(), assignments_.get(), distances_.get(), stream_);
        }
        {
            PhaseScope ps(*this, PH_UPDATE);
            launch_update(x, assignments_.get(), n, k, d_, ws_, c_cur_.get(), counts(), nullptr, stream_);
            group_cost_kernel<<<static_cast<unsigned>(n_groups), 256, 0, stream_>>>(distances_.get(), groups_dev.get(), sums_dev.get());
            SKM_LAUNCH_CHECK();
        }
        SKM_CUDA(cudaMemcpyAsync(counts_host(), counts(), sizeof(uint32_t) * k, cudaMemcpyDeviceToHost, stream_));
        SKM_CUDA(cudaMemcpyAsync(sums.get(), sums_dev.get(), sizeof(double) * n_groups, cudaMemcpyDeviceToHost, stream_));
        {
            PhaseScope ps(*this, PH_CONSOLIDATE);
            group_means_kernel<<<static_cast<unsigned>(k), 256, 0, stream_>>>(c_cur_.get(), c_prev_.get(), counts(), group_of_dev.get(), groups_dev.get(), d_);
            SKM_LAUNCH_CHECK();
        }
        tell_error();
        sync();
        check_told_error();
        // ConsolidateCentroids of every group (superkmeans.h:936-968)
        std::vector<const char*> failure(n_groups, nullptr);
#pragma omp parallel for schedule(dynamic) if (n_groups > 8)
        for (size_t q = 0; q < n_groups; ++q) {
            ops_of[q].clear();
            Group& g = groups[q];
            if (!g.active) continue;
            std::vector<uint32_t> s(counts_host() + g.y0, counts_host() + g.y0 + g.k);
            if (!split_can_terminate(s, g.rows, g.k)) {
                failure[q] = "cannot repopulate empty clusters: no cluster holds more than one point";
                continue;
            }
            state[q].n_split = split_clusters_hierarchical(s, g.rows, g.k, cfg_.seed, ops_of[q]);
            state[q].sizes.swap(s);
        }
        ops.clear();
        for (size_t q = 0; q < n_groups; ++q) {
            if (failure[q]) throw std::runtime_error(failure[q]);
            Group& g = groups[q];
            g.op0 = static_cast<uint32_t>(ops.size());
            g.ops = static_cast<uint32_t>(ops_of[q].size());
            for (SplitOp op : ops_of[q]) {
                op.dst += g.y0;
                op.src += g.y0;
                ops.push_back(op);
            }
        }
        {
            PhaseScope ps(*this, PH_CONSOLIDATE);
            if (!ops.empty()) {
                static_assert(sizeof(SplitOp) == sizeof(SplitOpDev), "layout");
                stage_.upload(split_ops_dev_.ensure(ops.size()), ops.data(), nullptr, ops.size(), sizeof(SplitOp), stream_);
                stage_.upload(groups_dev.get(), groups.data(), nullptr, n_groups, sizeof(Group), stream_);
                group_split_kernel<<<dim3(static_cast<unsigned>((d_ + 127) / 128), static_cast<unsigned>(n_groups)), 128, 0, stream_>>>(c_cur_.get(), d_, split_ops_dev_.get(),
                                                                                                                                        groups_dev.get());
                SKM_LAUNCH_CHECK();
            }
            if (cfg_.angular) {
                group_normalize_kernel<<<static_cast<unsigned>((k + 7) / 8), 256, 0, stream_>>>(c_cur_.get(), k, d_, group_of_dev.get(), groups_dev.get());
                SKM_LAUNCH_CHECK();
            }
        }
        {
            PhaseScope ps(*this, PH_SHIFT);
            group_shift_kernel<<<dim3(static_cast<unsigned>(n_groups), kShiftSlices), 256, 0, stream_>>>(c_cur_.get(), c_prev_.get(), d_, groups_dev.get(), shifts_dev(iter));
            SKM_LAUNCH_CHECK();
        }
        // only early stopping asks for the shift before the end
        if (cfg_.early_termination) {
            SKM_CUDA(cudaMemcpyAsync(shifts.get() + shift_words * iter, shifts_dev(iter), sizeof(double) * shift_words, cudaMemcpyDeviceToHost, stream_));
            sync();
        }
        for (size_t q = 0; q < n_groups; ++q) {
            Group& g = groups[q];
            if (!g.active) continue;
            State& st = state[q];
            st.prev_cost = st.cost;
            st.cost = static_cast<float>(sums.get()[q]);
            if (cfg_.early_termination) st.shift = shift_of(iter, q);
            st.cost_f64 = sums.get()[q];
            skm_iter_stats s{};
            s.iteration = iter + 1;
            s.objective = st.cost;
            s.shift = st.shift;
            s.split = st.n_split;
            s.recall = 0.0f;
            s.is_gemm_only = 1;
            s.not_pruned_pct = -1.0f;
            s.partial_d = 0u;
            st.stats.push_back(s);
            if (cfg_.early_termination && should_stop_early(st.shift, st.cost, st.prev_cost, cfg_.tol, iter)) {
                g.active = 0;
                tiles_current = false;
            }
        }
    }
    if (!cfg_.early_termination) {
        SKM_CUDA(cudaMemcpyAsync(shifts.get(), shifts_dev(0), sizeof(double) * shift_words * cfg_.iters_fineclustering, cudaMemcpyDeviceToHost, stream_));
        sync();
        for (size_t q = 0; q < n_groups; ++q) {
            for (skm_iter_stats& s : state[q].stats) state[q].shift = s.shift = shift_of(s.iteration - 1, q);
        }
    }
    for (size_t q = 0; q < n_groups; ++q) {
        for (const skm_iter_stats& s : state[q].stats) {
            stats_fine_.push_back(s);
            if (cfg_.verbose) print_iteration(s, partial_d_);
        }
        if (!state[q].stats.empty()) {
            cost_ = state[q].cost;
            prev_cost_ = state[q].prev_cost;
            shift_ = state[q].shift;
            n_split_ = state[q].n_split;
            last_cost_f64_ = state[q].cost_f64;
            sizes_host_ = state[q].sizes;
        }
    }
    // GetTrueAssignmentsFromIndirectionBuffer (:763-779) and the centroid copy (:416-423)
    launch_scatter_u32_offset(assignments_.get(), idx, final_assignments_.get(), n, static_cast<uint32_t>(fine_offset), stream_);
    SKM_CUDA(cudaMemcpyAsync(final_centroids_.get() + fine_offset * d_, c_cur_.get(), sizeof(float) * k * d_, cudaMemcpyDeviceToDevice, stream_));
}

} // namespace skmb
