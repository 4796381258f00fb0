// k nearest rows of Y for every row of Q, and the recall figure built on it.
//
// Used only by training with query vectors (SuperKMeans::GetGTAssignmentsAndDistances / ComputeRecall,
// superkmeans.h:1010-1087, on top of BatchComputer::FindKNearestNeighbors, batch_computers.h:191-274): once
// per Train for the ground truth (the objective_k nearest training points of every query) and once per
// iteration for the centroids a search would visit (the nearest ann_explore_fraction of the centroids).
//
// Y is walked in slabs of kSlab rows.  For a slab the dot products Q * Y_slab^T go to scratch with the
// fp32 tile GEMM; topk_merge_kernel (one CTA per query) turns them into distances
// ||q||^2 + ||y||^2 - 2 q.y, keeps those below the query's current k-th best in a shared-memory buffer
// and, whenever the buffer fills, sorts it (bitonic, 64-bit keys {ordered distance, index}) and keeps the
// best k.  Equal distances are ordered by index, as std::partial_sort on (distance, index) pairs does.
#include <cfloat>
#include <stdexcept>
#include <string>

#include "common.cuh"
#include "device_utils.cuh"

namespace skmb {

namespace {

constexpr int kTopkThreads = 256;
constexpr int kTopkBuf = 2048;   // keys held in shared memory; k <= kTopkMaxK leaves room for new candidates
constexpr size_t kSlab = 16384;

__device__ __forceinline__ unsigned long long make_key(float dist, uint32_t idx) {
    return (static_cast<unsigned long long>(float_to_ordered(dist)) << 32) | static_cast<unsigned long long>(idx);
}

// Ascending bitonic sort of buf[0 .. n) (n a power of two) by all threads of the CTA.
__device__ void bitonic_sort(unsigned long long* buf, int n) {
    for (int size = 2; size <= n; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (int t = threadIdx.x; t < n / 2; t += kTopkThreads) {
                const int lo = 2 * t - (t & (stride - 1));
                const int hi = lo + stride;
                const bool up = ((lo & size) == 0);
                const unsigned long long a = buf[lo], b = buf[hi];
                if ((a > b) == up) {
                    buf[lo] = b;
                    buf[hi] = a;
                }
            }
        }
    }
    __syncthreads();
}

// Where the lists of a pass go: the state that the next slab goes on with, or (out_idx given) the answers: indices and distances clamped at
// zero as FindKNearestNeighbors stores them; empty slots: index 0xFFFFFFFF, distance FLT_MAX.
struct TopkLists {
    unsigned long long* state;   // n_q x k keys, ascending, ~0 = empty
    uint32_t* out_idx;
    float* out_dist;
    __device__ __forceinline__ void put(size_t at, unsigned long long key) const {
        if (!out_idx) {
            state[at] = key;
            return;
        }
        const bool empty = key == ~0ull;
        out_idx[at] = empty ? 0xFFFFFFFFu : static_cast<uint32_t>(key & 0xFFFFFFFFull);
        if (out_dist) out_dist[at] = empty ? FLT_MAX : fmaxf(0.0f, ordered_to_float(static_cast<uint32_t>(key >> 32)));
    }
};

// dots: n_q x slab_ld dot products of this slab (columns [0, slab_n) valid, global indices col0 + c).  The first slab finds no state.
__global__ void __launch_bounds__(kTopkThreads) topk_merge_kernel(const float* __restrict__ dots, size_t slab_ld, size_t slab_n, size_t col0, const float* __restrict__ norms_q,
                                                                  const float* __restrict__ norms_y, uint32_t k, TopkLists lists) {
    __shared__ unsigned long long buf[kTopkBuf];
    __shared__ uint32_t count;
    __shared__ unsigned long long tau;
    const size_t q = blockIdx.x;
    const float nq = norms_q[q];
    const unsigned long long* st = lists.state + q * k;
    const uint32_t carried = col0 == 0 ? 0u : k;
    uint32_t held = carried;   // keys in the buffer, which every thread counts for itself: `count` may have moved on when it is read
    if (slab_n > 2 * kTopkThreads || carried) {
        for (int i = threadIdx.x; i < kTopkBuf; i += kTopkThreads) buf[i] = i < static_cast<int>(carried) ? st[i] : ~0ull;
    } else {
        for (int i = threadIdx.x; i < 2 * kTopkThreads; i += kTopkThreads) buf[i] = ~0ull;
    }
    if (threadIdx.x == 0) {
        count = carried;
        tau = carried ? st[k - 1] : ~0ull;
    }
    __syncthreads();
    const float* __restrict__ row = dots + q * slab_ld;
    for (size_t c0 = 0; c0 < slab_n; c0 += kTopkThreads) {
        const size_t c = c0 + threadIdx.x;
        const float dist = c < slab_n ? fmaf(-2.0f, row[c], nq) + norms_y[col0 + c] : 0.f;
        const unsigned long long key = make_key(dist, static_cast<uint32_t>(col0 + c));
        // (a place per warp, then per key)
        const bool kept = c < slab_n && key < tau;
        const uint32_t all = __ballot_sync(0xffffffffu, kept);
        if (all != 0) {
            const int lane = threadIdx.x & 31;
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&count, static_cast<uint32_t>(__popc(all)));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(all & ((1u << lane) - 1u));
            if (kept) buf[at] = key;   // below k + kTopkThreads * rounds, bounded by the flush below
        }
        held += static_cast<uint32_t>(__syncthreads_count(kept));
        // one more round adds at most kTopkThreads keys: flush while that still fits
        if (held + kTopkThreads > kTopkBuf) {
            bitonic_sort(buf, kTopkBuf);
            for (int i = k + threadIdx.x; i < kTopkBuf; i += kTopkThreads) buf[i] = ~0ull;
            if (threadIdx.x == 0) {
                count = k;
                tau = buf[k - 1];
            }
            held = k;
            __syncthreads();
        }
    }
    // what lies behind the keys held is empty: among 300 centroids a sort of 512 takes half the time of one of the whole buffer (9 us for 200
    // lists; places counted key by key: 12)
    int sorted = 2;
    while (sorted < static_cast<int>(held)) sorted <<= 1;
    bitonic_sort(buf, sorted);
    for (int i = threadIdx.x; i < static_cast<int>(k); i += kTopkThreads) lists.put(q * k + i, i < sorted ? buf[i] : ~0ull);
}

// found[q] = number of the query's ground-truth points whose current cluster is among the clusters the query
// would visit (superkmeans.h:1063-1086).
__global__ void __launch_bounds__(128) recall_count_kernel(const uint32_t* __restrict__ gt, uint32_t objective_k, const uint32_t* __restrict__ promising, uint32_t n_explore,
                                                           const uint32_t* __restrict__ assignments, size_t n_assignments, uint32_t* __restrict__ found) {
    __shared__ uint32_t total;
    const size_t q = blockIdx.x;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    uint32_t mine = 0;
    for (uint32_t j = threadIdx.x; j < objective_k; j += blockDim.x) {
        const uint32_t g = gt[q * objective_k + j];
        if (g >= n_assignments) continue;
        const uint32_t a = assignments[g];
        bool hit = false;
        for (uint32_t t = 0; t < n_explore && !hit; ++t) hit = promising[q * n_explore + t] == a;
        mine += hit ? 1u : 0u;
    }
    if (mine) atomicAdd(&total, mine);
    __syncthreads();
    if (threadIdx.x == 0) found[q] = total;
}

} // namespace

size_t topk_scratch_floats(size_t n_q) { return n_q * kSlab; }
size_t topk_max_k() { return kTopkBuf - 2 * kTopkThreads; }

void launch_topk_nn(const float* q, const float* y, size_t n_q, size_t n_y, size_t d, const float* norms_q, const float* norms_y, uint32_t k, uint32_t* out_idx,
                    float* out_dist, float* dots_scratch, unsigned long long* state, cudaStream_t stream) {
    if (n_q == 0 || k == 0) return;
    if (k > topk_max_k()) throw std::runtime_error("nearest-neighbour lists longer than " + std::to_string(topk_max_k()) + " entries are not supported");
    size_t c0 = 0;
    do {
        const size_t cn = std::min(kSlab, n_y - c0);
        launch_gemm_nt(q, d, y + c0 * d, d, dots_scratch, kSlab, n_q, cn, d, stream);
        const bool last = cn == n_y - c0;
        topk_merge_kernel<<<static_cast<unsigned>(n_q), kTopkThreads, 0, stream>>>(dots_scratch, kSlab, cn, c0, norms_q, norms_y, k,
                                                                                  TopkLists{state, last ? out_idx : nullptr, last ? out_dist : nullptr});
        SKM_LAUNCH_CHECK();
        c0 += kSlab;
    } while (c0 < n_y);
}

void launch_recall_count(const uint32_t* gt, uint32_t objective_k, const uint32_t* promising, uint32_t n_explore, const uint32_t* assignments, size_t n_assignments,
                         size_t n_q, uint32_t* found, cudaStream_t stream) {
    if (n_q == 0) return;
    recall_count_kernel<<<static_cast<unsigned>(n_q), 128, 0, stream>>>(gt, objective_k, promising, n_explore, assignments, n_assignments, found);
    SKM_LAUNCH_CHECK();
}

} // namespace skmb
