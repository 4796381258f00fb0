// Host-side pieces of the k-means hot path that must reproduce the reference bit for bit because
// they consume the random-number stream or take integer decisions: Forgy initialisation, cluster
// splitting, d' tuning, early stopping, dimension split, ADSampling ratios, fine-cluster
// allocation and the random orthogonal matrix.  Pure C++17, no CUDA: the same header is exercised
// by CPU-only tests through the skm_host_* entry points.
#pragma once

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <memory>
#include <numeric>
#include <random>
#include <thread>
#include <vector>

namespace skmb {

// Constants of the reference (include/superkmeans/common.h:89-115).
constexpr float kProportionHorizontalDim = 0.75f;
constexpr size_t kHDimSize = 64;
constexpr uint32_t kMinPartialD = 16;
constexpr size_t kDimensionThresholdForPruning = 128;
constexpr size_t kNClustersThresholdForPruning = 256;
constexpr size_t kXBatchSize = 4096;
constexpr size_t kYBatchSize = 1024;
constexpr size_t kVectorChunkSize = kYBatchSize;
constexpr float kCentroidPerturbationEps = 1.0f / 1024.0f;
constexpr float kPrunerInitialThreshold = 1.5f;
constexpr float kHierarchicalPrunerInitialThreshold = 1.1f;

struct DimensionSplit {
    size_t horizontal_d = 0;
    size_t vertical_d = 0;
};

// PDXLayout::GetDimensionSplit (include/superkmeans/pdx/layout.h:115-140): 75 % of the dimensions
// (25 % when d <= 256) go to the horizontal part, rounded to a multiple of 64; never all of them;
// none when d <= 64.
inline DimensionSplit dimension_split(size_t d) {
    float proportion = kProportionHorizontalDim;
    if (d <= 256) proportion = 0.25f;
    size_t horizontal_d = static_cast<size_t>(static_cast<double>(d) * proportion);
    size_t vertical_d = d - horizontal_d;
    if (horizontal_d % kHDimSize > 0) {
        horizontal_d = static_cast<size_t>(std::lround(
                           static_cast<double>(horizontal_d) / static_cast<double>(kHDimSize))) *
                       kHDimSize;
        vertical_d = d - horizontal_d;
    }
    if (!vertical_d) {
        horizontal_d = kHDimSize;
        vertical_d = d - horizontal_d;
    }
    if (d <= kHDimSize) {
        horizontal_d = 0;
        vertical_d = d;
    }
    return {horizontal_d, vertical_d};
}

// ADSamplingPruner::GetRatio / InitializeRatios (include/superkmeans/pdx/adsampling.h:93-99,
// :315-327): ratio[v] = v/d * (1 + eps0/sqrt(v))^2 in double, rounded to float; ratio[0] =
// ratio[d] = 1.
inline std::vector<float> make_ratios(size_t d, float epsilon0) {
    std::vector<float> r(d + 1);
    for (size_t v = 0; v <= d; ++v) {
        if (v == 0 || v == d) {
            r[v] = 1.0f;
            continue;
        }
        const double dv = static_cast<double>(v);
        const double t = 1.0 + epsilon0 / std::sqrt(dv);
        r[v] = static_cast<float>(dv / static_cast<double>(d) * t * t);
    }
    return r;
}

// Initial d' (include/superkmeans/superkmeans.h:211-215): half of vertical_d, at least 16, at most
// vertical_d.
inline uint32_t initial_partial_d(uint32_t vertical_d, uint32_t divisor = 2) {
    uint32_t p = std::max<uint32_t>(kMinPartialD, vertical_d / divisor);
    if (p > vertical_d) p = vertical_d;
    return p;
}

// SuperKMeans::GetNVectorsToSample (superkmeans.h:1269-1277) and the hierarchical override
// (hierarchical_superkmeans.h:559-567).
inline size_t n_vectors_to_sample(size_t n, size_t k, float sampling_fraction, uint32_t max_points_per_cluster, bool hierarchical) {
    if (hierarchical) {
        if (sampling_fraction == 1.0) return n;
        return static_cast<size_t>(std::floor(static_cast<double>(n) * sampling_fraction));
    }
    if (sampling_fraction == 1.0) return n;
    const size_t by_clusters = k * max_points_per_cluster;
    const size_t by_n = static_cast<size_t>(std::floor(static_cast<float>(n) * sampling_fraction));
    return std::min(by_n, by_clusters);
}

// The outputs of std::mt19937(seed) (Matsumoto and Nishimura's generator), a block of 624 at a time in loops without
// dependencies from one element to the next, which the compiler vectorises: 0.55 us a block with the vectors every x86-64 has
// (std::mt19937 takes 2.5), 0.3 us with AVX2.
class Mt19937Blocks {
  public:
    static constexpr size_t N = 624;
    explicit Mt19937Blocks(uint32_t seed) {
        x_[0] = seed;
        for (size_t i = 1; i < N; ++i) x_[i] = 1812433253u * (x_[i - 1] ^ (x_[i - 1] >> 30)) + static_cast<uint32_t>(i);
    }
    // the next N outputs
    void next(uint32_t* out) {
#if defined(__x86_64__)
        static const bool avx2 = __builtin_cpu_supports("avx2");
        if (avx2) return next_avx2(x_, out);
#endif
        step(x_, out);
    }

  private:
    static inline __attribute__((always_inline)) uint32_t twist(uint32_t hi, uint32_t lo) {
        const uint32_t v = (hi & 0x80000000u) | (lo & 0x7FFFFFFFu);
        return (v >> 1) ^ ((0u - (v & 1u)) & 0x9908B0DFu);
    }
    static inline __attribute__((always_inline)) void step(uint32_t* x, uint32_t* out) {
        constexpr size_t M = 397;
        uint32_t y[N];
        for (size_t i = 0; i < N - M; ++i) y[i] = x[i + M] ^ twist(x[i], x[i + 1]);
        for (size_t i = N - M; i < 2 * (N - M); ++i) y[i] = y[i - (N - M)] ^ twist(x[i], x[i + 1]);
        for (size_t i = 2 * (N - M); i < N - 1; ++i) y[i] = y[i - (N - M)] ^ twist(x[i], x[i + 1]);
        y[N - 1] = y[M - 1] ^ twist(x[N - 1], y[0]);
        for (size_t i = 0; i < N; ++i) {
            uint32_t v = y[i];
            x[i] = v;
            v ^= v >> 11;
            v ^= (v << 7) & 0x9D2C5680u;
            v ^= (v << 15) & 0xEFC60000u;
            out[i] = v ^ (v >> 18);
        }
    }
#if defined(__x86_64__)
    static __attribute__((target("avx2"))) void next_avx2(uint32_t* x, uint32_t* out) { step(x, out); }
#endif
    uint32_t x_[N];
};

// The same outputs one by one: a generator that std::shuffle takes in place of std::mt19937, with the same result.
class Mt19937Stream {
  public:
    using result_type = uint32_t;
    explicit Mt19937Stream(uint32_t seed) : blocks_(seed) {}
    static constexpr result_type min() { return 0; }
    static constexpr result_type max() { return 0xFFFFFFFFu; }
    result_type operator()() {
        if (at_ == Mt19937Blocks::N) {
            blocks_.next(out_);
            at_ = 0;
        }
        return out_[at_++];
    }

  private:
    Mt19937Blocks blocks_;
    uint32_t out_[Mt19937Blocks::N];
    size_t at_ = Mt19937Blocks::N;
};

// The first k entries of std::shuffle applied to [0, n) with std::mt19937(seed); 32-bit entries while they suffice, because
// the shuffle waits for memory.
inline std::vector<size_t> shuffled_indices(size_t n, size_t k, uint32_t seed) {
    Mt19937Stream rng(seed);
    if (n <= 0xFFFFFFFFu) {
        std::vector<uint32_t> idx(n);
        std::iota(idx.begin(), idx.end(), 0u);
        std::shuffle(idx.begin(), idx.end(), rng);
        return std::vector<size_t>(idx.begin(), idx.begin() + static_cast<std::ptrdiff_t>(std::min(k, n)));
    }
    std::vector<size_t> idx(n);
    std::iota(idx.begin(), idx.end(), size_t{0});
    std::shuffle(idx.begin(), idx.end(), rng);
    idx.resize(std::min(k, n));
    return idx;
}

// Forgy initialisation (superkmeans.h:1110-1123).  std::shuffle is library-specific; this engine and the oracle are both
// built with libstdc++.
inline std::vector<size_t> forgy_indices(size_t n_points, size_t k, uint32_t seed) { return shuffled_indices(n_points, k, seed); }

// Sampling permutation (superkmeans.h:1402-1407): a full shuffle of [0, n); the first n_samples
// entries are the sample.
inline std::vector<size_t> sampling_permutation(size_t n, uint32_t seed) { return shuffled_indices(n, n, seed); }

// One row operation produced by the split logic, applied to the row-major centroid matrix in list
// order by a device kernel (each dimension independently).
//   kind 0: row[dst] = row[src]; then even dims: dst *= 1+eps, src *= 1-eps; odd dims the opposite
//           (superkmeans.h:905-920).
//   kind 1: row[dst] = (wc*row[dst] + 1*row[src]) / (wc + 1)   (hierarchical_superkmeans.h:665-673).
struct SplitOp {
    uint32_t dst;
    uint32_t src;
    uint32_t kind;
    float wc;
};

// SuperKMeans::SplitClusters (superkmeans.h:890-928).  `sizes` is updated in place exactly like
// cluster_sizes.  Returns n_split.
inline size_t split_clusters_flat(std::vector<uint32_t>& sizes, size_t n_samples, size_t n_clusters, uint32_t seed, std::vector<SplitOp>& ops) {
    if (std::find(sizes.begin(), sizes.begin() + static_cast<std::ptrdiff_t>(n_clusters), 0u) == sizes.begin() + static_cast<std::ptrdiff_t>(n_clusters)) return 0;
    size_t n_split = 0;
    std::mt19937 rng(seed);
    // The walk below draws ~n_clusters numbers per empty cluster (tens of millions when a thousand clusters are empty), so
    // the acceptance probabilities are tabulated - with the reference's own expression, double division rounded to
    // float - and refreshed for the two clusters a split changes; the draws and comparisons are the reference's.
    const float denom = (float) (n_samples - n_clusters);
    auto prob = [&](size_t c) -> float { return (sizes[c] - 1.0) / denom; };
    std::vector<float> p(n_clusters);
    for (size_t c = 0; c < n_clusters; ++c) p[c] = prob(c);
    std::uniform_real_distribution<float> uniform(0, 1);   // stateless: one object draws what a fresh one per call would
    for (size_t ci = 0; ci < n_clusters; ci++) {
        if (sizes[ci] == 0) {
            size_t cj = 0;
            while (!(uniform(rng) < p[cj])) cj = (cj + 1 == n_clusters) ? 0 : cj + 1;
            ops.push_back({static_cast<uint32_t>(ci), static_cast<uint32_t>(cj), 0u, 0.0f});
            sizes[ci] = sizes[cj] / 2;
            sizes[cj] -= sizes[ci];
            p[ci] = prob(ci);
            p[cj] = prob(cj);
            n_split++;
        }
    }
    return n_split;
}

// HierarchicalSuperKMeans::SplitClusters (hierarchical_superkmeans.h:579-678): the same
// empty-cluster split followed by a pull of every cluster not larger than 25 % of the average
// towards a large cluster picked with probability proportional to its excess size.
inline size_t split_clusters_hierarchical(std::vector<uint32_t>& sizes, size_t n_samples, size_t n_clusters, uint32_t seed, std::vector<SplitOp>& ops) {
    constexpr float kCenterAdjustmentWeight = 7.0f;
    constexpr float kBalancingThreshold = 0.25f;
    size_t n_split = 0;
    std::mt19937 rng(seed);
    const size_t average_size = n_samples / n_clusters;
    const size_t threshold_size = static_cast<size_t>(static_cast<float>(average_size) * kBalancingThreshold);
    {
        // tabulated acceptance probabilities, as in split_clusters_flat (here the reference divides in float)
        const float denom = static_cast<float>(n_samples - n_clusters);
        auto prob = [&](size_t c) -> float { return (sizes[c] - 1.0f) / denom; };
        std::vector<float> p(n_clusters);
        for (size_t c = 0; c < n_clusters; ++c) p[c] = prob(c);
        std::uniform_real_distribution<float> uniform(0, 1);
        for (size_t ci = 0; ci < n_clusters; ci++) {
            if (sizes[ci] == 0) {
                size_t cj = 0;
                while (!(uniform(rng) < p[cj])) cj = (cj + 1 == n_clusters) ? 0 : cj + 1;
                ops.push_back({static_cast<uint32_t>(ci), static_cast<uint32_t>(cj), 0u, 0.0f});
                sizes[ci] = sizes[cj] / 2;
                sizes[cj] -= sizes[ci];
                p[ci] = prob(ci);
                p[cj] = prob(cj);
                n_split++;
            }
        }
    }
    for (size_t ci = 0; ci < n_clusters; ci++) {
        const size_t csize = sizes[ci];
        if (csize == 0 || csize > threshold_size) continue;
        size_t large;
        for (large = 0; true; large = (large + 1) % n_clusters) {
            const size_t large_size = sizes[large];
            if (large_size < average_size) continue;
            float p = static_cast<float>(large_size - average_size + 1) /
                      static_cast<float>(n_samples - average_size * n_clusters + n_clusters);
            float r = std::uniform_real_distribution<float>(0, 1)(rng);
            if (r < p) break;
        }
        const float wc = std::min(static_cast<float>(csize), kCenterAdjustmentWeight);
        ops.push_back({static_cast<uint32_t>(ci), static_cast<uint32_t>(large), 1u, wc});
        n_split++;
    }
    return n_split;
}

// The empty-cluster loop above never ends when no cluster has more than one point (every p <= 0).
// The reference has the same property; the engine reports it instead of spinning.
inline bool split_can_terminate(const std::vector<uint32_t>& sizes, size_t n_samples, size_t n_clusters) {
    bool any_empty = false;
    uint32_t max_size = 0;
    for (size_t c = 0; c < n_clusters; ++c) {
        any_empty |= sizes[c] == 0;
        max_size = std::max(max_size, sizes[c]);
    }
    if (!any_empty) return true;
    return max_size > 1 && n_samples > n_clusters;
}

struct TuneResult {
    float avg_not_pruned_pct;
    uint32_t new_partial_d;
    bool changed;
};

// SuperKMeans::TunePartialD (superkmeans.h:1230-1258).  The reference accumulates the per-point
// counts in a float; the engine passes the exact integer total.
inline TuneResult tune_partial_d(double not_pruned_total, size_t n_samples, size_t n_y, uint32_t partial_d, uint32_t vertical_d, float min_pct, float max_pct, float adjustment) {
    float avg = static_cast<float>(not_pruned_total);
    avg /= static_cast<float>(n_samples * n_y);
    uint32_t nd = partial_d;
    if (avg > max_pct) {
        auto increase = static_cast<uint32_t>(partial_d * adjustment * 2);
        nd = std::min(partial_d + std::max(increase, 1u), vertical_d);
    } else if (avg < min_pct) {
        auto decrease = static_cast<uint32_t>(partial_d * adjustment);
        nd = std::max(partial_d - std::max(decrease, 1u), kMinPartialD);
    }
    return {avg, nd, nd != partial_d};
}

// SuperKMeans::ShouldStopEarly (superkmeans.h:1294-1333).  With tracking_recall, best_recall and
// iters_without_improvement carry the recall history from call to call.
constexpr size_t kRecallConvergencePatience = 2;   // RECALL_CONVERGENCE_PATIENCE (common.h:111)
inline bool should_stop_early(float shift, float cost, float prev_cost, float tol, size_t iter_idx, bool tracking_recall = false, float recall = 0.0f,
                              float recall_tol = 0.0f, float* best_recall = nullptr, size_t* iters_without_improvement = nullptr) {
    if (shift < tol) return true;
    if (iter_idx > 0) {
        const float cost_delta = cost / prev_cost;
        if (cost_delta > 1 - tol) return true;
    }
    if (tracking_recall) {
        const float improvement = recall - *best_recall;
        if (improvement > recall_tol) {
            *best_recall = recall;
            *iters_without_improvement = 0;
        } else {
            ++*iters_without_improvement;
            if (*iters_without_improvement >= kRecallConvergencePatience) return true;
        }
    }
    return false;
}

// HierarchicalSuperKMeans::GetNMesoclusters (hierarchical_superkmeans.h:549-551).
inline size_t n_mesoclusters(size_t n_clusters) {
    return static_cast<size_t>(std::round(std::sqrt(n_clusters)));
}

// HierarchicalSuperKMeans::ArrangeFineClusters (hierarchical_superkmeans.h:718-761).
inline std::vector<size_t> arrange_fine_clusters(size_t n_clusters, size_t n_meso, size_t n_samples, const std::vector<uint32_t>& meso_sizes) {
    std::vector<size_t> out(n_meso);
    size_t clusters_remaining = n_clusters;
    size_t nonempty_remaining = 0;
    for (size_t i = 0; i < n_meso; ++i)
        if (meso_sizes[i] > 0) nonempty_remaining++;
    size_t samples_remaining = n_samples;
    for (size_t i = 0; i < n_meso; ++i) {
        if (i < n_meso - 1) {
            if (meso_sizes[i] == 0) {
                out[i] = 0;
            } else {
                nonempty_remaining--;
                const double proportion = static_cast<double>(clusters_remaining * meso_sizes[i]) /
                                          static_cast<double>(samples_remaining);
                size_t allocated = static_cast<size_t>(std::lround(proportion));
                allocated = std::min(allocated, clusters_remaining - nonempty_remaining);
                out[i] = std::max(allocated, size_t{1});
            }
        } else {
            out[i] = clusters_remaining;
        }
        clusters_remaining -= out[i];
        samples_remaining -= meso_sizes[i];
    }
    return out;
}

// A source of random bits that reads prepared ones.
struct BitsFromArray {
    using result_type = uint32_t;
    const uint32_t* next;
    static constexpr result_type min() { return 0; }
    static constexpr result_type max() { return 0xFFFFFFFFu; }
    result_type operator()() { return *next++; }
};

// The first `count` draws of std::normal_distribution<float>(0, 1) from std::mt19937(seed), made by several threads.
// libstdc++ uses Marsaglia's polar method: it takes the bits two at a time, accepts the pair if the point lies in the unit
// disc, and makes two draws of it.  So any even position of the bits is a place to start: one thread generates them (the
// only serial part, and the bound: 1.3 ms for the 3 million that d = 1536 needs), the others make the draws of one short stretch
// after the other, and whoever uses them can begin before the last is made.  First which pairs are accepted, without
// branches, then the logarithms: 3.5 ns a draw, against 10 in one loop that mispredicts every fifth pair.
class NormalDraws {
  public:
    NormalDraws(size_t count, uint32_t seed) : count_(count), seed_(seed) {
        threads_ = count < (size_t{1} << 15) ? 1u : std::min(8u, std::max(1u, std::thread::hardware_concurrency()));   // (more wait for the generator)
        // a pair is accepted with probability pi / 4; half a percent and 2000 pairs more than needed are a dozen standard deviations
        const double pairs = static_cast<double>((count + 1) / 2) / 0.7853 * 1.005 + 2000.0;
        const size_t blocks = static_cast<size_t>(2.0 * pairs / Mt19937Blocks::N) + 1;
        blocks_ = std::max<size_t>(16, (blocks + kMaxPieces - 1) / kMaxPieces);
        stretches_ = (blocks + blocks_ - 1) / blocks_;   // (kMaxPieces at most)
        made_.reset(new std::atomic<size_t>[stretches_]);
        for (size_t t = 0; t < stretches_; ++t) made_[t].store(kNotYet);
    }
    // Words of scratch for make(), which writes draws into `values` (the same number of floats).
    size_t scratch() const { return stretches_ * blocks_ * Mt19937Blocks::N; }
    // (before piece() is called)
    void values_at(float* values) { values_ = values; }
    void make(uint32_t* bits, float* values) {
        std::atomic<size_t> generated{0}, taken{0};
        auto work = [&] {
            for (size_t t; (t = taken.fetch_add(1)) < stretches_;) {
                while (generated.load(std::memory_order_acquire) <= t) std::this_thread::yield();
                made_[t].store(draw_stretch(bits + t * stretch(), values + t * stretch()), std::memory_order_release);
            }
        };
        // (starting a thread takes longer than a stretch: the first starts the others)
        std::vector<std::thread> pool;
        std::thread starter;
        try {
            if (threads_ > 1) {
                starter = std::thread([&] {
                    try {
                        for (unsigned t = 2; t < threads_; ++t) pool.emplace_back(work);
                    } catch (...) {
                        // (fewer threads then)
                    }
                    work();
                });
            }
        } catch (...) {
        }
        Mt19937Blocks generator(seed_);
        for (size_t t = 0; t < stretches_; ++t) {
            for (size_t b = 0; b < blocks_; ++b) generator.next(bits + t * stretch() + b * Mt19937Blocks::N);
            generated.store(t + 1, std::memory_order_release);
        }
        work();
        if (starter.joinable()) starter.join();
        for (auto& th : pool) th.join();
    }
    unsigned threads() const { return threads_; }
    static constexpr size_t kMaxPieces = 48;
    struct Piece {
        const float* values;
        size_t count;
    };
    // The draws in order, as up to pieces() pieces of `values`; piece(t) waits until make() has come to it.
    size_t pieces() const { return stretches_; }
    size_t stretch() const { return blocks_ * Mt19937Blocks::N; }   // from one piece to the next
    Piece piece(size_t t) const {
        size_t n;
        while ((n = made_[t].load(std::memory_order_acquire)) == kNotYet) std::this_thread::yield();
        return {values_ + t * stretch(), n};
    }

  private:
    static constexpr size_t kNotYet = ~size_t{0};
    size_t draw_stretch(const uint32_t* bits, float* out) const {
        constexpr size_t kBatch = 512;
        float x[kBatch], y[kBatch], r2[kBatch];
        BitsFromArray source{bits};
        size_t n = 0;
        for (size_t left = stretch() / 2; left > 0;) {
            const size_t pairs = std::min(left, kBatch);
            left -= pairs;
            size_t m = 0;
            for (size_t i = 0; i < pairs; ++i) {
                const float a = 2.0f * std::generate_canonical<float, 24>(source) - 1.0f;
                const float b = 2.0f * std::generate_canonical<float, 24>(source) - 1.0f;
                const float r = a * a + b * b;
                x[m] = a;
                y[m] = b;
                r2[m] = r;
                m += static_cast<size_t>((r <= 1.0f) & (r != 0.0f));
            }
            for (size_t i = 0; i < m; ++i) {
                const float mult = std::sqrt(-2.0f * std::log(r2[i]) / r2[i]);
                out[n++] = y[i] * mult;
                out[n++] = x[i] * mult;
            }
        }
        return n;
    }
    size_t count_;
    uint32_t seed_;
    unsigned threads_;
    size_t blocks_;      // generator blocks per stretch
    size_t stretches_;
    std::unique_ptr<std::atomic<size_t>[]> made_;   // draws of a stretch
    float* values_ = nullptr;
};

inline std::vector<float> normal_draws(size_t count, uint32_t seed) {
    NormalDraws draws(count, seed);
    std::unique_ptr<uint32_t[]> bits(new uint32_t[draws.scratch()]);
    std::unique_ptr<float[]> values(new float[draws.scratch()]);
    std::vector<float> out;
    out.reserve(count);
    draws.values_at(values.get());
    draws.make(bits.get(), values.get());
    for (size_t t = 0; t < draws.pieces() && out.size() < count; ++t) {
        const auto p = draws.piece(t);
        out.insert(out.end(), p.values, p.values + std::min(p.count, count - out.size()));
    }
    if (out.size() < count) {   // (practically impossible: too many pairs rejected)
        out.clear();
        std::mt19937 gen(seed);
        std::normal_distribution<float> dist(0.0f, 1.0f);
        for (size_t i = 0; i < count; ++i) out.push_back(dist(gen));
    }
    return out;
}

// The rotation of ADSamplingPruner's DCT branch (adsampling.h:53-73, :169-188) as an explicit matrix: a random sign
// per input dimension, then the orthonormal DCT-II (FFTW's REDFT10, 2 * sum_j x_j cos(pi (j + 1/2) k / d), scaled by
// sqrt(1 / 4d) for k = 0 and sqrt(1 / 2d) otherwise).  M[k][j] = scale_k * 2 cos(pi (j + 1/2) k / d) * sign_j, so that
// X * M^T is what a reference built with FFTW computes for power-of-two d >= 512.
inline std::vector<float> make_dct_rotation_matrix(size_t d, uint32_t seed) {
    std::mt19937 gen(seed);
    std::uniform_int_distribution<int> dist(0, 1);
    std::vector<double> sign(d);
    for (size_t j = 0; j < d; ++j) sign[j] = dist(gen) ? 1.0 : -1.0;
    std::vector<float> m(d * d);
    const double pi = 3.14159265358979323846;
    const double s0 = std::sqrt(1.0 / (4.0 * static_cast<double>(d))), s = std::sqrt(1.0 / (2.0 * static_cast<double>(d)));
    for (size_t k = 0; k < d; ++k) {
        const double scale = (k == 0 ? s0 : s) * 2.0;
        for (size_t j = 0; j < d; ++j) {
            m[k * d + j] = static_cast<float>(scale * std::cos(pi * (static_cast<double>(j) + 0.5) * static_cast<double>(k) / static_cast<double>(d)) * sign[j]);
        }
    }
    return m;
}

// Random orthogonal matrix of the ADSampling rotation (adsampling.h:76-85): a d x d matrix of
// N(0,1) draws from std::mt19937(seed), filled row by row, whose Householder-QR factor Q is the
// rotation.  Sign convention: each reflector maps its column to -sign(x0)*||x|| e1, as in the usual
// LAPACK/Eigen formulation, so Q agrees with the reference's up to floating-point rounding.
// Computed in double, rounded once to float.  Output row-major d x d.  (rotation_matrix.cu computes the same factor on the
// GPU; this one serves the callers without a device and the matrices that one declines.)
inline std::vector<float> make_rotation_matrix(size_t d, uint32_t seed) {
    const std::vector<float> draws = normal_draws(d * d, seed);
    std::vector<double> a(draws.begin(), draws.end());
    std::vector<double> beta(d, 0.0), w(d);
    for (size_t k = 0; k < d; ++k) {
        double norm2 = 0.0;
        for (size_t i = k; i < d; ++i) norm2 += a[i * d + k] * a[i * d + k];
        const double x0 = a[k * d + k];
        const double tail2 = norm2 - x0 * x0;
        if (tail2 <= 0.0 || k == d - 1) continue;
        const double alpha = (x0 >= 0.0) ? -std::sqrt(norm2) : std::sqrt(norm2);
        const double v0 = x0 - alpha;
        for (size_t i = k + 1; i < d; ++i) a[i * d + k] /= v0;
        beta[k] = -v0 / alpha;
        a[k * d + k] = alpha;
        const size_t m = d - k - 1;
        for (size_t j = 0; j < m; ++j) w[j] = a[k * d + k + 1 + j];
        for (size_t i = k + 1; i < d; ++i) {
            const double vi = a[i * d + k];
            const double* row = &a[i * d + k + 1];
            for (size_t j = 0; j < m; ++j) w[j] += vi * row[j];
        }
        const double b = beta[k];
        for (size_t j = 0; j < m; ++j) a[k * d + k + 1 + j] -= b * w[j];
#pragma omp parallel for if (m > 256)
        for (size_t i = k + 1; i < d; ++i) {
            const double vi = b * a[i * d + k];
            double* row = &a[i * d + k + 1];
            for (size_t j = 0; j < m; ++j) row[j] -= vi * w[j];
        }
    }
    std::vector<double> q(d * d, 0.0);
    for (size_t i = 0; i < d; ++i) q[i * d + i] = 1.0;
    for (size_t kk = d; kk-- > 0;) {
        const double b = beta[kk];
        if (b == 0.0) continue;
        const size_t m = d - kk;
        for (size_t j = 0; j < m; ++j) w[j] = q[kk * d + kk + j];
        for (size_t i = kk + 1; i < d; ++i) {
            const double vi = a[i * d + kk];
            const double* row = &q[i * d + kk];
            for (size_t j = 0; j < m; ++j) w[j] += vi * row[j];
        }
        for (size_t j = 0; j < m; ++j) q[kk * d + kk + j] -= b * w[j];
#pragma omp parallel for if (m > 256)
        for (size_t i = kk + 1; i < d; ++i) {
            const double vi = b * a[i * d + kk];
            double* row = &q[i * d + kk];
            for (size_t j = 0; j < m; ++j) row[j] -= vi * w[j];
        }
    }
    std::vector<float> out(d * d);
    for (size_t i = 0; i < d * d; ++i) out[i] = static_cast<float>(q[i]);
    return out;
}

// Offset of element (row, dim) inside the PDX-blocked copy of a row-major n x d matrix
// (layout.h:155-232): rows are grouped in chunks of 1024; inside a chunk of `cs` rows the first
// vertical_d dimensions are stored dimension-major ([vertical_d][cs]) and the remaining ones as
// consecutive blocks of 64 dimensions, each block row-major ([cs][64]).  The last chunk uses its
// own, smaller cs.
inline size_t pdx_offset(size_t row, size_t dim, size_t n, size_t d, size_t vertical_d) {
    const size_t chunk = row / kVectorChunkSize;
    const size_t v = row % kVectorChunkSize;
    const size_t cs = std::min(kVectorChunkSize, n - chunk * kVectorChunkSize);
    const size_t base = chunk * kVectorChunkSize * d;
    if (dim < vertical_d) return base + dim * cs + v;
    const size_t h = dim - vertical_d;
    return base + vertical_d * cs + (h / kHDimSize) * cs * kHDimSize + v * kHDimSize + (h % kHDimSize);
}

// The dense chain (kernels_chain.cu) goes through its points in slices, on tiles of kChainTileRows points.  While every tile of a launch can have
// a pair of SMs for each of the kChainUnits units of a chunk, the pairs of a tile tell each other what they found in scratch memory.
constexpr size_t kChainTileRows = 256;
constexpr size_t kChainUnits = 4;
inline bool chain_shares_tiles(size_t n, size_t sm_pairs) { return (n + kChainTileRows - 1) / kChainTileRows * kChainUnits <= sm_pairs; }
// Points that the scratch must have room for when n of them go through in slices of `slice`: the last slice, being shorter, may share its tiles
// where the others do not.
inline size_t chain_scratch_rows(size_t n, size_t slice, size_t sm_pairs) {
    size_t rows = 0;
    for (const size_t cnt : {std::min(n, slice), n % slice})
        if (chain_shares_tiles(cnt, sm_pairs)) rows = std::max(rows, cnt);
    return rows;
}

} // namespace skmb
