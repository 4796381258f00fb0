// See exact_assign.h.  What bounds the steps on a B200 (2M x 384 rows, 16 384 centroids): the filter is one fp16 product,
// 2 n k d flop where the three-product kernel does 6 n k d at half the rate; everything else streams the rows.
#include <cfloat>
#include <cmath>

#include "exact_assign.h"
#include "device_utils.cuh"
#include "kernels_tc.cuh"
#include "tc_ptx.cuh"

namespace skmb {

namespace {

using namespace tc;

// Largest values over all centroids, as bits of non-negative floats (ordered like integers; a NaN is larger than all).
enum Stat { kCentredNorm = 0, kResidual = 1, kPlainNorm = 2, kStats = 4 };

constexpr int kMeanSamples = 32;
constexpr float kSmallest = 1e-30f, kLargest = 1e30f;   // squared norms outside are not filtered

// Power of two that maps a vector of this squared norm into [-2^14, 2^14], where fp16 has its full precision down to
// elements 2^-28 of the norm.
__device__ __forceinline__ float fp16_scale(float sqnorm) {
    if (!(sqnorm > kSmallest) || !(sqnorm < kLargest)) return 1.0f;
    int e;
    frexpf(sqrtf(sqnorm), &e);
    return ldexpf(1.0f, 14 - e);
}

__device__ __forceinline__ void stat_max(uint32_t* stats, int which, float v) { atomicMax(stats + which, __float_as_uint(fabsf(v))); }

// Mean of some evenly spaced centroids: distances do not change when it is subtracted everywhere, the norms that scale the
// filter's error shrink to the spread of the data.
__global__ void __launch_bounds__(64) sample_mean_kernel(const float* __restrict__ y, size_t k, size_t d, float* __restrict__ mean, uint32_t* __restrict__ stats,
                                                         uint32_t* __restrict__ n_listed) {
    if (blockIdx.x == 0 && threadIdx.x < kStats) stats[threadIdx.x] = 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) *n_listed = 0u;
    const size_t j = static_cast<size_t>(blockIdx.x) * 64 + threadIdx.x;
    if (j >= d) return;
    float s = 0.f;   // (d = 0: the mean stays what it is)
#pragma unroll
    for (int q = 0; q < kMeanSamples; ++q) s += __ldg(y + (static_cast<size_t>(q) * k / kMeanSamples) * d + j);
    mean[j] = s * (1.0f / kMeanSamples);
}

// Squared norms of a row held by a warp, in the order of row_sqnorms_kernel, and of the row minus the mean.
struct RowNorms {
    float plain, centred;
};
template <bool VEC>
__device__ __forceinline__ RowNorms row_norms(const float* __restrict__ row, const float* __restrict__ mean, size_t d, int lane) {
    float a = 0.f, b = 0.f;
    if (VEC) {
        for (size_t j = static_cast<size_t>(lane) * 4; j < d; j += 128) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(row + j)), m = __ldg(reinterpret_cast<const float4*>(mean + j));
            a = fmaf(v.x, v.x, a); a = fmaf(v.y, v.y, a); a = fmaf(v.z, v.z, a); a = fmaf(v.w, v.w, a);
            float t;
            t = v.x - m.x; b = fmaf(t, t, b); t = v.y - m.y; b = fmaf(t, t, b); t = v.z - m.z; b = fmaf(t, t, b); t = v.w - m.w; b = fmaf(t, t, b);
        }
    } else {
        for (size_t j = lane; j < d; j += 32) {
            const float v = __ldg(row + j), t = v - __ldg(mean + j);
            a = fmaf(v, v, a);
            b = fmaf(t, t, b);
        }
    }
    return {warp_sum(a), warp_sum(b)};
}

// Writes the row minus the mean, times `scale`, as fp16 (columns d .. dp - 1 zero); returns the squared norm of the rounding
// error, in the row's own units.
template <bool VEC>
__device__ __forceinline__ float write_fp16_row(const float* __restrict__ row, const float* __restrict__ mean, size_t d, size_t dp, float scale, __half* __restrict__ out, int lane) {
    const float inv = 1.0f / scale;
    float err = 0.f;
    if (VEC) {
        for (size_t j = static_cast<size_t>(lane) * 4; j < dp; j += 128) {
            float t[4] = {0.f, 0.f, 0.f, 0.f};
            if (j < d) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(row + j)), m = __ldg(reinterpret_cast<const float4*>(mean + j));
                t[0] = v.x - m.x; t[1] = v.y - m.y; t[2] = v.z - m.z; t[3] = v.w - m.w;
            }
            __align__(8) __half h[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                h[q] = __float2half_rn(t[q] * scale);
                const float r = fmaf(-__half2float(h[q]), inv, t[q]);
                err = fmaf(r, r, err);
            }
            *reinterpret_cast<uint2*>(out + j) = *reinterpret_cast<const uint2*>(h);
        }
    } else {
        for (size_t j = lane; j < dp; j += 32) {
            const float t = j < d ? __ldg(row + j) - __ldg(mean + j) : 0.f;
            const __half h = __float2half_rn(t * scale);
            const float r = fmaf(-__half2float(h), inv, t);
            err = fmaf(r, r, err);
            out[j] = h;
        }
    }
    return warp_sum(err);
}

// One warp per centroid (and per padding column of the filter's last tile, which gets a norm that never wins).
template <bool VEC>
__global__ void __launch_bounds__(256) centroid_norms_kernel(const float* __restrict__ y, size_t k, size_t kp, size_t d, const float* __restrict__ mean, float* __restrict__ norms,
                                                             float* __restrict__ centred, uint32_t* __restrict__ stats) {
    const size_t c = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (c >= kp) return;
    if (c >= k) {
        if (lane == 0) centred[c] = FLT_MAX;
        return;
    }
    const RowNorms n = row_norms<VEC>(y + c * d, mean, d, lane);
    if (lane == 0) {
        norms[c] = n.plain;
        centred[c] = n.centred;
        stat_max(stats, kCentredNorm, n.centred);
        stat_max(stats, kPlainNorm, n.plain);
    }
}

template <bool VEC>
__global__ void __launch_bounds__(256) centroid_fp16_kernel(const float* __restrict__ y, size_t k, size_t d, size_t dp, const float* __restrict__ mean, uint32_t* __restrict__ stats,
                                                            __half* __restrict__ out) {
    const size_t c = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (c >= k) return;
    const int lane = threadIdx.x & 31;
    const float err = write_fp16_row<VEC>(y + c * d, mean, d, dp, fp16_scale(__uint_as_float(stats[kCentredNorm])), out + c * dp, lane);
    if (lane == 0) stat_max(stats, kResidual, err);
}

// With centroids that the filter cannot tell apart (copies of one another, one of a norm far above the others', one that is no number)
// every row ends in the list, and what the filter takes comes on top of the three-product kernel: 1M x 384 and 8192
// centroids, one of them 1e6 long: 39.6 ms, where the three products alone take 33 - 36.  So a batch that has listed most of its
// rows so far lists the others unseen (32.7).  Decided on the device, by the kernel before the filter, while nothing appends to the list.
constexpr uint32_t kSeenRows = 4096;
__device__ __forceinline__ bool hopeless(const uint32_t* n_listed, size_t rows_before) { return rows_before >= kSeenRows && 2 * static_cast<size_t>(*n_listed) > rows_before; }

// Per row: fp16 copy, norm, and {squared norm minus the mean, squared norm of the rounding error, squared norm, scale}.
// With U the row is read once, all of it in flight (rows of at most 128 U columns, VEC); without, twice.
template <bool VEC, int U>
__global__ void __launch_bounds__(256) row_fp16_kernel(const float* __restrict__ x, size_t n, size_t d, size_t dp, const float* __restrict__ mean, float* __restrict__ norms,
                                                       __half* __restrict__ out, float4* __restrict__ info, const uint32_t* __restrict__ n_listed, size_t rows_before,
                                                       uint32_t* __restrict__ unseen) {
    const size_t row = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    const bool give_up = hopeless(n_listed, rows_before);
    if (blockIdx.x == 0 && threadIdx.x == 0) *unseen = give_up ? 1u : 0u;
    if (row >= n) return;
    const int lane = threadIdx.x & 31;
    const float* xr = x + row * d;
    RowNorms nx;
    [[maybe_unused]] float4 v[U > 0 ? U : 1];
    if constexpr (U > 0) {
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = 4 * lane + 128 * u < d ? __ldg(reinterpret_cast<const float4*>(xr + 4 * lane + 128 * u)) : make_float4(0.f, 0.f, 0.f, 0.f);
        float a = 0.f, b = 0.f;   // (in the order of row_norms)
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (4 * lane + 128 * u < d) {
                const float4 m = __ldg(reinterpret_cast<const float4*>(mean + 4 * lane + 128 * u));
                a = fmaf(v[u].x, v[u].x, a); a = fmaf(v[u].y, v[u].y, a); a = fmaf(v[u].z, v[u].z, a); a = fmaf(v[u].w, v[u].w, a);
                v[u] = make_float4(v[u].x - m.x, v[u].y - m.y, v[u].z - m.z, v[u].w - m.w);
                b = fmaf(v[u].x, v[u].x, b); b = fmaf(v[u].y, v[u].y, b); b = fmaf(v[u].z, v[u].z, b); b = fmaf(v[u].w, v[u].w, b);
            }
        }
        nx = {warp_sum(a), warp_sum(b)};
    } else {
        nx = row_norms<VEC>(xr, mean, d, lane);
    }
    if (give_up) {
        if (lane == 0) norms[row] = nx.plain;
        return;
    }
    const float scale = fp16_scale(nx.centred);
    float err;
    if constexpr (U > 0) {
        const float inv = 1.0f / scale;
        err = 0.f;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (4 * lane + 128 * u < dp) {
                const float t[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
                __align__(8) __half h[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    h[q] = __float2half_rn(t[q] * scale);
                    const float r = fmaf(-__half2float(h[q]), inv, t[q]);
                    err = fmaf(r, r, err);
                }
                *reinterpret_cast<uint2*>(out + row * dp + 4 * lane + 128 * u) = *reinterpret_cast<const uint2*>(h);
            }
        }
        err = warp_sum(err);
    } else {
        err = write_fp16_row<VEC>(xr, mean, d, dp, scale, out + row * dp, lane);
    }
    if (lane != 0) return;
    norms[row] = nx.plain;
    info[row] = make_float4(nx.centred, err, nx.plain, scale);
}

// For the filter: {factor from accumulator to -2 x.c, width of the window above the smallest filtered distance in which the
// true nearest centroid lies (infinite: the row is not filtered)}.
__device__ __forceinline__ float2 filter_terms(const float4 r, const uint32_t* __restrict__ stats, uint32_t k_blocks) {
    const float c2 = __uint_as_float(__ldg(stats + kCentredNorm)), e2 = __uint_as_float(__ldg(stats + kResidual)), p2 = __uint_as_float(__ldg(stats + kPlainNorm));
    const bool usable = r.z < kLargest && p2 < kLargest && r.x < kLargest && c2 < kLargest && (r.x == 0.f || r.x > kSmallest) && (c2 == 0.f || c2 > kSmallest);
    // |x.c - x^.c^| <= |x - x^| |c| + |x^| |c - c^|, plus a truncation of at most 2^-22 of the running sum for each 16-wide
    // product added (counted twice); the norms are rounded up
    const float xn = sqrtf(r.x) * 1.0001f, xe = sqrtf(r.y) * 1.001f, cn = sqrtf(c2) * 1.0001f, ce = sqrtf(e2) * 1.001f;
    const float trunc = (static_cast<float>(k_blocks * 4) + 16.0f) * 4.8e-7f;
    const float bound = xe * cn + (xn + xe) * ce + trunc * (xn + xe) * (cn + ce);
    // twice the distance's error on both sides; pairs that the decision treats as near-ties (1e-4 of the distance), and
    // the rounding of the fp32 distances it compares
    const float window = 4.0f * bound + 2e-4f * (r.x + c2) + 4e-6f * (r.z + p2);
    return make_float2(-2.0f / (r.w * fp16_scale(c2)), usable ? window : INFINITY);
}

// -------------------------------------------------------------------------------------------------
// The filter: persistent pairs of CTAs (cta_group::2), a tile of 256 rows x 256 centroids at a time; each CTA holds its 128
// rows and half of the centroids, so that a byte of shared memory feeds twice the products and L2 delivers 64 bytes per SM
// and cycle at the tensor cores' nominal rate (a single CTA would need 96).
//   warp 0     TMA producer: 128 x 64 halves of rows and of centroids per stage, five stages, counted by the leader's barrier;
//   warp 1     MMA issuer (leader only), two accumulators of 256 columns;
//   warps 2-9  two threads per row, one for each half of the tile's columns: value = acc * factor + |c|^2, smallest four
//              with their indices and the fifth; merged at the end of the row.
// A value is looked at only when it is below the fifth smallest and inside the window above the smallest so far, which
// few are once a row has seen some centroids: the usual work on 32 columns is their minimum, two instructions a column, and
// the rest is kept out of line (inlined at every column it overflowed the instruction cache: 32 ms where this takes 21 ms
// at 2M x 384 and 16 384 centroids).  Every wait is bounded (see kernels_tc.cu).
constexpr int FK = 64;                                  // halves per stage and row: 128 bytes
constexpr int F_STAGES = 5;
constexpr uint32_t F_TILE_BYTES = 128 * FK * 2;         // rows, and half of the centroids, of a stage
constexpr uint32_t F_STAGE_BYTES = 2 * F_TILE_BYTES;
constexpr int F_THREADS = 320;
constexpr uint32_t F_CTRL_BYTES = 8192 + 8 * 32 * 33 * 4 + 2 * 128 * 9 * 4 + 256;
constexpr uint32_t F_SMEM_BYTES = F_STAGES * F_STAGE_BYTES + F_CTRL_BYTES + 1024;

struct FilterCtrl {
    alignas(16) float ny[4][2][256];   // per row quarter and accumulator
    float column[8][32][33];           // per epilogue warp: values of 32 columns that hold a candidate
    float half[2][9][128];             // smallest values and indices of the rows' second halves, by parity of the row tile
    uint64_t full[F_STAGES];           // (the leader's are used)
    uint64_t empty[F_STAGES];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];             // (the leader's are used)
    uint64_t half_full[2][4], half_empty[2][4];   // `half` written / read, by parity and row quarter
    uint32_t tmem_base;
};
static_assert(sizeof(FilterCtrl) <= F_CTRL_BYTES, "control block too large");

struct FilterParams {
    size_t n;              // rows of this launch
    size_t first;          // index of its first row inside the batch
    uint32_t k;
    uint32_t k_blocks;     // of 64 columns
    const AssignTile* tiles;   // grouped: what every row tile is assigned to
    size_t n_tiles;
    const float4* info;
    const uint32_t* stats;
    const float* norms_y;  // centred, padded to whole tiles
    uint4* cand;
    uint32_t* listed;
    uint32_t* n_listed;
    const uint32_t* unseen;   // nonzero: list all rows
    int* error;
    long long wait_limit;
    uint32_t producer_stop;   // see set_debug_wait_injection
};

struct Best {
    float v1 = FLT_MAX, v2 = FLT_MAX, v3 = FLT_MAX, v4 = FLT_MAX, v5 = FLT_MAX;
    uint32_t i1 = ~0u, i2 = ~0u, i3 = ~0u, i4 = ~0u;
    __device__ __forceinline__ void insert(float v, uint32_t i) {
        auto place = [&](float& w, uint32_t& j) {
            const bool less = v < w;
            const float tv = less ? w : v;
            const uint32_t ti = less ? j : i;
            w = less ? v : w;
            j = less ? i : j;
            v = tv;
            i = ti;
        };
        place(v1, i1);
        place(v2, i2);
        place(v3, i3);
        place(v4, i4);
        v5 = fminf(v5, v);
    }
};

// Columns of a column tile that are multiplied, half of them by the centroids of either CTA.  Groups of few centroids leave most of a tile
// empty (300 000 x 768 rows, groups of 50: 110 us a pass with whole tiles, 90 so); without groups it is the last tile at most.
template <bool GROUPED>
__device__ __forceinline__ uint32_t filter_columns(uint32_t k, uint32_t nt) {
    return GROUPED ? min(256u, (k - nt * 256 + 31) / 32 * 32) : 256u;
}

template <bool GROUPED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(F_THREADS, 1)
    filter_tc_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_y, const FilterParams p) {
    extern __shared__ uint8_t smem_raw[];
    if (!GROUPED && *p.unseen != 0) {   // (the same for all blocks)
        for (size_t row0 = static_cast<size_t>(blockIdx.x) * F_THREADS; row0 < p.n; row0 += static_cast<size_t>(gridDim.x) * F_THREADS) {
            const size_t row = row0 + threadIdx.x;
            const uint32_t mine = __ballot_sync(0xffffffffu, row < p.n), lane_id = threadIdx.x & 31;
            uint32_t at = 0;
            if (lane_id == 0) at = atomicAdd(p.n_listed, static_cast<uint32_t>(__popc(mine)));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (row < p.n) {
                p.listed[at + lane_id] = static_cast<uint32_t>(p.first + row);
                p.cand[row].x = ~0u;
            }
        }
        return;
    }
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
    const uint32_t smem_base = raw_addr + pad;
    FilterCtrl* ctrl = reinterpret_cast<FilterCtrl*>(smem_raw + pad + F_STAGES * F_STAGE_BYTES);
    const WaitCtx wctx{p.error, p.wait_limit};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();

    if (threadIdx.x == 0) {
        for (int s = 0; s < F_STAGES; ++s) {
            mbar_init(&ctrl->full[s], 1);
            mbar_init(&ctrl->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctrl->acc_full[b], 1);
            mbar_init(&ctrl->acc_empty[b], 16);   // a lane of each of the pair's epilogue warps
        }
        for (int q = 0; q < 8; ++q) {
            mbar_init(&ctrl->half_full[q >> 2][q & 3], 1);
            mbar_init(&ctrl->half_empty[q >> 2][q & 3], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (warp == 1) tmem_alloc_pair(&ctrl->tmem_base, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // the peer's barriers exist
    tc_fence_after();
    const uint32_t tmem_base = ctrl->tmem_base;

    const size_t n_row_tiles = GROUPED ? p.n_tiles : (p.n + 255) / 256;
    auto tile_at = [&](size_t rt) -> AssignTile {
        if (GROUPED) return p.tiles[rt];
        return {static_cast<uint32_t>(rt * 256), static_cast<uint32_t>(min(p.n - rt * 256, size_t{256})), 0u, p.k};
    };
    const size_t pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t kbt = 0;
            bool ok = true;
            for (size_t rt = pair; rt < n_row_tiles && ok; rt += n_pairs) {
                const AssignTile tile = tile_at(rt);
                const uint32_t col_tiles = (tile.k + 255) / 256;
                const int x_row = static_cast<int>(tile.row0 + rank * 128);
                for (uint32_t nt = 0; nt < col_tiles && ok; ++nt) {
                    const int y_row = static_cast<int>(tile.y0 + nt * 256 + rank * (filter_columns<GROUPED>(tile.k, nt) / 2));
                    for (uint32_t kb = 0; kb < p.k_blocks; ++kb, ++kbt) {
                        const uint32_t s = kbt % F_STAGES, ph = (kbt / F_STAGES) & 1u;
                        if ((p.producer_stop != 0 && kbt >= p.producer_stop) || !mbar_wait(&ctrl->empty[s], ph ^ 1u, wctx, 41)) {
                            ok = false;
                            break;
                        }
                        if (rank == 0) mbar_arrive_expect_tx(&ctrl->full[s], 2 * F_STAGE_BYTES);
                        const uint32_t bar = cluster_address(&ctrl->full[s], 0);
                        const uint32_t st = smem_base + s * F_STAGE_BYTES;
                        tma_load_2d_pair(st, &tmap_x, bar, static_cast<int>(kb * FK), x_row);
                        tma_load_2d_pair(st + F_TILE_BYTES, &tmap_y, bar, static_cast<int>(kb * FK), y_row);
                    }
                }
            }
            if (!ok) {
                // another role gave up: a millisecond for the copies that are in flight before the block's memory is let go
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000) {
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            uint32_t kbt = 0, t = 0;
            bool ok = true;
            for (size_t rt = pair; rt < n_row_tiles && ok; rt += n_pairs) {
                const uint32_t k = tile_at(rt).k, col_tiles = (k + 255) / 256;
                for (uint32_t nt = 0; nt < col_tiles && ok; ++nt, ++t) {
                    const uint32_t b = t & 1u, tph = (t >> 1) & 1u, idesc = make_idesc_f16(256, filter_columns<GROUPED>(k, nt));
                    if (!mbar_wait(&ctrl->acc_empty[b], tph ^ 1u, wctx, 42)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t acc = tmem_base + b * 256;
                    for (uint32_t kb = 0; kb < p.k_blocks; ++kb, ++kbt) {
                        const uint32_t s = kbt % F_STAGES, ph = (kbt / F_STAGES) & 1u;
                        if (!mbar_wait(&ctrl->full[s], ph, wctx, 43)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t st = smem_base + s * F_STAGE_BYTES;
#pragma unroll
                        for (uint32_t kk = 0; kk < FK / 16; ++kk)
                            umma_f16_pair(acc, make_desc_128(st + kk * 32), make_desc_128(st + F_TILE_BYTES + kk * 32), (kb | kk) != 0 ? 1u : 0u, idesc);
                        umma_commit_pair(&ctrl->empty[s]);
                    }
                    if (ok) umma_commit_pair(&ctrl->acc_full[b]);
                }
            }
        }
    } else {
        const uint32_t quarter = warp & 3, half = static_cast<uint32_t>(warp - 2) >> 2;
        const uint32_t lane_base = 32u * quarter;
        uint32_t t = 0, row_tiles = 0;
        bool ok = true;
        for (size_t rt = pair; rt < n_row_tiles && ok; rt += n_pairs, ++row_tiles) {
            const AssignTile tile = tile_at(rt);
            const uint32_t col_tiles = (tile.k + 255) / 256;
            const size_t row = static_cast<size_t>(tile.row0) + rank * 128 + lane_base + lane;
            const bool valid = rank * 128 + lane_base + lane < tile.rows;
            const float2 info = valid ? filter_terms(p.info[row], p.stats, p.k_blocks) : make_float2(0.f, 0.f);
            Best best;
            float limit = FLT_MAX;   // values from here on change nothing
            for (uint32_t nt = 0; nt < col_tiles && ok; ++nt, ++t) {
                const uint32_t b = t & 1u, tph = (t >> 1) & 1u;
                float* ny = ctrl->ny[quarter][b];
                // the two warps of a quarter fill (and read) their own halves
                if (GROUPED) {
                    // (the columns behind the group's are another group's centroids)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t c = nt * 256 + half * 128 + q * 32 + lane;
                        ny[half * 128 + q * 32 + lane] = c < tile.k ? __ldg(p.norms_y + tile.y0 + c) : FLT_MAX;
                    }
                } else {
                    *reinterpret_cast<float4*>(ny + half * 128 + lane * 4) = __ldg(reinterpret_cast<const float4*>(p.norms_y + static_cast<size_t>(nt) * 256 + half * 128 + lane * 4));
                }
                __syncwarp();
                if (!__all_sync(0xffffffffu, mbar_wait(&ctrl->acc_full[b], tph, wctx, 44))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + (lane_base << 16) + b * 256;
                auto look = [&](uint32_t (&r)[32], int ch) {
                    float least = FLT_MAX;
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 n4 = *reinterpret_cast<const float4*>(ny + ch * 32 + j);
                        const float a = fmaf(__uint_as_float(r[j]), info.x, n4.x), c = fmaf(__uint_as_float(r[j + 1]), info.x, n4.y);
                        const float e = fmaf(__uint_as_float(r[j + 2]), info.x, n4.z), g = fmaf(__uint_as_float(r[j + 3]), info.x, n4.w);
                        least = fminf(fminf(least, a), c);
                        least = fminf(fminf(least, e), g);
                        r[j] = __float_as_uint(a);
                        r[j + 1] = __float_as_uint(c);
                        r[j + 2] = __float_as_uint(e);
                        r[j + 3] = __float_as_uint(g);
                    }
                    if (!__any_sync(0xffffffffu, least < limit)) return;
                    uint32_t hits = 0;
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        ctrl->column[warp - 2][j][lane] = __uint_as_float(r[j]);
                        hits |= __uint_as_float(r[j]) < limit ? 1u << j : 0u;
                    }
#pragma unroll 1
                    while (hits) {
                        const int j = __ffs(hits) - 1;
                        hits &= hits - 1;
                        const float v = ctrl->column[warp - 2][j][lane];
                        if (v < limit) {
                            best.insert(v, tile.y0 + nt * 256 + ch * 32 + j);
                            limit = fminf(best.v5, best.v1 + info.y);
                        }
                    }
                    __syncwarp();
                };
                uint32_t ra[32], rb[32];
                const int slice0 = static_cast<int>(half) * 4;
                auto give_back = [&] {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster_read(cluster_address(&ctrl->acc_empty[b], 0));
                };
                if (GROUPED && filter_columns<GROUPED>(tile.k, nt) != 256) {
                    // only the columns that were multiplied: what stands in the others is older
                    const int end = min(slice0 + 4, static_cast<int>(filter_columns<GROUPED>(tile.k, nt) / 32));
#pragma unroll 1
                    for (int ch = slice0; ch < end; ++ch) {
                        tmem_ld32_issue(taddr + ch * 32, ra);
                        tmem_ld_wait(ra);
                        look(ra, ch);
                    }
                    give_back();
                    continue;
                }
                tmem_ld32_issue(taddr + slice0 * 32, ra);
                tmem_ld_wait(ra);
#pragma unroll 1
                for (int ch = slice0; ch < slice0 + 4; ch += 2) {
                    tmem_ld32_issue(taddr + (ch + 1) * 32, rb);
                    look(ra, ch);
                    tmem_ld_wait(rb);
                    if (ch == slice0) tmem_ld32_issue(taddr + (ch + 2) * 32, ra);
                    else give_back();
                    look(rb, ch + 1);
                    if (ch == slice0) tmem_ld_wait(ra);
                }
            }
            if (!ok) break;
            // merge the halves (two buffers, so that the second half need not wait for the first of the same row tile)
            const uint32_t par = row_tiles & 1u, use = row_tiles >> 1;
            float* mine = &ctrl->half[par][0][lane_base + lane];
            if (half == 1) {
                if (use > 0 && !__all_sync(0xffffffffu, mbar_wait(&ctrl->half_empty[par][quarter], (use - 1) & 1u, wctx, 45))) break;
                const float v[9] = {best.v1, best.v2, best.v3, best.v4, best.v5, __uint_as_float(best.i1), __uint_as_float(best.i2), __uint_as_float(best.i3), __uint_as_float(best.i4)};
#pragma unroll
                for (int q = 0; q < 9; ++q) mine[q * 128] = v[q];
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctrl->half_full[par][quarter]);
                continue;
            }
            if (!__all_sync(0xffffffffu, mbar_wait(&ctrl->half_full[par][quarter], use & 1u, wctx, 46))) break;
#pragma unroll
            for (int q = 0; q < 4; ++q) best.insert(mine[q * 128], __float_as_uint(mine[(5 + q) * 128]));
            best.v5 = fminf(best.v5, mine[4 * 128]);
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctrl->half_empty[par][quarter]);
            if (valid) {
                const float edge = best.v1 + info.y;
                uint4 c = make_uint4(best.i1, best.v2 <= edge ? best.i2 : ~0u, best.v3 <= edge ? best.i3 : ~0u, best.v4 <= edge ? best.i4 : ~0u);
                // more than four inside the window, or a row (or centroids) outside the range of the bound
                if (!(best.v5 > edge) || best.i1 == ~0u) {
                    c.x = ~0u;
                    p.listed[atomicAdd(p.n_listed, 1u)] = static_cast<uint32_t>(p.first + row);
                }
                p.cand[row] = c;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // nothing of the pair is in flight towards this CTA any more
    if (warp == 1) tmem_dealloc_pair(tmem_base, TMEM_COLS);
}

// The decision: fp32 distances of a row's candidates, one warp per row (see refine_top2_kernel, whose sums, ties and
// clamping these are).
// What bounds it is the latency of its loads, one behind the other for a row (candidates, centroids), so a warp asks for the next row's
// candidates and its first 512 columns before it decides the present one.
template <bool VEC>
__global__ void __launch_bounds__(256, 3) decide_kernel(const float* __restrict__ x, const float* __restrict__ y, size_t n, size_t k, size_t d, const float* __restrict__ norms_x,
                                                     const float* __restrict__ norms_y, const uint4* __restrict__ cand, uint32_t* __restrict__ out_knn, float* __restrict__ out_dist,
                                                     const int* __restrict__ error) {
    if (*reinterpret_cast<const volatile int*>(error) != 0) return;   // the candidates were not written
    const int lane = threadIdx.x & 31;
    constexpr int U = 4;
    const size_t step = static_cast<size_t>(gridDim.x) * 8;
    float4 v[U], v_next[U];
    uint4 c_next = make_uint4(~0u, ~0u, ~0u, ~0u);
    auto load_point = [&](float4 (&to)[U], size_t row, size_t j0) {
#pragma unroll
        for (int u = 0; u < U; ++u) to[u] = j0 + 128 * u < d ? __ldg(reinterpret_cast<const float4*>(x + row * d + j0 + 128 * u)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto ask = [&](size_t row) {
        if (row >= n) return;
        c_next = __ldg(cand + row);
        if (VEC && out_dist) load_point(v_next, row, 4 * lane);
    };
    size_t row = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    ask(row);
    for (; row < n; row += step) {
        const uint4 c4 = c_next;
        if (VEC && out_dist) {
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = v_next[u];
        }
        ask(row + step);
        if (c4.x >= k) continue;   // listed
        const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
        const int count = c4.y >= k ? 1 : (c4.z >= k ? 2 : (c4.w >= k ? 3 : 4));
        if (count == 1 && !out_dist) {
            if (lane == 0) out_knn[row] = c4.x;
            continue;
        }
        const float* xr = x + row * d;
        if (VEC && !out_dist) load_point(v, row, 4 * lane);
        const float* yr[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) yr[q] = y + static_cast<size_t>(q < count ? c[q] : c[0]) * d;
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        if (VEC) {
            for (size_t j0 = static_cast<size_t>(lane) * 4; j0 < d; j0 += 128 * U) {
                if (j0 >= 128 * U) load_point(v, row, j0);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (q < count) {
                        float4 w[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) w[u] = j0 + 128 * u < d ? __ldg(reinterpret_cast<const float4*>(yr[q] + j0 + 128 * u)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            if (j0 + 128 * u < d) {
                                s[q] = fmaf(v[u].x, w[u].x, s[q]); s[q] = fmaf(v[u].y, w[u].y, s[q]); s[q] = fmaf(v[u].z, w[u].z, s[q]); s[q] = fmaf(v[u].w, w[u].w, s[q]);
                            }
                        }
                    }
                }
            }
        } else {
            for (size_t j = lane; j < d; j += 32) {
                const float xv = __ldg(xr + j);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (q < count) s[q] = fmaf(xv, __ldg(yr[q] + j), s[q]);
            }
        }
        const float nx = norms_x[row];
        float e[4];
        float lowest = FLT_MAX;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            e[q] = FLT_MAX;
            if (q < count) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
                e[q] = fmaf(-2.0f, s[q], nx) + norms_y[c[q]];
                lowest = fminf(lowest, e[q]);
            }
        }
        // near-ties are settled with dot products accumulated in index order, a lane for each
        int close = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) close += (q < count && fabsf(e[q] - lowest) <= 1e-4f * fmaxf(fabsf(e[q]), fabsf(lowest))) ? 1 << q : 0;
        if (__popc(close) > 1) {
            float t = 0.f;
            if (lane < 4 && ((close >> lane) & 1)) {
                const float* yl = lane == 0 ? yr[0] : (lane == 1 ? yr[1] : (lane == 2 ? yr[2] : yr[3]));
                for (size_t j = 0; j < d; ++j) t = fmaf(xr[j], yl[j], t);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float tq = __shfl_sync(0xffffffffu, t, q);
                if ((close >> q) & 1) e[q] = fmaf(-2.0f, tq, nx) + norms_y[c[q]];
            }
        }
        if (lane == 0) {
            float be = e[0];
            uint32_t bi = c[0];
#pragma unroll
            for (int q = 1; q < 4; ++q) {
                if (q < count && (e[q] < be || (e[q] == be && c[q] < bi))) {
                    be = e[q];
                    bi = c[q];
                }
            }
            out_knn[row] = bi;
            if (out_dist) out_dist[row] = fmaxf(0.0f, be);
        }
    }
}

__global__ void __launch_bounds__(256) gather_listed_rows_kernel(const float* __restrict__ x, const uint32_t* __restrict__ idx, size_t n, size_t d, float* __restrict__ out) {
    const size_t i = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    const float* src = x + static_cast<size_t>(idx[i]) * d;
    for (size_t j = threadIdx.x & 31; j < d; j += 32) out[i * d + j] = __ldg(src + j);
}

// The listed rows of a grouped pass, few of them: a warp computes the fp32 distances of a row to all centroids of its group.
// With kDenseListed listed rows per tile and more this is the slower way (every row reads all centroids again), and
// decide_listed_tiles_kernel does them.
constexpr uint32_t kDenseListed = 32;
__global__ void __launch_bounds__(256) decide_listed_kernel(const float* __restrict__ x, const float* __restrict__ y, size_t d, const float* __restrict__ norms_x,
                                                            const float* __restrict__ norms_y, const AssignTile* __restrict__ tiles, size_t n_tiles,
                                                            const uint32_t* __restrict__ listed, const uint32_t* __restrict__ n_listed, uint32_t* __restrict__ out_knn,
                                                            float* __restrict__ out_dist, const int* __restrict__ error) {
    if (*reinterpret_cast<const volatile int*>(error) != 0) return;
    const int lane = threadIdx.x & 31;
    const uint32_t n = *n_listed;
    if (n >= kDenseListed * n_tiles) return;
    for (uint32_t i = blockIdx.x * 8 + (threadIdx.x >> 5); i < n; i += gridDim.x * 8) {
        const uint32_t row = listed[i];
        size_t lo = 0, hi = n_tiles;   // the last tile that begins at or before the row
        while (hi - lo > 1) {
            const size_t mid = (lo + hi) / 2;
            if (tiles[mid].row0 <= row) lo = mid;
            else hi = mid;
        }
        const AssignTile tile = tiles[lo];
        const float* xr = x + static_cast<size_t>(row) * d;
        const float nx = norms_x[row];
        unsigned long long best = ~0ull;
        for (uint32_t c = tile.y0; c < tile.y0 + tile.k; ++c) {
            const float* yr = y + static_cast<size_t>(c) * d;
            float s = 0.f;
            for (size_t j = lane; j < d; j += 32) s = fmaf(__ldg(xr + j), __ldg(yr + j), s);
            const unsigned long long key = pair_key(fmaf(-2.0f, warp_sum(s), nx) + norms_y[c], c);
            best = key < best ? key : best;
        }
        if (lane == 0) store_answer(best, row, out_knn, out_dist);
    }
}

// Many of them (clusters closer to each other than the rounding of the group's largest distances lets the filter see): 64 of a
// tile's listed rows per block (blockIdx.y: which 64) against 64 centroids of the group at a time, 4 x 4 distances per
// thread as in direct_assign.cu, bound by fp32 issue.  2.5M x 768 in 128 groups of 128 clusters, nearly all rows listed, eight
// exact passes: 116 ms, 962 with a warp per row.
constexpr int kListedRows = 64, kListedCols = 64, kListedDepth = 16;
template <bool VEC>
__global__ void __launch_bounds__(256) decide_listed_tiles_kernel(const float* __restrict__ x, const float* __restrict__ y, size_t d, const float* __restrict__ norms_x,
                                                                  const float* __restrict__ norms_y, const AssignTile* __restrict__ tiles, size_t n_tiles,
                                                                  const uint4* __restrict__ cand, const uint32_t* __restrict__ n_listed, uint32_t* __restrict__ out_knn,
                                                                  float* __restrict__ out_dist, const int* __restrict__ error) {
    __shared__ __align__(16) float sx[2][kListedDepth][kListedRows + 4], sy[2][kListedDepth][kListedCols + 4];
    __shared__ uint32_t rows[kListedRows];
    __shared__ uint32_t before[9];
    if (*n_listed < kDenseListed * n_tiles || *reinterpret_cast<const volatile int*>(error) != 0) return;
    const AssignTile tile = tiles[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // which rows: a thread per row of the tile
    const bool mine = threadIdx.x < tile.rows && cand[tile.row0 + threadIdx.x].x == ~0u;
    const uint32_t all = __ballot_sync(0xffffffffu, mine);
    if (lane == 0) before[warp + 1] = __popc(all);
    if (threadIdx.x == 0) before[0] = 0;
    if (threadIdx.x < kListedRows) rows[threadIdx.x] = ~0u;
    __syncthreads();
    uint32_t rank = __popc(all & ((1u << lane) - 1u)), total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < warp) rank += before[w + 1];
        total += before[w + 1];
    }
    const uint32_t first = blockIdx.y * kListedRows;
    if (first >= total) return;
    if (mine && rank >= first && rank < first + kListedRows) rows[rank - first] = tile.row0 + threadIdx.x;
    __syncthreads();

    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int lr = threadIdx.x >> 2, lc = 4 * (threadIdx.x & 3);
    const float* __restrict__ xr = rows[lr] != ~0u ? x + static_cast<size_t>(rows[lr]) * d : nullptr;
    auto load = [&](const float* __restrict__ row, size_t j) {
        if (!row || j >= d) return make_float4(0.f, 0.f, 0.f, 0.f);
        if (VEC) return __ldg(reinterpret_cast<const float4*>(row + j));
        float4 v = make_float4(__ldg(row + j), 0.f, 0.f, 0.f);
        if (j + 1 < d) v.y = __ldg(row + j + 1);
        if (j + 2 < d) v.z = __ldg(row + j + 2);
        if (j + 3 < d) v.w = __ldg(row + j + 3);
        return v;
    };
    float nx[4];
    unsigned long long best[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        nx[r] = rows[ty * 4 + r] != ~0u ? norms_x[rows[ty * 4 + r]] : 0.f;
        best[r] = ~0ull;
    }
    int buf = 0;
    for (uint32_t col0 = 0; col0 < tile.k; col0 += kListedCols) {
        const float* __restrict__ yr = col0 + lr < tile.k ? y + static_cast<size_t>(tile.y0 + col0 + lr) * d : nullptr;
        float acc[4][4] = {};
        float4 vx = load(xr, lc), vy = load(yr, lc);
        for (size_t j0 = 0; j0 < d; j0 += kListedDepth, buf ^= 1) {
            sx[buf][lc][lr] = vx.x; sx[buf][lc + 1][lr] = vx.y; sx[buf][lc + 2][lr] = vx.z; sx[buf][lc + 3][lr] = vx.w;
            sy[buf][lc][lr] = vy.x; sy[buf][lc + 1][lr] = vy.y; sy[buf][lc + 2][lr] = vy.z; sy[buf][lc + 3][lr] = vy.w;
            __syncthreads();
            if (j0 + kListedDepth < d) {
                vx = load(xr, j0 + kListedDepth + lc);
                vy = load(yr, j0 + kListedDepth + lc);
            }
#pragma unroll
            for (int q = 0; q < kListedDepth; ++q) {
                const float4 a = *reinterpret_cast<const float4*>(&sx[buf][q][ty * 4]);
                const float4 b = *reinterpret_cast<const float4*>(&sy[buf][q][tx * 4]);
                const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(av[r], bv[c], acc[r][c]);
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint32_t col = col0 + tx * 4 + c;
            if (col >= tile.k) continue;
            const float ny = __ldg(norms_y + tile.y0 + col);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const unsigned long long key = pair_key(fmaf(-2.0f, acc[r][c], nx[r]) + ny, tile.y0 + col);
                best[r] = key < best[r] ? key : best[r];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, best[r], o);
            best[r] = other < best[r] ? other : best[r];
        }
        if (tx == 0 && rows[ty * 4 + r] != ~0u) store_answer(best[r], rows[ty * 4 + r], out_knn, out_dist);
    }
}

constexpr size_t kWaveRows = 74 * 256;   // a row tile for every pair of SMs

bool aligned16(const float* p, size_t d) { return d % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
unsigned warps_grid(size_t rows) { return static_cast<unsigned>((rows + 7) / 8); }

} // namespace

AssignRoute assign_route(size_t n, size_t k, size_t d) {
    if (!tc::enabled()) return AssignRoute::blocks;
    const double elements = static_cast<double>(n) * static_cast<double>(d);
    const double columns = static_cast<double>((k + 255) / 256 * 256);
    auto rounds = [&](size_t rows, size_t workers) { return static_cast<double>((n + rows * workers - 1) / (rows * workers)); };
    const double direct = tc::producer_stop() != 0 ? 1e9 : direct_assign_seconds(n, k, d);   // (a test of waits wants a kernel that waits)
    // the three-product kernel: five launches, two passes over the rows, 10 us per tile of 128 x 256 and 0.33 us per 16
    // dimensions of it
    const double blocks = d % 4 != 0 ? 1e9 : 4e-5 + elements * 8.0 / 5e12 + rounds(128, 148) * (columns / 256.0) * (1e-5 + static_cast<double>(d) / 16.0 * 3.3e-7);
    // the filter: six launches and a round trip, three passes (14 bytes an element), 2 n k d flop in tiles of 256 x 256
    const double filter = 8e-5 + elements * 14.0 / 5e12 + rounds(256, 74) * 74.0 * 256.0 * columns * std::max<double>(static_cast<double>(d), 128.0) / 5e14;
    // (rows are listed by 32-bit indices)
    if (d <= 16384 && k < (size_t{1} << 31) && n >= 256 && n < (size_t{1} << 32) && filter < direct && filter < blocks) return AssignRoute::filter;
    return direct < blocks ? AssignRoute::direct : AssignRoute::blocks;
}

void DirectAssign::run(const float* x, const float* y, size_t n, size_t k, size_t d, float* norms_x, float* norms_y, uint32_t* knn, float* dist, cudaStream_t stream) {
    const bool fresh = arrived_.get() == nullptr;
    DirectScratch s;
    s.norms_x = norms_x;
    s.norms_y = norms_y;
    s.keys = keys_.ensure(direct_key_count(n));
    s.counters = counters_.ensure(direct_counter_count(n));
    s.arrived = arrived_.ensure(1);
    if (fresh) SKM_CUDA(cudaMemsetAsync(s.arrived, 0, sizeof(uint32_t), stream));
    launch_direct_assign(x, y, n, k, d, s, knn, dist, stream);
}

void ExactAssign::centroids(const float* y, size_t k, float* norms_y, bool with_mean, cudaStream_t stream) {
    y_ = y;
    norms_y_ = norms_y;
    k_ = k;
    kp_ = (k + 255) / 256 * 256;
    float* mean = mean_.ensure(dp_);
    float* centred = centred_norms_.ensure(kp_);
    uint32_t* stats = stats_.ensure(kStats);
    __half* yh = yh_.ensure(k * dp_);
    sample_mean_kernel<<<with_mean ? static_cast<unsigned>((d_ + 63) / 64) : 1u, 64, 0, stream>>>(y, k, with_mean ? d_ : 0, mean, stats, n_listed_.ensure(2));
    SKM_LAUNCH_CHECK();
    if (aligned16(y, d_)) {
        centroid_norms_kernel<true><<<warps_grid(kp_), 256, 0, stream>>>(y, k, kp_, d_, mean, norms_y, centred, stats);
        SKM_LAUNCH_CHECK();
        centroid_fp16_kernel<true><<<warps_grid(k), 256, 0, stream>>>(y, k, d_, dp_, mean, stats, yh);
    } else {
        centroid_norms_kernel<false><<<warps_grid(kp_), 256, 0, stream>>>(y, k, kp_, d_, mean, norms_y, centred, stats);
        SKM_LAUNCH_CHECK();
        centroid_fp16_kernel<false><<<warps_grid(k), 256, 0, stream>>>(y, k, d_, dp_, mean, stats, yh);
    }
    SKM_LAUNCH_CHECK();
}

// (before: rows of the batch that have gone through the filter already)
void ExactAssign::convert(const float* x, size_t n, size_t before, float* norms_x, cudaStream_t stream) {
    auto* kernel = !aligned16(x, d_) ? row_fp16_kernel<false, 0> : d_ <= 512 ? row_fp16_kernel<true, 4> : d_ <= 1024 ? row_fp16_kernel<true, 8> : row_fp16_kernel<true, 0>;
    kernel<<<warps_grid(n), 256, 0, stream>>>(x, n, d_, dp_, mean_.get(), norms_x, xh_.get(), row_info_.get(), n_listed_.get(), before, n_listed_.get() + 1);
    SKM_LAUNCH_CHECK();
}

// Filter and decision of the n converted rows x.
void ExactAssign::search(const float* x, size_t first, size_t n, const AssignTile* tiles, size_t n_tiles, const float* norms_x, uint32_t* out_knn, float* out_dist,
                         cudaStream_t stream) {
    int device = 0, sms = 0;
    SKM_CUDA(cudaGetDevice(&device));
    SKM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    FilterParams p{};
    p.n = n;
    p.first = first;
    p.k = static_cast<uint32_t>(k_);
    p.k_blocks = static_cast<uint32_t>((dp_ + FK - 1) / FK);
    p.tiles = tiles;
    p.n_tiles = tiles ? n_tiles : (n + 255) / 256;
    p.info = row_info_.get();
    p.stats = stats_.get();
    p.norms_y = centred_norms_.get();
    p.cand = cand_.ensure(n);
    p.listed = listed_.get();
    p.n_listed = n_listed_.get();
    p.unseen = n_listed_.get() + 1;
    p.error = error_word();
    p.wait_limit = wait_limit();
    p.producer_stop = producer_stop();
    const CUtensorMap tx = make_half_tmap(xh_.get(), dp_, n, 128), ty = make_half_tmap(yh_.get(), dp_, k_, 128);
    const unsigned grid = static_cast<unsigned>(2 * std::min<size_t>(static_cast<size_t>(sms / 2), p.n_tiles));
    auto* kernel = tiles ? filter_tc_kernel<true> : filter_tc_kernel<false>;
    SKM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(F_SMEM_BYTES)));
    kernel<<<grid, F_THREADS, F_SMEM_BYTES, stream>>>(tx, ty, p);
    SKM_LAUNCH_CHECK();
    const unsigned deciders = std::min<unsigned>(warps_grid(n), static_cast<unsigned>(sms) * 3);
    auto* decide = aligned16(x, d_) && aligned16(y_, d_) ? decide_kernel<true> : decide_kernel<false>;
    decide<<<deciders, 256, 0, stream>>>(x, y_, n, k_, d_, norms_x, norms_y_, cand_.get(), out_knn, out_dist, p.error);
    SKM_LAUNCH_CHECK();
}

// A gigabyte of fp16 rows, in whole waves of row tiles.
size_t ExactAssign::rows_at_once(size_t n) const {
    const size_t wave = kWaveRows;
    return std::min(n, std::max(wave, ((size_t{1} << 30) / (dp_ * sizeof(__half))) / wave * wave));
}

void ExactAssign::give_back() {
    xh_.release();
    yh_.release();
    row_info_.release();
    cand_.release();
    listed_.release();
}

bool ExactAssign::begin(const float* y, size_t k, size_t d, size_t batch_rows, size_t piece_rows, float* norms_y, cudaStream_t stream) {
    d_ = d;
    dp_ = (d + 7) / 8 * 8;
    try {
        listed_.ensure(batch_rows);
        const size_t per = rows_at_once(piece_rows);
        xh_.ensure(per * dp_);
        row_info_.ensure(per);
        cand_.ensure(per);
        yh_.ensure(k * dp_);
    } catch (const OutOfMemory&) {
        give_back();
        return false;
    }
    centroids(y, k, norms_y, true, stream);
    return true;
}

void ExactAssign::rows(const float* x, size_t first, size_t n, float* norms_x, uint32_t* out_knn, float* out_dist, cudaStream_t stream) {
    const size_t per = rows_at_once(n), wave = kWaveRows;
    xh_.ensure(per * dp_);
    row_info_.ensure(per);
    // the first launch of a batch of several waves is short, to see what the list comes to; it takes what is left of the last wave
    // (from about a millisecond on, of which the launches are one or two percent)
    const bool long_enough = static_cast<double>(n) * static_cast<double>(kp_) * std::max<double>(static_cast<double>(dp_), 128.0) > 5e11 && n > 2 * wave;
    const size_t look = first == 0 && long_enough ? (n % wave >= kSeenRows ? n % wave : wave) : per;
    size_t cnt;
    for (size_t r0 = 0; r0 < n; r0 += cnt) {
        cnt = std::min({per, n - r0, r0 == 0 ? look : per});
        convert(x + r0 * d_, cnt, first + r0, norms_x + r0, stream);
        search(x + r0 * d_, first + r0, cnt, nullptr, 0, norms_x + r0, out_knn + r0, out_dist ? out_dist + r0 : nullptr, stream);
    }
}

void ExactAssign::begin_groups(const float* x, size_t n, size_t d, const float* y, size_t k, float* norms_x, cudaStream_t stream) {
    listed_.ensure(n);
    d_ = d;
    dp_ = (d + 7) / 8 * 8;
    xh_.ensure(n * dp_);
    row_info_.ensure(n);
    sample_mean_kernel<<<static_cast<unsigned>((d + 63) / 64), 64, 0, stream>>>(y, k, d, mean_.ensure(dp_), stats_.ensure(kStats), n_listed_.ensure(2));
    SKM_LAUNCH_CHECK();
    convert(x, n, 0, norms_x, stream);
}

void ExactAssign::assign_groups(const float* x, size_t n, const float* y, size_t k, const AssignTile* tiles, size_t n_tiles, const float* norms_x, float* norms_y, uint32_t* out_knn,
                                float* out_dist, cudaStream_t stream) {
    if (n_tiles == 0) return;
    centroids(y, k, norms_y, false, stream);
    SKM_CUDA(cudaMemsetAsync(cand_.ensure(n), 0xFF, sizeof(uint4) * n, stream));   // rows of no tile: nothing to decide
    search(x, 0, n, tiles, n_tiles, norms_x, out_knn, out_dist, stream);
    decide_listed_kernel<<<592, 256, 0, stream>>>(x, y, d_, norms_x, norms_y, tiles, n_tiles, listed_.get(), n_listed_.get(), out_knn, out_dist, error_word());
    SKM_LAUNCH_CHECK();
    const dim3 grid(static_cast<unsigned>(n_tiles), 256 / kListedRows);
    if (aligned16(x, d_) && aligned16(y, d_))
        decide_listed_tiles_kernel<true><<<grid, 256, 0, stream>>>(x, y, d_, norms_x, norms_y, tiles, n_tiles, cand_.get(), n_listed_.get(), out_knn, out_dist, error_word());
    else
        decide_listed_tiles_kernel<false><<<grid, 256, 0, stream>>>(x, y, d_, norms_x, norms_y, tiles, n_tiles, cand_.get(), n_listed_.get(), out_knn, out_dist, error_word());
    SKM_LAUNCH_CHECK();
}

size_t ExactAssign::settle(cudaStream_t stream) {
    uint32_t* host = n_listed_host_.ensure(1);
    launch_tell_word(n_listed_.get(), host, stream);
    SKM_CUDA(cudaStreamSynchronize(stream));
    return *host;
}

void ExactAssign::finish(const float* x_listed, size_t at, size_t count, uint32_t* out_knn, float* out_dist, cudaStream_t stream) {
    if (count == 0) return;
    float* norms = l_norms_.ensure(count + k_);
    uint32_t* knn = l_knn_.ensure(count);
    float* dist = l_dist_.ensure(count);
    // a pass of the three-product kernel walks all centroids in one block per 128 rows: 0.2 ms or more however few rows
    if (direct_assign_seconds(count, k_, d_) < 2e-4) {
        direct_.run(x_listed, y_, count, k_, d_, norms, norms + count, knn, dist, stream);
    } else {
        launch_row_sqnorms(x_listed, count, d_, d_, norms, stream);
        skmb::launch_assign_full(x_listed, y_, count, k_, d_, norms, norms_y_, knn, dist, l_top2_.ensure(count), stream, l_split_.ensure(2 * k_ * d_));
    }
    launch_scatter_u32(listed_.get() + at, l_knn_.get(), out_knn, count, stream);
    if (out_dist) launch_scatter_u32(listed_.get() + at, reinterpret_cast<const uint32_t*>(l_dist_.get()), reinterpret_cast<uint32_t*>(out_dist), count, stream);
}

size_t ExactAssign::settle_on_device(const float* x_batch, uint32_t* out_knn, float* out_dist, cudaStream_t stream) {
    const size_t total = settle(stream);
    size_t per = std::max<size_t>(1, (size_t{1} << 30) / (sizeof(float) * d_)), count;   // (a gigabyte)
    for (size_t at = 0; at < total; at += count) {
        count = std::min(per, total - at);
        float* xl = nullptr;
        try {
            xl = l_rows_.ensure(count * d_);
        } catch (const OutOfMemory&) {
            if (count <= 1024) throw;
            per = count / 8;   // (smaller steps then)
            count = 0;
            continue;
        }
        gather_listed_rows_kernel<<<warps_grid(count), 256, 0, stream>>>(x_batch, listed_.get() + at, count, d_, xl);
        SKM_LAUNCH_CHECK();
        finish(xl, at, count, out_knn, out_dist, stream);
    }
    return total;
}

} // namespace skmb
