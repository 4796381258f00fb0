// Exact assignment of few rows, or to few centroids, in fp32 on all SMs.
//
// The tensor-core kernels give a block to 128 or 256 rows and let it walk all centroids: one query against 1000 centroids
// of 768 dimensions kept one SM busy for 100 us and the others idle, and their passes around it (conversion, decision) cost
// 60 us of launches and streams whatever the size.  Here the pairs themselves are divided:
//   up to 8 rows   a warp per centroid, the rows in shared memory; bound by the centroids' bytes from L2 or HBM;
//   more           64 x 64 tiles of rows x centroids, 4 x 4 or 8 x 4 per thread, bound by reads of shared memory: 15 - 20 T multiply-adds per second.
// Distances are ||x||^2 + ||y||^2 - 2 x.y, the smallest wins, the lower index on a tie, clamped at zero when stored.
#include <cfloat>

#include "common.cuh"
#include "device_utils.cuh"

namespace skmb {

namespace {

constexpr int kQueryRows = 8;
constexpr int kQueryBlocks = 1184;               // at most: eight per SM
constexpr size_t kQuerySmem = 48 * 1024;
constexpr int kCell = 64;                        // rows and centroids of a tile

// Sum over the row in the order of row_sqnorms_kernel.
template <bool VEC, class F>
__device__ __forceinline__ void for_columns(size_t d, int lane, F f) {
    if (VEC)
        for (size_t j = static_cast<size_t>(lane) * 4; j < d; j += 128) f(j);
    else
        for (size_t j = lane; j < d; j += 32) f(j);
}

// Every block leaves its smallest keys in `partial`; the last one to finish reduces them.  *arrived is zero before and after.
template <bool VEC, int ROWS>
__global__ void __launch_bounds__(256) query_kernel(const float* __restrict__ x, const float* __restrict__ y, int n, size_t k, size_t d, unsigned long long* __restrict__ partial,
                                                    uint32_t* __restrict__ arrived, uint32_t* __restrict__ knn, float* __restrict__ dist) {
    extern __shared__ __align__(16) float rows[];   // n x d
    __shared__ float row_norm[kQueryRows];
    __shared__ unsigned long long keys[8][kQueryRows];
    __shared__ bool last;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (size_t i = threadIdx.x; i < static_cast<size_t>(n) * d; i += 256) rows[i] = x[i];
    __syncthreads();
    if (warp < n) {
        float s = 0.f;
        const float* r = rows + static_cast<size_t>(warp) * d;
        for_columns<VEC>(d, lane, [&](size_t j) {
#pragma unroll
            for (int q = 0; q < (VEC ? 4 : 1); ++q) s = fmaf(r[j + q], r[j + q], s);
        });
        s = warp_sum(s);
        if (lane == 0) row_norm[warp] = s;
    }
    __syncthreads();
    unsigned long long best[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) best[r] = ~0ull;
    for (size_t c = static_cast<size_t>(blockIdx.x) * 8 + warp; c < k; c += static_cast<size_t>(gridDim.x) * 8) {
        const float* __restrict__ yr = y + c * d;
        float ny = 0.f, s[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) s[r] = 0.f;
        if (VEC) {
#pragma unroll 4
            for (size_t j = static_cast<size_t>(lane) * 4; j < d; j += 128) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(yr + j));
                ny = fmaf(v.x, v.x, ny); ny = fmaf(v.y, v.y, ny); ny = fmaf(v.z, v.z, ny); ny = fmaf(v.w, v.w, ny);
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    if (r < n) {
                        const float4 u = *reinterpret_cast<const float4*>(rows + static_cast<size_t>(r) * d + j);
                        s[r] = fmaf(u.x, v.x, s[r]); s[r] = fmaf(u.y, v.y, s[r]); s[r] = fmaf(u.z, v.z, s[r]); s[r] = fmaf(u.w, v.w, s[r]);
                    }
                }
            }
        } else {
#pragma unroll 4
            for (size_t j = lane; j < d; j += 32) {
                const float v = __ldg(yr + j);
                ny = fmaf(v, v, ny);
#pragma unroll
                for (int r = 0; r < ROWS; ++r)
                    if (r < n) s[r] = fmaf(rows[static_cast<size_t>(r) * d + j], v, s[r]);
            }
        }
        ny = warp_sum(ny);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if (r < n) {
                const unsigned long long key = pair_key(fmaf(-2.0f, warp_sum(s[r]), row_norm[r]) + ny, static_cast<uint32_t>(c));
                best[r] = key < best[r] ? key : best[r];
            }
        }
    }
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) keys[warp][r] = best[r];
    }
    __syncthreads();
    if (threadIdx.x < n) {
        unsigned long long b = keys[0][threadIdx.x];
        for (int w = 1; w < 8; ++w) b = keys[w][threadIdx.x] < b ? keys[w][threadIdx.x] : b;
        partial[static_cast<size_t>(blockIdx.x) * kQueryRows + threadIdx.x] = b;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(arrived, 1u) + 1 == gridDim.x;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (warp < n) {
        unsigned long long b = ~0ull;
        for (uint32_t i = lane; i < gridDim.x; i += 32) {
            const unsigned long long key = __ldcg(partial + static_cast<size_t>(i) * kQueryRows + warp);
            b = key < b ? key : b;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, b, o);
            b = other < b ? other : b;
        }
        if (lane == 0) store_answer(b, warp, knn, dist);
    }
    if (threadIdx.x == 0) *arrived = 0u;
}

// Squared norms of both sides (a warp per row), keys and row-tile counters at their starting values.
template <bool VEC>
__global__ void __launch_bounds__(256) tile_prepare_kernel(const float* __restrict__ x, const float* __restrict__ y, size_t n, size_t k, size_t d, float* __restrict__ norms_x,
                                                           float* __restrict__ norms_y, unsigned long long* __restrict__ keys, uint32_t* __restrict__ counters, size_t row_tiles) {
    const size_t i = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= n + k) return;
    const float* row = i < n ? x + i * d : y + (i - n) * d;
    float s = 0.f;
    for_columns<VEC>(d, lane, [&](size_t j) {
        if (VEC) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(row + j));
            s = fmaf(v.x, v.x, s); s = fmaf(v.y, v.y, s); s = fmaf(v.z, v.z, s); s = fmaf(v.w, v.w, s);
        } else {
            const float v = __ldg(row + j);
            s = fmaf(v, v, s);
        }
    });
    s = warp_sum(s);
    if (lane != 0) return;
    if (i < n) {
        norms_x[i] = s;
        keys[i] = ~0ull;
        if (i < row_tiles) counters[i] = 0u;
    } else {
        norms_y[i - n] = s;
    }
}

// A thread's part of a piece of D columns of rows [row0, row0 + 64): four columns of a row from `at` on.
template <bool VEC, int D>
__device__ __forceinline__ float4 load_cell(const float* __restrict__ m, size_t row0, size_t rows, size_t d, size_t j0, int at) {
    const size_t r = row0 + at + threadIdx.x / (D / 4), j = j0 + 4 * (threadIdx.x % (D / 4));
    if (r >= rows || j >= d) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float* p = m + r * d + j;
    if (VEC) return __ldg(reinterpret_cast<const float4*>(p));
    float4 v = make_float4(__ldg(p), 0.f, 0.f, 0.f);
    if (j + 1 < d) v.y = __ldg(p + 1);
    if (j + 2 < d) v.z = __ldg(p + 2);
    if (j + 3 < d) v.w = __ldg(p + 3);
    return v;
}

// In shared memory row r of column q lies at r ^ (q & 28): neither the reads nor, with 32 columns, the transposing stores have bank conflicts.
template <int D>
__device__ __forceinline__ void store_cell(float (*cell)[kCell], int at, float4 v) {
    const int q = 4 * (threadIdx.x % (D / 4)), r = (at + static_cast<int>(threadIdx.x / (D / 4))) ^ q;
    cell[q][r] = v.x; cell[q + 1][r] = v.y; cell[q + 2][r] = v.z; cell[q + 3][r] = v.w;
}

// A step costs at least the latency of a load from L2, which the step before covers: 32 columns take half as many as 16 (1000 x 1000 x 768:
// 55 us, with 16 columns 64; 3000 x 3000 x 384: 189, 209; 20 x 1000 x 768: 30, 38; 5000 x 300 x 128: 18.5, 19.8).
// R x 4 products a thread, D columns a step.
template <bool VEC, int R, int D>
__global__ void __launch_bounds__(1024 / R) tile_kernel(const float* __restrict__ x, const float* __restrict__ y, size_t n, size_t k, size_t d, const float* __restrict__ norms_x,
                                                   const float* __restrict__ norms_y, unsigned long long* __restrict__ keys, uint32_t* __restrict__ counters,
                                                   uint32_t* __restrict__ knn, float* __restrict__ dist) {
    constexpr int kAtOnce = 4096 / (R * D), kParts = kCell / kAtOnce;   // rows that a load takes, loads for a piece
    __shared__ __align__(16) float sx[2][D][kCell], sy[2][D][kCell];
    __shared__ bool last;
    const size_t row0 = static_cast<size_t>(blockIdx.y) * kCell, col0 = static_cast<size_t>(blockIdx.x) * kCell;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[R][4] = {};
    float4 vx[kParts], vy[kParts];
#pragma unroll
    for (int h = 0; h < kParts; ++h) {
        vx[h] = load_cell<VEC, D>(x, row0, n, d, 0, h * kAtOnce);
        vy[h] = load_cell<VEC, D>(y, col0, k, d, 0, h * kAtOnce);
    }
    int buf = 0;
    for (size_t j0 = 0; j0 < d; j0 += D, buf ^= 1) {
#pragma unroll
        for (int h = 0; h < kParts; ++h) {
            store_cell<D>(sx[buf], h * kAtOnce, vx[h]);
            store_cell<D>(sy[buf], h * kAtOnce, vy[h]);
        }
        __syncthreads();
        if (j0 + D < d) {
#pragma unroll
            for (int h = 0; h < kParts; ++h) {
                vx[h] = load_cell<VEC, D>(x, row0, n, d, j0 + D, h * kAtOnce);
                vy[h] = load_cell<VEC, D>(y, col0, k, d, j0 + D, h * kAtOnce);
            }
        }
#pragma unroll
        for (int half = 0; half < D; half += 16) {
            if (half > 0 && j0 + half >= d) break;   // (zeros)
#pragma unroll
            for (int q = half; q < half + 16; ++q) {
                float av[R];
#pragma unroll
                for (int r = 0; r < R; r += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(&sx[buf][q][(ty * R + r) ^ (q & 28)]);
                    av[r] = a.x; av[r + 1] = a.y; av[r + 2] = a.z; av[r + 3] = a.w;
                }
                const float4 b = *reinterpret_cast<const float4*>(&sy[buf][q][(tx * 4) ^ (q & 28)]);
                const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(av[r], bv[c], acc[r][c]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const size_t row = row0 + ty * R + r;
        unsigned long long best = ~0ull;
        if (row < n) {
            const float nx = norms_x[row];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const size_t col = col0 + tx * 4 + c;
                if (col < k) {
                    const unsigned long long key = pair_key(fmaf(-2.0f, acc[r][c], nx) + __ldg(norms_y + col), static_cast<uint32_t>(col));
                    best = key < best ? key : best;
                }
            }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
            best = other < best ? other : best;
        }
        if (tx == 0 && row < n) {
            if (gridDim.x == 1) store_answer(best, row, knn, dist);
            else atomicMin(keys + row, best);
        }
    }
    if (gridDim.x == 1) return;
    // the last tile of a row of tiles stores the answers
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counters + blockIdx.y, 1u) + 1 == gridDim.x;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < kCell && row0 + threadIdx.x < n) store_answer(__ldcg(keys + row0 + threadIdx.x), row0 + threadIdx.x, knn, dist);
}

template <bool VEC>
void launch_query(const float* x, const float* y, size_t n, size_t k, size_t d, const DirectScratch& s, uint32_t* knn, float* dist, cudaStream_t stream) {
    const unsigned grid = static_cast<unsigned>(std::min<size_t>((k + 7) / 8, kQueryBlocks));
    const size_t smem = n * d * sizeof(float);
    const int rows = static_cast<int>(n);
    if (n == 1) query_kernel<VEC, 1><<<grid, 256, smem, stream>>>(x, y, rows, k, d, s.keys, s.arrived, knn, dist);
    else if (n == 2) query_kernel<VEC, 2><<<grid, 256, smem, stream>>>(x, y, rows, k, d, s.keys, s.arrived, knn, dist);
    else if (n <= 4) query_kernel<VEC, 4><<<grid, 256, smem, stream>>>(x, y, rows, k, d, s.keys, s.arrived, knn, dist);
    else query_kernel<VEC, kQueryRows><<<grid, 256, smem, stream>>>(x, y, rows, k, d, s.keys, s.arrived, knn, dist);
    SKM_LAUNCH_CHECK();
}

template <bool VEC>
void launch_tiles(const float* x, const float* y, size_t n, size_t k, size_t d, const DirectScratch& s, uint32_t* knn, float* dist, cudaStream_t stream) {
    const size_t row_tiles = (n + kCell - 1) / kCell, col_tiles = (k + kCell - 1) / kCell;
    tile_prepare_kernel<VEC><<<static_cast<unsigned>((n + k + 7) / 8), 256, 0, stream>>>(x, y, n, k, d, s.norms_x, s.norms_y, s.keys, s.counters, row_tiles);
    SKM_LAUNCH_CHECK();
    // R + 4 reads of shared memory for 4 R products, which is what bounds the tiles: with 8 x 4 a thread they take 0.75 of the time, but
    // a block of its own on an SM has too few warps then to cover their latency.  600 x 20 x 64 (10 tiles): 5.1 us with 4 x 4 a thread, 6.5 with 8 x 4;
    // 5000 x 300 x 128 (395): 18.5 and 16.8; 1000 x 1000 x 768 (256): 55 and 51; 3000 x 3000 x 384: 189 and 172.
    const dim3 grid(static_cast<unsigned>(col_tiles), static_cast<unsigned>(row_tiles));
    // Up to 64 columns the tiles are mostly ends, which many blocks on an SM overlap: those of 16 columns a step take the least of it (5339 x 8002 x 32:
    // 141 us, 154 with 32 columns, 179 with 8 x 4 as well).
    if (row_tiles * col_tiles <= static_cast<size_t>(sm_count())) tile_kernel<VEC, 4, 32><<<grid, 256, 0, stream>>>(x, y, n, k, d, s.norms_x, s.norms_y, s.keys, s.counters, knn, dist);
    else if (d <= 64) tile_kernel<VEC, 4, 16><<<grid, 256, 0, stream>>>(x, y, n, k, d, s.norms_x, s.norms_y, s.keys, s.counters, knn, dist);
    else tile_kernel<VEC, 8, 32><<<grid, 128, 0, stream>>>(x, y, n, k, d, s.norms_x, s.norms_y, s.keys, s.counters, knn, dist);
    SKM_LAUNCH_CHECK();
}

} // namespace

size_t direct_key_count(size_t n) { return std::max<size_t>(n, static_cast<size_t>(kQueryBlocks) * kQueryRows); }
size_t direct_counter_count(size_t n) { return (n + kCell - 1) / kCell; }

double direct_assign_seconds(size_t n, size_t k, size_t d) { return 1.2e-5 + static_cast<double>(n) * static_cast<double>(k) * static_cast<double>(d) / 1.3e13; }

bool direct_assign_counts_arrivals(size_t n, size_t d) { return n <= kQueryRows && n * d * sizeof(float) <= kQuerySmem - 4096; }

void launch_direct_assign(const float* x, const float* y, size_t n, size_t k, size_t d, const DirectScratch& s, uint32_t* knn, float* dist, cudaStream_t stream) {
    if (n == 0 || k == 0) return;
    const bool vec = d % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
    if (direct_assign_counts_arrivals(n, d)) {
        if (vec) launch_query<true>(x, y, n, k, d, s, knn, dist, stream);
        else launch_query<false>(x, y, n, k, d, s, knn, dist, stream);
        return;
    }
    // row tiles are on grid.y (limit 65535)
    const size_t per = std::min(n, size_t{65535} * kCell);
    for (size_t r0 = 0; r0 < n; r0 += per) {
        DirectScratch t = s;
        t.norms_x += r0;
        t.keys += r0;
        const size_t cnt = std::min(per, n - r0);
        if (vec) launch_tiles<true>(x + r0 * d, y, cnt, k, d, t, knn + r0, dist ? dist + r0 : nullptr, stream);
        else launch_tiles<false>(x + r0 * d, y, cnt, k, d, t, knn + r0, dist ? dist + r0 : nullptr, stream);
    }
}

} // namespace skmb
