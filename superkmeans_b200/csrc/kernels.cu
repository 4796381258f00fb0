// CUDA kernels of the k-means hot path (sm_100a) and their launchers.
//
//   rotation / un-rotation      gemm_nt_kernel              (reference: adsampling.h:191-215, :273-298)
//   row norms                   row_sqnorms_kernel          (superkmeans.h:1147-1171)
//   exact assignment            assign_full_kernel          (batch_computers.h:104-171)
//   pruned assignment           assign_pruned_kernel        (batch_computers.h:297-409, pdxearch.h:118-327)
//   centroid update             radix sort + segmented sum  (superkmeans.h:729-765, :973-981)
//   consolidation               scale / split ops / pdxify / shift (superkmeans.h:936-998, layout.h:155-232)
#include "common.cuh"
#include "device_utils.cuh"
#include "gemm_simt.cuh"
#include "kernels_tc.cuh"

#include <atomic>
#include <cfloat>

namespace skmb {

// Number of kernels this library has launched in the process (reported by skm_kernel_launches).
static std::atomic<unsigned long long> g_kernel_launches{0};
unsigned long long kernel_launch_count() { return g_kernel_launches.load(); }
void note_kernel_launch() { g_kernel_launches.fetch_add(1, std::memory_order_relaxed); }
// =================================================================================================
// Row squared norms over the first `upto` columns: one warp per row.
// =================================================================================================
__global__ void __launch_bounds__(256) row_sqnorms_kernel(const float* __restrict__ x, size_t n, size_t ld, size_t upto, float* __restrict__ out) {
    const size_t row = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (row >= n) return;
    const int lane = threadIdx.x & 31;
    const float* p = x + row * ld;
    float acc = 0.f;
    const bool vec = (ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    const size_t upto4 = vec ? (upto & ~size_t{3}) : 0;
    for (size_t j = static_cast<size_t>(lane) * 4; j < upto4; j += 128) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(p + j));
        acc = fmaf(v.x, v.x, acc);
        acc = fmaf(v.y, v.y, acc);
        acc = fmaf(v.z, v.z, acc);
        acc = fmaf(v.w, v.w, acc);
    }
    for (size_t j = upto4 + lane; j < upto; j += 32) {
        const float v = __ldg(p + j);
        acc = fmaf(v, v, acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) out[row] = acc;
}

void launch_row_sqnorms(const float* x, size_t n, size_t ld, size_t upto, float* out, cudaStream_t stream) {
    if (n == 0) return;
    const unsigned grid = static_cast<unsigned>((n + 7) / 8);
    row_sqnorms_kernel<<<grid, 256, 0, stream>>>(x, n, ld, upto, out);
    SKM_LAUNCH_CHECK();
}

// =================================================================================================
// NT GEMM with a plain store epilogue (rotation, un-rotation).
// =================================================================================================
__global__ void __launch_bounds__(256, 2) gemm_nt_kernel(
    const float* __restrict__ a, size_t lda, const float* __restrict__ b, size_t ldb, float* __restrict__ out, size_t ldo, size_t n, size_t n_out, size_t k_dim
) {
    __shared__ GemmSmem smem;
    const size_t row0 = static_cast<size_t>(blockIdx.x) * kTileM;
    const size_t col0 = static_cast<size_t>(blockIdx.y) * kTileN;
    const int m_valid = static_cast<int>(min(static_cast<size_t>(kTileM), n - row0));
    const int n_valid = static_cast<int>(min(static_cast<size_t>(kTileN), n_out - col0));
    float acc[8][8];
    gemm_tile_nt(a + row0 * lda, lda, m_valid, b + col0 * ldb, ldb, n_valid, static_cast<int>(k_dim), smem, acc);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const bool vec = (ldo % 4 == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = tile_row_of(ty, i);
        if (r >= m_valid) continue;
        float* orow = out + (row0 + r) * ldo + col0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = tile_col_of(tx, h * 4);
            if (vec && c + 3 < n_valid) {
                *reinterpret_cast<float4*>(orow + c) = make_float4(acc[i][h * 4 + 0], acc[i][h * 4 + 1], acc[i][h * 4 + 2], acc[i][h * 4 + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (c + j < n_valid) orow[c + j] = acc[i][h * 4 + j];
            }
        }
    }
}

__global__ void __launch_bounds__(256, 4) gemm_nt_small_kernel(
    const float* __restrict__ a, size_t lda, const float* __restrict__ b, size_t ldb, float* __restrict__ out, size_t ldo, size_t n, size_t n_out, size_t k_dim
) {
    __shared__ GemmSmem32 smem;
    const size_t row0 = static_cast<size_t>(blockIdx.x) * 32, col0 = static_cast<size_t>(blockIdx.y) * kTileN;
    const int m_valid = static_cast<int>(min(size_t{32}, n - row0));
    const int n_valid = static_cast<int>(min(static_cast<size_t>(kTileN), n_out - col0));
    float acc[4][4];
    gemm_tile32_nt<true, false>(a + row0 * lda, lda, m_valid, nullptr, b + col0 * ldb, ldb, n_valid, static_cast<int>(k_dim), smem, acc);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (warp * 4 + i < m_valid && lane + 32 * j < n_valid) out[(row0 + warp * 4 + i) * ldo + col0 + lane + 32 * j] = acc[i][j];
}

int sm_count() {
    int device = 0, sms = 0;
    SKM_CUDA(cudaGetDevice(&device));
    SKM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    return std::max(sms, 1);
}

void launch_gemm_nt(const float* a, size_t lda, const float* b, size_t ldb, float* out, size_t ldo, size_t n, size_t n_out, size_t k_dim, cudaStream_t stream) {
    if (n == 0 || n_out == 0) return;
    // Tensor cores when TMA can address both operands: the rotation kernel cuts the accumulation into four chains summed
    // in fp32 registers, which keeps the result at the accuracy of this file's fp32 kernel (a single chain in tensor
    // memory would be ~1e-5 off, and rotated rows feed every later distance).
    if (tc::eligible(a, lda, b, ldb) && ldb == k_dim && k_dim >= 32) {
        tc::launch_rotate(a, lda, b, out, ldo, n, n_out, k_dim, stream);
        return;
    }
    // The point dimension is on grid.x (limit 2^31-1); output columns on grid.y.
    dim3 grid(static_cast<unsigned>((n + kTileM - 1) / kTileM), static_cast<unsigned>((n_out + kTileN - 1) / kTileN));
    // Few tiles take the time of one, which is shorter with 32 rows; from a tile for every second SM on they are no faster.  1000 x 355 by
    // 355 x 355 (24 tiles): 49 us with 128 rows, 20 with 32; 3000 rows (72): 51 and 35; 6000 (141): 52 and 66.
    if (2 * static_cast<size_t>(grid.x) * grid.y <= static_cast<size_t>(sm_count())) {
        grid.x = static_cast<unsigned>((n + 31) / 32);
        gemm_nt_small_kernel<<<grid, 256, 0, stream>>>(a, lda, b, ldb, out, ldo, n, n_out, k_dim);
    } else {
        gemm_nt_kernel<<<grid, 256, 0, stream>>>(a, lda, b, ldb, out, ldo, n, n_out, k_dim);
    }
    SKM_LAUNCH_CHECK();
}

// Rows that 16-byte loads cannot address have the fp32 tiles otherwise, whose sums of up to 64 products are closer to 64 bits than those of 22-bit
// halves (rms error relative to a row's length: d = 33: 1.8e-8 against 2.0e-8, 50: 1.8e-8 and 1.9e-8, 57: 1.8e-8 both, 101: 1.8e-8 and 1.3e-8, 1023:
// 1.8e-8 and 0.5e-8).  Aligned rows have the tf32 kernel otherwise: 3.4e-8 (d = 32) to 7.0e-8 (1536) against 1.9e-8 to 0.4e-8.
void launch_rotate_to_assign(const float* a, size_t lda, const float* b, float* out, size_t ldo, size_t n, size_t n_out, size_t k_dim, cudaStream_t stream) {
    const bool addressable = lda % 4 == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
    if (n != 0 && n_out != 0 && tc::enabled() && k_dim >= (addressable ? 32 : 64)) {
        try {
            tc::launch_rotate_halves(a, lda, b, out, ldo, n, n_out, k_dim, stream);
            return;
        } catch (const OutOfMemory&) {   // (of its scratch, before anything is launched; the fp32 tiles have none)
        }
    }
    launch_gemm_nt(a, lda, b, k_dim, out, ldo, n, n_out, k_dim, stream);
}

__global__ void transpose_square_kernel(const float* __restrict__ in, float* __restrict__ out, size_t n) {
    __shared__ float t[32][33];
    const size_t bx = static_cast<size_t>(blockIdx.x) * 32, by = static_cast<size_t>(blockIdx.y) * 32;
    for (int r = threadIdx.y; r < 32; r += 8) {
        const size_t i = by + r, j = bx + threadIdx.x;
        if (i < n && j < n) t[r][threadIdx.x] = in[i * n + j];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8) {
        const size_t i = bx + r, j = by + threadIdx.x;
        if (i < n && j < n) out[i * n + j] = t[threadIdx.x][r];
    }
}

void launch_transpose_square(const float* in, float* out, size_t n, cudaStream_t stream) {
    dim3 grid(static_cast<unsigned>((n + 31) / 32), static_cast<unsigned>((n + 31) / 32));
    transpose_square_kernel<<<grid, dim3(32, 8), 0, stream>>>(in, out, n);
    SKM_LAUNCH_CHECK();
}

// =================================================================================================
// Exact assignment.  One CTA owns 128 points and walks all centroid tiles; distances never leave
// registers.  Tie rules of the reference: first minimum inside a batch of 1024 centroids, a later
// batch wins only with a strictly smaller distance than the stored (clamped at 0) one.
// =================================================================================================
__global__ void __launch_bounds__(256, 2) assign_full_kernel(
    const float* __restrict__ x, const float* __restrict__ y, size_t n, size_t k, size_t d, const float* __restrict__ norms_x, const float* __restrict__ norms_y,
    uint32_t* __restrict__ out_knn, float* __restrict__ out_dist
) {
    __shared__ GemmSmem smem;
    const size_t row0 = static_cast<size_t>(blockIdx.x) * kTileM;
    const int m_valid = static_cast<int>(min(static_cast<size_t>(kTileM), n - row0));
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;

    __shared__ float s_nx[kTileM], s_best[kTileM];
    __shared__ uint32_t s_bidx[kTileM];
    if (threadIdx.x < kTileM) {
        s_nx[threadIdx.x] = (static_cast<int>(threadIdx.x) < m_valid) ? norms_x[row0 + threadIdx.x] : 0.f;
        s_best[threadIdx.x] = FLT_MAX;
        s_bidx[threadIdx.x] = 0;
    }
    float bmin[8];
    uint32_t bminidx[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        bmin[i] = FLT_MAX;
        bminidx[i] = 0;
    }
    __syncthreads();
    float acc[8][8];
    for (size_t col0 = 0; col0 < k; col0 += kTileN) {
        const int n_valid = static_cast<int>(min(static_cast<size_t>(kTileN), k - col0));
        gemm_tile_nt(x + row0 * d, d, m_valid, y + col0 * d, d, n_valid, static_cast<int>(d), smem, acc);
        float nyr[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = tile_col_of(tx, j);
            nyr[j] = (c < n_valid) ? __ldg(norms_y + col0 + c) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float nxv = s_nx[tile_row_of(ty, i)];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int c = tile_col_of(tx, j);
                if (c < n_valid) {
                    const float dist = fmaf(-2.0f, acc[i][j], nxv) + nyr[j];
                    if (dist < bmin[i]) {
                        bmin[i] = dist;
                        bminidx[i] = static_cast<uint32_t>(col0 + c);
                    }
                }
            }
        }
        const bool batch_end = ((col0 + kTileN) % kChunk == 0) || (col0 + kTileN >= k);
        if (batch_end) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float v = bmin[i];
                uint32_t vi = bminidx[i];
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
                    const uint32_t oi = __shfl_xor_sync(0xffffffffu, vi, o);
                    if (ov < v || (ov == v && oi < vi)) {
                        v = ov;
                        vi = oi;
                    }
                }
                if (tx == 0) {
                    const int r = tile_row_of(ty, i);
                    if (v < s_best[r]) {
                        s_best[r] = fmaxf(0.0f, v);
                        s_bidx[r] = vi;
                    }
                }
                bmin[i] = FLT_MAX;
                bminidx[i] = 0;
            }
        }
    }
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < m_valid) {
        out_knn[row0 + threadIdx.x] = s_bidx[threadIdx.x];
        out_dist[row0 + threadIdx.x] = s_best[threadIdx.x];
    }
}

void launch_assign_full(const float* x, const float* y, size_t n, size_t k, size_t d, const float* norms_x, const float* norms_y, uint32_t* out_knn, float* out_dist, uint2* top2_scratch, cudaStream_t stream, float* y_split) {
    if (n == 0) return;
    if (top2_scratch && tc::eligible(x, d, y, d)) {
        tc::launch_assign_full(x, y, n, k, d, norms_x, norms_y, out_knn, out_dist, top2_scratch, stream, y_split);
        return;
    }
    const unsigned grid = static_cast<unsigned>((n + kTileM - 1) / kTileM);
    assign_full_kernel<<<grid, 256, 0, stream>>>(x, y, n, k, d, norms_x, norms_y, out_knn, out_dist);
    SKM_LAUNCH_CHECK();
}

// =================================================================================================
// Pruned assignment.
//
// A persistent CTA takes tiles of 128 points.  For every chunk of 1024 centroids it
//   1. computes the partial dot products over the first d' dimensions, 128 centroids at a time,
//      and turns them into partial distances ||x||'^2 + ||c||'^2 - 2 x.c;
//   2. keeps only (point, centroid) pairs whose partial distance is below best * ratio[d'] (the
//      ADSampling test); survivors go to a per-CTA candidate list in global scratch;
//   3. walks the survivors, eight lanes per pair: adds the horizontal dimensions 64 at a time from
//      the PDX-blocked centroid copy, re-testing against best * ratio[dims seen] after each block,
//      then the remaining vertical dimensions [d', vertical_d) from the auxiliary row-major copy,
//      and finally competes for the per-point minimum of the chunk;
//   4. lowers `best` of each point before the next chunk.
// `best` is constant inside a chunk, so pairs are independent of each other.  The pair formed with
// the point's previous centroid is held back until the survivor count of the chunk is known: when
// it is the only survivor the chunk is skipped for that point, as the reference does.
// =================================================================================================
constexpr int kListCap = kTileM * kChunk;

struct PrunedRowState {
    float thr[kTileM];
    float best[kTileM];
    uint32_t bestidx[kTileM];
    uint32_t prev[kTileM];
    float nxs[kTileM];
    uint32_t cnt[kTileM];
    uint32_t npc[kTileM];
    float prev_pd[kTileM];
    uint32_t prev_flag[kTileM];
    unsigned long long chunk_key[kTileM];
    uint32_t active[kTileM];
    uint32_t list_count;
};

template <bool VEC>
__device__ __forceinline__ void pruned_process_pair(
    const PrunedParams& p, PrunedRowState& st, size_t row0, int r, uint32_t cl, float pd, size_t chunk, size_t c0, size_t cs, int gl, uint32_t gmask
) {
    const size_t c = c0 + cl;
    const float b = st.best[r];
    const float* __restrict__ q = p.x + (row0 + r) * p.d;
    uint32_t dims = p.partial_d;
    bool alive = true;
    const size_t n_hblocks = p.horizontal_d / kHBlock;
    const float* __restrict__ blk = p.y_pdx + chunk * kChunk * p.d + static_cast<size_t>(p.vertical_d) * cs + static_cast<size_t>(cl) * kHBlock;
    for (size_t hb = 0; hb < n_hblocks; ++hb) {
        const float* __restrict__ cp = blk + hb * cs * kHBlock + gl * 8;
        const float* __restrict__ qp = q + p.vertical_d + hb * kHBlock + gl * 8;
        float s = 0.f;
        if (VEC) {
            const float4 c0v = __ldg(reinterpret_cast<const float4*>(cp));
            const float4 c1v = __ldg(reinterpret_cast<const float4*>(cp + 4));
            const float4 q0v = __ldg(reinterpret_cast<const float4*>(qp));
            const float4 q1v = __ldg(reinterpret_cast<const float4*>(qp + 4));
            float t;
            t = q0v.x - c0v.x; s = fmaf(t, t, s);
            t = q0v.y - c0v.y; s = fmaf(t, t, s);
            t = q0v.z - c0v.z; s = fmaf(t, t, s);
            t = q0v.w - c0v.w; s = fmaf(t, t, s);
            t = q1v.x - c1v.x; s = fmaf(t, t, s);
            t = q1v.y - c1v.y; s = fmaf(t, t, s);
            t = q1v.z - c1v.z; s = fmaf(t, t, s);
            t = q1v.w - c1v.w; s = fmaf(t, t, s);
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float t = __ldg(qp + e) - __ldg(cp + e);
                s = fmaf(t, t, s);
            }
        }
        s += __shfl_xor_sync(gmask, s, 4);
        s += __shfl_xor_sync(gmask, s, 2);
        s += __shfl_xor_sync(gmask, s, 1);
        pd += s;
        dims += kHBlock;
        if (!(pd < b * __ldg(p.ratios + dims))) {
            alive = false;
            break;
        }
    }
    if (alive && p.partial_d < p.vertical_d) {
        const float* __restrict__ cp = p.y_aux + c * p.vertical_d + p.partial_d;
        const float* __restrict__ qp = q + p.partial_d;
        const uint32_t len = p.vertical_d - p.partial_d;
        float s = 0.f;
        for (uint32_t e = gl; e < len; e += 8) {
            const float t = __ldg(qp + e) - __ldg(cp + e);
            s = fmaf(t, t, s);
        }
        s += __shfl_xor_sync(gmask, s, 4);
        s += __shfl_xor_sync(gmask, s, 2);
        s += __shfl_xor_sync(gmask, s, 1);
        pd += s;
        if (!(pd < b)) alive = false;  // ratio[d] == 1
    }
    if (alive && gl == 0) {
        const unsigned long long key = (static_cast<unsigned long long>(float_to_ordered(pd)) << 32) | static_cast<unsigned long long>(c);
        atomicMin(&st.chunk_key[r], key);
    }
}

template <bool VEC>
__global__ void __launch_bounds__(256, 2) assign_pruned_kernel(const PrunedParams p) {
    __shared__ GemmSmem smem;
    __shared__ PrunedRowState st;
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int lane = tid & 31, warp = tid >> 5;
    const int g = tid >> 3, gl = tid & 7;
    const uint32_t gmask = 0xFFu << ((lane >> 3) * 8);
    uint2* __restrict__ list = p.scratch + static_cast<size_t>(blockIdx.x) * kListCap;
    const size_t n_tiles = (p.n + kTileM - 1) / kTileM;
    const size_t n_chunks = (p.k + kChunk - 1) / kChunk;
    const float ratio_first = __ldg(p.ratios + p.partial_d);

    for (size_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const size_t row0 = tile * kTileM;
        const int m_valid = static_cast<int>(min(static_cast<size_t>(kTileM), p.n - row0));

        // Exact distance to the previous centroid gives the first threshold (batch_computers.h:372-377).
        // When the caller has computed it already (p.best_in) it is taken from there; rows flagged in
        // p.skip belong to the dense kernel and are left untouched here.
        if (p.best_in) {
            if (tid < kTileM) {
                const bool active = tid < m_valid && !(p.skip && p.skip[row0 + tid]);
                st.best[tid] = active ? p.best_in[row0 + tid] : -1.0f;   // negative: no partial distance passes
                st.bestidx[tid] = active ? p.knn[row0 + tid] : 0u;
                st.prev[tid] = active ? p.knn[row0 + tid] : 0xFFFFFFFFu;
                st.nxs[tid] = (tid < m_valid) ? p.norms_x[row0 + tid] : 0.f;
                st.npc[tid] = 0;
                st.active[tid] = active ? 1u : 0u;
            }
        } else
        for (int r = warp; r < kTileM; r += 8) {
            if (lane == 0) st.active[r] = (r < m_valid) ? 1u : 0u;
            if (r < m_valid) {
                const uint32_t pa = p.knn[row0 + r];
                const float* __restrict__ xr = p.x + (row0 + r) * p.d;
                const float* __restrict__ yr = p.y + static_cast<size_t>(pa) * p.d;
                float s = 0.f;
                if (VEC) {
                    for (size_t j = static_cast<size_t>(lane) * 4; j < p.d; j += 128) {
                        const float4 a = __ldg(reinterpret_cast<const float4*>(xr + j));
                        const float4 b = __ldg(reinterpret_cast<const float4*>(yr + j));
                        float t;
                        t = a.x - b.x; s = fmaf(t, t, s);
                        t = a.y - b.y; s = fmaf(t, t, s);
                        t = a.z - b.z; s = fmaf(t, t, s);
                        t = a.w - b.w; s = fmaf(t, t, s);
                    }
                } else {
                    for (size_t j = lane; j < p.d; j += 32) {
                        const float t = __ldg(xr + j) - __ldg(yr + j);
                        s = fmaf(t, t, s);
                    }
                }
                s = warp_sum(s);
                if (lane == 0) {
                    st.best[r] = s;
                    st.bestidx[r] = pa;
                    st.prev[r] = pa;
                    st.nxs[r] = p.norms_x[row0 + r];
                    st.npc[r] = 0;
                }
            } else if (lane == 0) {
                st.best[r] = 0.f;
                st.bestidx[r] = 0;
                st.prev[r] = 0xFFFFFFFFu;
                st.nxs[r] = 0.f;
                st.npc[r] = 0;
            }
        }
        __syncthreads();

        for (size_t chunk = 0; chunk < n_chunks; ++chunk) {
            const size_t c0 = chunk * kChunk;
            const size_t cs = min(static_cast<size_t>(kChunk), p.k - c0);
            if (tid < kTileM) {
                st.thr[tid] = st.best[tid] * ratio_first;
                st.cnt[tid] = 0;
                st.prev_flag[tid] = 0;
                st.chunk_key[tid] = ~0ull;
            }
            if (tid == 0) st.list_count = 0;
            __syncthreads();

            float acc[8][8];
            for (size_t sub0 = 0; sub0 < cs; sub0 += kTileN) {
                const int n_valid = static_cast<int>(min(static_cast<size_t>(kTileN), cs - sub0));
                gemm_tile_nt(p.x + row0 * p.d, p.d, m_valid, p.y + (c0 + sub0) * p.d, p.d, n_valid, static_cast<int>(p.partial_d), smem, acc);
                float nyr[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = tile_col_of(tx, j);
                    nyr[j] = (c < n_valid) ? __ldg(p.norms_y + c0 + sub0 + c) : 0.f;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = tile_row_of(ty, i);
                    if (r >= m_valid) continue;
                    const float t = st.thr[r];
                    const float nxv = st.nxs[r];
                    const uint32_t pv = st.prev[r];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int c = tile_col_of(tx, j);
                        if (c < n_valid) {
                            const float pd = fmaf(-2.0f, acc[i][j], nxv) + nyr[j];
                            if (pd < t) {
                                atomicAdd(&st.cnt[r], 1u);
                                const uint32_t cl = static_cast<uint32_t>(sub0) + c;
                                if (static_cast<size_t>(pv) == c0 + cl) {
                                    st.prev_pd[r] = pd;
                                    st.prev_flag[r] = 1;
                                } else {
                                    const uint32_t pos = atomicAdd(&st.list_count, 1u);
                                    list[pos] = make_uint2((static_cast<uint32_t>(r) << 16) | cl, __float_as_uint(pd));
                                }
                            }
                        }
                    }
                }
            }
            __syncthreads();

            const uint32_t total = st.list_count;
            for (uint32_t e = g; e < total; e += 32) {
                const uint2 ent = list[e];
                pruned_process_pair<VEC>(p, st, row0, static_cast<int>(ent.x >> 16), ent.x & 0xFFFFu, __uint_as_float(ent.y), chunk, c0, cs, gl, gmask);
            }
            for (int r = g; r < kTileM; r += 32) {
                if (r < m_valid && st.prev_flag[r] && st.cnt[r] != 1u) {
                    pruned_process_pair<VEC>(p, st, row0, r, st.prev[r] - static_cast<uint32_t>(c0), st.prev_pd[r], chunk, c0, cs, gl, gmask);
                }
            }
            __syncthreads();
            if (tid < kTileM) {
                st.npc[tid] += st.cnt[tid];
                const unsigned long long key = st.chunk_key[tid];
                if (key != ~0ull) {
                    st.best[tid] = ordered_to_float(static_cast<uint32_t>(key >> 32));
                    st.bestidx[tid] = static_cast<uint32_t>(key & 0xFFFFFFFFull);
                }
            }
            __syncthreads();
        }
        if (tid < m_valid && st.active[tid]) {
            p.knn[row0 + tid] = st.bestidx[tid];
            p.dist[row0 + tid] = st.best[tid];
            p.not_pruned[row0 + tid] = st.npc[tid];
        }
        __syncthreads();
    }
}

int pruned_grid_size(int device) {
    int sms = 0;
    SKM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    return sms * 2;
}

size_t pruned_scratch_elems(int grid) { return static_cast<size_t>(grid) * kListCap; }

void launch_assign_pruned(const PrunedParams& p, int grid, cudaStream_t stream) {
    if (p.n == 0) return;
    const size_t n_tiles = (p.n + kTileM - 1) / kTileM;
    const int g = static_cast<int>(min(static_cast<size_t>(grid), n_tiles));
    const bool vec = (p.d % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.x) & 15) == 0) && ((reinterpret_cast<uintptr_t>(p.y) & 15) == 0) &&
                     ((reinterpret_cast<uintptr_t>(p.y_pdx) & 15) == 0);
    if (vec) {
        assign_pruned_kernel<true><<<g, 256, 0, stream>>>(p);
    } else {
        assign_pruned_kernel<false><<<g, 256, 0, stream>>>(p);
    }
    SKM_LAUNCH_CHECK();
}

// =================================================================================================
// Centroid update: stable LSD radix sort of point ids by assignment, then a segmented row sum in
// sorted order.  Everything is order-deterministic, so the same input gives bit-identical sums.
// =================================================================================================
// Elements handled by one warp, 32 at a time.  A warp's steps are a chain (each ranks its elements behind those of the
// steps before), and the digit table has 256 entries per unit: short units while there are fewer than a few warps per SM,
// long ones above.  At n = 6000 a pass takes 10 us where units of 2048 took 46 us.
static int sort_unit(size_t n) { return n < (size_t{1} << 17) ? 256 : (n < (size_t{1} << 20) ? 512 : 2048); }
constexpr int kSortAhead = 8;   // steps whose elements are loaded before the first of them is used

// Rows summed by one block of the segmented sum: 1024 where that gives every SM a block, else 128, because a block's rows
// are a chain of additions (95 us for 1024 rows, whatever the number of blocks; at n = 6000 a sum now takes 8 us).
static int update_tile_rows(size_t n) { return n >= (size_t{148} << 10) ? kUpdateTile : kUpdateTileSmall; }

static size_t sort_units_of(size_t n) { return (n + sort_unit(n) - 1) / sort_unit(n); }
static size_t tiles_of(size_t n) { return (n + update_tile_rows(n) - 1) / update_tile_rows(n); }

// A workspace made for n points also serves fewer, and fewer points can need more units and tiles.
static size_t update_sort_units(size_t n) {
    return std::max({sort_units_of(n), sort_units_of(std::min(n, (size_t{1} << 17) - 1)), sort_units_of(std::min(n, (size_t{1} << 20) - 1))});
}
// Up to 1024 clusters are sorted in one pass of ten bits: each of the five launches of a second pass takes 2 - 6 us however few the
// points are (30 000 points, 1000 clusters: 31 -> 19 us), and at 1M points the larger table is less than a pass over them.
// From there on eight bits at a time: the tables of a warp no longer fit a block of eight.
static int sort_bits(size_t k) { return k > 256 && k <= 1024 ? 10 : 8; }
size_t update_table_words(size_t n, size_t k) {
    const size_t words = (size_t{1} << (k > 256 ? 10 : 8)) * update_sort_units(n);
    return words + words / 2048 + 64;
}
size_t update_tiles(size_t n) { return std::max(tiles_of(n), tiles_of(std::min(n, (size_t{148} << 10) - 1))); }

template <int BITS>
__global__ void __launch_bounds__(256) sort_hist_kernel(const uint32_t* __restrict__ keys, size_t n, int shift, uint32_t* __restrict__ table, size_t n_units, int unit_size) {
    constexpr int DIGITS = 1 << BITS;
    __shared__ uint32_t h[8][DIGITS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = lane; i < DIGITS; i += 32) h[warp][i] = 0;
    __syncwarp();
    const size_t unit = static_cast<size_t>(blockIdx.x) * 8 + warp;
    if (unit < n_units) {
        const size_t base = unit * unit_size;
        for (int s0 = 0; s0 < unit_size / 32; s0 += kSortAhead) {
            uint32_t key[kSortAhead];
#pragma unroll
            for (int u = 0; u < kSortAhead; ++u) {
                const size_t idx = base + static_cast<size_t>(s0 + u) * 32 + lane;
                key[u] = idx < n ? keys[idx] : 0u;
            }
#pragma unroll
            for (int u = 0; u < kSortAhead; ++u)
                if (base + static_cast<size_t>(s0 + u) * 32 + lane < n) atomicAdd(&h[warp][(key[u] >> shift) & (DIGITS - 1u)], 1u);
        }
        __syncwarp();
        for (int i = lane; i < DIGITS; i += 32) table[static_cast<size_t>(i) * n_units + unit] = h[warp][i];
    }
}

// Exclusive scan of a uint32 array: (1) per-block scan of 2048 elements + block totals,
// (2) scan of the totals by one block, (3) add block offsets.
__global__ void __launch_bounds__(1024) scan_block_kernel(uint32_t* __restrict__ data, size_t n, uint32_t* __restrict__ totals) {
    __shared__ uint32_t ws[32];
    const size_t base = static_cast<size_t>(blockIdx.x) * 2048;
    const size_t i0 = base + static_cast<size_t>(threadIdx.x) * 2;
    const uint32_t a = (i0 < n) ? data[i0] : 0u;
    const uint32_t b = (i0 + 1 < n) ? data[i0 + 1] : 0u;
    uint32_t v = a + b;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = ws[lane];
        uint32_t winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, winc, o);
            if (lane >= o) winc += t;
        }
        ws[lane] = winc - w;
        if (lane == 31 && totals) totals[blockIdx.x] = winc;
    }
    __syncthreads();
    const uint32_t excl = ws[warp] + inc - v;
    if (i0 < n) data[i0] = excl;
    if (i0 + 1 < n) data[i0 + 1] = excl + a;
}

__global__ void __launch_bounds__(1024) scan_totals_kernel(uint32_t* __restrict__ totals, size_t m) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (size_t base = 0; base < m; base += 1024) {
        const size_t i = base + threadIdx.x;
        const uint32_t v = (i < m) ? totals[i] : 0u;
        uint32_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) ws[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const uint32_t w = ws[lane];
            uint32_t winc = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, winc, o);
                if (lane >= o) winc += t;
            }
            ws[lane] = winc - w;
        }
        __syncthreads();
        const uint32_t c = carry;
        if (i < m) totals[i] = c + ws[warp] + inc - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry = c + ws[warp] + inc;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(1024) scan_add_kernel(uint32_t* __restrict__ data, size_t n, const uint32_t* __restrict__ totals) {
    const size_t base = static_cast<size_t>(blockIdx.x) * 2048;
    const uint32_t off = totals[blockIdx.x];
    const size_t i0 = base + static_cast<size_t>(threadIdx.x) * 2;
    if (i0 < n) data[i0] += off;
    if (i0 + 1 < n) data[i0 + 1] += off;
}

void exclusive_scan_u32(uint32_t* data, size_t n, uint32_t* totals_tmp, cudaStream_t stream) {
    if (n == 0) return;
    const size_t blocks = (n + 2047) / 2048;
    scan_block_kernel<<<static_cast<unsigned>(blocks), 1024, 0, stream>>>(data, n, totals_tmp);
    SKM_LAUNCH_CHECK();
    if (blocks > 1) {
        scan_totals_kernel<<<1, 1024, 0, stream>>>(totals_tmp, blocks);
        SKM_LAUNCH_CHECK();
        scan_add_kernel<<<static_cast<unsigned>(blocks), 1024, 0, stream>>>(data, n, totals_tmp);
        SKM_LAUNCH_CHECK();
    }
}

// Stable scatter: each warp re-reads its unit in order; lanes with equal digits are ranked by lane.
template <int BITS>
__global__ void __launch_bounds__(256) sort_scatter_kernel(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, size_t n, int shift,
    const uint32_t* __restrict__ table, size_t n_units, int unit_size, uint32_t* __restrict__ seg_offsets, size_t k
) {
    constexpr int DIGITS = 1 << BITS;
    __shared__ uint32_t base_s[8][DIGITS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t unit = static_cast<size_t>(blockIdx.x) * 8 + warp;
    // the only pass knows where every key begins
    if (seg_offsets && blockIdx.x == 0)
        for (size_t c = threadIdx.x; c <= k; c += 256) seg_offsets[c] = c < DIGITS ? table[c * n_units] : static_cast<uint32_t>(n);
    if (unit >= n_units) return;
    for (int i = lane; i < DIGITS; i += 32) base_s[warp][i] = table[static_cast<size_t>(i) * n_units + unit];
    __syncwarp();
    const size_t base = unit * unit_size;
    const uint32_t lt_mask = (1u << lane) - 1u;
    for (int s0 = 0; s0 < unit_size / 32; s0 += kSortAhead) {
        uint32_t keys[kSortAhead], vals[kSortAhead];
#pragma unroll
        for (int u = 0; u < kSortAhead; ++u) {
            const size_t idx = base + static_cast<size_t>(s0 + u) * 32 + lane;
            const bool valid = idx < n;
            keys[u] = valid ? keys_in[idx] : 0u;
            vals[u] = valid ? (vals_in ? vals_in[idx] : static_cast<uint32_t>(idx)) : 0u;
        }
#pragma unroll
        for (int u = 0; u < kSortAhead; ++u) {
            const bool valid = base + static_cast<size_t>(s0 + u) * 32 + lane < n;
            const uint32_t digit = valid ? ((keys[u] >> shift) & (DIGITS - 1u)) : 0xFFFFFFFFu;
            const uint32_t peers = __match_any_sync(0xffffffffu, digit);
            const uint32_t rank = __popc(peers & lt_mask);
            if (valid) {
                const uint32_t pos = base_s[warp][digit] + rank;
                keys_out[pos] = keys[u];
                vals_out[pos] = vals[u];
            }
            __syncwarp();
            if (valid && rank == 0) base_s[warp][digit] += __popc(peers);
            __syncwarp();
        }
    }
}

// seg_offsets[c] = first sorted position whose key is >= c, for c in [0, k]
__global__ void segment_offsets_kernel(const uint32_t* __restrict__ sorted_keys, size_t n, size_t k, uint32_t* __restrict__ off) {
    const size_t p = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const uint32_t key = sorted_keys[p];
    const uint32_t lo = (p == 0) ? 0u : sorted_keys[p - 1] + 1u;
    for (uint32_t c = lo; c <= key && c <= k; ++c) off[c] = static_cast<uint32_t>(p);
    if (p == n - 1) {
        for (size_t c = static_cast<size_t>(key) + 1; c <= k; ++c) off[c] = static_cast<uint32_t>(n);
    }
}

// One CTA sums the rows of TILE consecutive sorted points for a slab of 4 columns per thread.  The
// first segment of the tile goes to partial slot 2t, the last one (if different) to slot 2t+1, and
// segments that lie strictly inside the tile are final and go straight to `sums`.
template <bool VEC, int TILE>
__global__ void __launch_bounds__(256) segsum_tile_kernel(
    const float* __restrict__ x, const uint32_t* __restrict__ sorted_keys, const uint32_t* __restrict__ order, size_t n, size_t d, float* __restrict__ sums, float* __restrict__ partials
) {
    __shared__ uint32_t skey[TILE];
    __shared__ uint32_t sid[TILE];
    const size_t tile = blockIdx.x;
    const size_t p0 = tile * TILE;
    const int cnt = static_cast<int>(min(static_cast<size_t>(TILE), n - p0));
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
        skey[i] = sorted_keys[p0 + i];
        sid[i] = order[p0 + i];
    }
    __syncthreads();
    const size_t colbase = static_cast<size_t>(blockIdx.y) * 4 * blockDim.x;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    size_t col[4];
    bool cv[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        col[e] = VEC ? (colbase + static_cast<size_t>(threadIdx.x) * 4 + e) : (colbase + threadIdx.x + blockDim.x * e);
        cv[e] = col[e] < d;
    }
    auto flush = [&](uint32_t key, int kind) {
        float* dst = (kind == 0) ? (partials + (tile * 2) * d) : (kind == 1 ? (partials + (tile * 2 + 1) * d) : (sums + static_cast<size_t>(key) * d));
        if (VEC) {
            if (cv[0]) *reinterpret_cast<float4*>(dst + col[0]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (cv[e]) dst[col[e]] = acc[e];
        }
        acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
    };
    uint32_t cur = skey[0];
    bool first = true;
    constexpr int U = 8;
    for (int i0 = 0; i0 < cnt; i0 += U) {
        float v[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u;
            if (i < cnt) {
                const float* row = x + static_cast<size_t>(sid[i]) * d;
                if (VEC) {
                    if (cv[0]) {
                        const float4 t = __ldg(reinterpret_cast<const float4*>(row + col[0]));
                        v[u][0] = t.x; v[u][1] = t.y; v[u][2] = t.z; v[u][3] = t.w;
                    } else {
                        v[u][0] = v[u][1] = v[u][2] = v[u][3] = 0.f;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[u][e] = cv[e] ? __ldg(row + col[e]) : 0.f;
                }
            } else {
                v[u][0] = v[u][1] = v[u][2] = v[u][3] = 0.f;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u;
            if (i < cnt) {
                const uint32_t kk = skey[i];
                if (kk != cur) {
                    flush(cur, first ? 0 : 2);
                    first = false;
                    cur = kk;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[e] += v[u][e];
            }
        }
    }
    flush(cur, first ? 0 : 1);
}

// Combines the tile partials of every cluster whose points are not strictly inside one tile, in
// tile order; empty clusters get zeros.
template <bool VEC, int TILE>
__global__ void __launch_bounds__(256) segsum_fix_kernel(const uint32_t* __restrict__ off, size_t n, size_t d, const float* __restrict__ partials, float* __restrict__ sums, uint32_t* __restrict__ counts) {
    const size_t c = blockIdx.x;
    const size_t s = off[c], e = off[c + 1];
    if (blockIdx.y == 0 && threadIdx.x == 0) counts[c] = static_cast<uint32_t>(e - s);
    const size_t colbase = static_cast<size_t>(blockIdx.y) * 4 * blockDim.x;
    size_t col[4];
    bool cv[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        col[q] = VEC ? (colbase + static_cast<size_t>(threadIdx.x) * 4 + q) : (colbase + threadIdx.x + blockDim.x * q);
        cv[q] = col[q] < d;
    }
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (s < e) {
        const size_t t0 = s / TILE, t1 = (e - 1) / TILE;
        const size_t tile_end = min((t0 + 1) * TILE, n);
        const bool direct = (t0 == t1) && (s > t0 * TILE) && (e < tile_end);
        if (direct) return;
        for (size_t t = t0; t <= t1; ++t) {
            const size_t slot = (s <= t * TILE) ? (2 * t) : (2 * t + 1);
            const float* src = partials + slot * d;
            if (VEC) {
                if (cv[0]) {
                    const float4 v = *reinterpret_cast<const float4*>(src + col[0]);
                    acc[0] += v.x; acc[1] += v.y; acc[2] += v.z; acc[3] += v.w;
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (cv[q]) acc[q] += src[col[q]];
            }
        }
    }
    float* dst = sums + c * d;
    if (VEC) {
        if (cv[0]) *reinterpret_cast<float4*>(dst + col[0]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (cv[q]) dst[col[q]] = acc[q];
    }
}

// Reductions of the per-point distance (double) and not-pruned counts (u64) in a fixed order: every block leaves its sums in
// the scratch, and the block that finds it is the last adds them up.
constexpr int kReduceBlocks = 512;
static_assert(kReduceScratchDoubles >= 2 * kReduceBlocks + 1, "reduction scratch");

__device__ __forceinline__ bool last_block(double* scratch) {
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned* ticket = reinterpret_cast<unsigned*>(scratch + 2 * kReduceBlocks);
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
        if (last) *ticket = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

__device__ __forceinline__ void block_tree(double* sd, unsigned long long* su) {
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sd[threadIdx.x] += sd[threadIdx.x + o];
            su[threadIdx.x] += su[threadIdx.x + o];
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) reduce_stats_kernel(UpdateStats u, size_t n, double* scratch) {
    __shared__ double sd[256];
    __shared__ unsigned long long su[256];
    double a = 0.0;
    unsigned long long b = 0;
    for (size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; i < n; i += static_cast<size_t>(kReduceBlocks) * 256) {
        a += static_cast<double>(u.dist[i]);
        if (u.not_pruned) b += u.not_pruned[i];
    }
    sd[threadIdx.x] = a;
    su[threadIdx.x] = b;
    block_tree(sd, su);
    unsigned long long* bu = reinterpret_cast<unsigned long long*>(scratch + kReduceBlocks);
    if (threadIdx.x == 0) {
        scratch[blockIdx.x] = sd[0];
        bu[blockIdx.x] = su[0];
    }
    if (!last_block(scratch)) return;
    a = 0.0;
    b = 0;
    for (int i = threadIdx.x; i < kReduceBlocks; i += 256) {
        a += __ldcg(scratch + i);
        b += __ldcg(bu + i);
    }
    sd[threadIdx.x] = a;
    su[threadIdx.x] = b;
    block_tree(sd, su);
    if (threadIdx.x == 0) {
        IterationReport& r = *u.report;
        r.wcss = sd[0];
        r.not_pruned = static_cast<double>(su[0]);
        r.error = u.error ? *u.error : 0;
    }
}

// Stable LSD radix sort of the indices 0 .. n-1 by key (keys < k): *sorted_keys and *order point into ws.keys_* / ws.vals_*.
template <int BITS>
static void launch_sort_pass(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, size_t n, int shift, const UpdateWorkspace& ws, uint32_t* seg_offsets, size_t k,
                             cudaStream_t stream) {
    const size_t n_units = sort_units_of(n), words = n_units << BITS;
    const unsigned blocks = static_cast<unsigned>((n_units + 7) / 8);
    sort_hist_kernel<BITS><<<blocks, 256, 0, stream>>>(kin, n, shift, ws.digit_table, n_units, sort_unit(n));
    SKM_LAUNCH_CHECK();
    exclusive_scan_u32(ws.digit_table, words, ws.digit_table + words, stream);   // (block totals behind the table)
    sort_scatter_kernel<BITS><<<blocks, 256, 0, stream>>>(kin, vin, kout, vout, n, shift, ws.digit_table, n_units, sort_unit(n), seg_offsets, k);
    SKM_LAUNCH_CHECK();
}

bool launch_sort_by_key(const uint32_t* keys, size_t n, size_t k, UpdateWorkspace& ws, const uint32_t** sorted_keys_out, const uint32_t** order_out, uint32_t* seg_offsets,
                        cudaStream_t stream) {
    int bits = 1;
    while ((size_t{1} << bits) < k) ++bits;
    const int per_pass = sort_bits(k), passes = (bits + per_pass - 1) / per_pass;
    if (passes > 1) seg_offsets = nullptr;
    const uint32_t* kin = keys;
    const uint32_t* vin = nullptr;
    uint32_t* kout = ws.keys_a;
    uint32_t* vout = ws.vals_a;
    for (int pass = 0; pass < passes; ++pass) {
        if (per_pass == 10) launch_sort_pass<10>(kin, vin, kout, vout, n, pass * 10, ws, seg_offsets, k, stream);
        else launch_sort_pass<8>(kin, vin, kout, vout, n, pass * 8, ws, seg_offsets, k, stream);
        kin = kout;
        vin = vout;
        kout = (kout == ws.keys_a) ? ws.keys_b : ws.keys_a;
        vout = (vout == ws.vals_a) ? ws.vals_b : ws.vals_a;
    }
    *sorted_keys_out = kin;
    *order_out = vin;
    return seg_offsets != nullptr;
}

template <bool VEC, int TILE>
static void launch_segsum(const float* x, const uint32_t* sorted_keys, const uint32_t* order, size_t n, size_t k, size_t d, UpdateWorkspace& ws, float* sums, uint32_t* counts,
                          cudaStream_t stream) {
    // four columns per thread, no more warps than the columns need
    const unsigned threads = static_cast<unsigned>(std::min<size_t>(256, ((d + 3) / 4 + 31) / 32 * 32));
    const unsigned slabs = static_cast<unsigned>((d + 4 * threads - 1) / (4 * threads));
    segsum_tile_kernel<VEC, TILE><<<dim3(static_cast<unsigned>(tiles_of(n)), slabs), threads, 0, stream>>>(x, sorted_keys, order, n, d, sums, ws.tile_partials);
    SKM_LAUNCH_CHECK();
    segsum_fix_kernel<VEC, TILE><<<dim3(static_cast<unsigned>(k), slabs), threads, 0, stream>>>(ws.seg_offsets, n, d, ws.tile_partials, sums, counts);
    SKM_LAUNCH_CHECK();
}

void launch_update(const float* x, const uint32_t* assign, size_t n, size_t k, size_t d, UpdateWorkspace& ws, float* sums, uint32_t* counts, const UpdateStats* stats,
                   cudaStream_t stream) {
    if (n == 0) return;
    const uint32_t* sorted_keys = nullptr;
    const uint32_t* order = nullptr;
    if (!launch_sort_by_key(assign, n, k, ws, &sorted_keys, &order, ws.seg_offsets, stream)) {
        segment_offsets_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(sorted_keys, n, k, ws.seg_offsets);
        SKM_LAUNCH_CHECK();
    }
    const bool vec = (d % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    const bool big = update_tile_rows(n) == kUpdateTile;
    if (vec && big) launch_segsum<true, kUpdateTile>(x, sorted_keys, order, n, k, d, ws, sums, counts, stream);
    else if (vec) launch_segsum<true, kUpdateTileSmall>(x, sorted_keys, order, n, k, d, ws, sums, counts, stream);
    else if (big) launch_segsum<false, kUpdateTile>(x, sorted_keys, order, n, k, d, ws, sums, counts, stream);
    else launch_segsum<false, kUpdateTileSmall>(x, sorted_keys, order, n, k, d, ws, sums, counts, stream);
    if (stats) {
        reduce_stats_kernel<<<kReduceBlocks, 256, 0, stream>>>(*stats, n, ws.reduce_scratch);
        SKM_LAUNCH_CHECK();
    }
}

// =================================================================================================
// Consolidation
// =================================================================================================
// Every thread owns one dimension and replays the row operations in list order.
__global__ void apply_split_ops_kernel(float* __restrict__ c, size_t d, const SplitOpDev* __restrict__ ops, size_t n_ops) {
    const size_t j = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= d) return;
    for (size_t o = 0; o < n_ops; ++o) apply_split_op(c, d, j, ops[o]);
}

void launch_apply_split_ops(float* c, size_t d, const SplitOpDev* ops, size_t n_ops, cudaStream_t stream) {
    if (n_ops == 0) return;
    apply_split_ops_kernel<<<static_cast<unsigned>((d + 127) / 128), 128, 0, stream>>>(c, d, ops, n_ops);
    SKM_LAUNCH_CHECK();
}

// Where dimension j of row v of a chunk of cs rows lies in the chunk's PDX block.
__device__ __forceinline__ size_t pdx_offset(size_t j, size_t v, size_t cs, size_t vertical_d) {
    if (j < vertical_d) return j * cs + v;
    const size_t h = j - vertical_d;
    return vertical_d * cs + (h / kHBlock) * cs * kHBlock + v * kHBlock + (h % kHBlock);
}

__global__ void pdxify_kernel(const float* __restrict__ c, float* __restrict__ pdx, float* __restrict__ aux, size_t k, size_t d, size_t vertical_d) {
    const size_t row = blockIdx.x;
    const size_t chunk = row / kChunk, v = row % kChunk;
    const size_t cs = min(static_cast<size_t>(kChunk), k - chunk * kChunk);
    float* __restrict__ out = pdx + chunk * kChunk * d;
    const float* src = c + row * d;
    for (size_t j = threadIdx.x; j < d; j += blockDim.x) {
        const float val = src[j];
        out[pdx_offset(j, v, cs, vertical_d)] = val;
        if (aux && j < vertical_d) aux[row * vertical_d + j] = val;
    }
}

void launch_pdxify(const float* c, float* pdx, float* aux, size_t k, size_t d, size_t vertical_d, cudaStream_t stream) {
    if (k == 0) return;
    pdxify_kernel<<<static_cast<unsigned>(k), 256, 0, stream>>>(c, pdx, aux, k, d, vertical_d);
    SKM_LAUNCH_CHECK();
}

// A warp per row; every lane keeps to its own dimensions.  What bounds it is the launch: with k = 1000 it replaces five of
// them, and with the report's single copy four waits of the host: a Train of 2000 x 64, k = 20, took 2.1 ms and takes 1.6.
__global__ void __launch_bounds__(256) consolidate_kernel(const ConsolidateParams p) {
    __shared__ double sd[256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bool finish = true;
    if (p.counts && p.normalize) {
        bool empty = false;
        for (size_t i = threadIdx.x; i < p.k; i += 256) empty |= p.counts[i] == 0;
        finish = __syncthreads_or(empty || p.splits_follow) == 0;
    }
    double total = 0.0;
    for (size_t row = static_cast<size_t>(blockIdx.x) * 8 + warp; row < p.k; row += static_cast<size_t>(gridDim.x) * 8) {
        float* __restrict__ c = p.c + row * p.d;
        const float* __restrict__ prev = p.prev + row * p.d;
        const size_t chunk = row / kChunk, v = row % kChunk;
        const size_t cs = min(static_cast<size_t>(kChunk), p.k - chunk * kChunk);
        float* __restrict__ pdx = p.pdx + chunk * kChunk * p.d;
        float* __restrict__ aux = p.aux + row * p.vertical_d;
        const uint32_t cnt = p.counts ? p.counts[row] : 0;
        const float mult = cnt ? static_cast<float>(1.0 / static_cast<double>(cnt)) : 1.0f;
        if (p.normalize) {
            for (size_t j = lane; j < p.d; j += 32) c[j] = __fmul_rn(c[j], mult);
            if (!finish) continue;
            normalize_row(c, p.d, lane);
        }
        const float scale = p.normalize ? 1.0f : mult;
        float s = 0.f;
        constexpr int U = 8;   // loads in flight: the stores between them would hold them up
        for (size_t j0 = lane; j0 < p.d; j0 += 32 * U) {
            float cv[U], pv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const size_t j = min(j0 + 32 * u, p.d - 1);
                cv[u] = c[j];
                pv[u] = prev[j];
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const size_t j = j0 + 32 * u;
                if (j >= p.d) break;
                const float val = __fmul_rn(cv[u], scale);
                c[j] = val;
                pdx[pdx_offset(j, v, cs, p.vertical_d)] = val;
                if (j < p.vertical_d) aux[j] = val;
                const float t = val - pv[u];
                s = fmaf(t, t, s);
            }
        }
        s = warp_sum(s);
        total += static_cast<double>(s);
    }
    if (lane == 0) sd[warp] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += sd[w];
        p.reduce_scratch[blockIdx.x] = t;
    }
    if (!last_block(p.reduce_scratch)) return;
    double a = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += 256) a += __ldcg(p.reduce_scratch + i);
    sd[threadIdx.x] = a;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) sd[threadIdx.x] += sd[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) p.report->shift = sd[0];
    __syncthreads();
    for (size_t i = threadIdx.x; i < p.told_words; i += 256) p.told[i] = __ldcg(p.tell + i);
}

// UpdateCentroids, ComputeCost, ConsolidateCentroids and ComputeShift of a small problem in one launch, a block per cluster: it looks for its
// points among all of them (a piece at a time, their rows in a fixed order), adds their rows up, and has the cluster's centroid.
constexpr int kSmallPiece = 4096;
constexpr int kSmallLoads = 8;   // rows in flight per thread
constexpr uint32_t kSmallChain = 32;   // rows, or sums of rows, added one after the other: no more than in a tile of the large update
__global__ void __launch_bounds__(256) small_update_kernel(const float* __restrict__ x, const uint32_t* __restrict__ assign, size_t n, const UpdateStats u, uint32_t* __restrict__ counts,
                                                           const ConsolidateParams p) {
    __shared__ uint32_t ids[kSmallPiece];
    __shared__ float4 parts[256];
    __shared__ uint32_t found[8];
    __shared__ double sd[3][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t cluster = blockIdx.x;
    const uint32_t groups = static_cast<uint32_t>(p.d / 4), rows = 256 / groups;   // columns four at a time, rows beside each other
    const uint32_t g = threadIdx.x % groups, r = threadIdx.x / groups;
    double cost = 0.0;
    unsigned long long not_pruned = 0;
    uint32_t count = 0, loads = 0;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f), total = sum;
    for (size_t base = 0; base < n; base += kSmallPiece) {
        uint32_t mask = 0;
#pragma unroll
        for (int i = 0; i < kSmallPiece / 256; ++i) {
            const size_t at = base + i * 256 + threadIdx.x;
            if (at < n && __ldg(assign + at) == cluster) mask |= 1u << i;
        }
        const uint32_t mine = __popc(mask);
        uint32_t before = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += t;
        }
        if (lane == 31) found[warp] = before;
        before -= mine;
        __syncthreads();
        uint32_t m = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            if (w < warp) before += found[w];
            m += found[w];
        }
        for (; mask; mask &= mask - 1) {
            const uint32_t at = static_cast<uint32_t>(base) + (__ffs(mask) - 1) * 256 + threadIdx.x;
            ids[before++] = at;
            cost += static_cast<double>(u.dist[at]);
            if (u.not_pruned) not_pruned += u.not_pruned[at];
        }
        __syncthreads();
        count += m;
        if (r < rows) {
            for (uint32_t j = r; j < m; j += rows * kSmallLoads) {
                float4 v[kSmallLoads];
#pragma unroll
                for (int q = 0; q < kSmallLoads; ++q)
                    v[q] = j + q * rows < m ? __ldg(reinterpret_cast<const float4*>(x + static_cast<size_t>(ids[j + q * rows]) * p.d) + g) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int q = 0; q < kSmallLoads; ++q) {
                    sum.x += v[q].x;
                    sum.y += v[q].y;
                    sum.z += v[q].z;
                    sum.w += v[q].w;
                }
                if (++loads % (kSmallChain / kSmallLoads) == 0) {
                    total = make_float4(total.x + sum.x, total.y + sum.y, total.z + sum.z, total.w + sum.w);
                    sum = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        }
        __syncthreads();
    }
    sum = make_float4(total.x + sum.x, total.y + sum.y, total.z + sum.z, total.w + sum.w);
    parts[threadIdx.x] = sum;
    __syncthreads();
    float s = 0.f;
    if (r == 0) {
        total = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t q = 1; q < rows; ++q) {
            const float4 t = parts[q * groups + g];
            sum.x += t.x;
            sum.y += t.y;
            sum.z += t.z;
            sum.w += t.w;
            if (q % kSmallChain == 0) {
                total = make_float4(total.x + sum.x, total.y + sum.y, total.z + sum.z, total.w + sum.w);
                sum = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        sum = make_float4(total.x + sum.x, total.y + sum.y, total.z + sum.z, total.w + sum.w);
        const float mult = count ? static_cast<float>(1.0 / static_cast<double>(count)) : 1.0f;
        const float val[4] = {__fmul_rn(sum.x, mult), __fmul_rn(sum.y, mult), __fmul_rn(sum.z, mult), __fmul_rn(sum.w, mult)};
        const size_t chunk = cluster / kChunk, v = cluster % kChunk;
        const size_t cs = min(static_cast<size_t>(kChunk), p.k - chunk * kChunk);
        float* __restrict__ pdx = p.pdx + chunk * kChunk * p.d;
        const float4 prev = *reinterpret_cast<const float4*>(p.prev + cluster * p.d + 4 * g);
        const float pv[4] = {prev.x, prev.y, prev.z, prev.w};
        *reinterpret_cast<float4*>(p.c + cluster * p.d + 4 * g) = make_float4(val[0], val[1], val[2], val[3]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const size_t j = 4 * g + q;
            pdx[pdx_offset(j, v, cs, p.vertical_d)] = val[q];
            if (j < p.vertical_d) p.aux[cluster * p.vertical_d + j] = val[q];
            const float t = val[q] - pv[q];
            s = fmaf(t, t, s);
        }
    }
    // sums over the block, then over the blocks, always in the same order
    double a[3] = {static_cast<double>(s), cost, static_cast<double>(not_pruned)};   // (counts below 2^53)
    auto block_sums = [&](double (&v)[3]) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
            if (lane == 0) sd[i][warp] = v[i];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            v[i] = 0.0;
            for (int w = 0; w < 8; ++w) v[i] += sd[i][w];
        }
        __syncthreads();
    };
    block_sums(a);
    if (threadIdx.x == 0) {
        counts[cluster] = count;
        for (int i = 0; i < 3; ++i) p.reduce_scratch[3 * cluster + i] = a[i];
    }
    if (!last_block(p.reduce_scratch)) return;
    a[0] = a[1] = a[2] = 0.0;
    for (size_t c = threadIdx.x; c < p.k; c += 256)
        for (int i = 0; i < 3; ++i) a[i] += __ldcg(p.reduce_scratch + 3 * c + i);
    block_sums(a);
    if (threadIdx.x == 0) {
        p.report->shift = a[0];
        p.report->wcss = a[1];
        p.report->not_pruned = a[2];
        p.report->error = u.error ? *u.error : 0;
    }
    __syncthreads();
    for (size_t i = threadIdx.x; i < p.told_words; i += 256) p.told[i] = __ldcg(p.tell + i);
}

bool small_update(size_t n, size_t k, size_t d) { return d % 4 == 0 && d <= 1024 && 3 * k <= 2 * kReduceBlocks && n * d <= (size_t{1} << 19); }

void launch_small_update(const float* x, const uint32_t* assign, size_t n, uint32_t* counts, const UpdateStats& stats, const ConsolidateParams& p, cudaStream_t stream) {
    small_update_kernel<<<static_cast<unsigned>(p.k), 256, 0, stream>>>(x, assign, n, stats, counts, p);
    SKM_LAUNCH_CHECK();
}

__global__ void __launch_bounds__(256) tell_host_kernel(const uint4* __restrict__ from, uint4* __restrict__ to, size_t words) {
    for (size_t i = threadIdx.x; i < words; i += 256) to[i] = from[i];
}

__global__ void tell_word_kernel(const uint32_t* __restrict__ from, uint32_t* __restrict__ to) { *to = *from; }

void launch_tell_word(const void* from, void* to, cudaStream_t stream) {
    tell_word_kernel<<<1, 1, 0, stream>>>(static_cast<const uint32_t*>(from), static_cast<uint32_t*>(to));
    SKM_LAUNCH_CHECK();
}

void launch_tell_host(const void* from, void* to, size_t bytes, cudaStream_t stream) {
    tell_host_kernel<<<1, 256, 0, stream>>>(static_cast<const uint4*>(from), static_cast<uint4*>(to), bytes / 16);
    SKM_LAUNCH_CHECK();
}

void launch_consolidate(const ConsolidateParams& p, cudaStream_t stream) {
    const unsigned blocks = static_cast<unsigned>(std::min(static_cast<size_t>(kReduceBlocks), (p.k + 7) / 8));
    consolidate_kernel<<<blocks, 256, 0, stream>>>(p);
    SKM_LAUNCH_CHECK();
}

// =================================================================================================
// Gather / scatter by index
// =================================================================================================
// A warp per row, four 16-byte loads in flight per lane (VEC: 16-byte aligned rows).  300 000 x 768: 0.66 ms with a block per row and
// 4-byte loads, 0.27 so.
template <bool VEC>
__global__ void __launch_bounds__(256) gather_rows_kernel(const float* __restrict__ in, const uint64_t* __restrict__ idx, float* __restrict__ out, size_t n_out, size_t d) {
    const size_t row = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (row >= n_out) return;
    const int lane = threadIdx.x & 31;
    const uint64_t from = idx[row];
    // "no row here" (held by another shard): zeros
    const bool none = from == ~uint64_t{0};
    const float* __restrict__ src = in + (none ? 0 : from) * d;
    float* __restrict__ dst = out + row * d;
    if (VEC) {
        for (size_t j0 = static_cast<size_t>(lane) * 4; j0 < d; j0 += 512) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = !none && j0 + 128 * u < d ? __ldg(reinterpret_cast<const float4*>(src + j0 + 128 * u)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j0 + 128 * u < d) *reinterpret_cast<float4*>(dst + j0 + 128 * u) = v[u];
        }
    } else {
#pragma unroll 4
        for (size_t j = lane; j < d; j += 32) dst[j] = none ? 0.f : __ldg(src + j);
    }
}

void launch_gather_rows(const float* in, const uint64_t* idx, float* out, size_t n_out, size_t d, cudaStream_t stream) {
    if (n_out == 0) return;
    const unsigned grid = static_cast<unsigned>((n_out + 7) / 8);
    if (d % 4 == 0 && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) gather_rows_kernel<true><<<grid, 256, 0, stream>>>(in, idx, out, n_out, d);
    else gather_rows_kernel<false><<<grid, 256, 0, stream>>>(in, idx, out, n_out, d);
    SKM_LAUNCH_CHECK();
}

__global__ void gather_f32_kernel(const float* __restrict__ in, const uint64_t* __restrict__ idx, float* __restrict__ out, size_t n_out) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n_out) out[i] = in[idx[i]];
}

void launch_gather_f32(const float* in, const uint64_t* idx, float* out, size_t n_out, cudaStream_t stream) {
    if (n_out == 0) return;
    gather_f32_kernel<<<static_cast<unsigned>((n_out + 255) / 256), 256, 0, stream>>>(in, idx, out, n_out);
    SKM_LAUNCH_CHECK();
}

__global__ void scatter_u32_offset_kernel(const uint32_t* __restrict__ in, const uint64_t* __restrict__ idx, uint32_t* __restrict__ out, size_t n, uint32_t offset) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) out[idx[i]] = in[i] + offset;
}

void launch_scatter_u32_offset(const uint32_t* in, const uint64_t* idx, uint32_t* out, size_t n, uint32_t offset, cudaStream_t stream) {
    if (n == 0) return;
    scatter_u32_offset_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(in, idx, out, n, offset);
    SKM_LAUNCH_CHECK();
}

} // namespace skmb
