// The random orthogonal matrix of the ADSampling rotation (adsampling.h:76-85) from its Gaussian draws, on the GPU.
//
// The matrix is the Q factor of the d x d draws with the signs of a Householder QR; host_logic.h computes it column by
// column on the host (0.25 s at d = 768, 1.2 s at d = 1536 on 16 cores: twice d rank-one updates of a matrix that
// does not stay in cache).  Householder steps are a chain of d reductions here too, so Q is computed another way, in
// double throughout, from products whose chains are d / 32 long:
//
//   1. G = A^T A, G = R^T R (blocked Cholesky), Q = A R^-1 (rows are independent of each other);
//   2. E = Q^T Q - I (at most cond(A)^2 * 1e-16), Q <- Q (I - up(E)), up = strict upper part + half the diagonal: the first
//      order of a second Cholesky QR.  Each turn squares E; repeated until E^2 is below the rounding of double;
//   3. this Q has a positive diagonal in R; Householder's sign for column k is minus the sign of entry (k, k) of what is
//      left of the column after k reflections, which is the k-th pivot of the elimination of Q - S without pivoting,
//      S = diag(signs), chosen as the elimination goes (the reconstruction of Householder vectors from an orthonormal
//      basis: Ballard, Demmel, Grigori, Jacquelin, Nguyen, Solomonik, 2014); the last column keeps its sign.
//
// Steps 1 and 3 are right-looking over 32-wide panels with one launch per panel: every block of the trailing matrix
// recomputes the 32 x 32 products it needs of the panel (three small products instead of one, against a launch and a
// round trip saved), and the block that holds the next diagonal factorises it at once.  Measured (kernels, one B200): d = 768
// 1.2 ms, of which 0.25 ms are the solve of step 1 (0.88 with one batch of loads in flight instead of four; d = 1536: 2.5 - 3.0 ms
// before) and 0.75 ms (d = 1536: 1.9) the two chains of d / 32 dependent launches.
//
// A matrix too close to singular for this (or too wide for step 1's row buffer, or for the memory that is left: the scratch is 32 bytes
// an element) is declined: the caller takes the host's.
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "engine.h"

namespace skmb {

namespace {

constexpr int NB = 32;    // panel width of the factorisations
constexpr int GT = 64;    // tile of the products: GT x GN
constexpr int GN = 32;
constexpr int kProductThreads = GT / 4 * GN / 4;
constexpr int GK = 16;
constexpr int kThreads = 256;
constexpr size_t kSolveSmem = 200 * 1024;
constexpr int kSolveMaxRows = 16;

// A column of blocks per piece; pinned memory is read in place.
__global__ void __launch_bounds__(kThreads) collect_draws_kernel(const DrawPieces p, float* __restrict__ out) {
    const uint32_t t = blockIdx.y;
    const float* from = p.values + t * p.stretch;
    const size_t at = p.start[t], n = p.start[t + 1] - at;
    for (size_t i = static_cast<size_t>(blockIdx.x) * kThreads + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * kThreads) out[at + i] = from[i];
}

// Double copy of the draws, padded with the identity to a multiple of GT, so that nothing below has edges.
__global__ void widen_draws_kernel(const float* __restrict__ draws, size_t d, size_t dp, double* __restrict__ a) {
    const size_t j = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (j >= dp) return;
    a[i * dp + j] = (i < d && j < d) ? static_cast<double>(draws[i * d + j]) : (i == j ? 1.0 : 0.0);
}

// kGram: out = a^T a, blocks on and above the diagonal; with `minus_identity` I is subtracted and *largest becomes the
// largest |entry| as an ordered integer (all ones for a NaN).   !kGram: out = a - a up(e).
// Tiles of 64 x 32, 4 x 4 per thread, the next 16 of K in registers meanwhile: twice the blocks of 64 x 64, so that most SMs have two that
// wait for memory in turn (d = 768: 0.14 -> 0.085 ms a product, d = 1536: 0.6 -> 0.4).
template <bool kGram>
__global__ void __launch_bounds__(kProductThreads) product_kernel(const double* __restrict__ a, const double* __restrict__ e, size_t dp, double* __restrict__ out, bool minus_identity,
                                                                  unsigned long long* __restrict__ largest) {
    __shared__ __align__(16) double sa[GK][GT + 2];
    __shared__ __align__(16) double sb[GK][GN + 2];
    const size_t i0 = static_cast<size_t>(blockIdx.y) * GT, j0 = static_cast<size_t>(blockIdx.x) * GN;
    if (kGram && j0 + GN <= i0) return;
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    double acc[4][4] = {};
    const size_t k_end = kGram ? dp : j0 + GN;   // up(e) is zero below the diagonal
    constexpr int NA = GK * GT / kProductThreads, NBV = GK * GN / kProductThreads;
    double va[NA], vb[NBV];
    auto fetch = [&](size_t k0) {
#pragma unroll
        for (int u = 0; u < NA; ++u) {
            const int q = threadIdx.x + u * kProductThreads;
            if (kGram) va[u] = a[(k0 + (q / GT)) * dp + i0 + q % GT];
            else va[u] = a[(i0 + q / GK) * dp + k0 + q % GK];
        }
#pragma unroll
        for (int u = 0; u < NBV; ++u) {
            const int q = threadIdx.x + u * kProductThreads;
            const size_t row = k0 + q / GN, col = j0 + q % GN;
            if (kGram) vb[u] = a[row * dp + col];
            else vb[u] = row < col ? e[row * dp + col] : (row == col ? 0.5 * e[row * dp + col] : 0.0);
        }
    };
    fetch(0);
    for (size_t k0 = 0; k0 < k_end; k0 += GK) {
#pragma unroll
        for (int u = 0; u < NA; ++u) {
            const int q = threadIdx.x + u * kProductThreads;
            if (kGram) sa[q / GT][q % GT] = va[u];
            else sa[q % GK][q / GK] = va[u];
        }
#pragma unroll
        for (int u = 0; u < NBV; ++u) {
            const int q = threadIdx.x + u * kProductThreads;
            sb[q / GN][q % GN] = vb[u];
        }
        __syncthreads();
        if (k0 + GK < k_end) fetch(k0 + GK);
#pragma unroll
        for (int kk = 0; kk < GK; ++kk) {
            double av[4], bv[4];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const double2 u = *reinterpret_cast<const double2*>(&sa[kk][ty * 4 + q * 2]);
                const double2 v = *reinterpret_cast<const double2*>(&sb[kk][tx * 4 + q * 2]);
                av[2 * q] = u.x;
                av[2 * q + 1] = u.y;
                bv[2 * q] = v.x;
                bv[2 * q + 1] = v.y;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] = fma(av[r], bv[c], acc[r][c]);
        }
        __syncthreads();
    }
    double worst = 0.0;
    bool broken = false;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const size_t i = i0 + ty * 4 + r;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const size_t j = j0 + tx * 4 + c;
            double v = acc[r][c];
            if (!kGram) v = a[i * dp + j] - v;
            else if (minus_identity && i == j) v -= 1.0;
            out[i * dp + j] = v;
            worst = fmax(worst, fabs(v));
            broken |= v != v;
        }
    }
    if (kGram && largest) {
        // non-negative doubles are ordered like their bit patterns
        unsigned long long key = broken ? ~0ull : static_cast<unsigned long long>(__double_as_longlong(worst));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
            key = other > key ? other : key;
        }
        if ((threadIdx.x & 31) == 0) atomicMax(largest, key);
    }
}

// ---- 32 x 32 blocks in shared memory, 256 threads: thread (tx, ty) holds rows ty, ty + 8, ty + 16, ty + 24 of column tx
using Block = double[NB][NB + 1];

__device__ __forceinline__ void load_block(Block& s, const double* __restrict__ g, size_t ld, int tx, int ty) {
#pragma unroll
    for (int q = 0; q < 4; ++q) s[ty + 8 * q][tx] = g[static_cast<size_t>(ty + 8 * q) * ld + tx];
}

// r = a^T b (kTransA) or a b
template <bool kTransA>
__device__ __forceinline__ void multiply(const Block& a, const Block& b, double (&r)[4], int tx, int ty) {
#pragma unroll
    for (int q = 0; q < 4; ++q) r[q] = 0.0;
#pragma unroll 8
    for (int k = 0; k < NB; ++k) {
        const double bv = b[k][tx];
#pragma unroll
        for (int q = 0; q < 4; ++q) r[q] = fma(kTransA ? a[k][ty + 8 * q] : a[ty + 8 * q][k], bv, r[q]);
    }
}

// Cholesky factor of the block held in v (v is used up) and its inverse: r = upper factor, r_inv = its inverse.
__device__ void factor_block(double (&v)[4], double (&row)[2][NB], Block& rs, double* __restrict__ r, size_t ld, double* __restrict__ r_inv, unsigned long long* __restrict__ broken,
                             int tx, int ty) {
#pragma unroll
    for (int pq = 0; pq < 4; ++pq) {   // (split so that v is indexed by constants)
        for (int p = 8 * pq; p < 8 * pq + 8; ++p) {
            double* pivot_row = row[p & 1];
            if (ty == (p & 7)) pivot_row[tx] = v[pq];
            __syncthreads();
            double pivot = pivot_row[p];
            if (!(pivot > 0.0)) {
                if (tx == 0 && ty == 0) atomicMax(broken, ~0ull);
                pivot = 1.0;
            }
            const double scale = 1.0 / sqrt(pivot);
            const double rc = pivot_row[tx] * scale;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = ty + 8 * q;
                if (i == p) rs[p][tx] = tx >= p ? rc : 0.0;
                if (i > p) v[q] = fma(-(pivot_row[i] * scale), rc, v[q]);
            }
        }
    }
    __syncthreads();
    double x[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = ty + 8 * q;
        x[q] = i == tx ? 1.0 : 0.0;
        r[static_cast<size_t>(i) * ld + tx] = rs[i][tx];
    }
#pragma unroll
    for (int pq = 3; pq >= 0; --pq) {
        for (int p = 8 * pq + 7; p >= 8 * pq; --p) {
            double* solved = row[p & 1];
            if (ty == (p & 7)) {
                x[pq] /= rs[p][p];
                solved[tx] = x[pq];
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = ty + 8 * q;
                if (i < p) x[q] = fma(-rs[i][p], solved[tx], x[q]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) r_inv[(ty + 8 * q) * NB + tx] = x[q];
}

// Inverse of (block - S) by in-place Gauss-Jordan elimination without pivoting; S is chosen pivot by pivot so that every
// pivot has magnitude at least one.
__device__ void invert_block_signed(double (&v)[4], double (&row)[2][NB], double (&col)[2][NB], double* __restrict__ inverse, float* __restrict__ signs, size_t first, size_t d,
                                    int tx, int ty) {
#pragma unroll
    for (int pq = 0; pq < 4; ++pq) {   // (split so that v is indexed by constants)
        for (int p = 8 * pq; p < 8 * pq + 8; ++p) {
            double* pr = row[p & 1];
            double* pc = col[p & 1];
            if (ty == (p & 7)) pr[tx] = v[pq];
            if (tx == p) {
#pragma unroll
                for (int q = 0; q < 4; ++q) pc[ty + 8 * q] = v[q];
            }
            __syncthreads();
            const double w = pr[p];
            const double s = w >= 0.0 ? -1.0 : 1.0;
            const double inv = 1.0 / (w - s);
            // the last column is not reflected
            if (tx == 0 && ty == 0) signs[first + p] = static_cast<float>(first + p + 1 == d ? -s : s);
            const double scaled = (tx == p ? 1.0 : pr[tx]) * inv;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = ty + 8 * q;
                if (i == p) v[q] = scaled;
                else v[q] = (tx == p ? 0.0 : v[q]) - pc[i] * scaled;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) inverse[(ty + 8 * q) * NB + tx] = v[q];
}

// First diagonal block of either factorisation.
template <bool kCholesky>
__global__ void __launch_bounds__(kThreads) first_block_kernel(const double* __restrict__ m, size_t dp, double* __restrict__ r, double* __restrict__ inverses, float* __restrict__ signs,
                                                               size_t d, unsigned long long* __restrict__ broken) {
    __shared__ Block rs;
    __shared__ double row[2][NB], col[2][NB];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = m[static_cast<size_t>(ty + 8 * q) * dp + tx];
    if (kCholesky) factor_block(v, row, rs, r, dp, inverses, broken, tx, ty);
    else invert_block_signed(v, row, col, inverses, signs, 0, d, tx, ty);
}

// Panel k of either factorisation: block (i, j) behind the panel, i and j counted from k + 1.
//   Cholesky (i <= j): T = R_kk^-T G_k*, G_ij -= T_i^T T_j; row i = k + 1 also stores the factor's row k.
//   signs:             W_ij -= W_ik (W_kk - S_k)^-1 W_kj
template <bool kCholesky>
__global__ void __launch_bounds__(kThreads) panel_kernel(double* __restrict__ m, size_t dp, size_t k, double* __restrict__ r, double* __restrict__ inverses, float* __restrict__ signs,
                                                         size_t d, unsigned long long* __restrict__ broken) {
    const size_t i = k + 1 + blockIdx.y, j = k + 1 + blockIdx.x;
    if (kCholesky && j < i) return;
    __shared__ Block s_inv, s_a, s_b, s_t;
    __shared__ double row[2][NB], col[2][NB];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    load_block(s_inv, inverses + k * NB * NB, NB, tx, ty);
    load_block(s_b, m + (k * NB) * dp + j * NB, dp, tx, ty);
    if (kCholesky) load_block(s_a, m + (k * NB) * dp + i * NB, dp, tx, ty);
    else load_block(s_a, m + (i * NB) * dp + k * NB, dp, tx, ty);
    double* block = m + (i * NB) * dp + j * NB;
    double v[4], t[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = block[static_cast<size_t>(ty + 8 * q) * dp + tx];
    __syncthreads();
    multiply<kCholesky>(s_inv, s_b, t, tx, ty);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        s_t[ty + 8 * q][tx] = t[q];
        if (kCholesky && i == k + 1) r[(k * NB + ty + 8 * q) * dp + j * NB + tx] = t[q];
    }
    if (kCholesky) {
        multiply<true>(s_inv, s_a, t, tx, ty);
        __syncthreads();   // everyone has read s_a
#pragma unroll
        for (int q = 0; q < 4; ++q) s_a[ty + 8 * q][tx] = t[q];
    }
    __syncthreads();
    multiply<kCholesky>(s_a, s_t, t, tx, ty);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v[q] -= t[q];
        block[static_cast<size_t>(ty + 8 * q) * dp + tx] = v[q];
    }
    if (i == k + 1 && j == k + 1) {
        double* inverse = inverses + (k + 1) * NB * NB;
        __syncthreads();   // s_t is free again
        if (kCholesky) factor_block(v, row, s_t, r + ((k + 1) * NB) * dp + (k + 1) * NB, dp, inverse, broken, tx, ty);
        else invert_block_signed(v, row, col, inverse, signs, (k + 1) * NB, d, tx, ty);
    }
}

// Rows of Q = A R^-1, panel after panel; every warp keeps the solved part of its rows in shared memory, a lane per column.
// `rows` rows per block (a multiple of 8, or fewer than 8).
template <int kRowsPerWarp>
__global__ void __launch_bounds__(kThreads) solve_rows_kernel(const double* __restrict__ a, const double* __restrict__ r, const double* __restrict__ inverses, size_t dp, int rows,
                                                              double* __restrict__ q_out) {
    extern __shared__ double solved[];   // rows x dp
    __shared__ double rest[8][kRowsPerWarp][NB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp >= rows) return;   // warps work on their own rows and never meet
    const size_t row0 = static_cast<size_t>(blockIdx.x) * rows;
    double* mine[kRowsPerWarp];
    size_t row[kRowsPerWarp];
#pragma unroll
    for (int u = 0; u < kRowsPerWarp; ++u) {
        mine[u] = solved + static_cast<size_t>(warp + 8 * u) * dp;
        row[u] = min(row0 + warp + 8 * u, dp - 1);
    }
    for (size_t kb = 0; kb < dp; kb += NB) {
        double acc[kRowsPerWarp], part[kRowsPerWarp][4] = {};   // four chains: one alone is bound by the FMA's latency
#pragma unroll
        for (int u = 0; u < kRowsPerWarp; ++u) acc[u] = a[row[u] * dp + kb + lane];
        const double* __restrict__ rp = r + kb + lane;
        // four batches of loads in flight: the loop waits for L2, not for the FMAs
        double rv[4][16];
        auto load = [&](double (&v)[16], size_t j0) {
            if (j0 >= kb) return;
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = __ldg(rp + (j0 + q) * dp);
        };
#pragma unroll
        for (int b = 0; b < 4; ++b) load(rv[b], 16 * b);
        for (size_t j0 = 0; j0 < kb; j0 += 64) {
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const size_t j = j0 + 16 * b;
                if (j >= kb) break;
#pragma unroll
                for (int q = 0; q < 16; ++q)
#pragma unroll
                    for (int u = 0; u < kRowsPerWarp; ++u) part[u][q & 3] = fma(mine[u][j + q], rv[b][q], part[u][q & 3]);
                load(rv[b], j + 64);
            }
        }
        const double* __restrict__ inv = inverses + (kb / NB) * NB * NB + lane;
        double iv[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) iv[b] = __ldg(inv + b * NB);
#pragma unroll
        for (int u = 0; u < kRowsPerWarp; ++u) rest[warp][u][lane] = acc[u] - ((part[u][0] + part[u][1]) + (part[u][2] + part[u][3]));
        __syncwarp();
        double x[kRowsPerWarp] = {};
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int u = 0; u < kRowsPerWarp; ++u) x[u] = fma(rest[warp][u][b], iv[b], x[u]);
#pragma unroll
        for (int u = 0; u < kRowsPerWarp; ++u) {
            mine[u][kb + lane] = x[u];
            if (row0 + warp + 8 * u < dp) q_out[row[u] * dp + kb + lane] = x[u];
        }
        __syncwarp();
    }
}

__global__ void signed_columns_kernel(const double* __restrict__ q, const float* __restrict__ signs, size_t d, size_t dp, float* __restrict__ out) {
    const size_t j = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (j < d) out[i * d + j] = static_cast<float>(q[i * dp + j] * signs[j]);
}

template <bool kCholesky>
void factorise(double* m, size_t dp, double* r, double* inverses, float* signs, size_t d, unsigned long long* broken, cudaStream_t stream) {
    first_block_kernel<kCholesky><<<1, kThreads, 0, stream>>>(m, dp, r, inverses, signs, d, broken);
    SKM_LAUNCH_CHECK();
    const size_t panels = dp / NB;
    for (size_t k = 0; k + 1 < panels; ++k) {
        const unsigned left = static_cast<unsigned>(panels - 1 - k);
        panel_kernel<kCholesky><<<dim3(left, left), kThreads, 0, stream>>>(m, dp, k, r, inverses, signs, d, broken);
        SKM_LAUNCH_CHECK();
    }
}

} // namespace

void launch_collect_draws(const DrawPieces& p, float* out, cudaStream_t stream) {
    if (p.n == 0) return;
    collect_draws_kernel<<<dim3(16, p.n), kThreads, 0, stream>>>(p, out);
    SKM_LAUNCH_CHECK();
}

static bool factorise_on_device(const float* draws, size_t d, float* out, cudaStream_t stream) {
    const size_t dp = (d + GT - 1) / GT * GT;
    // rows per block of the solve: as many as the row buffer holds, but no more than leave a block for most SMs
    int rows = kSolveMaxRows;
    while (rows > 1 && (static_cast<size_t>(rows) * dp * sizeof(double) > kSolveSmem || (rows > 8 && dp < 1536))) rows /= 2;
    if (static_cast<size_t>(rows) * dp * sizeof(double) > kSolveSmem) return false;

    DeviceBuffer<double> a_buf, q_buf, g_buf, r_buf, inv_buf;
    DeviceBuffer<float> signs_buf;
    DeviceBuffer<unsigned long long> worst_buf;
    double* a = a_buf.ensure(dp * dp);
    double* q = q_buf.ensure(dp * dp);
    double* g = g_buf.ensure(dp * dp);
    double* r = r_buf.ensure(dp * dp);
    double* inverses = inv_buf.ensure(dp * NB);
    float* signs = signs_buf.ensure(dp);
    unsigned long long* worst = worst_buf.ensure(1);
    const dim3 cells(static_cast<unsigned>((dp + 255) / 256), static_cast<unsigned>(dp));
    const dim3 tiles(static_cast<unsigned>(dp / GN), static_cast<unsigned>(dp / GT));

    widen_draws_kernel<<<cells, 256, 0, stream>>>(draws, d, dp, a);
    SKM_LAUNCH_CHECK();
    SKM_CUDA(cudaMemsetAsync(worst, 0, sizeof(unsigned long long), stream));
    product_kernel<true><<<tiles, kProductThreads, 0, stream>>>(a, nullptr, dp, g, false, nullptr);
    SKM_LAUNCH_CHECK();
    factorise<true>(g, dp, r, inverses, nullptr, d, worst, stream);
    const size_t smem = static_cast<size_t>(rows) * dp * sizeof(double);
    const unsigned blocks = static_cast<unsigned>((dp + rows - 1) / rows);
    if (rows == kSolveMaxRows) {
        SKM_CUDA(cudaFuncSetAttribute(solve_rows_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSolveSmem)));
        solve_rows_kernel<2><<<blocks, kThreads, smem, stream>>>(a, r, inverses, dp, rows, q);
    } else {
        SKM_CUDA(cudaFuncSetAttribute(solve_rows_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSolveSmem)));
        solve_rows_kernel<1><<<blocks, kThreads, smem, stream>>>(a, r, inverses, dp, rows, q);
    }
    SKM_LAUNCH_CHECK();

    // each turn squares the distance from orthonormality
    double* cur = q;
    double* next = a;
    for (int turn = 0;; ++turn) {
        product_kernel<true><<<tiles, kProductThreads, 0, stream>>>(cur, nullptr, dp, g, true, worst);
        SKM_LAUNCH_CHECK();
        product_kernel<false><<<tiles, kProductThreads, 0, stream>>>(cur, g, dp, next, false, nullptr);
        SKM_LAUNCH_CHECK();
        std::swap(cur, next);
        unsigned long long bits = 0;
        SKM_CUDA(cudaMemcpyAsync(&bits, worst, sizeof(bits), cudaMemcpyDeviceToHost, stream));
        SKM_CUDA(cudaMemsetAsync(worst, 0, sizeof(unsigned long long), stream));
        SKM_CUDA(cudaStreamSynchronize(stream));
        double e;
        static_assert(sizeof(e) == sizeof(bits), "one word");
        std::memcpy(&e, &bits, sizeof(e));   // a NaN when a pivot or a product was none
        if (!(e < 0.01) || turn == 4) return false;
        if (e * e * static_cast<double>(d) < 1e-15) break;
    }
    SKM_CUDA(cudaMemcpyAsync(next, cur, sizeof(double) * dp * dp, cudaMemcpyDeviceToDevice, stream));
    factorise<false>(next, dp, nullptr, inverses, signs, d, worst, stream);
    signed_columns_kernel<<<dim3(static_cast<unsigned>((d + 255) / 256), static_cast<unsigned>(d)), 256, 0, stream>>>(cur, signs, d, dp, out);
    SKM_LAUNCH_CHECK();
    return true;
}

bool make_rotation_matrix_on_device(const float* draws, size_t d, float* out, cudaStream_t stream) {
    try {
        return factorise_on_device(draws, d, out, stream);
    } catch (const OutOfMemory&) {
        return false;
    }
}

} // namespace skmb
