// The random orthogonal matrix of the ADSampling rotation (adsampling.h:76-85) from its Gaussian draws, on the GPU.
//
// The matrix is the Q factor of the d x d draws with the signs of a Householder QR; host_logic.h computes it column by
// column on the host (0.25 s at d = 768, 1.2 s at d = 1536 on 16 cores: twice d rank-one updates of a matrix that
// does not stay in cache).  Householder steps are a chain of d reductions here too, so Q is computed another way, in
// double throughout, from products and one chain of d / 32 launches:
//
//   1. G = A^T A;
//   2. panel after panel of 32 columns, three eliminations side by side:
//        Cholesky   G = R^T R;
//        solve      Q = A R^-1, the panel's columns of Q and what they leave of the columns behind them;
//        signs      this Q has a positive diagonal in R.  Householder's sign for column k is minus the sign of entry (k, k) of what is
//                   left of the column after k reflections, which is the k-th pivot of the elimination of Q - S without
//                   pivoting, S = diag(signs), chosen as the elimination goes (the reconstruction of Householder vectors from an
//                   orthonormal basis: Ballard, Demmel, Grigori, Jacquelin, Nguyen, Solomonik, 2014); the last column keeps its
//                   sign.  As Q - S = L U means A - S R = L (U R), the elimination is done on A - S R, whose pivots have the same
//                   signs, a panel behind the Cholesky factor that it takes its rows of R from: it need not wait for Q;
//   3. E = Q^T Q - I (at most cond(A)^2 * 1e-16), Q <- Q (I - up(E)), up = strict upper part + half the diagonal: the first
//      order of a second Cholesky QR.  Each turn squares E; repeated until that is far below the rounding of the result.
//
// A launch of the chain is a grid of 64 x 64 tiles of the three trailing matrices, each of which recomputes the 32 x 64 products that
// it needs of the panel (half of its work, against another launch and a round trip), and two blocks that make the next
// diagonal block of either elimination and invert it: one warp each, a lane per column in registers, because 32 dependent
// pivots are what the launch takes when the tiles are few.
// One B200, kernels behind the draws, against a chain of launches for each elimination with the solve between them: d = 768: 1.4 -> 0.5 ms
// (0.29 of them the chain), d = 1024: 2.3 -> 0.8, d = 1536: 5.2 -> 2.0 (1.18 the chain, whose first launches are bound by fp64 issue
// at 60 us each, the last by their pivots at 9).
//
// A matrix too close to singular for this (or too wide for the memory that is left: the scratch is 40 bytes an element) is declined:
// the caller takes the host's.
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "engine.h"

namespace skmb {

namespace {

constexpr int NB = 32;    // panel width of the eliminations
constexpr int GT = 64;    // tiles of the trailing matrices, and of the products: GT x GN
constexpr int GN = 32;
constexpr int kProductThreads = GT / 4 * GN / 4;
constexpr int GK = 16;
constexpr int kThreads = 256;

// A column of blocks per piece; pinned memory is read in place.
__global__ void __launch_bounds__(kThreads) collect_draws_kernel(const DrawPieces p, float* __restrict__ out) {
    const uint32_t t = blockIdx.y;
    const float* from = p.values + t * p.stretch;
    const size_t at = p.start[t], n = p.start[t + 1] - at;
    for (size_t i = static_cast<size_t>(blockIdx.x) * kThreads + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * kThreads) out[at + i] = from[i];
}

// Two double copies of the draws, padded with the identity to a multiple of GT, so that nothing below has edges.
__global__ void widen_draws_kernel(const float* __restrict__ draws, size_t d, size_t dp, double* __restrict__ a, double* __restrict__ w) {
    const size_t j = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (j >= dp) return;
    const double v = (i < d && j < d) ? static_cast<double>(draws[i * d + j]) : (i == j ? 1.0 : 0.0);
    a[i * dp + j] = v;
    w[i * dp + j] = v;
}

// 4 x 4 products per thread for one value of the reduction index; a and b hold the tile's rows and columns for it.  Thread (tx, ty) has rows
// 4 ty .. and columns 2 tx, 2 tx + 1, kHalf + 2 tx and the next: the lanes' 16-byte reads of b then lie side by side (four columns in a row
// are read in twice the time, and shared memory is the bound).
template <int kHalf>
__device__ __forceinline__ void multiply_add_4x4(const double* __restrict__ a, const double* __restrict__ b, double (&acc)[4][4], int tx, int ty) {
    double av[4], bv[4];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const double2 u = *reinterpret_cast<const double2*>(a + ty * 4 + q * 2);
        const double2 v = *reinterpret_cast<const double2*>(b + tx * 2 + q * kHalf);
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
// the column of acc[..][c]
template <int kHalf>
__device__ __forceinline__ int column_of(int tx, int c) {
    return tx * 2 + (c & 1) + (c >> 1) * kHalf;
}

// kGram: out = a^T a, tiles on and above the diagonal; with `minus_identity` I is subtracted and *largest becomes the
// largest |entry| as an ordered integer (all ones for a NaN).   !kGram: out = a - a up(e).
// Tiles of 64 x 32, the next 16 of K in registers while the present ones are multiplied: twice the blocks of 64 x 64, which leave a last
// wave nearly empty (d = 1536: 300 on 296 places).  The tiles with the longest sums come first.
template <bool kGram>
__global__ void __launch_bounds__(kProductThreads) product_kernel(const double* __restrict__ a, const double* __restrict__ e, size_t dp, double* __restrict__ out, bool minus_identity,
                                                              unsigned long long* __restrict__ largest) {
    __shared__ __align__(16) double sa[2][GK][GT + 2];
    __shared__ __align__(16) double sb[2][GK][GN + 2];
    const size_t j0 = static_cast<size_t>(gridDim.y - 1 - blockIdx.y) * GN, i0 = static_cast<size_t>(blockIdx.x) * GT;
    if (kGram && j0 + GN <= i0) return;
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    double acc[4][4] = {};
    const size_t k_end = kGram ? dp : j0 + GN;   // up(e) is zero below the diagonal
    constexpr int NA = GK * GT / kProductThreads, NV = GK * GN / kProductThreads;
    double va[NA], vb[NV];
    auto fetch = [&](size_t k0) {
#pragma unroll
        for (int u = 0; u < NA; ++u) {
            const int q = threadIdx.x + u * kProductThreads;
            if (kGram) va[u] = a[(k0 + (q / GT)) * dp + i0 + q % GT];
            else va[u] = a[(i0 + q / GK) * dp + k0 + q % GK];
        }
#pragma unroll
        for (int u = 0; u < NV; ++u) {
            const int q = threadIdx.x + u * kProductThreads;
            const size_t row = k0 + q / GN, col = j0 + q % GN;
            if (kGram) vb[u] = a[row * dp + col];
            else vb[u] = row < col ? e[row * dp + col] : (row == col ? 0.5 * e[row * dp + col] : 0.0);
        }
    };
    fetch(0);
    int s = 0;
    for (size_t k0 = 0; k0 < k_end; k0 += GK, s ^= 1) {
#pragma unroll
        for (int u = 0; u < NA; ++u) {
            const int q = threadIdx.x + u * kProductThreads;
            if (kGram) sa[s][q / GT][q % GT] = va[u];
            else sa[s][q % GK][q / GK] = va[u];
        }
#pragma unroll
        for (int u = 0; u < NV; ++u) {
            const int q = threadIdx.x + u * kProductThreads;
            sb[s][q / GN][q % GN] = vb[u];
        }
        __syncthreads();   // (whoever still multiplies the other buffer has passed this of the step before)
        if (k0 + GK < k_end) fetch(k0 + GK);
#pragma unroll
        for (int kk = 0; kk < GK; ++kk) multiply_add_4x4<GN / 2>(sa[s][kk], sb[s][kk], acc, tx, ty);
    }
    double worst = 0.0;
    bool broken = false;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const size_t i = i0 + ty * 4 + r;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const size_t j = j0 + column_of<GN / 2>(tx, c);
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

// ---- the chain

struct Chain {
    size_t dp, d, panels;
    double* g;                // A^T A; above the diagonal: what is left of it
    double* a;                // A: what is left of it for the solve
    double* w;                // A: ... and for the signs
    double* q;                // out
    double* r;                // R, rows of the panels behind the present one
    double* r_inverse;        // per panel 32 x 32: the inverse of R's diagonal block
    double* s_inverse;        // ... the transposed inverse of the diagonal block of A - S R
    float* signs;             // out, per column
    unsigned long long* broken;
};

using Block = double[NB][NB + 2];     // (rows start on 16 bytes)
using Panel = double[NB][GT + 2];

struct ChainShared {
    Block x;
    Panel pi, pj;
};

__device__ __forceinline__ void load_block(Block& s, const double* __restrict__ from, size_t ld) {
#pragma unroll
    for (int u = 0; u < NB * NB / kThreads; ++u) {
        const int q = threadIdx.x + u * kThreads;
        s[q / NB][q % NB] = from[static_cast<size_t>(q / NB) * ld + q % NB];
    }
}

// p = x^T p, in place
__device__ __forceinline__ void apply_transposed(const Block& x, Panel& p) {
    const int c = (threadIdx.x & 31) * 2, r = (threadIdx.x >> 5) * 4;
    double acc[4][2] = {};
#pragma unroll 8
    for (int k = 0; k < NB; ++k) {
        const double2 v = *reinterpret_cast<const double2*>(&p[k][c]);
        const double2 u0 = *reinterpret_cast<const double2*>(&x[k][r]), u1 = *reinterpret_cast<const double2*>(&x[k][r + 2]);
        const double u[4] = {u0.x, u0.y, u1.x, u1.y};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            acc[q][0] = fma(u[q], v.x, acc[q][0]);
            acc[q][1] = fma(u[q], v.y, acc[q][1]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) *reinterpret_cast<double2*>(&p[r + q][c]) = make_double2(acc[q][0], acc[q][1]);
    __syncthreads();
}

// Columns first .. first + 63 of rows row0 .. row0 + 31, zero from dp on; minus S R for the signs' rows.
__device__ __forceinline__ void load_panel_rows(Panel& p, const double* __restrict__ from, size_t dp, size_t row0, size_t first, const double* __restrict__ r, const float* __restrict__ signs) {
#pragma unroll
    for (int u = 0; u < NB * GT / kThreads; ++u) {
        const int q = threadIdx.x + u * kThreads;
        const size_t i = row0 + q / GT, j = first + q % GT;
        double v = 0.0;
        if (j < dp) {
            v = from[i * dp + j];
            if (signs) v -= static_cast<double>(signs[i]) * r[i * dp + j];
        }
        p[q / GT][q % GT] = v;
    }
}

// Rows first .. first + 63 of columns col0 .. col0 + 31, transposed, zero from dp on.
__device__ __forceinline__ void load_panel_columns(Panel& p, const double* __restrict__ from, size_t dp, size_t first, size_t col0) {
#pragma unroll
    for (int u = 0; u < NB * GT / kThreads; ++u) {
        const int q = threadIdx.x + u * kThreads;
        const size_t i = first + q / NB;
        p[q % NB][q / NB] = i < dp ? from[i * dp + col0 + q % NB] : 0.0;
    }
}

// m[I ..][J ..] -= pi^T pj, but for the block (skip, skip)
__device__ __forceinline__ void update_tile(double* __restrict__ m, size_t dp, size_t i0, size_t j0, const Panel& pi, const Panel& pj, size_t skip) {
    constexpr int kHalf = GT / 2;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const size_t i = i0 + ty * 4;
    bool mine[2];   // (each pair of columns lies in a block of its own)
    double2 old[4][2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const size_t j = j0 + tx * 2 + c * kHalf;
        mine[c] = i < dp && j < dp && !(i / NB == skip && j / NB == skip);
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (mine[c]) old[r][c] = *reinterpret_cast<const double2*>(m + (i + r) * dp + j);
    }
    double acc[4][4] = {};
#pragma unroll 8
    for (int k = 0; k < NB; ++k) multiply_add_4x4<kHalf>(pi[k], pj[k], acc, tx, ty);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const size_t j = j0 + tx * 2 + c * kHalf;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (mine[c]) *reinterpret_cast<double2*>(m + (i + r) * dp + j) = make_double2(old[r][c].x - acc[r][2 * c], old[r][c].y - acc[r][2 * c + 1]);
    }
}

// 32 x 32 blocks, 2 x 2 values per thread of 256: acc = u^T v
__device__ __forceinline__ void multiply_blocks(const Block& u, const Block& v, double (&acc)[2][2], int r, int c) {
    acc[0][0] = acc[0][1] = acc[1][0] = acc[1][1] = 0.0;
#pragma unroll 8
    for (int q = 0; q < NB; ++q) {
        const double2 a = *reinterpret_cast<const double2*>(&u[q][r]), b = *reinterpret_cast<const double2*>(&v[q][c]);
        acc[0][0] = fma(a.x, b.x, acc[0][0]);
        acc[0][1] = fma(a.x, b.y, acc[0][1]);
        acc[1][0] = fma(a.y, b.x, acc[1][0]);
        acc[1][1] = fma(a.y, b.y, acc[1][1]);
    }
}

// out = from - left^T T, T = x^T y (kept in `t`; left may be t)
__device__ __forceinline__ void update_block(const Block& x, const Block& y, Block& t, const Block& left, const double* __restrict__ from, size_t ld, Block& out) {
    const int c = (threadIdx.x & 15) * 2, r = (threadIdx.x >> 4) * 2;
    double2 old[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) old[q] = *reinterpret_cast<const double2*>(from + static_cast<size_t>(r + q) * ld + c);
    double acc[2][2];
    multiply_blocks(x, y, acc, r, c);
#pragma unroll
    for (int q = 0; q < 2; ++q) *reinterpret_cast<double2*>(&t[r + q][c]) = make_double2(acc[q][0], acc[q][1]);
    __syncthreads();
    multiply_blocks(left, t, acc, r, c);
    __syncthreads();   // (out may be one of those)
#pragma unroll
    for (int q = 0; q < 2; ++q) *reinterpret_cast<double2*>(&out[r + q][c]) = make_double2(old[q].x - acc[q][0], old[q].y - acc[q][1]);
    __syncthreads();
}

__device__ __forceinline__ double from_lane(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

// The first two warps of a block, of which one waits until the other has come here.
__device__ __forceinline__ void announce(int barrier) { asm volatile("bar.arrive %0, 64;" ::"r"(barrier) : "memory"); }
__device__ __forceinline__ void await(int barrier) { asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory"); }

// Cholesky factor R of the block m and its inverse: elimination of the block, by the first warp, and eight pivots behind it of the identity,
// by the second, a lane per column, gives L D L^T and L^-1; R = D^1/2 L^T, R^-1 = L^-T D^-1/2.  On return rows holds R (on and above
// the diagonal), inverse its inverse.
__device__ void factor_block(const Block& m, Block& inverse, Block& rows, double* roots, unsigned long long* __restrict__ broken) {
    constexpr int kAhead = 8;
    const int c = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        double v[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) v[i] = m[i][c];
#pragma unroll
        for (int p = 0; p < NB; ++p) {
            double pivot = from_lane(v[p], p);
            if (!(pivot > 0.0)) {
                if (c == 0) atomicMax(broken, ~0ull);
                pivot = 1.0;
            }
            const double root = rsqrt(pivot);    // 1 / R_pp
            const double row = v[p] * root;      // row p of R, from column p on
            rows[p][c] = row;
            if (c == 0) roots[p] = root;
            __syncwarp();
#pragma unroll
            for (int i = p + 1; i < NB; ++i) v[i] = fma(-rows[p][i], row, v[i]);
            if ((p + 1) % kAhead == 0) announce(1 + p / kAhead);
        }
    } else if (threadIdx.x < 64) {
        double z[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) z[i] = i == c ? 1.0 : 0.0;
#pragma unroll
        for (int p = 0; p < NB; ++p) {
            if (p % kAhead == 0) await(1 + p / kAhead);
            const double mine = z[p] * roots[p];   // row p of D^-1/2 L^-1, up to column p
            inverse[c][p] = c <= p ? mine : 0.0;
#pragma unroll
            for (int i = p + 1; i < NB; ++i) z[i] = fma(-rows[p][i], mine, z[i]);
        }
    }
    __syncthreads();
}

// Inverse of (m - S R) by in-place Gauss-Jordan elimination without pivoting, by all threads: thread (tx, ty) holds rows ty, ty + 8, ty + 16 and
// ty + 24 of column tx.  S is chosen pivot by pivot so that no pivot is smaller than R's.  On return m holds the transposed inverse.  (By
// one warp, with whole columns in registers as above, it took 40 us.)
__device__ void invert_block_signed(Block& m, const Block& r, double (&row)[2][NB], double (&col)[2][NB], float* __restrict__ signs, size_t first, size_t d) {
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = m[ty + 8 * q][tx];
    __syncthreads();
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
            // the last column is not reflected
            if (tx == 0 && ty == 0) signs[first + p] = static_cast<float>(first + p + 1 == d ? -s : s);
            const double inv = 1.0 / (w - s * r[p][p]);
            const double scaled = (tx == p ? 1.0 : pr[tx] - s * r[p][tx]) * inv;   // (R is zero below the diagonal)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = ty + 8 * q;
                if (i == p) v[q] = scaled;
                else v[q] = (tx == p ? 0.0 : v[q]) - pc[i] * scaled;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) m[tx][ty + 8 * q] = v[q];
    __syncthreads();
}

// First diagonal block of R.
__global__ void __launch_bounds__(kThreads) first_block_kernel(const Chain p) {
    __shared__ __align__(16) Block m, inverse, rows;
    __shared__ double roots[NB];
    load_block(m, p.g, p.dp);
    __syncthreads();
    factor_block(m, inverse, rows, roots, p.broken);
    for (int q = threadIdx.x; q < NB * NB; q += kThreads) {
        p.r[static_cast<size_t>(q / NB) * p.dp + q % NB] = q % NB >= q / NB ? rows[q / NB][q % NB] : 0.0;
        p.r_inverse[q] = inverse[q / NB][q % NB];
    }
}

// Launch k of the chain: Cholesky and solve of panel k (R's diagonal block k is there), signs of panel k - 1, and the diagonal
// blocks k + 1 and k that the next launch needs of them.
__global__ void __launch_bounds__(kThreads, 2) panel_kernel(const Chain p, const size_t k) {
    __shared__ __align__(16) union {
        ChainShared tile;
        Block blocks[4];
    } shared;
    __shared__ double roots[NB], pivot_row[2][NB], pivot_col[2][NB];
    ChainShared& sh = shared.tile;
    const size_t dp = p.dp, behind = p.panels - 1 - k;   // panels behind k
    const unsigned nb = static_cast<unsigned>((behind + 1) / 2), n_rows = static_cast<unsigned>(dp / GT);
    const unsigned n_factor = nb * (nb + 1) / 2, n_solve = n_rows * (nb > 0 ? nb : 1), n_signs = k > 0 ? static_cast<unsigned>((behind + 2) / 2) : 0u;
    unsigned t = blockIdx.x;
    if (t == 0) {
        if (behind == 0) return;
        // ---- R's diagonal block k + 1
        Block &x = shared.blocks[0], &y = shared.blocks[1], &m = shared.blocks[2], &rows = shared.blocks[3];
        load_block(x, p.r_inverse + k * NB * NB, NB);
        load_block(y, p.g + k * NB * dp + (k + 1) * NB, dp);
        __syncthreads();
        update_block(x, y, rows, rows, p.g + ((k + 1) * NB) * dp + (k + 1) * NB, dp, m);
        factor_block(m, x, rows, roots, p.broken);
        double* r = p.r + ((k + 1) * NB) * dp + (k + 1) * NB;
        double* inverse = p.r_inverse + (k + 1) * NB * NB;
        for (int q = threadIdx.x; q < NB * NB; q += kThreads) {
            r[static_cast<size_t>(q / NB) * dp + q % NB] = q % NB >= q / NB ? rows[q / NB][q % NB] : 0.0;
            inverse[q] = x[q / NB][q % NB];
        }
        return;
    }
    if (t == 1) {
        // ---- the signs' diagonal block k
        Block &x = shared.blocks[0], &y = shared.blocks[1], &left = shared.blocks[2], &m = shared.blocks[3];
        const double* from = p.w + (k * NB) * dp + k * NB;
        if (k == 0) {
            load_block(m, from, dp);
        } else {
            const size_t before = (k - 1) * NB;
            load_block(x, p.s_inverse + before * NB, NB);
#pragma unroll
            for (int u = 0; u < NB * NB / kThreads; ++u) {
                const int q = threadIdx.x + u * kThreads;
                const size_t i = before + q / NB, j = k * NB + q % NB;
                y[q / NB][q % NB] = p.w[i * dp + j] - static_cast<double>(p.signs[i]) * p.r[i * dp + j];
                left[q % NB][q / NB] = p.w[(k * NB + q / NB) * dp + before + q % NB];
            }
            __syncthreads();
            update_block(x, y, m, left, from, dp, m);
        }
        load_block(y, p.r + (k * NB) * dp + k * NB, dp);
        __syncthreads();
        invert_block_signed(m, y, pivot_row, pivot_col, p.signs, k * NB, p.d);
        double* inverse = p.s_inverse + k * NB * NB;
        for (int q = threadIdx.x; q < NB * NB; q += kThreads) inverse[q] = m[q / NB][q % NB];
        return;
    }
    t -= 2;
    if (t < n_factor) {
        unsigned bi = 0;
        while (t >= nb - bi) {
            t -= nb - bi;
            ++bi;
        }
        const size_t i0 = (k + 1) * NB + static_cast<size_t>(bi) * GT, j0 = i0 + static_cast<size_t>(t) * GT;
        load_block(sh.x, p.r_inverse + k * NB * NB, NB);
        load_panel_rows(sh.pi, p.g, dp, k * NB, i0, nullptr, nullptr);
        if (t != 0) load_panel_rows(sh.pj, p.g, dp, k * NB, j0, nullptr, nullptr);
        __syncthreads();
        apply_transposed(sh.x, sh.pi);
        if (t != 0) apply_transposed(sh.x, sh.pj);
        const Panel& pj = t != 0 ? sh.pj : sh.pi;
        if (bi == 0) {   // row k of R
#pragma unroll
            for (int u = 0; u < NB * GT / kThreads; ++u) {
                const int q = threadIdx.x + u * kThreads;
                if (j0 + q % GT < dp) p.r[(k * NB + q / GT) * dp + j0 + q % GT] = pj[q / GT][q % GT];
            }
        }
        update_tile(p.g, dp, i0, j0, sh.pi, pj, k + 1);
        return;
    }
    t -= n_factor;
    if (t < n_solve) {
        const size_t i0 = static_cast<size_t>(t % n_rows) * GT, j0 = (k + 1) * NB + static_cast<size_t>(t / n_rows) * GT;
        load_block(sh.x, p.r_inverse + k * NB * NB, NB);
        load_panel_columns(sh.pi, p.a, dp, i0, k * NB);
        if (nb > 0) load_panel_rows(sh.pj, p.g, dp, k * NB, j0, nullptr, nullptr);
        __syncthreads();
        apply_transposed(sh.x, sh.pi);   // Q's columns of the panel, transposed
        if (t < n_rows) {
#pragma unroll
            for (int u = 0; u < NB * GT / kThreads; ++u) {
                const int q = threadIdx.x + u * kThreads;
                p.q[(i0 + q / NB) * dp + k * NB + q % NB] = sh.pi[q % NB][q / NB];
            }
        }
        if (nb == 0) return;
        apply_transposed(sh.x, sh.pj);
        update_tile(p.a, dp, i0, j0, sh.pi, sh.pj, ~size_t{0});
        return;
    }
    t -= n_solve;
    {
        const size_t m = k - 1, i0 = k * NB + static_cast<size_t>(t % n_signs) * GT, j0 = k * NB + static_cast<size_t>(t / n_signs) * GT;
        load_block(sh.x, p.s_inverse + m * NB * NB, NB);
        load_panel_columns(sh.pi, p.w, dp, i0, m * NB);
        load_panel_rows(sh.pj, p.w, dp, m * NB, j0, p.r, p.signs);
        __syncthreads();
        apply_transposed(sh.x, sh.pj);
        update_tile(p.w, dp, i0, j0, sh.pi, sh.pj, k);
    }
}

__global__ void signed_columns_kernel(const double* __restrict__ q, const float* __restrict__ signs, size_t d, size_t dp, float* __restrict__ out) {
    const size_t j = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (j < d) out[i * d + j] = static_cast<float>(q[i * dp + j] * signs[j]);
}

void run_chain(const Chain& p, cudaStream_t stream) {
    first_block_kernel<<<1, kThreads, 0, stream>>>(p);
    SKM_LAUNCH_CHECK();
    for (size_t k = 0; k < p.panels; ++k) {
        const size_t behind = p.panels - 1 - k, nb = (behind + 1) / 2, rows = p.dp / GT, signs = k > 0 ? (behind + 2) / 2 : 0;
        const size_t blocks = 2 + nb * (nb + 1) / 2 + rows * std::max<size_t>(nb, 1) + signs * signs;
        panel_kernel<<<static_cast<unsigned>(blocks), kThreads, 0, stream>>>(p, k);
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
    DeviceBuffer<double> a_buf, w_buf, q_buf, g_buf, r_buf, inv_buf;
    DeviceBuffer<float> signs_buf;
    DeviceBuffer<unsigned long long> worst_buf;
    PinnedBuffer<unsigned long long> bits;
    bits.ensure(1);
    double* a = a_buf.ensure(dp * dp);
    double* w = w_buf.ensure(dp * dp);
    double* q = q_buf.ensure(dp * dp);
    double* g = g_buf.ensure(dp * dp);
    double* r = r_buf.ensure(dp * dp);
    double* inverses = inv_buf.ensure(2 * dp * NB);
    float* signs = signs_buf.ensure(dp);
    unsigned long long* worst = worst_buf.ensure(1);
    const dim3 cells(static_cast<unsigned>((dp + 255) / 256), static_cast<unsigned>(dp));
    const dim3 tiles(static_cast<unsigned>(dp / GT), static_cast<unsigned>(dp / GN));

    widen_draws_kernel<<<cells, 256, 0, stream>>>(draws, d, dp, a, w);
    SKM_LAUNCH_CHECK();
    SKM_CUDA(cudaMemsetAsync(worst, 0, sizeof(unsigned long long), stream));
    product_kernel<true><<<tiles, kProductThreads, 0, stream>>>(a, nullptr, dp, g, false, nullptr);
    SKM_LAUNCH_CHECK();
    run_chain(Chain{dp, d, dp / NB, g, a, w, q, r, inverses, inverses + dp * NB, signs, worst}, stream);

    // each turn squares the distance from orthonormality
    double* cur = q;
    double* next = a;
    for (int turn = 0;; ++turn) {
        if (turn > 0) SKM_CUDA(cudaMemsetAsync(worst, 0, sizeof(unsigned long long), stream));
        product_kernel<true><<<tiles, kProductThreads, 0, stream>>>(cur, nullptr, dp, g, true, worst);
        SKM_LAUNCH_CHECK();
        product_kernel<false><<<tiles, kProductThreads, 0, stream>>>(cur, g, dp, next, false, nullptr);
        SKM_LAUNCH_CHECK();
        std::swap(cur, next);
        // (a copy to pageable memory would keep other threads' calls waiting as long as the chain takes: 0.4 ms in which no rows are uploaded)
        SKM_CUDA(cudaMemcpyAsync(bits.get(), worst, sizeof(unsigned long long), cudaMemcpyDeviceToHost, stream));
        SKM_CUDA(cudaStreamSynchronize(stream));
        double e;
        static_assert(sizeof(e) == sizeof(unsigned long long), "one word");
        std::memcpy(&e, bits.get(), sizeof(e));   // a NaN when a pivot or a product was none
        if (!(e < 0.01) || turn == 4) return false;
        // What is left is at most d e^2: the result is rounded to 24 bits.
        if (e * e * static_cast<double>(d) < 1e-12) break;
    }
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
