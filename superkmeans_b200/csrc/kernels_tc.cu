// Tensor-core (tcgen05) kernels for sm_100a: X * Y^T with fp32 operands and fp32-level accuracy.
//
// Every fp32 operand value v is split into hi = tf32(v) and lo = tf32(v - hi); the product is accumulated as
// hi*hi + hi*lo + lo*hi (three kind::tf32 MMAs per k-step, fp32 accumulation in tensor memory), which restores
// fp32-level accuracy of the products.  The points (X) are split in shared memory by splitter warps; the
// centroids (Y), which every CTA re-reads, can arrive already split from global memory (split_tf32_kernel).
//
// gemm_tc_kernel: one persistent CTA per SM, 448 threads:
//   warp 0       TMA producer: cp.async.bulk.tensor loads of a 128 x 16 tile of X and a 256 x 16 tile of Y
//                (hi and lo when pre-split; 64-byte swizzle) into a 4-stage ring;
//   warp 1       MMA issuer: tcgen05.mma (M = 128, N = 256, K = 8) into one of two 256-column accumulators in
//                tensor memory, tcgen05.commit to release stages / publish tiles;
//   warps 2-5    splitters: rewrite each landed X (and raw Y) tile in place as its hi part and write the lo part
//                beside it (element-wise, so the swizzle pattern never has to be decoded);
//   warps 6-9    epilogue: tcgen05.ld, one thread per row.  Three epilogues: the two smallest
//                ||x||^2 + ||y||^2 - 2 x.y per row (exact assignment), a plain store, and the first ADSampling
//                test as union bits or counts (its lists: kernels_first_test.cu);
//   warps 10-13  second half of the epilogue warps in the union and counting modes (idle otherwise).
// Rows / columns / k beyond the matrix edges are zero-filled by TMA, so any n, k and K work as long as the row
// pitch is a multiple of 16 bytes.
//
// Every wait on an mbarrier is bounded: on expiry the kernel records an error code, all roles leave their loops,
// tensor memory is released and the kernel returns.
#include <cuda.h>

#include <cfloat>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <stdexcept>

#include "common.cuh"
#include "kernels_tc.cuh"
#include "tc_ptx.cuh"

namespace skmb {
namespace tc {

struct Params {
    size_t n;         // rows of X
    size_t k;         // rows of Y
    uint32_t kdim;    // reduction length
    // arg-min epilogue
    const float* norms_x;
    const float* norms_y;
    uint32_t* out_knn;
    float* out_dist;
    uint2* out_top2;  // per row: the two best candidate indices found by the tensor-core pass
    // store epilogue
    float* out;
    size_t ldo;
    int* error;
    long long wait_limit;   // SM cycles after which a wait gives up
    // union and counting epilogues: rows [tile0 * 128, (tile0 + n_tiles) * 128) are processed; norms_x / norms_y
    // hold the norms over the first kdim dimensions
    size_t tile0;
    size_t n_tiles;        // 0 = all row tiles (other modes)
    const float* best_in;  // n: exact distance to the previous centroid
    const uint32_t* skip;  // n or null: 1 = row handled elsewhere
    float ratio_first;     // ratios[kdim]
    // union mode: when set, entry t of the launch's tile range works on row tile tile_map[t]
    // (rows tile_map[t] * 128 ...) instead of row tile tile0 + t; lists and union words stay indexed by t
    const uint32_t* tile_map;
    // union epilogue (MODE_UNION): bit c of union_bits[t * union_words + c / 32] is set when at least one row of the
    // tile passes the (slightly widened) first test against centroid c
    uint32_t* union_bits;
    uint32_t union_words;
    // counting epilogue (MODE_COUNT): count_out[row] += number of centroids whose partial distance over the first kdim
    // dimensions is below thr_rows[row * thr_chunks + chunk of 1024 the centroid lies in]
    const float* thr_rows;
    uint32_t thr_chunks;
    uint32_t* count_out;
    // Y arrives already split: tmap_y covers the hi parts, tmap_ylo the lo parts, and the splitter warps
    // only treat X
    bool y_presplit;
    // test hook: when non-zero the producer stops after this many k-blocks, so that the roles behind it wait for
    // data that never arrives, run into the wait limit and the kernel returns with an error code
    uint32_t debug_producer_stop;
};

enum { MODE_ARGMIN = 0, MODE_STORE = 1, MODE_UNION = 2, MODE_COUNT = 3 };
constexpr float kUnionSlack = 1.0f / 512.0f;   // see the union epilogue

template <int MODE>
__global__ void __launch_bounds__(NUM_THREADS, 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_y,
                                                                 const __grid_constant__ CUtensorMap tmap_ylo, const Params p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
    uint8_t* smem = smem_raw + pad;
    const uint32_t smem_base = raw_addr + pad;
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem + STAGES * STAGE_BYTES);
    const WaitCtx wctx{p.error, p.wait_limit};

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&ctrl->full[s], 1);
            mbar_init(&ctrl->conv[s], 128);
            mbar_init(&ctrl->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctrl->tmem_full[b], 1);
            mbar_init(&ctrl->tmem_empty[b], (MODE == MODE_UNION || MODE == MODE_COUNT) ? 256 : 128);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (warp == 1) tmem_alloc(&ctrl->tmem_base, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = ctrl->tmem_base;

    constexpr bool kTiled = (MODE == MODE_UNION || MODE == MODE_COUNT);   // works on a given range / list of row tiles
    const size_t rt_begin = kTiled ? p.tile0 : 0;
    const size_t n_row_tiles = kTiled ? p.tile0 + p.n_tiles : (p.n + BM - 1) / BM;
    // row tile that entry rt of the loops below stands for
    auto tile_of = [&](size_t rt) -> size_t { return (kTiled && p.tile_map) ? static_cast<size_t>(__ldg(p.tile_map + (rt - rt_begin))) : rt; };
    const uint32_t n_col_tiles = static_cast<uint32_t>((p.k + BN - 1) / BN);
    const uint32_t nkb = (p.kdim + BK - 1) / BK;

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            uint32_t kbt = 0;
            bool ok = true;
            for (size_t rt = rt_begin + blockIdx.x; rt < n_row_tiles && ok; rt += gridDim.x) {
                const size_t x_row = tile_of(rt) * BM;
                for (uint32_t nt = 0; nt < n_col_tiles && ok; ++nt) {
                    for (uint32_t kb = 0; kb < nkb; ++kb, ++kbt) {
                        const uint32_t s = kbt % STAGES, ph = (kbt / STAGES) & 1u;
                        if (p.debug_producer_stop != 0 && kbt >= p.debug_producer_stop) {
                            ok = false;
                            break;
                        }
                        if (!mbar_wait(&ctrl->empty[s], ph ^ 1u, wctx, 1)) {
                            ok = false;
                            break;
                        }
                        // (the union pass multiplies hi parts only and never loads the lo parts of Y)
                        const bool load_ylo = p.y_presplit && MODE != MODE_UNION;
                        mbar_arrive_expect_tx(&ctrl->full[s], A_TILE_BYTES + (load_ylo ? 2 * B_TILE_BYTES : B_TILE_BYTES));
                        const uint32_t st = smem_base + s * STAGE_BYTES;
                        tma_load_2d(st + OFF_A_HI, &tmap_x, &ctrl->full[s], static_cast<int>(kb * BK), static_cast<int>(x_row));
                        tma_load_2d(st + OFF_B_HI, &tmap_y, &ctrl->full[s], static_cast<int>(kb * BK), static_cast<int>(nt * BN));
                        if (load_ylo) tma_load_2d(st + OFF_B_LO, &tmap_ylo, &ctrl->full[s], static_cast<int>(kb * BK), static_cast<int>(nt * BN));
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (lane == 0) {
            uint32_t kbt = 0, t = 0;
            bool ok = true;
            for (size_t rt = rt_begin + blockIdx.x; rt < n_row_tiles && ok; rt += gridDim.x) {
                for (uint32_t nt = 0; nt < n_col_tiles && ok; ++nt, ++t) {
                    const uint32_t b = t & 1u, tph = (t >> 1) & 1u;
                    if (!mbar_wait(&ctrl->tmem_empty[b], tph ^ 1u, wctx, 2)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t acc = tmem_base + b * BN;
                    // (columns behind the last are not multiplied: 300 000 x 768 rows, k = 50: 390 -> 340 us)
                    const uint32_t idesc = make_idesc(static_cast<uint32_t>(min(static_cast<size_t>(BN), (p.k - static_cast<size_t>(nt) * BN + 15) / 16 * 16)));
                    for (uint32_t kb = 0; kb < nkb; ++kb, ++kbt) {
                        const uint32_t s = kbt % STAGES, ph = (kbt / STAGES) & 1u;
                        if (!mbar_wait(&ctrl->conv[s], ph, wctx, 3)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t st = smem_base + s * STAGE_BYTES;
#pragma unroll
                        for (uint32_t kk = 0; kk < BK / 8; ++kk) {
                            const uint64_t a_hi = make_desc(st + OFF_A_HI + kk * 32);
                            const uint64_t a_lo = make_desc(st + OFF_A_LO + kk * 32);
                            const uint64_t b_hi = make_desc(st + OFF_B_HI + kk * 32);
                            const uint64_t b_lo = make_desc(st + OFF_B_LO + kk * 32);
                            umma_tf32(acc, a_hi, b_hi, (kb | kk) != 0 ? 1u : 0u, idesc);
                            if (MODE != MODE_UNION) {
                                umma_tf32(acc, a_hi, b_lo, 1u, idesc);
                                umma_tf32(acc, a_lo, b_hi, 1u, idesc);
                            }
                        }
                        umma_commit(&ctrl->empty[s]);
                    }
                    if (ok) umma_commit(&ctrl->tmem_full[b]);
                }
            }
        }
    } else if (warp < 6) {
        // ---------------------------------------------------------------- hi / lo splitters
        const int cid = threadIdx.x - 64;
        uint32_t kbt = 0;
        bool ok = true;
        for (size_t rt = rt_begin + blockIdx.x; rt < n_row_tiles && ok; rt += gridDim.x) {
            for (uint32_t nt = 0; nt < n_col_tiles && ok; ++nt) {
                for (uint32_t kb = 0; kb < nkb; ++kb, ++kbt) {
                    const uint32_t s = kbt % STAGES, ph = (kbt / STAGES) & 1u;
                    if (!mbar_wait(&ctrl->full[s], ph, wctx, 4)) {
                        ok = false;
                        break;
                    }
                    uint8_t* st = smem + s * STAGE_BYTES;
                    float4* a_hi = reinterpret_cast<float4*>(st + OFF_A_HI);
                    float4* a_lo = reinterpret_cast<float4*>(st + OFF_A_LO);
                    float4* b_hi = reinterpret_cast<float4*>(st + OFF_B_HI);
                    float4* b_lo = reinterpret_cast<float4*>(st + OFF_B_LO);
#pragma unroll
                    for (int i = 0; i < static_cast<int>(A_TILE_BYTES / 16 / 128); ++i) {
                        float4 hi, lo;
                        split4(a_hi[cid + 128 * i], hi, lo);
                        a_hi[cid + 128 * i] = hi;
                        a_lo[cid + 128 * i] = lo;
                    }
                    if (!p.y_presplit) {
#pragma unroll
                        for (int i = 0; i < static_cast<int>(B_TILE_BYTES / 16 / 128); ++i) {
                            float4 hi, lo;
                            split4(b_hi[cid + 128 * i], hi, lo);
                            b_hi[cid + 128 * i] = hi;
                            b_lo[cid + 128 * i] = lo;
                        }
                    }
                    fence_proxy_async();
                    mbar_arrive(&ctrl->conv[s]);
                }
            }
        }
    } else if (warp < 10 || kTiled) {
        // ---------------------------------------------------------------- epilogue
        // Union and counting modes: eight warps, two per quarter of the tile's rows; warps 6-9 take columns 0-127 of
        // every 256-column tile, warps 10-13 columns 128-255.
        const uint32_t half = kTiled ? static_cast<uint32_t>(warp - 6) >> 2 : 0u;
        const uint32_t lane_base = 32u * (warp & 3);    // tensor-memory lanes this warp may read
        const uint32_t row_in_tile = lane_base + lane;
        uint32_t t = 0;
        bool ok = true;
        for (size_t rt = rt_begin + blockIdx.x; rt < n_row_tiles && ok; rt += gridDim.x) {
            const size_t row = tile_of(rt) * BM + row_in_tile;
            const bool row_valid = row < p.n;
            // Best and runner-up of the tensor-core distances.  They are only candidates: the accumulator
            // in tensor memory truncates, which biases long sums by up to ~1e-5 relative, so the winner and
            // its distance are settled afterwards in fp32 by refine_top2_kernel.
            float nx = 0.f, d1 = FLT_MAX, d2 = FLT_MAX;
            uint32_t i1 = 0, i2 = 0xFFFFFFFFu;
            if ((MODE == MODE_ARGMIN || kTiled) && row_valid) nx = p.norms_x[row];
            float thr = -FLT_MAX;
            uint32_t* my_union = nullptr;
            if (MODE == MODE_UNION) {
                my_union = p.union_bits + (rt - rt_begin) * static_cast<size_t>(p.union_words);
                // The union must contain every pair that the chain kernel's own first test will pass.  This pass multiplies
                // the tf32 hi parts only (one product instead of three): x.c is then off by at most 2^-10 |x| |c|, the
                // partial distance by at most 2^-10 (|x|^2 + |c|^2).  The test is widened by twice that (kUnionSlack; the
                // |c|^2 share is folded into the centroid norms below), plus a little for norms summed in another order.
                if (row_valid && !(p.skip && p.skip[row])) {
                    const float t0 = p.best_in[row] * p.ratio_first;
                    thr = fmaf(t0, 1e-4f, t0) + (kUnionSlack + 1e-6f) * nx;
                }
            }
            uint32_t counted = 0;   // MODE_COUNT
            for (uint32_t nt = 0; nt < n_col_tiles && ok; ++nt, ++t) {
                const uint32_t b = t & 1u, tph = (t >> 1) & 1u;
                const size_t col0 = static_cast<size_t>(nt) * BN;
                float* ny = ctrl->ny[warp & 3][b];
                if (MODE == MODE_COUNT && (nt & 3u) == 0) thr = row_valid ? __ldg(p.thr_rows + row * p.thr_chunks + (nt >> 2)) : -FLT_MAX;
                if (MODE == MODE_ARGMIN) {
                    // each warp keeps its own copy, so no cross-warp barrier is needed
                    for (int j = lane; j < BN; j += 32) ny[j] = (col0 + j < p.k) ? __ldg(p.norms_y + col0 + j) : 0.f;
                    __syncwarp();
                }
                if (kTiled) {
                    // the two warps of a row quarter fill (and read) disjoint halves of the shared copy
                    const float ny_scale = MODE == MODE_UNION ? 1.0f - kUnionSlack : 1.0f;
                    for (int j = half * (BN / 2) + lane; j < static_cast<int>((half + 1) * (BN / 2)); j += 32) ny[j] = (col0 + j < p.k) ? ny_scale * __ldg(p.norms_y + col0 + j) : 0.f;
                    __syncwarp();
                }
                // warp-uniform outcome: the tensor-memory loads below must be executed by the whole warp
                if (!__all_sync(0xffffffffu, mbar_wait(&ctrl->tmem_full[b], tph, wctx, 5))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + (lane_base << 16) + b * BN;
                const int ch_begin = kTiled ? static_cast<int>(half) * (BN / 64) : 0;
                const int ch_end = kTiled ? ch_begin + BN / 64 : static_cast<int>(min(static_cast<size_t>(BN / 32), (p.k - col0 + 31) / 32));
#pragma unroll 1
                for (int ch = ch_begin; ch < ch_end; ++ch) {
                    uint32_t r[32];
                    tmem_ld32(taddr + ch * 32, r);
                    if (MODE == MODE_ARGMIN) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const size_t c = col0 + ch * 32 + j;
                            if (c < p.k) {
                                const float dist = fmaf(-2.0f, __uint_as_float(r[j]), nx) + ny[ch * 32 + j];
                                if (dist < d2) {
                                    if (dist < d1) {
                                        d2 = d1;
                                        i2 = i1;
                                        d1 = dist;
                                        i1 = static_cast<uint32_t>(c);
                                    } else {
                                        d2 = dist;
                                        i2 = static_cast<uint32_t>(c);
                                    }
                                }
                            }
                        }
                    } else if (MODE == MODE_UNION) {
                        // first test for 32 centroids; only which centroids pass for ANY row of the tile is kept
                        uint32_t mask = 0;
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const float4 nyv = *reinterpret_cast<const float4*>(ny + ch * 32 + j);
                            const float p0 = fmaf(-2.0f, __uint_as_float(r[j + 0]), nx) + nyv.x;
                            const float p1 = fmaf(-2.0f, __uint_as_float(r[j + 1]), nx) + nyv.y;
                            const float p2 = fmaf(-2.0f, __uint_as_float(r[j + 2]), nx) + nyv.z;
                            const float p3 = fmaf(-2.0f, __uint_as_float(r[j + 3]), nx) + nyv.w;
                            mask |= (p0 < thr ? (1u << j) : 0u) | (p1 < thr ? (2u << j) : 0u) | (p2 < thr ? (4u << j) : 0u) | (p3 < thr ? (8u << j) : 0u);
                        }
                        const size_t first = col0 + static_cast<size_t>(ch) * 32;
                        const uint32_t n_valid = first >= p.k ? 0u : static_cast<uint32_t>(min(static_cast<size_t>(32), p.k - first));
                        mask &= n_valid >= 32u ? 0xFFFFFFFFu : ((1u << n_valid) - 1u);
                        const uint32_t any = __reduce_or_sync(0xffffffffu, mask);
                        if (any != 0 && lane == 0) atomicOr(my_union + (first >> 5), any);
                    } else if (MODE == MODE_COUNT) {
                        uint32_t mask = 0;
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const float4 nyv = *reinterpret_cast<const float4*>(ny + ch * 32 + j);
                            const float p0 = fmaf(-2.0f, __uint_as_float(r[j + 0]), nx) + nyv.x;
                            const float p1 = fmaf(-2.0f, __uint_as_float(r[j + 1]), nx) + nyv.y;
                            const float p2 = fmaf(-2.0f, __uint_as_float(r[j + 2]), nx) + nyv.z;
                            const float p3 = fmaf(-2.0f, __uint_as_float(r[j + 3]), nx) + nyv.w;
                            mask |= (p0 < thr ? (1u << j) : 0u) | (p1 < thr ? (2u << j) : 0u) | (p2 < thr ? (4u << j) : 0u) | (p3 < thr ? (8u << j) : 0u);
                        }
                        const size_t first = col0 + static_cast<size_t>(ch) * 32;
                        const uint32_t n_valid = first >= p.k ? 0u : static_cast<uint32_t>(min(static_cast<size_t>(32), p.k - first));
                        mask &= n_valid >= 32u ? 0xFFFFFFFFu : ((1u << n_valid) - 1u);
                        counted += __popc(mask);
                    } else if (row_valid) {
                        float* orow = p.out + row * p.ldo + col0 + ch * 32;
                        const size_t left = (col0 + ch * 32 < p.k) ? (p.k - (col0 + ch * 32)) : 0;
                        if (left >= 32 && (p.ldo % 4 == 0)) {
#pragma unroll
                            for (int j = 0; j < 32; j += 4)
                                *reinterpret_cast<float4*>(orow + j) =
                                    make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (static_cast<size_t>(j) < left) orow[j] = __uint_as_float(r[j]);
                        }
                    }
                }
                tc_fence_before();
                mbar_arrive(&ctrl->tmem_empty[b]);
            }
            if (MODE == MODE_ARGMIN && ok && row_valid) p.out_top2[row] = make_uint2(i1, i2);
            if (MODE == MODE_COUNT && ok && row_valid && counted != 0) atomicAdd(p.count_out + row, counted);   // the row's other half adds its own
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// After the chain: the exact squared distance (direct differences, fp32) of a point to the chain's
// winner and to the two runner-ups; the smallest wins, the winner keeps its place on ties.
__global__ void __launch_bounds__(256) refine_chain_kernel(const float* __restrict__ x, const float* __restrict__ y, size_t n, size_t k, size_t d,
                                                           const uint2* __restrict__ top2, const uint32_t* knn, const int* __restrict__ error,
                                                           const uint32_t* __restrict__ tile_map, const uint32_t* __restrict__ idx, const uint32_t* not_pruned,
                                                           uint32_t* knn_out, float* __restrict__ dist_out, uint32_t* not_pruned_out) {
    // with a tile map the grid covers the rows of the listed 128-row tiles, else rows 0 .. n-1; row i of the chain's arrays is row idx[i]
    // of x and of what is written, or row i
    size_t row = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (tile_map) row = static_cast<size_t>(tile_map[row / BM]) * BM + (row % BM);
    if (row >= n) return;
    // a chain kernel that gave up on a wait leaves its outputs unwritten: nothing to refine, and no index to trust
    if (*reinterpret_cast<const volatile int*>(error) != 0) return;
    const int lane = threadIdx.x & 31;
    const uint32_t w = knn[row];
    const uint2 t = top2[row];
    if (w >= k) return;
    uint32_t cand[3] = {w, t.x < k ? t.x : 0xFFFFFFFFu, t.y < k ? t.y : 0xFFFFFFFFu};
    if (cand[1] == 0xFFFFFFFFu || cand[1] == w) cand[1] = w;
    if (cand[2] == 0xFFFFFFFFu || cand[2] == w) cand[2] = w;
    const size_t to = idx ? idx[row] : row;
    const float* xr = x + to * d;
    const float* y0 = y + static_cast<size_t>(cand[0]) * d;
    const float* y1 = y + static_cast<size_t>(cand[1]) * d;
    const float* y2 = y + static_cast<size_t>(cand[2]) * d;
    float s0 = 0.f, s1 = 0.f, s2 = 0.f;
    for (size_t j = static_cast<size_t>(lane) * 4; j < d; j += 128) {
        const float4 xv = __ldg(reinterpret_cast<const float4*>(xr + j));
        const float4 a = __ldg(reinterpret_cast<const float4*>(y0 + j));
        const float4 b = __ldg(reinterpret_cast<const float4*>(y1 + j));
        const float4 c = __ldg(reinterpret_cast<const float4*>(y2 + j));
        float u;
        u = xv.x - a.x; s0 = fmaf(u, u, s0); u = xv.y - a.y; s0 = fmaf(u, u, s0); u = xv.z - a.z; s0 = fmaf(u, u, s0); u = xv.w - a.w; s0 = fmaf(u, u, s0);
        u = xv.x - b.x; s1 = fmaf(u, u, s1); u = xv.y - b.y; s1 = fmaf(u, u, s1); u = xv.z - b.z; s1 = fmaf(u, u, s1); u = xv.w - b.w; s1 = fmaf(u, u, s1);
        u = xv.x - c.x; s2 = fmaf(u, u, s2); u = xv.y - c.y; s2 = fmaf(u, u, s2); u = xv.z - c.z; s2 = fmaf(u, u, s2); u = xv.w - c.w; s2 = fmaf(u, u, s2);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
        uint32_t bi = cand[0];
        float bd = s0;
        if (s1 < bd || (s1 == bd && cand[1] < bi && cand[1] != w && bi != w)) {
            bd = s1;
            bi = cand[1];
        }
        if (s2 < bd || (s2 == bd && cand[2] < bi && bi != w)) {
            bd = s2;
            bi = cand[2];
        }
        knn_out[to] = bi;
        dist_out[to] = bd;
        if (not_pruned_out) not_pruned_out[to] = not_pruned[row];
    }
}

// Settles the assignment in fp32: one warp per row recomputes ||x||^2 + ||y||^2 - 2 x.y for the two
// candidates with fp32 fused multiply-adds, keeps the smaller (the lower index on a tie) and stores
// the distance clamped at zero, as the reference does (batch_computers.h:160-166).
__global__ void __launch_bounds__(256) refine_top2_kernel(
    const float* __restrict__ x, const float* __restrict__ y, size_t n, size_t k, size_t d, const float* __restrict__ norms_x, const float* __restrict__ norms_y,
    const uint2* __restrict__ top2, uint32_t* __restrict__ out_knn, float* __restrict__ out_dist, const int* __restrict__ error
) {
    const size_t row = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (row >= n) return;
    // a tensor-core pass that gave up on a wait leaves the candidate pairs unwritten
    if (*reinterpret_cast<const volatile int*>(error) != 0) return;
    const int lane = threadIdx.x & 31;
    const uint2 cand = top2[row];
    if (cand.x >= k) return;
    const bool two = cand.y < k;
    const float* xr = x + row * d;
    const float* y1 = y + static_cast<size_t>(cand.x) * d;
    const float* y2 = y + static_cast<size_t>(two ? cand.y : cand.x) * d;
    float a1 = 0.f, a2 = 0.f;
    for (size_t j = static_cast<size_t>(lane) * 4; j < d; j += 128) {  // d % 4 == 0 on this path
        const float4 xv = __ldg(reinterpret_cast<const float4*>(xr + j));
        const float4 u = __ldg(reinterpret_cast<const float4*>(y1 + j));
        const float4 v = __ldg(reinterpret_cast<const float4*>(y2 + j));
        a1 = fmaf(xv.x, u.x, a1); a1 = fmaf(xv.y, u.y, a1); a1 = fmaf(xv.z, u.z, a1); a1 = fmaf(xv.w, u.w, a1);
        a2 = fmaf(xv.x, v.x, a2); a2 = fmaf(xv.y, v.y, a2); a2 = fmaf(xv.z, v.z, a2); a2 = fmaf(xv.w, v.w, a2);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        a2 += __shfl_xor_sync(0xffffffffu, a2, o);
    }
    if (lane == 0) {
        const float nx = norms_x[row];
        float e1 = fmaf(-2.0f, a1, nx) + norms_y[cand.x];
        uint32_t w = cand.x;
        if (two) {
            float e2 = fmaf(-2.0f, a2, nx) + norms_y[cand.y];
            if (fabsf(e1 - e2) <= 1e-4f * fmaxf(fabsf(e1), fabsf(e2))) {
                // Near-tie (typically the twin centroids left by a cluster split): settle it with the dot
                // products accumulated strictly in index order, the order of the fp32 SIMT kernel.
                float s1 = 0.f, s2 = 0.f;
                for (size_t j = 0; j < d; ++j) {
                    const float xv = xr[j];
                    s1 = fmaf(xv, y1[j], s1);
                    s2 = fmaf(xv, y2[j], s2);
                }
                e1 = fmaf(-2.0f, s1, nx) + norms_y[cand.x];
                e2 = fmaf(-2.0f, s2, nx) + norms_y[cand.y];
            }
            if (e2 < e1 || (e2 == e1 && cand.y < cand.x)) {
                e1 = e2;
                w = cand.y;
            }
        }
        out_knn[row] = w;
        out_dist[row] = fmaxf(0.0f, e1);
    }
}

// hi = tf32(v), lo = tf32(v - hi) for every element (the split the splitter warps would do in shared memory)
__global__ void __launch_bounds__(256) split_tf32_kernel(const float4* __restrict__ in, float4* __restrict__ hi, float4* __restrict__ lo, size_t n4) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n4) return;
    float4 h, l;
    split4(__ldg(in + i), h, l);
    hi[i] = h;
    lo[i] = l;
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                   CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(p);
        }
    });
    if (!fn) throw CudaError("cuTensorMapEncodeTiled is not available from this driver");
    return fn;
}

// Row-major fp32 matrix [rows][ld] of which the first `extent` columns are visible; boxes of 16
// columns x box_rows rows, 64-byte swizzle, zero fill outside.
CUtensorMap make_tmap_of(CUtensorMapDataType type, size_t element, CUtensorMapSwizzle swizzle, const void* base, size_t extent, size_t rows, size_t ld, uint32_t box_cols,
                         uint32_t box_rows) {
    CUtensorMap m;
    const cuuint64_t dims[2] = {extent, rows};
    const cuuint64_t strides[1] = {ld * element};
    const cuuint32_t box[2] = {box_cols, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = encode_fn()(&m, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw CudaError("cuTensorMapEncodeTiled failed with code " + std::to_string(static_cast<int>(r)));
    return m;
}

CUtensorMap make_tmap(const float* base, size_t extent, size_t rows, size_t ld, uint32_t box_rows) {
    return make_tmap_of(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, sizeof(float), CU_TENSOR_MAP_SWIZZLE_64B, base, extent, rows, ld, BK, box_rows);
}

// Splits y (rows x ld, 16-byte aligned, ld % 4 == 0) into y_split[0 .. rows*ld) = hi and y_split[rows*ld ..) = lo.
void presplit(const float* y, size_t rows, size_t ld, float* y_split, cudaStream_t stream) {
    const size_t n4 = rows * ld / 4;
    if (n4 == 0) return;
    split_tf32_kernel<<<static_cast<unsigned>((n4 + 255) / 256), 256, 0, stream>>>(reinterpret_cast<const float4*>(y), reinterpret_cast<float4*>(y_split),
                                                                                   reinterpret_cast<float4*>(y_split + rows * ld), n4);
    note_kernel_launch();
    SKM_CUDA(cudaGetLastError());
}

int* error_flag(int device) {
    static std::mutex mu;
    static int* flags[64] = {nullptr};
    std::lock_guard<std::mutex> lock(mu);
    if (!flags[device]) {
        note_device_alloc();
        SKM_CUDA(cudaMalloc(&flags[device], sizeof(int)));
        SKM_CUDA(cudaMemset(flags[device], 0, sizeof(int)));
    }
    return flags[device];
}

int sm_count(int device) {
    int sms = 0;
    SKM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    return sms;
}

template <int MODE>
void launch(const CUtensorMap& tx, const CUtensorMap& ty, const CUtensorMap& tylo, const Params& p, cudaStream_t stream) {
    SKM_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SMEM_BYTES)));
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    const size_t row_tiles = (p.n + BM - 1) / BM;
    const int grid = static_cast<int>(std::min<size_t>(row_tiles, static_cast<size_t>(sm_count(device))));
    gemm_tc_kernel<MODE><<<grid, NUM_THREADS, SMEM_BYTES, stream>>>(tx, ty, tylo, p);
    note_kernel_launch();
    SKM_CUDA(cudaGetLastError());
}

bool g_enabled = true;
uint32_t g_debug_producer_stop = 0;
long long g_wait_limit = WAIT_LIMIT_CYCLES;

} // namespace

long long wait_limit() { return g_wait_limit; }

void set_debug_wait_injection(long long wait_limit_cycles, uint32_t producer_stops_after_kblocks) {
    g_wait_limit = wait_limit_cycles > 0 ? wait_limit_cycles : WAIT_LIMIT_CYCLES;
    g_debug_producer_stop = producer_stops_after_kblocks;
}

uint32_t producer_stop() { return g_debug_producer_stop; }

void launch_presplit(const float* y, size_t rows, size_t ld, float* y_split, cudaStream_t stream) { presplit(y, rows, ld, y_split, stream); }

CUtensorMap make_half_tmap(const void* base, size_t cols, size_t rows, uint32_t box_rows, size_t pitch) {
    return make_tmap_of(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, CU_TENSOR_MAP_SWIZZLE_128B, base, cols, rows, pitch ? pitch : cols, 64, box_rows);
}

CUtensorMap make_row_major_tmap_128(const float* base, size_t extent, size_t rows, size_t ld, uint32_t box_rows) {
    return make_tmap_of(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, sizeof(float), CU_TENSOR_MAP_SWIZZLE_128B, base, extent, rows, ld, 32, box_rows);
}
CUtensorMap make_row_major_tmap(const float* base, size_t extent, size_t rows, size_t ld, uint32_t box_rows) { return make_tmap(base, extent, rows, ld, box_rows); }

int* error_word() {
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    return error_flag(device);
}

void set_enabled(bool on) { g_enabled = on; }
bool enabled() { return g_enabled; }

bool eligible(const float* x, size_t ldx, const float* y, size_t ldy) {
    if (!g_enabled) return false;
    if (ldx % 4 != 0 || ldy % 4 != 0) return false;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(y) & 15)) return false;
    return true;
}

void launch_assign_full(const float* x, const float* y, size_t n, size_t k, size_t d, const float* norms_x, const float* norms_y, uint32_t* out_knn, float* out_dist,
                        uint2* top2_scratch, cudaStream_t stream, float* y_split) {
    if (n == 0 || k == 0) return;
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    if (y_split) presplit(y, k, d, y_split, stream);
    const CUtensorMap tx = make_tmap(x, d, n, d, BM);
    const CUtensorMap ty = make_tmap(y_split ? y_split : y, d, k, d, BN);
    const CUtensorMap tylo = y_split ? make_tmap(y_split + k * d, d, k, d, BN) : ty;
    Params p{};
    p.y_presplit = y_split != nullptr;
    p.n = n;
    p.k = k;
    p.kdim = static_cast<uint32_t>(d);
    p.norms_x = norms_x;
    p.norms_y = norms_y;
    p.out_knn = out_knn;
    p.out_dist = out_dist;
    p.out_top2 = top2_scratch;
    p.error = error_flag(device);
    p.wait_limit = g_wait_limit;
    p.debug_producer_stop = g_debug_producer_stop;
    launch<MODE_ARGMIN>(tx, ty, tylo, p, stream);
    refine_top2_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(x, y, n, k, d, norms_x, norms_y, top2_scratch, out_knn, out_dist, p.error);
    note_kernel_launch();
    SKM_CUDA(cudaGetLastError());
}

void launch_assign_full_flagged(const float* x, const float* y, size_t n, size_t k, size_t d, const float* norms_x, const float* norms_y, uint32_t* out_knn, float* out_dist,
                                uint2* top2_scratch, int* error_word, cudaStream_t stream) {
    if (n == 0 || k == 0) return;
    const CUtensorMap tx = make_tmap(x, d, n, d, BM);
    const CUtensorMap ty = make_tmap(y, d, k, d, BN);
    Params p{};
    p.n = n;
    p.k = k;
    p.kdim = static_cast<uint32_t>(d);
    p.norms_x = norms_x;
    p.norms_y = norms_y;
    p.out_knn = out_knn;
    p.out_dist = out_dist;
    p.out_top2 = top2_scratch;
    p.error = error_word;
    p.wait_limit = g_wait_limit;
    launch<MODE_ARGMIN>(tx, ty, ty, p, stream);
    refine_top2_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(x, y, n, k, d, norms_x, norms_y, top2_scratch, out_knn, out_dist, p.error);
    note_kernel_launch();
    SKM_CUDA(cudaGetLastError());
}

void launch_count_first_test(const float* x, size_t n, size_t k, size_t d, uint32_t partial_d, const float* norms_x, const float* norms_y, const float* thr_rows,
                             uint32_t thr_chunks, uint32_t* count_out, const float* y_split, cudaStream_t stream) {
    if (n == 0 || k == 0) return;
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    const CUtensorMap tx = make_tmap(x, partial_d, n, d, BM);
    const CUtensorMap ty = make_tmap(y_split, partial_d, k, d, BN);
    const CUtensorMap tylo = make_tmap(y_split + k * d, partial_d, k, d, BN);
    Params p{};
    p.y_presplit = true;
    p.n = n;
    p.k = k;
    p.kdim = partial_d;
    p.norms_x = norms_x;
    p.norms_y = norms_y;
    p.error = error_flag(device);
    p.wait_limit = g_wait_limit;
    p.tile0 = 0;
    p.n_tiles = (n + BM - 1) / BM;
    p.thr_rows = thr_rows;
    p.thr_chunks = thr_chunks;
    p.count_out = count_out;
    SKM_CUDA(cudaMemsetAsync(count_out, 0, sizeof(uint32_t) * n, stream));
    SKM_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<MODE_COUNT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SMEM_BYTES)));
    const int grid = static_cast<int>(std::min<size_t>(p.n_tiles, static_cast<size_t>(sm_count(device))));
    gemm_tc_kernel<MODE_COUNT><<<grid, NUM_THREADS, SMEM_BYTES, stream>>>(tx, ty, tylo, p);
    note_kernel_launch();
    SKM_CUDA(cudaGetLastError());
}

void launch_union(const float* x, size_t n, size_t k, size_t d, uint32_t partial_d, const float* norms_x, const float* norms_y, const float* best_in, float ratio_first,
                  const uint32_t* tile_map, size_t n_tiles, uint32_t* union_bits, uint32_t union_words, const float* y_split, cudaStream_t stream) {
    if (n_tiles == 0 || k == 0) return;
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    const CUtensorMap tx = make_tmap(x, partial_d, n, d, BM);
    const CUtensorMap ty = make_tmap(y_split, partial_d, k, d, BN);
    const CUtensorMap tylo = make_tmap(y_split + k * d, partial_d, k, d, BN);
    Params p{};
    p.y_presplit = true;
    p.n = n;
    p.k = k;
    p.kdim = partial_d;
    p.norms_x = norms_x;
    p.norms_y = norms_y;
    p.error = error_flag(device);
    p.wait_limit = g_wait_limit;
    p.tile0 = 0;
    p.n_tiles = n_tiles;
    p.best_in = best_in;
    p.ratio_first = ratio_first;
    p.tile_map = tile_map;
    p.union_bits = union_bits;
    p.union_words = union_words;
    SKM_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<MODE_UNION>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SMEM_BYTES)));
    const int grid = static_cast<int>(std::min<size_t>(n_tiles, static_cast<size_t>(sm_count(device))));
    gemm_tc_kernel<MODE_UNION><<<grid, NUM_THREADS, SMEM_BYTES, stream>>>(tx, ty, tylo, p);
    note_kernel_launch();
    SKM_CUDA(cudaGetLastError());
}

void launch_gemm_nt(const float* a, size_t lda, const float* b, size_t ldb, float* out, size_t ldo, size_t n, size_t n_out, size_t k_dim, cudaStream_t stream) {
    if (n == 0 || n_out == 0) return;
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    const CUtensorMap tx = make_tmap(a, k_dim, n, lda, BM);
    const CUtensorMap ty = make_tmap(b, k_dim, n_out, ldb, BN);
    Params p{};
    p.n = n;
    p.k = n_out;
    p.kdim = static_cast<uint32_t>(k_dim);
    p.out = out;
    p.ldo = ldo;
    p.error = error_flag(device);
    p.wait_limit = g_wait_limit;
    launch<MODE_STORE>(tx, ty, ty, p, stream);
}

void launch_refine_chain_tiles(const float* x, const float* y, size_t n, size_t k, size_t d, const uint2* top2, uint32_t* knn, float* dist, const uint32_t* tile_map,
                               size_t n_tiles, cudaStream_t stream) {
    if (n_tiles == 0) return;
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    refine_chain_kernel<<<static_cast<unsigned>(n_tiles * (BM / 8)), 256, 0, stream>>>(x, y, n, k, d, top2, knn, error_flag(device), tile_map, nullptr, nullptr, knn, dist, nullptr);
    SKM_LAUNCH_CHECK();
}

void launch_refine_chain(const float* x, const float* y, size_t n, size_t k, size_t d, const uint2* top2, const uint32_t* idx, const uint32_t* knn, const uint32_t* not_pruned,
                         uint32_t* knn_out, float* dist_out, uint32_t* not_pruned_out, cudaStream_t stream) {
    if (n == 0) return;
    refine_chain_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(x, y, n, k, d, top2, knn, error_word(), nullptr, idx, not_pruned, knn_out, dist_out, not_pruned_out);
    SKM_LAUNCH_CHECK();
}

// Reads (and clears) the error code left by the last kernels on this device.  Synchronises `stream`.
int fetch_error(cudaStream_t stream) {
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    int* flag = error_flag(device);
    int host = 0;
    SKM_CUDA(cudaMemcpyAsync(&host, flag, sizeof(int), cudaMemcpyDeviceToHost, stream));
    SKM_CUDA(cudaStreamSynchronize(stream));
    if (host != 0) SKM_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), stream));
    return host;
}

} // namespace tc
} // namespace skmb
