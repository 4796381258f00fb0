// Pruned assignment as a dense chain on the tensor cores: what the reference does for one point and a chunk of 1024 centroids
// (batch_computers.h:297-409, pdx/pdxearch.h:118-327) is a sequence of tests "partial distance < best * ratio[dimensions seen]": after
// the first d' dimensions, after every further 64 horizontal dimensions, and after the remaining vertical dimensions
// (pdx/pdxearch.h:118-217); `best` is fixed inside the chunk and lowered at its end (:290-324).  Here the partial distances come from
// accumulators in tensor memory that keep growing along that same order of dimensions: after each segment the threads of a row read
// them (without clearing), turn them into ||x||^2 + ||c||^2 - 2 x.c over the dimensions seen so far with precomputed cumulative
// norms, and update a bit mask of surviving centroids.
//
// Points and centroids come as fp16 pairs v * scale = hi + lo, products are hi*hi + hi*lo + lo*hi with fp32 accumulation.  The scale is a power of
// two per row: values down to 2^-17 of the row's norm have 22 bits (as two tf32 parts have), smaller ones are off by 2^-39 of the norm at most, which is
// far below what the accumulator's truncation and the norms' rounding leave (2^-24 of the norms).  Against 64 bits the chain is closer than
// with tf32 parts, which take twice as many truncated additions: of 60 000 points these have another count of first-test survivors: 1024 columns,
// k = 4000: 81 (tf32: 128) and, unstructured, 106 (229); 1536, k = 2048: 37 (67) and 67 (125); 768, k = 1000: 13 (15) and 3 (6); columns scaled from 1 to
// 1e-6: 21 (28).
// Their columns are laid out in the order of the chain, every segment from a multiple of 64 on with zeros behind it, so that a segment is a run
// of whole stages whatever d' is.  A pass writes the halves of its points (chain_points_kernel, which also gathers them and makes their
// cumulative norms) and of the centroids anyway.
//
// Persistent pairs of CTAs (cta_group::2) on tiles of 256 points x 256 centroids (a unit), 18 warps:
//   warp 0      TMA producer: 128 x 64 halves of each of the four parts per stage and CTA, three stages;
//   warp 1      MMA issuer (the leader's), two accumulators of 256 columns;
//   warps 2-17  tests, a warp per 32 points and 64 columns of a unit; the four threads of a point exchange what they found at the end of
//               every chunk.
// The two accumulators belong to two neighbouring units that advance through the segments in turn, so the tensor pipe works on one
// unit while the tests read the other.
// What bounds it is the tests (their issue and latency, as in kernels_first_test.cu) and, beside the walk, the SMs shared with it.  One
// B200, the phase of the chain against three tf32 products on single CTAs whose points four warps split in shared memory.  All points in the chain
// (unstructured rows): 250 000 x 1024, k = 1000, two passes: 6.9 ms -> 4.5; 100 000 x 256, k = 2000, three: 3.7 -> 1.7; 60 000 x 512, k = 500, four: 1.65 -> 1.08.
// Nine passes of a Train with the walk beside it: 1M x 1024, k = 4000: 23.3 -> 18.2 (the walk has fewer SMs meanwhile: 18.2 -> 20.5), 250 000 x 1536,
// k = 2048: 5.8 - 6.4 -> 6.0, 30 000 x 768, k = 1000: 0.80 -> 0.71 - 0.76.
// Every wait is bounded (see kernels_tc.cu).
#include <cfloat>
#include <cmath>

#include "common.cuh"
#include "device_utils.cuh"
#include "host_logic.h"
#include "kernels_tc.cuh"
#include "tc_ptx.cuh"

namespace skmb {
namespace tc {

namespace {

constexpr int CK = 64;                     // columns of a stage
constexpr int CN = 256;                    // centroids of a unit
constexpr int C_STAGES = 3;
constexpr uint32_t C_PART_BYTES = 128 * CK * 2;
constexpr uint32_t C_STAGE_BYTES = 4 * C_PART_BYTES;   // points hi, lo, centroids hi, lo
constexpr int C_TEST_WARPS = 16;
constexpr int C_THREADS = 64 + 32 * C_TEST_WARPS;
constexpr uint32_t kMaxSegments = 64;

// What the four threads of a point (one per 64 columns) tell each other at the end of a chunk, and a pair of blocks that looks
// at one unit of the chunk only tells merge_chain_kernel.
struct ChainPartial {
    uint32_t cnt;          // survivors of the first test in this chunk
    uint32_t prev_first;   // the previous centroid is among them
    float cb;              // best final distance of the chunk, FLT_MAX if none
    uint32_t cbi;
    float t1, t2;          // the two smallest final distances of the row so far (candidates for the refinement)
    uint32_t i1, i2;
};

struct ChainCtrl {
    ChainPartial xchg[4][128];               // [columns 64 q ..][row]
    alignas(16) float ny[C_TEST_WARPS][64];  // centroid norms of the warp's columns at the current checkpoint
    alignas(16) float fy[C_TEST_WARPS][64];  // and their factors
    float seg_ratio[kMaxSegments];           // ratios[dimensions seen after segment s]
    uint64_t full[C_STAGES];                 // (the leader's are used)
    uint64_t empty[C_STAGES];
    uint64_t acc_ready[2];                   // accumulator a holds the chain up to the current segment
    uint64_t acc_loaded[2];                  // (the leader's are used) every row has read it
    uint64_t told[4], heard[4];              // per 32 rows: the four warps have written, and read, xchg
    uint32_t tmem_base;
};
constexpr uint32_t C_CTRL_BYTES = 26 * 1024;
static_assert(sizeof(ChainCtrl) <= C_CTRL_BYTES, "control block too large");
constexpr uint32_t C_SMEM_BYTES = C_STAGES * C_STAGE_BYTES + C_CTRL_BYTES + 1024;

struct ChainMaps {
    CUtensorMap xhi, xlo, yhi, ylo;
};

struct ChainParams {
    size_t n, k;
    ChainShape shape;
    uint32_t n_seg;
    const float* factor_x;          // per row: -2 / scale
    const float* factor_y;          // per centroid: 1 / scale
    const float* norms_x;           // n x n_seg cumulative squared norms of the points
    const float* norms_y;           // n_seg x k (checkpoint-major), of the centroids
    const float* ratios;
    const float* best_in;           // exact distance to the previous centroid
    uint32_t* knn;                  // in: previous assignment, out: new
    float* dist;
    uint32_t* not_pruned;
    uint2* top2;                    // out: the two smallest final distances seen by the chain, per point
    uint32_t chunk_begin, chunk_end;   // chunks of 1024 centroids
    ChainPartial* partial;             // with SLICES
    int* error;
    long long wait_limit;
    uint32_t producer_stop;            // see set_debug_wait_injection
};

// Order of work shared by all roles: tile of 256 points, chunk of 1024 centroids, pair of 256-centroid units, segment, unit of the
// pair.  `a` (0 / 1) is the unit's accumulator.
#define CHAIN_FOR_EACH_UNIT_SEGMENT(...)                                                                  \
    for (size_t item = blockIdx.x >> 1; item < n_row_tiles * SLICES && ok; item += gridDim.x >> 1) {      \
        [[maybe_unused]] const size_t rt = item / SLICES;                                                 \
        for (uint32_t chunk = p.chunk_begin; chunk < p.chunk_end && ok; ++chunk) {                        \
            const size_t c0 = static_cast<size_t>(chunk) * kChunk;                                        \
            const uint32_t cs = static_cast<uint32_t>(min(static_cast<size_t>(kChunk), p.k - c0));        \
            const uint32_t unit0 = static_cast<uint32_t>(item % SLICES);                                  \
            const uint32_t all_units = (cs + CN - 1) / CN;                                                \
            const uint32_t n_units = SLICES > 1 ? min(unit0 + 1, all_units) : all_units;                  \
            for (uint32_t pair = 0; unit0 + pair * 2 < n_units && ok; ++pair) {                           \
                for (uint32_t seg = 0; seg < p.n_seg && ok; ++seg) {                                      \
                    [[maybe_unused]] const uint32_t seg_begin = p.shape.begin(seg), seg_length = p.shape.length(seg); \
                    for (uint32_t a = 0; a < 2 && ok; ++a) {                                              \
                        const uint32_t unit = unit0 + pair * 2 + a;                                       \
                        if (unit >= n_units) break;                                                       \
                        __VA_ARGS__                                                                       \
                    }                                                                                     \
                }                                                                                         \
            }                                                                                             \
        }                                                                                                 \
    }

// SLICES: 1, or 4 for a pair of blocks per unit of the only chunk, whose findings go to partial[slice][row].
template <uint32_t SLICES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(C_THREADS, 1) chain_tc_kernel(const __grid_constant__ ChainMaps maps, const ChainParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
    const uint32_t smem_base = raw_addr + pad;
    ChainCtrl* ctrl = reinterpret_cast<ChainCtrl*>(smem_raw + pad + C_STAGES * C_STAGE_BYTES);
    const WaitCtx wctx{p.error, p.wait_limit};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();

    if (threadIdx.x == 0) {
        for (int s = 0; s < C_STAGES; ++s) {
            mbar_init(&ctrl->full[s], 1);
            mbar_init(&ctrl->empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&ctrl->acc_ready[a], 1);
            mbar_init(&ctrl->acc_loaded[a], 2 * C_TEST_WARPS);   // a lane of each of the pair's test warps
        }
        for (int q = 0; q < 4; ++q) {
            mbar_init(&ctrl->told[q], 4);
            mbar_init(&ctrl->heard[q], 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (threadIdx.x >= 64 && threadIdx.x - 64 < p.n_seg) ctrl->seg_ratio[threadIdx.x - 64] = __ldg(p.ratios + p.shape.dims_after(threadIdx.x - 64));
    if (warp == 1) tmem_alloc_pair(&ctrl->tmem_base, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // the peer's barriers exist
    tc_fence_after();
    const uint32_t tmem_base = ctrl->tmem_base;
    const size_t n_row_tiles = (p.n + 255) / 256;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t kbt = 0;
            bool ok = true;
            CHAIN_FOR_EACH_UNIT_SEGMENT({
                const int x_row = static_cast<int>(rt * 256 + rank * 128), y_row = static_cast<int>(c0 + static_cast<size_t>(unit) * CN + rank * 128);
                for (uint32_t j = 0; j < seg_length; j += CK, ++kbt) {
                    const uint32_t s = kbt % C_STAGES, ph = (kbt / C_STAGES) & 1u;
                    if ((p.producer_stop != 0 && kbt >= p.producer_stop) || !mbar_wait(&ctrl->empty[s], ph ^ 1u, wctx, 11)) {
                        ok = false;
                        break;
                    }
                    if (rank == 0) mbar_arrive_expect_tx(&ctrl->full[s], 2 * C_STAGE_BYTES);
                    const uint32_t bar = cluster_address(&ctrl->full[s], 0);
                    const uint32_t st = smem_base + s * C_STAGE_BYTES;
                    const int col = static_cast<int>(seg_begin + j);
                    tma_load_2d_pair(st, &maps.xhi, bar, col, x_row);
                    tma_load_2d_pair(st + C_PART_BYTES, &maps.xlo, bar, col, x_row);
                    tma_load_2d_pair(st + 2 * C_PART_BYTES, &maps.yhi, bar, col, y_row);
                    tma_load_2d_pair(st + 3 * C_PART_BYTES, &maps.ylo, bar, col, y_row);
                }
            })
            if (!ok) {
                // another role gave up: a millisecond for the copies that are in flight before the block's memory is let go
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000) {
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = make_idesc_f16(256, CN);
            uint32_t kbt = 0;
            uint32_t uses[2] = {0, 0};
            bool ok = true;
            CHAIN_FOR_EACH_UNIT_SEGMENT({
                // the rows must have read this accumulator's previous checkpoint before it grows (or restarts)
                if (uses[a] > 0 && !mbar_wait(&ctrl->acc_loaded[a], (uses[a] - 1) & 1u, wctx, 12)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t acc = tmem_base + a * CN;
                for (uint32_t j = 0; j < seg_length; j += CK, ++kbt) {
                    const uint32_t s = kbt % C_STAGES, ph = (kbt / C_STAGES) & 1u;
                    if (!mbar_wait(&ctrl->full[s], ph, wctx, 13)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t st = smem_base + s * C_STAGE_BYTES;
                    // (nothing but zeros behind the segment)
                    const uint32_t steps = min(static_cast<uint32_t>(CK / 16), (seg_length - j + 15) / 16);
                    for (uint32_t kk = 0; kk < steps; ++kk) {
                        const uint64_t xh = make_desc_128(st + kk * 32), xl = make_desc_128(st + C_PART_BYTES + kk * 32);
                        const uint64_t yh = make_desc_128(st + 2 * C_PART_BYTES + kk * 32), yl = make_desc_128(st + 3 * C_PART_BYTES + kk * 32);
                        umma_f16_pair(acc, xh, yh, (seg | j | kk) != 0 ? 1u : 0u, idesc);
                        umma_f16_pair(acc, xh, yl, 1u, idesc);
                        umma_f16_pair(acc, xl, yh, 1u, idesc);
                    }
                    umma_commit_pair(&ctrl->empty[s]);
                }
                if (ok) umma_commit_pair(&ctrl->acc_ready[a]);
                ++uses[a];
            })
        }
    } else {
        // ---------------------------------------------------------------- tests at every checkpoint
        const uint32_t quarter = warp & 3, part = static_cast<uint32_t>(warp - 2) >> 2;   // rows 32 quarter.., columns 64 part..
        const uint32_t lane_base = 32u * quarter, row_in_tile = lane_base + lane;
        float* ny = ctrl->ny[warp - 2];
        float* fy = ctrl->fy[warp - 2];
        uint32_t uses[2] = {0, 0};
        uint32_t exchanges = 0;
        bool ok = true;
        size_t cur_item = ~size_t{0};
        uint32_t cur_chunk = 0xFFFFFFFFu;
        size_t row = 0;
        bool row_valid = false;
        float best = -1.f, cb = FLT_MAX, t1 = FLT_MAX, t2 = FLT_MAX, factor = 0.f;
        uint32_t bestidx = 0, prev = 0xFFFFFFFFu, npc = 0, cnt = 0, cbi = 0, i1 = 0xFFFFFFFFu, i2 = 0xFFFFFFFFu;
        uint32_t o1 = 0xFFFFFFFFu, o2 = 0xFFFFFFFFu;   // merged runner-ups of the row, set at every chunk end
        bool prev_first = false;
        uint32_t alive0[2] = {0, 0}, alive1[2] = {0, 0};   // survivors of the unit in accumulator 0 and 1, columns 0-31 and 32-63
        // End of a chunk: the four threads of the row exchange what they found in their columns and all apply the same update.  Returns
        // false when a wait ran out.
        auto close_chunk = [&]() -> bool {
            if (exchanges > 0 && !__all_sync(0xffffffffu, mbar_wait(&ctrl->heard[quarter], (exchanges - 1) & 1u, wctx, 17))) return false;
            ctrl->xchg[part][row_in_tile] = ChainPartial{cnt, prev_first ? 1u : 0u, cb, cbi, t1, t2, i1, i2};
            __threadfence_block();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctrl->told[quarter]);
            if (!__all_sync(0xffffffffu, mbar_wait(&ctrl->told[quarter], exchanges & 1u, wctx, 16))) return false;
            ++exchanges;
            uint32_t cnt_all = 0, prev_all = 0, mbi = 0;
            float mb = FLT_MAX, v1 = FLT_MAX, v2 = FLT_MAX;
            o1 = o2 = 0xFFFFFFFFu;
#pragma unroll 1
            for (int q = 0; q < 4; ++q) {
                const ChainPartial c = ctrl->xchg[q][row_in_tile];
                cnt_all += c.cnt;
                prev_all |= c.prev_first;
                if (c.cb < mb || (c.cb == mb && c.cbi < mbi)) {
                    mb = c.cb;
                    mbi = c.cbi;
                }
                // the two smallest of all, for the end of the row (the threads' own pairs cover disjoint columns and stay as they are)
                if (c.t1 < v1) {
                    o2 = v1 < c.t2 ? o1 : c.i2;
                    v2 = fminf(v1, c.t2);
                    o1 = c.i1;
                    v1 = c.t1;
                } else if (c.t1 < v2) {
                    o2 = c.i1;
                    v2 = c.t1;
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctrl->heard[quarter]);
            npc += cnt_all;
            // pdxearch.h:140-143: the previous centroid as the only survivor leaves the candidate untouched
            if (mb < FLT_MAX && !(cnt_all == 1u && prev_all)) {
                best = mb;
                bestidx = mbi;
            }
            if (SLICES > 1 && part == 0 && row_valid) p.partial[cur_item % SLICES * p.n + row] = ChainPartial{cnt_all, prev_all, mb, mbi, v1, v2, o1, o2};
            cnt = 0;
            prev_first = false;
            cb = FLT_MAX;
            cbi = 0;
            return true;
        };
        auto close_row = [&]() {
            if (row_valid && part == 0 && SLICES == 1) {
                p.knn[row] = bestidx;
                p.dist[row] = best;
                p.not_pruned[row] = npc;
                p.top2[row] = make_uint2(o1, o2);
            }
        };
        CHAIN_FOR_EACH_UNIT_SEGMENT({
            if (item != cur_item) {
                if (cur_item != ~size_t{0}) {
                    if (!close_chunk()) {
                        ok = false;
                        break;
                    }
                    close_row();
                }
                cur_item = item;
                cur_chunk = chunk;
                row = rt * 256 + rank * 128 + row_in_tile;
                row_valid = row < p.n;
                best = row_valid ? p.best_in[row] : -1.f;
                factor = row_valid ? p.factor_x[row] : 0.f;
                prev = row_valid ? p.knn[row] : 0xFFFFFFFFu;
                bestidx = row_valid ? prev : 0u;
                npc = 0;
                cnt = 0;
                prev_first = false;
                cb = FLT_MAX;
                cbi = 0;
                t1 = t2 = FLT_MAX;
                i1 = i2 = 0xFFFFFFFFu;
            } else if (chunk != cur_chunk) {
                if (!close_chunk()) {
                    ok = false;
                    break;
                }
                cur_chunk = chunk;
            }
            const size_t col0 = c0 + static_cast<size_t>(unit) * CN + part * 64;
            const uint32_t cols_valid = static_cast<uint32_t>(min(static_cast<size_t>(64), p.k - min(col0, p.k)));
            const float thr = best * ctrl->seg_ratio[seg];
            const float nx = row_valid ? __ldg(p.norms_x + row * p.n_seg + seg) : 0.f;
            const bool first = seg == 0, last = (seg + 1 == p.n_seg);
            {
                const float* __restrict__ src = p.norms_y + static_cast<size_t>(seg) * p.k + col0;
                float n2[2];
                float f2[2];
#pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {
                    const bool in = q * 32 + lane < cols_valid;
                    n2[q] = in ? __ldg(src + q * 32 + lane) : 0.f;
                    f2[q] = in ? __ldg(p.factor_y + col0 + q * 32 + lane) : 0.f;
                }
                __syncwarp();
#pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {
                    ny[q * 32 + lane] = n2[q];
                    fy[q * 32 + lane] = f2[q];
                }
                __syncwarp();
            }
            if (!__all_sync(0xffffffffu, mbar_wait(&ctrl->acc_ready[a], uses[a] & 1u, wctx, 15))) {
                ok = false;
                break;
            }
            ++uses[a];
            tc_fence_after();
            const uint32_t taddr = tmem_base + (lane_base << 16) + a * CN + part * 64;
            const uint64_t nx2 = pack2(nx, nx), factor2 = pack2(factor, factor), minus_thr2 = pack2(-thr, -thr);
            uint32_t alive_lo = a ? alive1[0] : alive0[0], alive_hi = a ? alive1[1] : alive0[1];
#pragma unroll 1
            for (uint32_t ch = 0; ch < 2; ++ch) {
                uint32_t r[32];
                tmem_ld32(taddr + ch * 32, r);
                if (ch == 1) {
                    // everything of this checkpoint is in registers: the accumulator may grow again
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster_read(cluster_address(&ctrl->acc_loaded[a], 0));
                }
                // two columns per instruction; the sign of (distance - threshold) is the column's bit
                uint32_t bits[4] = {0, 0, 0, 0};
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const float4 n0 = *reinterpret_cast<const float4*>(ny + ch * 32 + 8 * h), n1 = *reinterpret_cast<const float4*>(ny + ch * 32 + 8 * h + 4);
                    const float4 f0 = *reinterpret_cast<const float4*>(fy + ch * 32 + 8 * h), f1 = *reinterpret_cast<const float4*>(fy + ch * 32 + 8 * h + 4);
                    const uint64_t nyv[4] = {pack2(n0.x, n0.y), pack2(n0.z, n0.w), pack2(n1.x, n1.y), pack2(n1.z, n1.w)};
                    const uint64_t fv[4] = {pack2(f0.x, f0.y), pack2(f0.z, f0.w), pack2(f1.x, f1.y), pack2(f1.z, f1.w)};
#pragma unroll
                    for (int q = 3; q >= 0; --q) {
                        uint32_t& lo = r[8 * h + 2 * q];
                        uint32_t& hi = r[8 * h + 2 * q + 1];
                        // (the sum takes one factor after the other: their product may be no float)
                        const uint64_t pd = add2(fma2(mul2(factor2, pack2(__uint_as_float(lo), __uint_as_float(hi))), fv[q], nx2), nyv[q]);
                        const uint64_t over = add2(pd, minus_thr2);
                        lo = static_cast<uint32_t>(pd);
                        hi = static_cast<uint32_t>(pd >> 32);
                        bits[h] = __funnelshift_l(static_cast<uint32_t>(over >> 32), bits[h], 1);
                        bits[h] = __funnelshift_l(static_cast<uint32_t>(over), bits[h], 1);
                    }
                }
                uint32_t al = bits[0] | bits[1] << 8 | bits[2] << 16 | bits[3] << 24;
                uint32_t compete = 0;   // at the last checkpoint
                if (first) {
                    const uint32_t lo = ch * 32;
                    al &= (cols_valid >= lo + 32) ? 0xFFFFFFFFu : (cols_valid > lo ? ((1u << (cols_valid - lo)) - 1u) : 0u);
                    cnt += __popc(al);
                    const size_t at = static_cast<size_t>(prev) - (col0 + lo);   // (wraps when the previous centroid is before these columns)
                    if (at < 32 && ((al >> at) & 1u)) prev_first = true;
                    compete = al;
                } else {
                    compete = ch ? alive_hi : alive_lo;
                    al &= compete;
                }
                if (ch) alive_hi = al;
                else alive_lo = al;
                if (last && __any_sync(0xffffffffu, compete != 0)) {
                    // Last checkpoint: the pairs alive until here compete, those below the threshold (which is `best`: ratio[d] == 1) for the chain's
                    // winner.  Its distances are truncated, by 3e-5 of the norms at d = 1536, so that a centroid a little nearer than the previous one may
                    // end above it: the runner-ups are taken from all of them, and the fp32 refinement afterwards decides.
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        if ((compete >> j) & 1u) {
                            const float pd = __uint_as_float(r[j]);
                            const uint32_t gc = static_cast<uint32_t>(col0 + ch * 32 + j);
                            if (pd < t2) {
                                const bool nearer = pd < t1;
                                t2 = nearer ? t1 : pd;
                                i2 = nearer ? i1 : gc;
                                t1 = nearer ? pd : t1;
                                i1 = nearer ? gc : i1;
                            }
                            if (((al >> j) & 1u) && pd < cb) {
                                cb = pd;
                                cbi = gc;
                            }
                        }
                    }
                }
            }
            if (a) {
                alive1[0] = alive_lo;
                alive1[1] = alive_hi;
            } else {
                alive0[0] = alive_lo;
                alive0[1] = alive_hi;
            }
        })
        if (ok && cur_item != ~size_t{0}) {
            if (close_chunk()) close_row();
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync();   // nothing of the pair is in flight towards this CTA any more
    if (warp == 1) tmem_dealloc_pair(tmem_base, TMEM_COLS);
}
#undef CHAIN_FOR_EACH_UNIT_SEGMENT

// The end of a chunk (close_chunk above) for rows whose units were looked at by blocks of their own.  `state` carries a row from chunk
// to chunk, `best` is the threshold that the next chunk's blocks read.
struct ChainState {
    uint32_t bestidx, npc;
    float t1, t2;
    uint32_t i1, i2;
};

__global__ void __launch_bounds__(128) merge_chain_kernel(const ChainPartial* __restrict__ partial, uint32_t n_units, size_t n, bool first, bool last, const float* __restrict__ best_in,
                                                          float* __restrict__ best_state, ChainState* __restrict__ state, uint32_t* __restrict__ knn, float* __restrict__ dist,
                                                          uint32_t* __restrict__ not_pruned, uint2* __restrict__ top2, const int* __restrict__ error) {
    const size_t row = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    // (partials of a chain that gave up on a wait are not read)
    if (row >= n || *reinterpret_cast<const volatile int*>(error) != 0) return;
    ChainState st{};
    float best;
    if (first) {
        st = {knn[row], 0u, FLT_MAX, FLT_MAX, 0xFFFFFFFFu, 0xFFFFFFFFu};
        best = best_in[row];
    } else {
        st = state[row];
        best = best_state[row];
    }
    uint32_t cnt = 0, prev_first = 0, mbi = 0;
    float mb = FLT_MAX;
    for (uint32_t u = 0; u < n_units; ++u) {
        const ChainPartial q = partial[u * n + row];
        cnt += q.cnt;
        prev_first |= q.prev_first;
        if (q.cb < mb || (q.cb == mb && q.cbi < mbi)) {
            mb = q.cb;
            mbi = q.cbi;
        }
        if (q.t1 < st.t1) {
            if (st.t1 < q.t2) {
                st.t2 = st.t1;
                st.i2 = st.i1;
            } else {
                st.t2 = q.t2;
                st.i2 = q.i2;
            }
            st.t1 = q.t1;
            st.i1 = q.i1;
        } else if (q.t1 < st.t2) {
            st.t2 = q.t1;
            st.i2 = q.i1;
        }
    }
    st.npc += cnt;
    if (mb < FLT_MAX && !(cnt == 1u && prev_first)) {
        best = mb;
        st.bestidx = mbi;
    }
    if (!last) {
        state[row] = st;
        best_state[row] = best;
        return;
    }
    knn[row] = st.bestidx;
    dist[row] = best;
    not_pruned[row] = st.npc;
    top2[row] = make_uint2(st.i1, st.i2);
}

// Power of two that maps the largest element of a row below 2^14, for rows whose squared norm is no normal number any more: shorter than 1e-19, which fp32
// tells apart all the same, or longer than 1.8e19, of which some checkpoints are still finite.
__device__ __forceinline__ float scale_of_largest(const float* __restrict__ row, uint32_t d, int lane) {
    float m = 0.f;
    for (uint32_t j = lane; j < d; j += 32) m = fmaxf(m, fabsf(__ldg(row + j)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (!(m > 0.f) || m > FLT_MAX) return 1.0f;
    int e;
    frexpf(m, &e);
    return ldexpf(1.0f, min(14 - e, 126));
}

// A row of points or centroids for the chain, by a warp: cumulative squared norms at the checkpoints, then the halves in the order of the
// chain (ChainShape), zeros behind every segment.  Returns the scale.
__device__ __forceinline__ float chain_row(const float* __restrict__ row, const ChainShape& s, float* norms, size_t norms_stride, __half* __restrict__ hi, __half* __restrict__ lo,
                                           int lane) {
    const float sqnorm = chain_norms_row(row, s.partial_d, s.vertical_d, s.horizontal_d, lane, norms, norms_stride);
    const float scale = has_split_scale(sqnorm) ? split_scale(sqnorm) : scale_of_largest(row, s.d, lane);
    const uint32_t pitch = s.pitch(), h0 = s.begin(1), t0 = h0 + s.horizontal_d;
    for (uint32_t c = 4 * lane; c < pitch; c += 128) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (c >= h0 && c < t0) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(row + s.vertical_d + (c - h0)));
            v[0] = t.x;
            v[1] = t.y;
            v[2] = t.z;
            v[3] = t.w;
        } else {
            const uint32_t first = c < h0 ? c : s.partial_d + (c - t0), end = c < h0 ? s.partial_d : s.vertical_d;   // (on no boundary behind d')
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                if (first + q < end) v[q] = __ldg(row + first + q);
        }
        __align__(8) __half h[4], l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            h[q] = __float2half_rn(v[q] * scale);
            l[q] = __float2half_rn(v[q] * scale - __half2float(h[q]));
        }
        *reinterpret_cast<uint2*>(hi + c) = *reinterpret_cast<const uint2*>(h);
        *reinterpret_cast<uint2*>(lo + c) = *reinterpret_cast<const uint2*>(l);
    }
    return scale;
}

// Points idx[i] (or i): halves, factors, norms and, gathered, their state.
__global__ void __launch_bounds__(256) chain_points_kernel(const float* __restrict__ x, const uint32_t* __restrict__ idx, const float* __restrict__ best, const uint32_t* __restrict__ knn,
                                                           size_t n, const ChainShape s, const ChainHalves out, float* __restrict__ best_out, uint32_t* __restrict__ knn_out) {
    const size_t i = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    const int lane = threadIdx.x & 31;
    const size_t row = idx ? idx[i] : i, pitch = s.pitch(), n_seg = s.n_seg();
    const float scale = chain_row(x + row * s.d, s, out.norms + i * n_seg, 1, out.hi + i * pitch, out.lo + i * pitch, lane);
    if (lane == 0) {
        out.factor[i] = -2.0f / scale;
        if (idx) {
            best_out[i] = best[row];
            knn_out[i] = knn[row];
        }
    }
}

__global__ void __launch_bounds__(256) chain_centroids_kernel(const float* __restrict__ y, size_t k, const ChainShape s, const ChainHalves out) {
    const size_t c = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (c >= k) return;
    const int lane = threadIdx.x & 31;
    const size_t pitch = s.pitch();
    const float scale = chain_row(y + c * s.d, s, out.norms + c, k, out.hi + c * pitch, out.lo + c * pitch, lane);
    if (lane == 0) out.factor[c] = 1.0f / scale;
}

} // namespace

void launch_chain_points(const float* x, const uint32_t* idx, const float* best, const uint32_t* knn, size_t n, const ChainShape& shape, const ChainHalves& out, float* best_out,
                         uint32_t* knn_out, cudaStream_t stream) {
    if (n == 0) return;
    chain_points_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(x, idx, best, knn, n, shape, out, best_out, knn_out);
    SKM_LAUNCH_CHECK();
}

void launch_chain_centroids(const float* y, size_t k, const ChainShape& shape, const ChainHalves& out, cudaStream_t stream) {
    if (k == 0) return;
    chain_centroids_kernel<<<static_cast<unsigned>((k + 7) / 8), 256, 0, stream>>>(y, k, shape, out);
    SKM_LAUNCH_CHECK();
}

// Few rows: a pair of blocks per tile leaves most SMs idle.  While every tile can have four pairs, each takes one of the (at most four)
// units of a chunk, a launch per chunk, and merge_chain_kernel does what the tile's rows do at the end of a chunk.
constexpr uint32_t kChainSlices = kChunk / CN;
static_assert(kChainSlices == kChainUnits && kChainTileRows == 256, "chain_shares_tiles counts them");
int sm_pairs() {
    int device = 0, sms = 0;
    SKM_CUDA(cudaGetDevice(&device));
    SKM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    return sms / 2;
}
size_t chain_scratch_bytes(size_t rows) { return rows * (kChainSlices * sizeof(ChainPartial) + sizeof(ChainState) + sizeof(float)); }

void launch_chain(size_t n, size_t k, const ChainShape& shape, const ChainHalves& x, const ChainHalves& y, const float* ratios, const float* best_in, uint32_t* knn, float* dist,
                  uint32_t* not_pruned, uint2* top2, const ChainScratch& scratch, cudaStream_t stream, const std::function<void()>& beside) {
    if (n == 0 || k == 0) return;
    const size_t pitch = shape.pitch();
    ChainMaps maps;
    maps.xhi = make_half_tmap(x.hi, pitch, n, 128);
    maps.xlo = make_half_tmap(x.lo, pitch, n, 128);
    maps.yhi = make_half_tmap(y.hi, pitch, k, 128);
    maps.ylo = make_half_tmap(y.lo, pitch, k, 128);
    ChainParams p{};
    p.n = n;
    p.k = k;
    p.shape = shape;
    p.n_seg = shape.n_seg();
    if (p.n_seg > kMaxSegments) throw std::invalid_argument("dimensionality too large for the tensor-core chain");
    p.factor_x = x.factor;
    p.factor_y = y.factor;
    p.norms_x = x.norms;
    p.norms_y = y.norms;
    p.ratios = ratios;
    p.best_in = best_in;
    p.knn = knn;
    p.dist = dist;
    p.not_pruned = not_pruned;
    p.top2 = top2;
    p.error = error_word();
    p.wait_limit = wait_limit();
    p.producer_stop = producer_stop();
    const size_t row_tiles = (n + 255) / 256;
    const uint32_t n_chunks = static_cast<uint32_t>((k + kChunk - 1) / kChunk);
    if (n > scratch.rows || !chain_shares_tiles(n, static_cast<size_t>(sm_pairs()))) {
        p.chunk_end = n_chunks;
        SKM_CUDA(cudaFuncSetAttribute(chain_tc_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(C_SMEM_BYTES)));
        chain_tc_kernel<1><<<static_cast<unsigned>(2 * std::min<size_t>(row_tiles, static_cast<size_t>(sm_pairs()))), C_THREADS, C_SMEM_BYTES, stream>>>(maps, p);
        SKM_LAUNCH_CHECK();
        if (beside) beside();
        return;
    }
    SKM_CUDA(cudaFuncSetAttribute(chain_tc_kernel<kChainSlices>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(C_SMEM_BYTES)));
    p.partial = static_cast<ChainPartial*>(scratch.p);
    ChainState* state = reinterpret_cast<ChainState*>(p.partial + kChainSlices * n);
    float* best = reinterpret_cast<float*>(state + n);
    for (uint32_t c = 0; c < n_chunks; ++c) {
        const size_t cs = std::min<size_t>(kChunk, k - static_cast<size_t>(c) * kChunk);
        p.chunk_begin = c;
        p.chunk_end = c + 1;
        p.best_in = c == 0 ? best_in : best;
        chain_tc_kernel<kChainSlices><<<static_cast<unsigned>(2 * row_tiles * kChainSlices), C_THREADS, C_SMEM_BYTES, stream>>>(maps, p);
        SKM_LAUNCH_CHECK();
        if (c == 0 && beside) beside();
        merge_chain_kernel<<<static_cast<unsigned>((n + 127) / 128), 128, 0, stream>>>(p.partial, static_cast<uint32_t>((cs + CN - 1) / CN), n, c == 0, c + 1 == n_chunks, best_in, best,
                                                                                      state, knn, dist, not_pruned, top2, p.error);
        SKM_LAUNCH_CHECK();
    }
}

} // namespace tc
} // namespace skmb
