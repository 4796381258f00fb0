// First ADSampling test on the tensor cores (batch_computers.h:297-409, pdxearch.h:118-143): the partial distances over the
// first d' dimensions of every (point, centroid) pair against best * ratio[d'], survivors to candidate lists that
// walk_lists_kernel takes up.
//
// Points and centroids come as fp16 pairs v * scale = hi + lo (scale a power of two, 22 bits: what two tf32 parts hold), and
// a product is hi*hi + hi*lo + lo*hi with fp32 accumulation: fp32-level accuracy at twice the rate of tf32.  The points are
// split once per training, over the dimensions d' can reach, not in every tile, each with a scale of its own.  The centroids share
// one while the smallest is no shorter than a thousandth of the longest, and have their own otherwise (kOneScaleSpread).
//
// Persistent pairs of CTAs (cta_group::2) on tiles of 256 rows x 256 centroids, as in exact_assign.cu:
//   warp 0     TMA producer: 128 x 64 halves of each of the four parts per stage, three stages;
//   warp 1     MMA issuer (leader only), two accumulators of 256 columns;
//   warps 2-17 test, a warp per 32 rows and 64 columns: partial distance = ||x||^2 + ||c||^2 - 2 x.c, survivors appended to
//              the warp's list.  The test is what bounds the kernel, its latency more than its 200 instructions per 32
//              columns: hence four warps per scheduler (with two it took 6500 cycles per tile), two columns per instruction
//              and no scan for the places in the list.  1M x 1024, k = 4000, nine passes: 27.2 ms with one column per
//              instruction and a scan by shuffles, 25.0 so, and 20.1 since the accumulators are given back without a release
//              at cluster scope, which waited for the lists' stores (a third of all stalls).
// Every wait is bounded (see kernels_tc.cu).
#include <cfloat>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "device_utils.cuh"
#include "kernels_tc.cuh"
#include "tc_ptx.cuh"

namespace skmb {
namespace tc {

namespace {

constexpr int TK = 64;
constexpr int T_STAGES = 3;
constexpr uint32_t T_PART_BYTES = 128 * TK * 2;
constexpr uint32_t T_STAGE_BYTES = 4 * T_PART_BYTES;   // rows hi, rows lo, centroids hi, centroids lo
constexpr int T_TEST_WARPS = 16;
constexpr int T_THREADS = 64 + 32 * T_TEST_WARPS;
constexpr uint32_t T_CTRL_BYTES = 2 * 8192 + T_TEST_WARPS * 8 * 32 * 4 + 256;
constexpr uint32_t T_SMEM_BYTES = T_STAGES * T_STAGE_BYTES + T_CTRL_BYTES + 1024;

struct TestCtrl {
    alignas(16) float ny[4][2][256];   // per row quarter and accumulator
    alignas(16) float fy[4][2][256];   // so the centroids' factors, where they differ
    float column[T_TEST_WARPS][8 * 32];   // per test warp: 8 values of each of its lanes
    uint32_t filled[T_TEST_WARPS];
    uint64_t full[T_STAGES];           // (the leader's are used)
    uint64_t empty[T_STAGES];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];             // (the leader's are used)
    uint32_t tmem_base;
};
static_assert(sizeof(TestCtrl) <= T_CTRL_BYTES, "control block too large");

struct TestMaps {
    CUtensorMap xhi, xlo, yhi, ylo;
};

struct TestParams {
    size_t n, k;
    uint32_t k_blocks, partial_d;
    size_t tile0, n_tiles;       // of 128 rows
    const uint32_t* tile_map;    // null: tile0, tile0 + 1, ...
    const float* factor_x;       // per row: -2 / scale
    const float* factor_y;       // per centroid: 1 / scale; behind them: not zero if they are all alike
    const float* norms_x;
    const float* norms_y;
    const float* best_in;
    uint32_t* flags;             // may be null: per row, nonzero = leave this point out
    uint32_t limit_slope;        // 2^-32: a row with kFirstTestLimitStart and this many survivors per column of a warp is left out from there on, and
    uint32_t* dropped;           // appended here (its flag set)
    uint32_t* n_dropped;
    float ratio_first;
    uint2* lists;
    uint32_t* list_offs;
    uint32_t cap_group;
    int* error;
    long long wait_limit;
    uint32_t producer_stop;      // see set_debug_wait_injection
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(T_THREADS, 1) first_test_kernel(const __grid_constant__ TestMaps maps, const TestParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
    const uint32_t smem_base = raw_addr + pad;
    TestCtrl* ctrl = reinterpret_cast<TestCtrl*>(smem_raw + pad + T_STAGES * T_STAGE_BYTES);
    const WaitCtx wctx{p.error, p.wait_limit};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();

    if (threadIdx.x == 0) {
        for (int s = 0; s < T_STAGES; ++s) {
            mbar_init(&ctrl->full[s], 1);
            mbar_init(&ctrl->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctrl->acc_full[b], 1);
            mbar_init(&ctrl->acc_empty[b], 2 * T_TEST_WARPS);   // a lane of each of the pair's test warps
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

    const size_t pair_tiles = (p.n_tiles + 1) / 2;
    const uint32_t col_tiles = static_cast<uint32_t>((p.k + 255) / 256);
    const size_t pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    // this CTA's row tile of pair tile t (the second one of the last pair may not exist: a tile behind the last row)
    auto tile_of = [&](size_t t) -> size_t {
        const size_t q = 2 * t + rank;
        if (q >= p.n_tiles) return (p.n + 127) / 128;
        return p.tile_map ? static_cast<size_t>(__ldg(p.tile_map + q)) : p.tile0 + q;
    };

    if (warp == 0) {
        if (lane == 0) {
            uint32_t kbt = 0;
            bool ok = true;
            for (size_t t = pair; t < pair_tiles && ok; t += n_pairs) {
                const int x_row = static_cast<int>(tile_of(t) * 128);
                for (uint32_t nt = 0; nt < col_tiles && ok; ++nt) {
                    const int y_row = static_cast<int>(nt * 256 + rank * 128);
                    for (uint32_t kb = 0; kb < p.k_blocks; ++kb, ++kbt) {
                        const uint32_t s = kbt % T_STAGES, ph = (kbt / T_STAGES) & 1u;
                        if ((p.producer_stop != 0 && kbt >= p.producer_stop) || !mbar_wait(&ctrl->empty[s], ph ^ 1u, wctx, 51)) {
                            ok = false;
                            break;
                        }
                        if (rank == 0) mbar_arrive_expect_tx(&ctrl->full[s], 2 * T_STAGE_BYTES);
                        const uint32_t bar = cluster_address(&ctrl->full[s], 0);
                        const uint32_t st = smem_base + s * T_STAGE_BYTES;
                        const int col = static_cast<int>(kb * TK);
                        tma_load_2d_pair(st, &maps.xhi, bar, col, x_row);
                        tma_load_2d_pair(st + T_PART_BYTES, &maps.xlo, bar, col, x_row);
                        tma_load_2d_pair(st + 2 * T_PART_BYTES, &maps.yhi, bar, col, y_row);
                        tma_load_2d_pair(st + 3 * T_PART_BYTES, &maps.ylo, bar, col, y_row);
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
            constexpr uint32_t idesc = make_idesc_f16(256, 256);
            uint32_t kbt = 0, u = 0;
            bool ok = true;
            for (size_t t = pair; t < pair_tiles && ok; t += n_pairs) {
                for (uint32_t nt = 0; nt < col_tiles && ok; ++nt, ++u) {
                    const uint32_t b = u & 1u, uph = (u >> 1) & 1u;
                    if (!mbar_wait(&ctrl->acc_empty[b], uph ^ 1u, wctx, 52)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t acc = tmem_base + b * 256;
                    for (uint32_t kb = 0; kb < p.k_blocks; ++kb, ++kbt) {
                        const uint32_t s = kbt % T_STAGES, ph = (kbt / T_STAGES) & 1u;
                        if (!mbar_wait(&ctrl->full[s], ph, wctx, 53)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t st = smem_base + s * T_STAGE_BYTES;
                        // (nothing but zeros behind partial_d)
                        const uint32_t steps = min(static_cast<uint32_t>(TK / 16), (p.partial_d - kb * TK + 15) / 16);
                        for (uint32_t kk = 0; kk < steps; ++kk) {
                            const uint64_t xh = make_desc_128(st + kk * 32), xl = make_desc_128(st + T_PART_BYTES + kk * 32);
                            const uint64_t yh = make_desc_128(st + 2 * T_PART_BYTES + kk * 32), yl = make_desc_128(st + 3 * T_PART_BYTES + kk * 32);
                            umma_f16_pair(acc, xh, yh, (kb | kk) != 0 ? 1u : 0u, idesc);
                            umma_f16_pair(acc, xh, yl, 1u, idesc);
                            umma_f16_pair(acc, xl, yh, 1u, idesc);
                        }
                        umma_commit_pair(&ctrl->empty[s]);
                    }
                    if (ok) umma_commit_pair(&ctrl->acc_full[b]);
                }
            }
        }
    } else {
        const uint32_t quarter = warp & 3, part = static_cast<uint32_t>(warp - 2) >> 2;   // rows 32 quarter.., columns 64 part..
        const uint32_t lane_base = 32u * quarter;
        float* column = ctrl->column[warp - 2] + lane;
        uint32_t* filled = &ctrl->filled[warp - 2];   // pairs in the warp's list
        const bool one_scale = p.factor_y[p.k] != 0.f;
        const float fy = one_scale ? p.factor_y[0] : 1.0f;
        uint32_t u = 0;
        bool ok = true;
        for (size_t t = pair; t < pair_tiles && ok; t += n_pairs) {
            const size_t q = 2 * t + rank;
            const bool listed = q < p.n_tiles;
            const size_t row = tile_of(t) * 128 + lane_base + lane;
            const bool valid = listed && row < p.n;
            const float nx = valid ? p.norms_x[row] : 0.f;
            const float factor = valid ? p.factor_x[row] * fy : 0.f;
            const uint64_t nx2 = pack2(nx, nx), factor2 = pack2(factor, factor);
            float thr = valid && !(p.flags && p.flags[row]) ? p.best_in[row] * p.ratio_first : -FLT_MAX;
            uint32_t survivors = 0;
            const size_t group = (listed ? q : 0) * kListsPerTile + part * 4 + quarter;
            uint2* my_list = p.lists + group * p.cap_group;
            uint32_t* my_offs = p.list_offs + group * ((p.k + 1023) / 1024 + 1);
            if (lane == 0) *filled = 0;
            __syncwarp();
            for (uint32_t nt = 0; nt < col_tiles && ok; ++nt, ++u) {
                const uint32_t b = u & 1u, uph = (u >> 1) & 1u;
                const uint32_t col0 = nt * 256 + part * 64;
                float* ny = ctrl->ny[quarter][b] + part * 64;   // the four warps of a quarter fill (and read) their own parts
                if ((nt & 3u) == 0 && lane == 0 && listed) my_offs[nt >> 2] = *filled;
#pragma unroll
                for (int i = 0; i < 2; ++i) ny[i * 32 + lane] = col0 + i * 32 + lane < p.k ? __ldg(p.norms_y + col0 + i * 32 + lane) : INFINITY;   // never below a threshold
                float* fys = ctrl->fy[quarter][b] + part * 64;
                if (!one_scale) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) fys[i * 32 + lane] = col0 + i * 32 + lane < p.k ? __ldg(p.factor_y + col0 + i * 32 + lane) : 0.f;
                }
                __syncwarp();
                if (!__all_sync(0xffffffffu, mbar_wait(&ctrl->acc_full[b], uph, wctx, 54))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + (lane_base << 16) + b * 256 + part * 64;
                const uint64_t minus_thr2 = pack2(-thr, -thr);
                auto test = [&](uint32_t (&r)[32], int ch, auto own_scales) {
                    // two columns per instruction; the sign of (distance - threshold) is the column's bit
                    uint32_t bits[4] = {0, 0, 0, 0};
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        const float4 n0 = *reinterpret_cast<const float4*>(ny + ch * 32 + 8 * h), n1 = *reinterpret_cast<const float4*>(ny + ch * 32 + 8 * h + 4);
                        const uint64_t nyv[4] = {pack2(n0.x, n0.y), pack2(n0.z, n0.w), pack2(n1.x, n1.y), pack2(n1.z, n1.w)};
                        uint64_t factors[4] = {factor2, factor2, factor2, factor2};
                        if constexpr (decltype(own_scales)::value) {
                            const float4 f0 = *reinterpret_cast<const float4*>(fys + ch * 32 + 8 * h), f1 = *reinterpret_cast<const float4*>(fys + ch * 32 + 8 * h + 4);
                            factors[0] = mul2(factor2, pack2(f0.x, f0.y));
                            factors[1] = mul2(factor2, pack2(f0.z, f0.w));
                            factors[2] = mul2(factor2, pack2(f1.x, f1.y));
                            factors[3] = mul2(factor2, pack2(f1.z, f1.w));
                        }
#pragma unroll
                        for (int q = 3; q >= 0; --q) {
                            uint32_t& lo = r[8 * h + 2 * q];
                            uint32_t& hi = r[8 * h + 2 * q + 1];
                            const uint64_t pd = add2(fma2(factors[q], pack2(__uint_as_float(lo), __uint_as_float(hi)), nx2), nyv[q]);
                            const uint64_t over = add2(pd, minus_thr2);
                            lo = static_cast<uint32_t>(pd);
                            hi = static_cast<uint32_t>(pd >> 32);
                            bits[h] = __funnelshift_l(static_cast<uint32_t>(over >> 32), bits[h], 1);
                            bits[h] = __funnelshift_l(static_cast<uint32_t>(over), bits[h], 1);
                        }
                    }
                    const uint32_t mask = bits[0] | bits[1] << 8 | bits[2] << 16 | bits[3] << 24;
                    if (!__any_sync(0xffffffffu, mask != 0)) return;
                    // where a lane's survivors go, in any order: a list is read chunk by chunk
                    const uint32_t cnt = __popc(mask);
                    survivors += cnt;
                    uint32_t pos = cnt != 0 ? atomicAdd(filled, cnt) : 0u;
                    // They are few and found bit by bit, their values through a column of shared memory of the lane's own,
                    // because registers cannot be indexed (unrolled over the columns, this outgrows the instruction cache).
                    const uint32_t colbits = ((col0 + ch * 32) << 5) | static_cast<uint32_t>(lane);
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        uint32_t sub = bits[h];
                        if (!__any_sync(0xffffffffu, sub != 0)) continue;
#pragma unroll
                        for (int j = 0; j < 8; ++j) column[j * 32] = __uint_as_float(r[8 * h + j]);
#pragma unroll 1
                        while (sub) {
                            const uint32_t j = __ffs(sub) - 1;
                            sub &= sub - 1;
                            if (pos < p.cap_group) my_list[pos] = make_uint2(colbits + ((8u * h + j) << 5), __float_as_uint(column[j * 32]));
                            ++pos;
                        }
                        __syncwarp();
                    }
                };
#pragma unroll 1
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t r[32];
                    tmem_ld32(taddr + ch * 32, r);
                    if (ch == 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster_read(cluster_address(&ctrl->acc_empty[b], 0));
                    }
                    if (one_scale) test(r, ch, std::false_type{});
                    else test(r, ch, std::true_type{});
                }
                // Too many survivors, or on the way there: from the start of a point that keeps 10 %, the sloped line saves three
                // quarters of the pairs that would be listed in vain.
                const bool drop = survivors >= kFirstTestLimitStart + __umulhi((nt + 1) * 64, p.limit_slope);
                if (__any_sync(0xffffffffu, drop)) {
                    if (drop) {
                        survivors = 0;
                        thr = -FLT_MAX;
                        if (atomicExch(p.flags + row, 1u) == 0) p.dropped[atomicAdd(p.n_dropped, 1u)] = static_cast<uint32_t>(row);
                    }
                    __syncwarp();
                }
            }
            if (ok && lane == 0 && listed) my_offs[(p.k + 1023) / 1024] = *filled;
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // nothing of the pair is in flight towards this CTA any more
    if (warp == 1) tmem_dealloc_pair(tmem_base, TMEM_COLS);
}

// Largest ratio of two centroids' squared norms under one scale: a centroid 2^-10 as long as the longest still has its elements
// to 2^-29 of its norm, all of d' <= 16 384 together to 2^-22.  (With one scale for all, a single centroid of norm 1e10 among
// unit ones left nothing of these, and one of 1e7 a partial distance that was 1e-4 off.)  With a scale
// per centroid nine passes over 600 000 x 1024, k = 4000, take 13.6 - 15.1 ms, with one for all 12.0.
constexpr float kOneScaleSpread = 1048576.0f;

// (rows are 16-byte aligned and a multiple of 4 long, as everywhere on the tensor-core path)
__device__ __forceinline__ float4 leading_columns(const float* __restrict__ row, uint32_t j, uint32_t cols) {
    if (j >= cols) return make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v = __ldg(reinterpret_cast<const float4*>(row + j));
    if (j + 1 >= cols) v.y = 0.f;
    if (j + 2 >= cols) v.z = 0.f;
    if (j + 3 >= cols) v.w = 0.f;
    return v;
}

__device__ __forceinline__ void split_half_row(const float* __restrict__ row, uint32_t cols, uint32_t pitch, float scale, __half* __restrict__ hi, __half* __restrict__ lo, int lane) {
    for (uint32_t j = 4 * lane; j < pitch; j += 128) {
        const float4 v4 = leading_columns(row, j, cols);
        const float v[4] = {v4.x * scale, v4.y * scale, v4.z * scale, v4.w * scale};
        __align__(8) __half h[4], l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            h[q] = __float2half_rn(v[q]);
            l[q] = __float2half_rn(v[q] - __half2float(h[q]));
        }
        *reinterpret_cast<uint2*>(hi + j) = *reinterpret_cast<const uint2*>(h);
        *reinterpret_cast<uint2*>(lo + j) = *reinterpret_cast<const uint2*>(l);
    }
}

// The first `cols` columns of the points, a scale per row; one warp per row.
__global__ void __launch_bounds__(256) split_points_kernel(const float* __restrict__ x, size_t n, size_t d, uint32_t cols, uint32_t pitch, __half* __restrict__ hi,
                                                           __half* __restrict__ lo, float* __restrict__ factor) {
    const size_t row = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (row >= n) return;
    const int lane = threadIdx.x & 31;
    const float* xr = x + row * d;
    float s = 0.f;
    for (uint32_t j = 4 * lane; j < cols; j += 128) {
        const float4 v = leading_columns(xr, j, cols);
        s = fmaf(v.x, v.x, s); s = fmaf(v.y, v.y, s); s = fmaf(v.z, v.z, s); s = fmaf(v.w, v.w, s);
    }
    const float scale = split_scale(warp_sum(s));
    split_half_row(xr, cols, pitch, scale, hi + row * pitch, lo + row * pitch, lane);
    if (lane == 0) factor[row] = -2.0f / scale;
}

// The centroids: every block finds the largest and the smallest of the k squared norms over the columns in question (but for zeros and
// what is no number, which no scale helps).
__global__ void __launch_bounds__(256) split_centroids_kernel(const float* __restrict__ y, size_t k, size_t d, uint32_t cols, uint32_t pitch, const float* __restrict__ norms,
                                                              __half* __restrict__ hi, __half* __restrict__ lo, float* __restrict__ factor) {
    __shared__ float largest[8], smallest[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float m = 0.f, s = FLT_MAX;
    for (size_t c = threadIdx.x; c < k; c += 256) {
        const float v = __ldg(norms + c);
        m = fmaxf(m, v);
        if (v > 0.f) s = fminf(s, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        s = fminf(s, __shfl_xor_sync(0xffffffffu, s, o));
    }
    if (lane == 0) {
        largest[warp] = m;
        smallest[warp] = s;
    }
    __syncthreads();
    m = largest[0];
    s = smallest[0];
    for (int w = 1; w < 8; ++w) {
        m = fmaxf(m, largest[w]);
        s = fminf(s, smallest[w]);
    }
    const bool one_scale = m <= kOneScaleSpread * s || m == 0.f;
    if (blockIdx.x == 0 && threadIdx.x == 0) factor[k] = one_scale ? 1.0f : 0.0f;
    for (size_t c = static_cast<size_t>(blockIdx.x) * 8 + warp; c < k; c += static_cast<size_t>(gridDim.x) * 8) {
        const float scale = split_scale(one_scale ? m : __ldg(norms + c));
        split_half_row(y + c * d, cols, pitch, scale, hi + c * pitch, lo + c * pitch, lane);
        if (lane == 0) factor[c] = 1.0f / scale;
    }
}

} // namespace

void launch_split_points(const float* x, size_t n, size_t d, uint32_t cols, const SplitHalves& out, cudaStream_t stream) {
    if (n == 0) return;
    split_points_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(x, n, d, cols, out.pitch, out.hi, out.lo, out.factor);
    SKM_LAUNCH_CHECK();
}

void launch_split_centroids(const float* y, size_t k, size_t d, uint32_t cols, const float* norms, const SplitHalves& out, cudaStream_t stream) {
    if (k == 0) return;
    split_centroids_kernel<<<static_cast<unsigned>(std::min<size_t>(296, (k + 7) / 8)), 256, 0, stream>>>(y, k, d, cols, out.pitch, norms, out.hi, out.lo, out.factor);
    SKM_LAUNCH_CHECK();
}

void launch_first_test(const SplitHalves& x, const SplitHalves& y, size_t n, size_t k, uint32_t partial_d, const float* norms_x, const float* norms_y, const float* best_in,
                       float ratio_first, size_t tile0, size_t n_tiles, uint2* lists, uint32_t* list_offs, uint32_t cap_group, const FirstTestRows& rows, cudaStream_t stream) {
    if (n_tiles == 0 || k == 0) return;
    int device = 0, sms = 0;
    SKM_CUDA(cudaGetDevice(&device));
    SKM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    TestMaps maps;
    maps.xhi = make_half_tmap(x.hi, partial_d, n, 128, x.pitch);
    maps.xlo = make_half_tmap(x.lo, partial_d, n, 128, x.pitch);
    maps.yhi = make_half_tmap(y.hi, partial_d, k, 128, y.pitch);
    maps.ylo = make_half_tmap(y.lo, partial_d, k, 128, y.pitch);
    TestParams p{};
    p.n = n;
    p.k = k;
    p.k_blocks = (partial_d + TK - 1) / TK;
    p.partial_d = partial_d;
    p.tile0 = tile0;
    p.n_tiles = n_tiles;
    p.tile_map = rows.tile_map;
    p.factor_x = x.factor;
    p.factor_y = y.factor;
    p.norms_x = norms_x;
    p.norms_y = norms_y;
    p.best_in = best_in;
    p.flags = rows.flags;
    // a line from kFirstTestLimitStart at no column to the limit at all columns of a warp; without a limit one that no row reaches
    p.limit_slope = 0xFFFFFFFFu;
    if (rows.limit != 0xFFFFFFFFu) p.limit_slope = static_cast<uint32_t>(4294967296.0 * (rows.limit - std::min(rows.limit, kFirstTestLimitStart)) / (64.0 * ((k + 255) / 256)));
    p.dropped = rows.dropped;
    p.n_dropped = rows.n_dropped;
    p.ratio_first = ratio_first;
    p.lists = lists;
    p.list_offs = list_offs;
    p.cap_group = cap_group;
    p.error = error_word();
    p.wait_limit = wait_limit();
    p.producer_stop = producer_stop();
    SKM_CUDA(cudaFuncSetAttribute(first_test_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(T_SMEM_BYTES)));
    const unsigned grid = static_cast<unsigned>(2 * std::min<size_t>(static_cast<size_t>(sms / 2), (n_tiles + 1) / 2));
    first_test_kernel<<<grid, T_THREADS, T_SMEM_BYTES, stream>>>(maps, p);
    SKM_LAUNCH_CHECK();
}

} // namespace tc
} // namespace skmb
