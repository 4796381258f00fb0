// Rotation on the tensor cores: out = A * B^T for row-major fp32 A [n][K] and B [n_out][K] (ADSamplingPruner::Rotate with
// B = M, Unrotate with B = M^T; adsampling.h:191-215, :273-298), with fp32-level accuracy.
//
// Both operands are split into tf32 hi + lo parts in shared memory and multiplied as hi*hi + hi*lo + lo*hi (see
// kernels_tc.cu).  What limits the accuracy of that scheme is the accumulator in tensor memory, which truncates on every
// addition: a chain of K products ends up about K * 1e-8 (relative to |a| |b|) low.  Rotated rows feed every distance
// computed afterwards, so the chain is cut: the reduction dimension is divided among kAcc accumulators, each summing a
// quarter of K, and the epilogue adds the four partial sums in fp32 registers.  With K = 1024 that leaves ~2e-6, the
// level of a sequential fp32 accumulation.
//
// B arrives split; A is split in shared memory, whose bandwidth is what bounds a three-product scheme: tiles of 128 x 128 on
// single CTAs with both operands split in place moved 112 KB of it per 16 columns of K for 384 cycles of tensor work
// (896 cycles).  Pairs of CTAs on tiles of 256 x 256 move 96 KB for 768 cycles.  As four accumulators of 256 columns do not
// fit, a quarter of K at a time goes through one of two, and the epilogue adds it to its sums in registers while the next
// one runs.
// One B200, products counted three times: 300 000 x 768: 2.67 ms -> 1.74 (399 -> 612 TF/s); 150 000 x 1536: 5.01 -> 3.23 (658 TF/s).
//
// Persistent pairs of CTAs (cta_group::2), 384 threads, which leaves the epilogue's threads 168 registers for their 128 sums:
//   warp 0      TMA producer: A, B hi and B lo, 128 rows x 32 columns each per stage and CTA, 128-byte swizzle (with rows of
//               64 bytes the copies were the bound);
//   warp 1      MMA issuer (the leader's; M = 256, N = 256, K = 8);
//   warps 2-3   split the A tile of every other stage into hi / lo parts in place;
//   warps 4-11  epilogue, a thread per row and 128 columns.
// Every wait is bounded (see kernels_tc.cu).
#include <stdexcept>
#include <string>

#include "common.cuh"
#include "kernels_tc.cuh"
#include "tc_ptx.cuh"

namespace skmb {
namespace tc {

namespace {

constexpr int RN = 256;                  // output columns per tile
constexpr int RK = 32;                   // columns of K per stage
constexpr int kAcc = 4;                  // parts of K, whole blocks of BK columns, with an accumulator each
constexpr int ROT_STAGES = 3;
constexpr int ROT_SPLIT_WARPS = 2;
constexpr int ROT_EPI_WARPS = 8;
constexpr int ROT_THREADS = 64 + 32 * (ROT_SPLIT_WARPS + ROT_EPI_WARPS);
constexpr uint32_t ROT_TILE_BYTES = 128 * RK * 4;
constexpr uint32_t ROT_STAGE_BYTES = 4 * ROT_TILE_BYTES;   // A hi (as loaded: A), A lo, B hi, B lo
constexpr uint32_t ROT_CTRL_BYTES = 1024;
constexpr uint32_t ROT_SMEM_BYTES = ROT_STAGES * ROT_STAGE_BYTES + ROT_CTRL_BYTES + 1024;
// as make_idesc, for a pair: M = 256, N = 256
constexpr uint32_t ROT_IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((RN >> 3) << 17) | ((256u >> 4) << 24);

struct RotParams {
    size_t n, n_out;
    uint32_t kdim;
    float* out;
    size_t ldo;
    bool wide_stores;     // rows of out start on 32-byte boundaries
    int* error;
    long long wait_limit;
    uint32_t producer_stop;   // see set_debug_wait_injection
};

struct RotCtrl {
    uint64_t full[ROT_STAGES];    // this CTA's copies
    uint64_t conv[ROT_STAGES];    // (the leader's are used) copied and split in both CTAs
    uint64_t empty[ROT_STAGES];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];        // (the leader's are used)
    uint32_t tmem_base;
};
static_assert(sizeof(RotCtrl) <= ROT_CTRL_BYTES, "control block too large");

__device__ __forceinline__ void store8(float* p, const float* v) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(ROT_THREADS, 1)
    rotate_tc_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_bhi, const __grid_constant__ CUtensorMap tmap_blo, const RotParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
    uint8_t* smem = smem_raw + pad;
    const uint32_t smem_base = raw_addr + pad;
    RotCtrl* ctrl = reinterpret_cast<RotCtrl*>(smem + ROT_STAGES * ROT_STAGE_BYTES);
    const WaitCtx wctx{p.error, p.wait_limit};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();

    if (threadIdx.x == 0) {
        for (int s = 0; s < ROT_STAGES; ++s) {
            mbar_init(&ctrl->full[s], 1);
            mbar_init(&ctrl->conv[s], 2);
            mbar_init(&ctrl->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctrl->acc_full[b], 1);
            mbar_init(&ctrl->acc_empty[b], 2 * ROT_EPI_WARPS);
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

    const uint32_t n_col_tiles = static_cast<uint32_t>((p.n_out + RN - 1) / RN);
    const size_t n_tiles = (p.n + 255) / 256 * n_col_tiles;   // 256 x 256, the column tiles of a row tile one after the other
    const uint32_t n_stages = (p.kdim + RK - 1) / RK;
    const uint32_t nkb = (p.kdim + BK - 1) / BK, kb_per_acc = (nkb + kAcc - 1) / kAcc;
    const size_t first = blockIdx.x >> 1, step = gridDim.x >> 1;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (size_t t = first; t < n_tiles && ok; t += step) {
                const int a_row = static_cast<int>(t / n_col_tiles * 256 + rank * 128), b_row = static_cast<int>(t % n_col_tiles * RN + rank * 128);
                for (uint32_t k = 0; k < n_stages; ++k, ++it) {
                    const uint32_t s = it % ROT_STAGES, ph = (it / ROT_STAGES) & 1u;
                    if ((p.producer_stop != 0 && it >= p.producer_stop) || !mbar_wait(&ctrl->empty[s], ph ^ 1u, wctx, 31)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&ctrl->full[s], 3 * ROT_TILE_BYTES);
                    const uint32_t st = smem_base + s * ROT_STAGE_BYTES;
                    const int col = static_cast<int>(k * RK);
                    tma_load_2d(st, &tmap_a, &ctrl->full[s], col, a_row);
                    tma_load_2d(st + 2 * ROT_TILE_BYTES, &tmap_bhi, &ctrl->full[s], col, b_row);
                    tma_load_2d(st + 3 * ROT_TILE_BYTES, &tmap_blo, &ctrl->full[s], col, b_row);
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
            uint32_t it = 0, u = 0;
            bool ok = true;
            for (size_t t = first; t < n_tiles && ok; t += step) {
                for (uint32_t k = 0; k < n_stages && ok; ++k, ++it) {
                    const uint32_t s = it % ROT_STAGES, ph = (it / ROT_STAGES) & 1u;
                    if (!mbar_wait(&ctrl->conv[s], ph, wctx, 33)) {
                        ok = false;
                        break;
                    }
                    const uint32_t st = smem_base + s * ROT_STAGE_BYTES;
#pragma unroll
                    for (uint32_t h = 0; h < RK / BK; ++h) {
                        const uint32_t kb = k * (RK / BK) + h, b = u & 1u;
                        if (kb >= nkb) break;
                        const bool fresh = kb % kb_per_acc == 0;
                        if (fresh && !mbar_wait(&ctrl->acc_empty[b], ((u >> 1) & 1u) ^ 1u, wctx, 32)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t acc = tmem_base + b * RN;
#pragma unroll
                        for (uint32_t kk = h * (BK / 8); kk < (h + 1) * (BK / 8); ++kk) {
                            const uint64_t a_hi = make_desc_128(st + kk * 32), a_lo = make_desc_128(st + ROT_TILE_BYTES + kk * 32);
                            const uint64_t b_hi = make_desc_128(st + 2 * ROT_TILE_BYTES + kk * 32), b_lo = make_desc_128(st + 3 * ROT_TILE_BYTES + kk * 32);
                            umma_tf32_pair(acc, a_hi, b_hi, fresh && kk == h * (BK / 8) ? 0u : 1u, ROT_IDESC);
                            umma_tf32_pair(acc, a_hi, b_lo, 1u, ROT_IDESC);
                            umma_tf32_pair(acc, a_lo, b_hi, 1u, ROT_IDESC);
                        }
                        if ((kb + 1) % kb_per_acc == 0 || kb + 1 == nkb) {
                            umma_commit_pair(&ctrl->acc_full[b]);
                            ++u;
                        }
                    }
                    if (ok) umma_commit_pair(&ctrl->empty[s]);
                }
            }
        }
    } else if (warp < 2 + ROT_SPLIT_WARPS) {
        uint32_t it = 0;
        bool ok = true;
        for (size_t t = first; t < n_tiles && ok; t += step) {
            for (uint32_t k = 0; k < n_stages; ++k, ++it) {
                if (it % ROT_SPLIT_WARPS != static_cast<uint32_t>(warp - 2)) continue;
                const uint32_t s = it % ROT_STAGES, ph = (it / ROT_STAGES) & 1u;
                if (!__all_sync(0xffffffffu, mbar_wait(&ctrl->full[s], ph, wctx, 34))) {
                    ok = false;
                    break;
                }
                float4* a_hi = reinterpret_cast<float4*>(smem + s * ROT_STAGE_BYTES) + lane;
                float4* a_lo = reinterpret_cast<float4*>(smem + s * ROT_STAGE_BYTES + ROT_TILE_BYTES) + lane;
                constexpr int U = 16;
#pragma unroll
                for (int i0 = 0; i0 < static_cast<int>(ROT_TILE_BYTES / 16 / 32); i0 += U) {
                    float4 v[U];
#pragma unroll
                    for (int i = 0; i < U; ++i) v[i] = a_hi[32 * (i0 + i)];
#pragma unroll
                    for (int i = 0; i < U; ++i) {
                        float4 hi, lo;
                        split4(v[i], hi, lo);
                        a_hi[32 * (i0 + i)] = hi;
                        a_lo[32 * (i0 + i)] = lo;
                    }
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(cluster_address(&ctrl->conv[s], 0));
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue
        const uint32_t lane_base = 32u * (warp & 3), half = static_cast<uint32_t>(warp - 2 - ROT_SPLIT_WARPS) >> 2;
        uint32_t u = 0;
        bool ok = true;
        for (size_t t = first; t < n_tiles && ok; t += step) {
            const size_t row = t / n_col_tiles * 256 + rank * 128 + lane_base + lane;
            const size_t col0 = t % n_col_tiles * RN + half * 128;
            float v[128];
            for (uint32_t kb0 = 0; kb0 < nkb; kb0 += kb_per_acc, ++u) {
                const uint32_t b = u & 1u;
                if (!__all_sync(0xffffffffu, mbar_wait(&ctrl->acc_full[b], (u >> 1) & 1u, wctx, 35))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + (lane_base << 16) + b * RN + half * 128;
                const bool fresh = kb0 == 0;
#pragma unroll
                for (int ch = 0; ch < 8; ++ch) {
                    uint32_t r[16];
                    tmem_ld16(taddr + ch * 16, r);
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[ch * 16 + j] = fresh ? __uint_as_float(r[j]) : v[ch * 16 + j] + __uint_as_float(r[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster_read(cluster_address(&ctrl->acc_empty[b], 0));
            }
            if (!ok || row >= p.n) continue;
            float* orow = p.out + row * p.ldo + col0;
            const size_t left = col0 < p.n_out ? p.n_out - col0 : 0;
            if (left >= 128 && p.wide_stores) {
#pragma unroll
                for (int j = 0; j < 128; j += 8) store8(orow + j, v + j);   // whole sectors
            } else {
#pragma unroll
                for (int j = 0; j < 128; ++j)
                    if (static_cast<size_t>(j) < left) orow[j] = v[j];
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync();   // nothing of the pair is in flight towards this CTA any more
    if (warp == 1) tmem_dealloc_pair(tmem_base, TMEM_COLS);
}

} // namespace

void launch_rotate(const float* a, size_t lda, const float* b, float* out, size_t ldo, size_t n, size_t n_out, size_t k_dim, cudaStream_t stream) {
    if (n == 0 || n_out == 0) return;
    int device = 0;
    SKM_CUDA(cudaGetDevice(&device));
    const MemoryBlock split = device_alloc(2 * n_out * k_dim * sizeof(float));
    float* b_split = static_cast<float*>(split.p);
    try {
        launch_presplit(b, n_out, k_dim, b_split, stream);
        RotParams p{};
        p.n = n;
        p.n_out = n_out;
        p.kdim = static_cast<uint32_t>(k_dim);
        p.out = out;
        p.ldo = ldo;
        p.wide_stores = ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 31) == 0;
        p.error = error_word();
        p.wait_limit = wait_limit();
        p.producer_stop = producer_stop();
        SKM_CUDA(cudaFuncSetAttribute(rotate_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ROT_SMEM_BYTES)));
        int sms = 0;
        SKM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
        const size_t tiles = (n + 255) / 256 * ((n_out + RN - 1) / RN);
        const unsigned grid = 2 * static_cast<unsigned>(std::min<size_t>(tiles, static_cast<size_t>(sms / 2)));
        rotate_tc_kernel<<<grid, ROT_THREADS, ROT_SMEM_BYTES, stream>>>(make_row_major_tmap_128(a, k_dim, n, lda, 128), make_row_major_tmap_128(b_split, k_dim, n_out, k_dim, 128),
                                                                        make_row_major_tmap_128(b_split + n_out * k_dim, k_dim, n_out, k_dim, 128), p);
        SKM_LAUNCH_CHECK();
    } catch (...) {
        device_free(split);
        throw;
    }
    device_free(split);   // (its next owner's stream waits for this one)
}

} // namespace tc
} // namespace skmb
