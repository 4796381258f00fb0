// Rotation on the tensor cores as in kernels_tc_rotate.cu, out = A * B^T for row-major fp32 A [n][K] and B [n_out][K], from fp16 halves: for
// rows that a trained model is applied to (AssignTrainingPoints).  The rows of a training itself stay with the tf32 kernel: another last digit in
// every row moves many points, and a training amplifies that (a point that changes its mesocluster shifts the first centroids of every
// point behind it): with these rows the same seed gave centroids that were off by 0.01 to 0.2.  (The dense chain's fp16 halves are another matter: what it finds is
// settled in fp32, so that they show only in a pair at a threshold: of nine trainings eight kept every bit, one was 3e-4 off.)
//
// Both operands are sums of two fp16 numbers, v * scale = hi + lo, to 22 bits of every value down to 2^-17 of the largest that shares its scale; a product is
// hi*hi + hi*lo + lo*hi with fp32 accumulation, at twice the rate of tf32.  B arrives so, with a power of two per row as its scale.  A's
// scale is one per row and 64 columns: that much is a stage, and the thread that has a row of it finds the largest element and writes the
// halves over the row, in place.  The accumulator in tensor memory truncates on every addition, so that a long chain of products ends up
// low (about 1e-8 a term, relative to |a| |b|): a chain here is those 64 columns, whose sum the epilogue multiplies by 1 / scale and adds
// to its fp32 registers while the next ones go into the other accumulator.
// One B200, products counted three times, against the tf32 kernel: 300 000 x 768: 1.75 ms -> 1.05 (608 -> 1007 TF/s),
// 250 000 x 1536: 5.29 -> 3.10, 20 000 x 768: 0.16 -> 0.10, 100 000 x 770 (copied first): 3.23 -> 1.40.  Error against fp64 with an orthonormal B, relative to
// a row's length, rms (largest of 2000 rows): 1.9e-8 (1.2e-7) at K = 32, 1.2e-8 (8e-8) at 132, 0.4e-8 (4e-8) at 1536; the tf32 kernel: 3.4e-8 (2.1e-7), 3.5e-8
// (1.9e-7), 7.0e-8 (3.9e-7); the fp32 tiles: 1.8e-8 (2 - 3e-7) at any width.
//
// Persistent pairs of CTAs (cta_group::2) on tiles of 256 x 256 in turn, four groups of four warps that share the block's registers
// unevenly (setmaxnreg): 64 a thread for the first, 112 for the second (a row of 64 values) and 168 for the others (128 sums):
//   warp 0       TMA producer: A (fp32) and B's halves, 128 rows x 64 columns each per stage and CTA, 128-byte swizzle;
//   warp 1       MMA issuer (the leader's; M = 256, N = 256, K = 16);
//   warps 4-7    split A, a thread per row;
//   warps 8-15   epilogue, a thread per row and 128 columns.
// Rows that TMA cannot address are copied to a scratch with a padded pitch first, a piece at a time that stays in L2.
// Every wait is bounded (see kernels_tc.cu).
#include <algorithm>

#include "common.cuh"
#include "kernels_tc.cuh"
#include "tc_ptx.cuh"

namespace skmb {
namespace tc {

namespace {

constexpr int RN = 256;                  // output columns per tile
constexpr int RK = 64;                   // columns of K per stage
constexpr int ROT_STAGES = 3;
constexpr int ROT_SPLIT_WARPS = 4;
constexpr int ROT_EPI_WARPS = 8;
constexpr int ROT_THREADS = 512;
constexpr uint32_t ROT_FACTORS = 8;      // stages whose factors are kept: the splitters are at most five ahead of the epilogue
constexpr uint32_t ROT_PART_BYTES = 128 * RK * 2;
constexpr uint32_t ROT_STAGE_BYTES = 4 * ROT_PART_BYTES;   // A (32 columns of fp32 each, then hi and lo), B hi, B lo
constexpr uint32_t ROT_CTRL_BYTES = 5120;
constexpr uint32_t ROT_SMEM_BYTES = ROT_STAGES * ROT_STAGE_BYTES + ROT_CTRL_BYTES + 1024;
constexpr int kScaleBits = 14;           // scaled values are below 2^14

struct HalfMaps {
    CUtensorMap a, bhi, blo;
};

struct HalfParams {
    size_t n, n_out;
    uint32_t kdim;
    const float* factor_b;    // per row of B: what its halves are to be multiplied by, times 2^14
    float* out;
    size_t ldo;
    bool wide_stores;         // rows of out start on 32-byte boundaries
    int* error;
    long long wait_limit;
    uint32_t producer_stop;   // see set_debug_wait_injection
};

struct HalfCtrl {
    float factor_a[ROT_FACTORS][128];
    uint64_t full[ROT_STAGES];    // this CTA's copies
    uint64_t conv[ROT_STAGES];    // (the leader's are used) copied and split in both CTAs
    uint64_t empty[ROT_STAGES];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];        // (the leader's are used)
    uint64_t factors[ROT_FACTORS];
    uint32_t tmem_base;
};
static_assert(sizeof(HalfCtrl) <= ROT_CTRL_BYTES, "control block too large");

template <int kRegs>
__device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs)); }
template <int kRegs>
__device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs)); }
static_assert(64 + 112 + 2 * 168 <= 4 * 128, "no more than the block is launched with");

__device__ __forceinline__ void store8(float* p, const float* v) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

// Exponent of the power of two that maps values up to this magnitude into [2^13, 2^14): hi + lo then hold 22 bits of every value down to
// 2^-17 of the largest, and smaller ones to 2^-38 of it.  112 at most, so that 2^-14 over it is a normal number.
__device__ __forceinline__ int scale_bits(float largest) { return min(kScaleBits - (static_cast<int>(__float_as_uint(largest) >> 23) - 126), 112); }
__device__ __forceinline__ float power_of_two(int e) { return __uint_as_float(static_cast<uint32_t>(127 + e) << 23); }

__device__ __forceinline__ float largest_of(float m, const float4& v) { return fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w))); }

// Two values as hi and lo pairs.
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// B's halves and factors, a warp per row (zeros from kdim to the pitch).
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ b, size_t rows, uint32_t kdim, uint32_t pitch, __half* __restrict__ hi, __half* __restrict__ lo,
                                                         float* __restrict__ factor) {
    const size_t row = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    const float* src = b + row * kdim;
    float m = 0.f;
#pragma unroll 8
    for (uint32_t j = lane; j < kdim; j += 32) m = fmaxf(m, fabsf(__ldg(src + j)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int e = scale_bits(m);
    const float scale = power_of_two(e);
    if (lane == 0) factor[row] = power_of_two(kScaleBits - e);
    for (uint32_t j = 2 * lane; j < pitch; j += 64) {
        uint32_t h, l;
        split_pair(j < kdim ? __ldg(src + j) * scale : 0.f, j + 1 < kdim ? __ldg(src + j + 1) * scale : 0.f, h, l);
        *reinterpret_cast<uint32_t*>(hi + row * pitch + j) = h;
        *reinterpret_cast<uint32_t*>(lo + row * pitch + j) = l;
    }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(ROT_THREADS, 1) rotate_halves_kernel(const __grid_constant__ HalfMaps maps, const HalfParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
    uint8_t* smem = smem_raw + pad;
    const uint32_t smem_base = raw_addr + pad;
    HalfCtrl* ctrl = reinterpret_cast<HalfCtrl*>(smem + ROT_STAGES * ROT_STAGE_BYTES);
    const WaitCtx wctx{p.error, p.wait_limit};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();

    if (threadIdx.x == 0) {
        for (int s = 0; s < ROT_STAGES; ++s) {
            mbar_init(&ctrl->full[s], 1);
            mbar_init(&ctrl->conv[s], 2 * ROT_SPLIT_WARPS);
            mbar_init(&ctrl->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctrl->acc_full[b], 1);
            mbar_init(&ctrl->acc_empty[b], 2 * ROT_EPI_WARPS);
        }
        for (uint32_t f = 0; f < ROT_FACTORS; ++f) mbar_init(&ctrl->factors[f], ROT_SPLIT_WARPS);
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
    const size_t first = blockIdx.x >> 1, step = gridDim.x >> 1;

    if (warp < 4) {
        fewer_registers<64>();
        if (warp == 0 && lane == 0) {
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
                    mbar_arrive_expect_tx(&ctrl->full[s], ROT_STAGE_BYTES);
                    const uint32_t st = smem_base + s * ROT_STAGE_BYTES;
                    const int col = static_cast<int>(k * RK);
                    tma_load_2d(st, &maps.a, &ctrl->full[s], col, a_row);
                    tma_load_2d(st + ROT_PART_BYTES, &maps.a, &ctrl->full[s], col + 32, a_row);
                    tma_load_2d(st + 2 * ROT_PART_BYTES, &maps.bhi, &ctrl->full[s], col, b_row);
                    tma_load_2d(st + 3 * ROT_PART_BYTES, &maps.blo, &ctrl->full[s], col, b_row);
                }
            }
            if (!ok) {
                // another role gave up: a millisecond for the copies that are in flight before the block's memory is let go
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000) {
                }
            }
        } else if (warp == 1 && lane == 0 && rank == 0) {
            constexpr uint32_t idesc = make_idesc_f16(256, RN);
            uint32_t it = 0;
            bool ok = true;
            for (size_t t = first; t < n_tiles && ok; t += step) {
                for (uint32_t k = 0; k < n_stages; ++k, ++it) {
                    const uint32_t s = it % ROT_STAGES, ph = (it / ROT_STAGES) & 1u, b = it & 1u;
                    if (!mbar_wait(&ctrl->acc_empty[b], ((it >> 1) & 1u) ^ 1u, wctx, 32) || !mbar_wait(&ctrl->conv[s], ph, wctx, 33)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t acc = tmem_base + b * RN, st = smem_base + s * ROT_STAGE_BYTES;
                    // (nothing but zeros behind kdim)
                    const uint32_t steps = min(static_cast<uint32_t>(RK / 16), (p.kdim - k * RK + 15) / 16);
                    auto part = [&](uint32_t which, uint32_t kk) { return make_desc_128(st + which * ROT_PART_BYTES + kk * 32); };
                    // the small products first: every addition truncates by the accumulator's magnitude
                    for (uint32_t kk = 0; kk < steps; ++kk) {
                        umma_f16_pair(acc, part(0, kk), part(3, kk), kk != 0 ? 1u : 0u, idesc);
                        umma_f16_pair(acc, part(1, kk), part(2, kk), 1u, idesc);
                    }
                    for (uint32_t kk = 0; kk < steps; ++kk) umma_f16_pair(acc, part(0, kk), part(2, kk), 1u, idesc);
                    umma_commit_pair(&ctrl->empty[s]);
                    umma_commit_pair(&ctrl->acc_full[b]);
                }
            }
        }
    } else if (warp < 4 + ROT_SPLIT_WARPS) {
        fewer_registers<112>();
        const uint32_t row = threadIdx.x - 128;
        uint32_t it = 0;
        bool ok = true;
        for (size_t t = first; t < n_tiles && ok; t += step) {
            for (uint32_t k = 0; k < n_stages; ++k, ++it) {
                const uint32_t s = it % ROT_STAGES, ph = (it / ROT_STAGES) & 1u;
                if (!__all_sync(0xffffffffu, mbar_wait(&ctrl->full[s], ph, wctx, 34))) {
                    ok = false;
                    break;
                }
                // 16-byte unit u of row r lies at unit u ^ (r & 7): columns 4 u .. of fp32 (two boxes of 32), or 8 u .. of halves
                uint8_t* at = smem + s * ROT_STAGE_BYTES + row * 128;
                float4 v[16];
#pragma unroll
                for (uint32_t u = 0; u < 16; ++u) v[u] = *reinterpret_cast<const float4*>(at + (u >> 3) * ROT_PART_BYTES + (((u & 7) ^ (row & 7)) << 4));
                float m = 0.f;
#pragma unroll
                for (int u = 0; u < 16; ++u) m = largest_of(m, v[u]);
                const int e = scale_bits(m);
                const float scale = power_of_two(e);
                ctrl->factor_a[it % ROT_FACTORS][row] = power_of_two(-kScaleBits - e);
#pragma unroll
                for (uint32_t u = 0; u < 8; ++u) {
                    uint4 hi, lo;
                    split_pair(v[2 * u].x * scale, v[2 * u].y * scale, hi.x, lo.x);
                    split_pair(v[2 * u].z * scale, v[2 * u].w * scale, hi.y, lo.y);
                    split_pair(v[2 * u + 1].x * scale, v[2 * u + 1].y * scale, hi.z, lo.z);
                    split_pair(v[2 * u + 1].z * scale, v[2 * u + 1].w * scale, hi.w, lo.w);
                    *reinterpret_cast<uint4*>(at + ((u ^ (row & 7)) << 4)) = hi;
                    *reinterpret_cast<uint4*>(at + ROT_PART_BYTES + ((u ^ (row & 7)) << 4)) = lo;
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&ctrl->factors[it % ROT_FACTORS]);
                    mbar_arrive_cluster(cluster_address(&ctrl->conv[s], 0));
                }
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue
        more_registers<168>();
        const uint32_t lane_base = 32u * (warp & 3), half = static_cast<uint32_t>(warp - 8) >> 2;
        uint32_t it = 0;
        bool ok = true;
        for (size_t t = first; t < n_tiles && ok; t += step) {
            const size_t row = t / n_col_tiles * 256 + rank * 128 + lane_base + lane;
            const size_t col0 = t % n_col_tiles * RN + half * 128;
            float v[128];
#pragma unroll
            for (int j = 0; j < 128; ++j) v[j] = 0.f;
            for (uint32_t k = 0; k < n_stages; ++k, ++it) {
                const uint32_t b = it & 1u, f = it % ROT_FACTORS;
                if (!__all_sync(0xffffffffu, mbar_wait(&ctrl->factors[f], (it / ROT_FACTORS) & 1u, wctx, 36) && mbar_wait(&ctrl->acc_full[b], (it >> 1) & 1u, wctx, 35))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const float factor = ctrl->factor_a[f][lane_base + lane];
                const uint32_t taddr = tmem_base + (lane_base << 16) + b * RN + half * 128;
#pragma unroll
                for (int ch = 0; ch < 8; ++ch) {
                    uint32_t r[16];
                    tmem_ld16(taddr + ch * 16, r);
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[ch * 16 + j] = fmaf(__uint_as_float(r[j]), factor, v[ch * 16 + j]);
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
                for (int j = 0; j < 128; j += 8) {
                    const float4 f0 = __ldg(reinterpret_cast<const float4*>(p.factor_b + col0 + j)), f1 = __ldg(reinterpret_cast<const float4*>(p.factor_b + col0 + j + 4));
                    const float w[8] = {v[j] * f0.x, v[j + 1] * f0.y, v[j + 2] * f0.z, v[j + 3] * f0.w, v[j + 4] * f1.x, v[j + 5] * f1.y, v[j + 6] * f1.z, v[j + 7] * f1.w};
                    store8(orow + j, w);   // whole sectors
                }
            } else {
#pragma unroll
                for (int j = 0; j < 128; ++j)
                    if (static_cast<size_t>(j) < left) orow[j] = v[j] * __ldg(p.factor_b + col0 + j);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync();   // nothing of the pair is in flight towards this CTA any more
    if (warp == 1) tmem_dealloc_pair(tmem_base, TMEM_COLS);
}

__global__ void __launch_bounds__(256) pad_rows_kernel(const float* __restrict__ in, size_t lda, size_t n, uint32_t k, uint32_t pitch, float* __restrict__ out) {
    const size_t row = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (row >= n) return;
    for (uint32_t j = threadIdx.x & 31; j < pitch; j += 32) out[row * pitch + j] = j < k ? __ldg(in + row * lda + j) : 0.f;
}

} // namespace

void launch_rotate_halves(const float* a, size_t lda, const float* b, float* out, size_t ldo, size_t n, size_t n_out, size_t k_dim, cudaStream_t stream) {
    if (n == 0 || n_out == 0) return;
    int device = 0, sms = 0;
    SKM_CUDA(cudaGetDevice(&device));
    SKM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const bool addressable = lda % 4 == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
    const size_t pitch = (k_dim + 7) / 8 * 8, halves = n_out * pitch, factors = (n_out + 3) / 4 * 4;
    // B's halves and factors, and the padded rows of a piece (32 MB, in whole tiles)
    const size_t pitch_a = (k_dim + 3) / 4 * 4, piece = addressable ? n : std::min(n, std::max<size_t>(1, (size_t{8} << 20) / pitch_a / 256) * 256);
    const MemoryBlock block = device_alloc(2 * halves * sizeof(__half) + (factors + (addressable ? 0 : piece * pitch_a)) * sizeof(float));
    try {
        __half* b_hi = static_cast<__half*>(block.p);
        __half* b_lo = b_hi + halves;
        float* factor_b = reinterpret_cast<float*>(b_lo + halves);
        float* padded = factor_b + factors;
        split_rows_kernel<<<static_cast<unsigned>((n_out + 7) / 8), 256, 0, stream>>>(b, n_out, static_cast<uint32_t>(k_dim), static_cast<uint32_t>(pitch), b_hi, b_lo, factor_b);
        SKM_LAUNCH_CHECK();
        HalfParams p{};
        p.n_out = n_out;
        p.kdim = static_cast<uint32_t>(k_dim);
        p.factor_b = factor_b;
        p.ldo = ldo;
        p.wide_stores = ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 31) == 0;
        p.error = error_word();
        p.wait_limit = wait_limit();
        p.producer_stop = producer_stop();
        HalfMaps maps;
        maps.bhi = make_half_tmap(b_hi, k_dim, n_out, 128, pitch);
        maps.blo = make_half_tmap(b_lo, k_dim, n_out, 128, pitch);
        SKM_CUDA(cudaFuncSetAttribute(rotate_halves_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ROT_SMEM_BYTES)));
        for (size_t r0 = 0; r0 < n; r0 += piece) {
            p.n = std::min(piece, n - r0);
            p.out = out + r0 * ldo;
            if (addressable) {
                maps.a = make_row_major_tmap_128(a, k_dim, n, lda, 128);
            } else {
                pad_rows_kernel<<<static_cast<unsigned>((p.n + 7) / 8), 256, 0, stream>>>(a + r0 * lda, lda, p.n, static_cast<uint32_t>(k_dim), static_cast<uint32_t>(pitch_a), padded);
                SKM_LAUNCH_CHECK();
                maps.a = make_row_major_tmap_128(padded, k_dim, p.n, pitch_a, 128);
            }
            const size_t tiles = (p.n + 255) / 256 * ((n_out + RN - 1) / RN);
            const unsigned grid = 2 * static_cast<unsigned>(std::min<size_t>(tiles, static_cast<size_t>(sms / 2)));
            rotate_halves_kernel<<<grid, ROT_THREADS, ROT_SMEM_BYTES, stream>>>(maps, p);
            SKM_LAUNCH_CHECK();
        }
    } catch (...) {
        device_free(block);
        throw;
    }
    device_free(block);   // (its next owner's stream waits for this one)
}

} // namespace tc
} // namespace skmb
