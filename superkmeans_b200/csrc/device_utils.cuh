// Small device-side helpers shared by the kernel files.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace skmb {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Monotone map float -> uint32 (preserves <), so that (key << 32 | index) orders by distance then
// by index under an unsigned 64-bit minimum.  A NaN that an operation made (0x7fffffff) comes last.  The last step is hidden from the
// compiler, which would set the sign bit with a floating-point negation, and that leaves a NaN as it is: it then came first.
// (Asking for it instead took 1 us of the 20 of a call of 5000 x 300 x 128.)
__device__ __forceinline__ uint32_t float_to_ordered(float f) {
    const uint32_t b = __float_as_uint(f), flip = static_cast<uint32_t>(static_cast<int32_t>(b) >> 31) | 0x80000000u;
    uint32_t key;
    asm("xor.b32 %0, %1, %2;" : "=r"(key) : "r"(b), "r"(flip));
    return key;
}
__device__ __forceinline__ float ordered_to_float(uint32_t o) {
    const uint32_t b = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
    return __uint_as_float(b);
}
// Ordered by distance, then by index.
__device__ __forceinline__ unsigned long long pair_key(float dist, uint32_t index) {
    return (static_cast<unsigned long long>(float_to_ordered(dist)) << 32) | index;
}
__device__ __forceinline__ void store_answer(unsigned long long key, size_t row, uint32_t* __restrict__ knn, float* __restrict__ dist) {
    knn[row] = static_cast<uint32_t>(key);
    if (dist) dist[row] = fmaxf(0.0f, ordered_to_float(static_cast<uint32_t>(key >> 32)));
}

// One row operation of a split (host_logic.h, SplitOp) for dimension j.
template <class Op>
__device__ __forceinline__ void apply_split_op(float* __restrict__ c, size_t d, size_t j, const Op op) {
    const float up = 1.0f + (1.0f / 1024.0f), down = 1.0f - (1.0f / 1024.0f);
    float* pd = c + static_cast<size_t>(op.dst) * d + j;
    float* ps = c + static_cast<size_t>(op.src) * d + j;
    if (op.kind == 0) {
        const float v = *ps;
        if ((j & 1) == 0) {
            *pd = __fmul_rn(v, up);
            *ps = __fmul_rn(v, down);
        } else {
            *pd = __fmul_rn(v, down);
            *ps = __fmul_rn(v, up);
        }
    } else {
        float val = __fmul_rn(op.wc, *pd);
        val = __fadd_rn(val, *ps);
        *pd = __fdiv_rn(val, __fadd_rn(op.wc, 1.0f));
    }
}

// Unit length, by one warp.
__device__ __forceinline__ void normalize_row(float* __restrict__ p, size_t d, int lane) {
    float s = 0.f;
    for (size_t j = lane; j < d; j += 32) s = fmaf(p[j], p[j], s);
    s = warp_sum(s);
    const float inv = 1.0f / sqrtf(s);
    for (size_t j = lane; j < d; j += 32) p[j] *= inv;
}

// Cumulative squared norm of `row` after each checkpoint of the chain: [0, d'), then each horizontal
// block [vd + 64 b, vd + 64 (b+1)), then [d', vd) when d' < vd.  One warp per row; `out` has n_ck
// entries and is written by lane 0; every lane returns the last of them.
__device__ __forceinline__ float chain_norms_row(const float* __restrict__ row, uint32_t partial_d, uint32_t vertical_d, uint32_t horizontal_d, int lane, float* out,
                                                size_t out_stride = 1) {
    float cum = 0.f;
    uint32_t ck = 0;
    {
        float s = 0.f;
        for (uint32_t j = lane; j < partial_d; j += 32) s = fmaf(__ldg(row + j), __ldg(row + j), s);
        cum += warp_sum(s);
        if (lane == 0) out[ck * out_stride] = cum;
        ++ck;
    }
    for (uint32_t h = 0; h < horizontal_d; h += kHBlock) {
        const float a = __ldg(row + vertical_d + h + lane), b = __ldg(row + vertical_d + h + 32 + lane);
        cum += warp_sum(fmaf(a, a, b * b));
        if (lane == 0) out[ck * out_stride] = cum;
        ++ck;
    }
    if (partial_d < vertical_d) {
        float s = 0.f;
        for (uint32_t j = partial_d + lane; j < vertical_d; j += 32) s = fmaf(__ldg(row + j), __ldg(row + j), s);
        cum += warp_sum(s);
        if (lane == 0) out[ck * out_stride] = cum;
    }
    return cum;
}

} // namespace skmb
