// Second half of the pruned assignment with candidate lists made on the tensor cores.
//
// The first ADSampling test (after d' dimensions) is evaluated for every (point, centroid) pair by the
// tensor cores (kernels_first_test.cu) against the loosest threshold a point can
// have, the exact distance to its previous centroid times ratio[d'].  Pairs that pass are written to
// sixteen lists per tile of 128 points (32 rows x 64 of the columns of every 256-centroid tile), in
// centroid-tile order, with the list position at every 1024-centroid boundary.
//
// walk_lists_kernel then does, for 32 points at a time and chunk after chunk, what the reference's
// search does inside one chunk (pdx/pdxearch.h:118-327, distance_computers/batch_computers.h:297-409):
//   * re-tests every listed pair against the point's CURRENT best (which earlier chunks may have
//     lowered) and counts the survivors per point (the not-pruned counter); the pair with the point's previous
//     centroid is only counted: its exact distance is the starting `best` and cannot undercut it;
//   * advances the surviving pairs by 64 horizontal dimensions (256 contiguous bytes of the PDX block), re-tests and
//     compacts, a lane group of eight per pair; when few are left each is followed to its end with four blocks'
//     loads in flight;
//   * adds the vertical dimensions [d', vertical_d), recomputes in fp32 any final distance that comes within
//     rounding of the tensor-core part of `best`, takes the per-point minimum, lowers `best`.
// `best` is constant inside a chunk, so pairs are independent and any processing order gives the same
// result.
//
// The walk waits on gathers, and its pairs are few: a warp owns its 32 points and their four lists, so that no warp waits
// for another.  (With a block per 128 points, a dozen block-wide barriers per chunk took as many stalls as the loads: ncu
// showed 7 of 19 cycles per instruction at barriers, L2 at 12 %.)
#include <cfloat>

#include "common.cuh"
#include "device_utils.cuh"

namespace skmb {

namespace {

constexpr int kWalkThreads = 64;
constexpr int kWalkWarps = kWalkThreads / 32;
constexpr int kWalkRows = 32;                     // points of a warp: the row group of its lists
constexpr uint32_t kWalkCap = 512;                // pairs a warp holds at a time
constexpr uint32_t kWalkFew = 8;                  // pairs that are followed to their end instead of block by block (at 16: walk 5 - 10 % longer)
constexpr int kWalkLists = kListsPerTile / 4;     // lists of a row group

struct WarpShared {
    uint2 list[kWalkCap];          // {local centroid << 5 | row, partial distance}
    unsigned long long key[kWalkRows];
    float best[kWalkRows];
    float thr[kWalkRows];
    float margin[kWalkRows];       // how close to `best` a final distance must be to be recomputed exactly
    uint32_t prev[kWalkRows];
    uint32_t cnt[kWalkRows];       // survivors of the first test in this chunk
};

__device__ __forceinline__ float sqdiff8(const float4 a0, const float4 a1, const float4 b0, const float4 b1) {
    float s0, s1, t;
    t = a0.x - b0.x; s0 = t * t;
    t = a0.y - b0.y; s1 = t * t;
    t = a0.z - b0.z; s0 = fmaf(t, t, s0);
    t = a0.w - b0.w; s1 = fmaf(t, t, s1);
    t = a1.x - b1.x; s0 = fmaf(t, t, s0);
    t = a1.y - b1.y; s1 = fmaf(t, t, s1);
    t = a1.z - b1.z; s0 = fmaf(t, t, s0);
    t = a1.w - b1.w; s1 = fmaf(t, t, s1);
    return s0 + s1;
}

// Sum over each group of eight lanes.  (The whole warp takes part in every shuffle: with masks of their own the four groups
// would be executed one after the other.)
__device__ __forceinline__ float group_sum(float s) {
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s;
}

// One 64-dimension block for the m pairs of `list`, eight at a time (two per lane group), compacted in place; returns the new
// number.  The control flow is the same for the whole warp.
__device__ __forceinline__ uint32_t walk_block(uint2* list, uint32_t m, const float* __restrict__ blk, const float* __restrict__ xblk, size_t d, const float* best, float ratio,
                                               int lane) {
    constexpr int U = 2;
    const uint32_t g = lane >> 3, below = (1u << lane) - 1u;
    uint32_t j = 0;
    for (uint32_t i = 0; i < m; i += 4 * U) {
        uint2 e[U];
        float4 c0[U], c1[U], x0[U], x1[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            e[u] = list[min(i + 4 * u + g, m - 1)];
            const float* c = blk + static_cast<size_t>(e[u].x >> 5) * kHBlock;
            const float* q = xblk + static_cast<size_t>(e[u].x & 31u) * d;
            c0[u] = __ldg(reinterpret_cast<const float4*>(c));
            c1[u] = __ldg(reinterpret_cast<const float4*>(c + 4));
            x0[u] = __ldg(reinterpret_cast<const float4*>(q));
            x1[u] = __ldg(reinterpret_cast<const float4*>(q + 4));
        }
        float pd[U];
#pragma unroll
        for (int u = 0; u < U; ++u) pd[u] = __uint_as_float(e[u].y) + group_sum(sqdiff8(x0[u], x1[u], c0[u], c1[u]));
        __syncwarp();   // these eight have been read
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool keep = (lane & 7) == 0 && i + 4 * u + g < m && pd[u] < best[e[u].x & 31u] * ratio;
            const uint32_t kept = __ballot_sync(0xffffffffu, keep);
            if (keep) list[j + __popc(kept & below)] = make_uint2(e[u].x, __float_as_uint(pd[u]));
            j += __popc(kept);
        }
    }
    __syncwarp();
    return j;
}

// The horizontal blocks [hb, n_h) of a pair per lane group, four blocks' loads in flight at a time; sums and tests as in
// walk_block.  Returns whether the group's pair is still alive.
__device__ __forceinline__ bool walk_rest(bool alive, const float* __restrict__ cblk, size_t cstride, const float* __restrict__ xblk, uint32_t hb, uint32_t n_h, float best,
                                          const float* __restrict__ ratios, int gl, float& pd, unsigned long long& steps) {
    constexpr int A = 4;
    for (; hb < n_h && __any_sync(0xffffffffu, alive); hb += A) {
        float s[A];
#pragma unroll
        for (int a = 0; a < A; ++a) {
            s[a] = 0.f;
            if (alive) {
                const uint32_t b = min(hb + a, n_h - 1);
                const float4* c = reinterpret_cast<const float4*>(cblk + b * cstride);
                const float4* x = reinterpret_cast<const float4*>(xblk + b * kHBlock);
                s[a] = sqdiff8(__ldg(x), __ldg(x + 1), __ldg(c), __ldg(c + 1));
            }
        }
#pragma unroll
        for (int a = 0; a < A; ++a) s[a] = group_sum(s[a]);
#pragma unroll
        for (int a = 0; a < A; ++a) {
            if (alive && hb + a < n_h) {
                pd += s[a];
                steps += gl == 0 ? 1u : 0u;
                alive = pd < best * __ldg(ratios + (hb + a + 1) * kHBlock);
            }
        }
    }
    return alive;
}

// Blocks of two warps, so that the few row groups of a small problem still reach every SM, and twelve of them to an SM: the
// registers of four more are worth more as loads in flight.  One B200, nine passes of a Train each, against a block of 128
// points before: 1M x 1024, k = 4000: 12.0 ms (21.0 before; 12.2 with sixteen blocks to an SM); 100k x 1536, k = 2000: 4.2 (6.1);
// 30 000 x 768, k = 1000: 0.63 (0.59; 0.78 with sixteen).  (With the share of the points that went to the dense chain then; the first
// test now drops fewer of them, see kHardShare, and the first of the three takes 18.2 ms here.)
constexpr int kWalkCtasPerSm = 12;

__global__ void __launch_bounds__(kWalkThreads, kWalkCtasPerSm) walk_lists_kernel(const WalkParams w, const uint32_t share) {
    __shared__ WarpShared all[kWalkWarps];
    if (w.upstream_error && *reinterpret_cast<const volatile int*>(w.upstream_error) != 0) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    WarpShared& sh = all[warp];
    const int g = lane >> 3, gl = lane & 7;
    const uint32_t below = (1u << lane) - 1u;
    const size_t n_chunks = (w.k + kChunk - 1) / kChunk;
    const uint32_t n_h = w.horizontal_d / kHBlock;
    const uint32_t vlen = w.vertical_d - w.partial_d;
    const float ratio_first = __ldg(w.ratios + w.partial_d);
    unsigned long long steps_done = 0;

    for (size_t unit = static_cast<size_t>(blockIdx.x) * kWalkWarps + warp; unit < w.n_tiles * 4 * share; unit += static_cast<size_t>(gridDim.x) * kWalkWarps) {
        const size_t group = unit / share, tile = group >> 2;
        const uint32_t quarter = static_cast<uint32_t>(group & 3);
        const size_t row0 = (w.tile_map ? static_cast<size_t>(w.tile_map[tile]) : w.tile0 + tile) * kTileM + quarter * kWalkRows;
        const size_t row = row0 + lane;
        // lane c < kWalkLists looks after list c of the row group
        const size_t list_id = tile * kListsPerTile + static_cast<size_t>(lane & (kWalkLists - 1)) * 4 + quarter;
        const uint32_t* offs = w.list_offs + list_id * (n_chunks + 1);
        const bool overflow = __any_sync(0xffffffffu, __ldg(offs + n_chunks) > w.cap_group);
        bool active = row < w.n && !(w.skip && w.skip[row]) && lane * share / kWalkRows == unit % share;
        if (active && overflow) {
            // a list did not fit: its points go to the dense kernel
            w.redo[row] = 1u;
            atomicAdd(w.redo_count, 1u);
            active = false;
        }
        if (!__any_sync(0xffffffffu, active)) continue;
        float best = active ? w.best_in[row] : -FLT_MAX;
        uint32_t bestidx = active ? w.knn[row] : 0u;
        uint32_t npc = 0;
        __syncwarp();
        sh.best[lane] = best;
        sh.prev[lane] = active ? bestidx : 0xFFFFFFFFu;
        sh.margin[lane] = 1e-5f * (active ? w.norms_x[row] : 0.f);   // the tensor-core part of a distance is within ~3e-6 of the norms over d'
        const float* __restrict__ xrows = w.x + row0 * w.d;

        uint32_t begin = __ldg(offs);
        for (size_t chunk = 0; chunk < n_chunks; ++chunk) {
            const size_t c0 = chunk * kChunk;
            const size_t cs = min(static_cast<size_t>(kChunk), w.k - c0);
            const uint32_t end = __ldg(offs + chunk + 1);
            const float* __restrict__ blk_chunk = w.y_pdx + chunk * kChunk * w.d + static_cast<size_t>(w.vertical_d) * cs + gl * 8;
            sh.thr[lane] = best * ratio_first;
            sh.cnt[lane] = 0;
            sh.key[lane] = ~0ull;
            __syncwarp();

            uint32_t m = 0;   // pairs held, warp-uniform
            auto walk = [&]() {
                __syncwarp();
                uint32_t hb = 0;
                while (hb < n_h && m > kWalkFew) {
                    steps_done += lane == 0 ? m : 0u;
                    m = walk_block(sh.list, m, blk_chunk + hb * cs * kHBlock, xrows + w.vertical_d + hb * kHBlock + gl * 8, w.d, sh.best, __ldg(w.ratios + w.partial_d + (hb + 1) * kHBlock),
                                   lane);
                    ++hb;
                }
                for (uint32_t i = 0; i < m; i += 4) {
                    const uint2 ent = sh.list[min(i + g, m - 1)];
                    const uint32_t r = ent.x & 31u, cl = ent.x >> 5;
                    const size_t c = c0 + cl;
                    const float row_best = sh.best[r];
                    float pd = __uint_as_float(ent.y);
                    const float* __restrict__ xr = xrows + static_cast<size_t>(r) * w.d;
                    const bool alive = walk_rest(i + g < m, blk_chunk + static_cast<size_t>(cl) * kHBlock, cs * kHBlock, xr + w.vertical_d + gl * 8, hb, n_h, row_best,
                                                 w.ratios + w.partial_d, gl, pd, steps_done);
                    if (!__any_sync(0xffffffffu, alive)) continue;
                    // ---- vertical dimensions [d', vertical_d)
                    float s = 0.f;
                    if (vlen != 0 && alive) {
                        const float* __restrict__ cp = w.y_aux + c * w.vertical_d + w.partial_d;
                        const float* __restrict__ qp = xr + w.partial_d;
                        // scalar head up to a 16-byte boundary (both rows start at a multiple of four floats, so
                        // they share it), float4 body, scalar rest
                        const uint32_t head = min(vlen, (4u - (w.partial_d & 3u)) & 3u);
                        const uint32_t n4 = (vlen - head) >> 2;
                        const uint32_t rest0 = head + (n4 << 2);
                        if (static_cast<uint32_t>(gl) < head) {
                            const float t = __ldg(qp + gl) - __ldg(cp + gl);
                            s = t * t;
                        }
                        if (rest0 + gl < vlen) {
                            const float t = __ldg(qp + rest0 + gl) - __ldg(cp + rest0 + gl);
                            s = fmaf(t, t, s);
                        }
                        const float4* q4 = reinterpret_cast<const float4*>(qp + head);
                        const float4* c4 = reinterpret_cast<const float4*>(cp + head);
#pragma unroll 4
                        for (uint32_t jj = gl; jj < n4; jj += 8) {
                            const float4 a = __ldg(q4 + jj), b = __ldg(c4 + jj);
                            float t;
                            t = a.x - b.x; s = fmaf(t, t, s);
                            t = a.y - b.y; s = fmaf(t, t, s);
                            t = a.z - b.z; s = fmaf(t, t, s);
                            t = a.w - b.w; s = fmaf(t, t, s);
                        }
                    }
                    pd += group_sum(s);
                    // The first d' dimensions of pd come from the tensor cores (a few 1e-6 of the norms off).  A pair that
                    // would win, or lose, by less than that is settled with the distance recomputed from direct differences
                    // in fp32.
                    const bool close = alive && pd < row_best + sh.margin[r];
                    if (!__any_sync(0xffffffffu, close)) continue;
                    float s0 = 0.f, s1 = 0.f;
                    if (close) {
                        const float4* q4 = reinterpret_cast<const float4*>(xr);
                        const float4* c4 = reinterpret_cast<const float4*>(w.y + c * w.d);
#pragma unroll 4
                        for (uint32_t jj = gl; jj < w.d / 4; jj += 8) {
                            const float4 a = __ldg(q4 + jj), b = __ldg(c4 + jj);
                            float t;
                            t = a.x - b.x; s0 = fmaf(t, t, s0);
                            t = a.y - b.y; s1 = fmaf(t, t, s1);
                            t = a.z - b.z; s0 = fmaf(t, t, s0);
                            t = a.w - b.w; s1 = fmaf(t, t, s1);
                        }
                    }
                    const float exact = group_sum(s0 + s1);
                    if (close && gl == 0 && exact < row_best)
                        atomicMin(&sh.key[r], (static_cast<unsigned long long>(float_to_ordered(exact)) << 32) | static_cast<unsigned long long>(c));
                }
                __syncwarp();
                m = 0;
            };

            // the chunk's pairs, 32 of each of the four lists at a time
            const uint32_t mine = end - begin;
            uint32_t longest = mine;
#pragma unroll
            for (int o = 1; o < kWalkLists; o <<= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
            for (uint32_t i0 = 0; i0 < longest; i0 += 32) {
                uint2 raw[kWalkLists];
#pragma unroll
                for (int c = 0; c < kWalkLists; ++c) {
                    const uint32_t b = __shfl_sync(0xffffffffu, begin, c), l = __shfl_sync(0xffffffffu, mine, c);
                    const size_t base = (tile * kListsPerTile + static_cast<size_t>(c) * 4 + quarter) * w.cap_group;
                    raw[c] = i0 + lane < l ? __ldg(w.lists + base + b + i0 + lane) : make_uint2(0u, 0x7F800000u);   // (infinity: no pair)
                }
#pragma unroll
                for (int c = 0; c < kWalkLists; ++c) {
                    const uint32_t r = raw[c].x & 31u, col = raw[c].x >> 5;
                    const bool pass = __uint_as_float(raw[c].y) < sh.thr[r];
                    if (pass) atomicAdd(&sh.cnt[r], 1u);
                    const bool keep = pass && col != sh.prev[r];
                    const uint32_t kept = __ballot_sync(0xffffffffu, keep);
                    if (keep) sh.list[m + __popc(kept & below)] = make_uint2(((col - static_cast<uint32_t>(c0)) << 5) | r, raw[c].y);
                    m += __popc(kept);
                }
                if (m > kWalkCap - 32 * kWalkLists) walk();
            }
            if (m != 0) walk();
            __syncwarp();
            begin = end;
            npc += sh.cnt[lane];
            const unsigned long long key = sh.key[lane];
            if (key != ~0ull) {
                best = ordered_to_float(static_cast<uint32_t>(key >> 32));
                bestidx = static_cast<uint32_t>(key & 0xFFFFFFFFull);
                sh.best[lane] = best;
            }
            __syncwarp();
        }
        if (active) {
            w.knn[row] = bestidx;
            w.dist[row] = best;
            w.not_pruned[row] = npc;
        }
    }
    if (gl == 0 && steps_done) atomicAdd(w.pair_steps, steps_done);
}

} // namespace

void launch_walk_lists(const WalkParams& w, int device, cudaStream_t stream) {
    if (w.n_tiles == 0) return;
    int sms = 0;
    SKM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    // Few points: their lists are shared by two or four warps (each reads them all and walks the pairs of its own points), while that
    // makes no more than two warps for every place there is: a warp's pairs are a chain of gathers.  30 000 x 768, k = 1000, nine passes: 98
    // us a pass with one warp, 81 with two, 77 with four, 94 with eight; 250 000 points: no difference up to four.
    const size_t places = static_cast<size_t>(sms) * kWalkCtasPerSm * kWalkWarps;
    uint32_t share = 1;
    while (share < 4 && w.n_tiles * 4 * share * 2 <= 2 * places) share *= 2;
    const unsigned grid = static_cast<unsigned>(std::min<size_t>((w.n_tiles * 4 * share + kWalkWarps - 1) / kWalkWarps, static_cast<size_t>(sms) * kWalkCtasPerSm));
    walk_lists_kernel<<<grid, kWalkThreads, 0, stream>>>(w, share);
    SKM_LAUNCH_CHECK();
}

} // namespace skmb
