// lbvh.cu -- linear BVH builder (BLAS over triangles, TLAS over instance boxes).
//
// Replaces the driver-side builds of BottomLevelAS / TopLevelAS
// (render/acceleration_structure.cpp:55-194), which the reference leaves opaque:
//   1. primitive boxes (triangles: min/max of the three vertices)
//   2. centroid bounds (order-preserving uint atomics: exact, order independent)
//   3. 30-bit Morton codes of the centroids, normalised to the cube of the largest centroid extent
//   4. stable LSD radix sort of (code, primitive) in four 8-bit passes, one onesweep kernel each
//   5. Karras 2012 hierarchy (n-1 internal nodes; equal codes split on the index) and its boxes, bottom
//      up: one thread per leaf climbs; the second arrival at a split goes on with the node
// Refit keeps the topology and recomputes the boxes in a climb of its own.
#include <cooperative_groups.h>

#include <atomic>
#include <cstdlib>

#include "rg_internal.cuh"

namespace rg {

namespace {

namespace cg = cooperative_groups;

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortRounds = 8;
static_assert(kSortWarps * kSortRounds * 32 == kSortTileKeys, "one onesweep tile per block");
constexpr uint32_t kNoBox = 0xFFFFFFFFu;        // a box word not yet written (no union of boxes is this NaN)
constexpr uint32_t kMortonMaxBlocks = 608;  // grid-stride: bounds the global histogram atomics

__global__ void k_tri_boxes(const rg_vertex* __restrict__ v, const uint32_t* __restrict__ idx, uint32_t vOff, uint32_t iOff,
                            uint32_t n, float* __restrict__ boxes) {
    chain_wait();
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    float lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
        const float* pos = v[vOff + idx[iOff + 3 * p + k]].position;
        for (int a = 0; a < 3; ++a) {
            float x = pos[a];
            lo[a] = k == 0 ? x : fminf(lo[a], x);
            hi[a] = k == 0 ? x : fmaxf(hi[a], x);
        }
    }
    float* o = boxes + 6 * (size_t)p;
    o[0] = lo[0]; o[1] = lo[1]; o[2] = lo[2]; o[3] = hi[0]; o[4] = hi[1]; o[5] = hi[2];
}

// triangle records in leaf order: v0 (w = primitive id), v1, v2
__global__ void k_tri_records(const rg_vertex* __restrict__ v, const uint32_t* __restrict__ idx, uint32_t vOff, uint32_t iOff,
                              const uint32_t* __restrict__ order, uint32_t n, float4* __restrict__ tris) {
    chain_wait();
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    uint32_t p = order[k];
    const float* a = v[vOff + idx[iOff + 3 * p + 0]].position;
    const float* b = v[vOff + idx[iOff + 3 * p + 1]].position;
    const float* c = v[vOff + idx[iOff + 3 * p + 2]].position;
    tris[3 * (size_t)k + 0] = make_float4(a[0], a[1], a[2], __uint_as_float(p));
    tris[3 * (size_t)k + 1] = make_float4(b[0], b[1], b[2], 0.0f);
    tris[3 * (size_t)k + 2] = make_float4(c[0], c[1], c[2], 0.0f);
}

__device__ inline void centroid(const float* b, float* c) {
    if (!(b[0] <= b[3])) {  // empty box (invalid instance): keyed at the origin
        c[0] = c[1] = c[2] = 0.0f;
        return;
    }
    for (int a = 0; a < 3; ++a) c[a] = __fmul_rn(__fadd_rn(b[a], b[3 + a]), 0.5f);
}

// the centroid bounds as words that start at zero: ~f2ord of the minima, f2ord of the maxima
__global__ void __launch_bounds__(256) k_centroid_bounds(const float* __restrict__ boxes, uint32_t n, uint32_t* bounds) {
    chain_wait();
    __shared__ float red[6][8];
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        float c[3];
        centroid(boxes + 6 * (size_t)p, c);
        for (int a = 0; a < 3; ++a) {
            mn[a] = fminf(mn[a], c[a]);
            mx[a] = fmaxf(mx[a], c[a]);
        }
    }
    for (int off = 16; off > 0; off >>= 1)
        for (int a = 0; a < 3; ++a) {
            mn[a] = fminf(mn[a], __shfl_xor_sync(0xFFFFFFFFu, mn[a], off));
            mx[a] = fmaxf(mx[a], __shfl_xor_sync(0xFFFFFFFFu, mx[a], off));
        }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int a = 0; a < 3; ++a) {
            red[a][w] = mn[a];
            red[3 + a][w] = mx[a];
        }
    __syncthreads();
    // one atomic per block and bound (same-address atomics from every warp serialise in L2)
    if (threadIdx.x < 3) {
        const int a = threadIdx.x;
        float lo = red[a][0], hi = red[3 + a][0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
            lo = fminf(lo, red[a][k]);
            hi = fmaxf(hi, red[3 + a][k]);
        }
        if (lo <= hi) {  // the block saw a centroid
            atomicMax(&bounds[a], ~f2ord(lo));
            atomicMax(&bounds[3 + a], f2ord(hi));
        }
    }
}

// codes, the sort's input (keys, and values = primitive ids in every buffer that a pass writes values
// to, so that each word is a valid primitive id whatever a pass writes), cleared arrival words of the
// hierarchy, and the four digit histograms of the sort (grid-stride; one shared-memory histogram per
// block, flushed with global atomics)
__global__ void __launch_bounds__(256) k_morton(const float* __restrict__ boxes, uint32_t n, const uint32_t* __restrict__ bounds,
                                                uint32_t* morton, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                uint32_t* __restrict__ valsAlt, uint32_t* order, uint32_t* __restrict__ arrivals,
                                                uint32_t* __restrict__ nodeBoxes, uint32_t* __restrict__ hist) {
    chain_wait();
    __shared__ uint32_t h[4 * 256];
    for (int i = threadIdx.x; i < 4 * 256; i += 256) h[i] = 0;
    // every axis is scaled by the LARGEST centroid extent (a cube), so a thin axis spends few of its
    // 10 bits and the hierarchy splits mostly along the long axes
    float lo[3], inv[3];
    float emax = 0.0f;
    for (int a = 0; a < 3; ++a) {
        lo[a] = ord2f(~bounds[a]);
        emax = fmaxf(emax, __fsub_rn(ord2f(bounds[3 + a]), lo[a]));
    }
    for (int a = 0; a < 3; ++a) inv[a] = emax > 0.0f ? __fdiv_rn(1.0f, emax) : 0.0f;
    __syncthreads();
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        float c[3];
        centroid(boxes + 6 * (size_t)p, c);
        uint32_t x = quant10(c[0], lo[0], inv[0]), y = quant10(c[1], lo[1], inv[1]), z = quant10(c[2], lo[2], inv[2]);
        uint32_t m = (expand10(x) << 2) | (expand10(y) << 1) | expand10(z);
        morton[p] = m;
        keys[p] = m;
        vals[p] = p;
        valsAlt[p] = p;
        order[p] = p;
        if (p + 1 < n) {
            arrivals[p] = 0u;
            for (int a = 0; a < 6; ++a) nodeBoxes[6 * (size_t)p + a] = kNoBox;
        }
#pragma unroll
        for (int d = 0; d < 4; ++d) atomicAdd(&h[256 * d + ((m >> (8 * d)) & 0xFFu)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * 256; i += 256)
        if (h[i]) atomicAdd(&hist[i], h[i]);
}

// ---- onesweep LSD radix sort (Adinets & Merrill 2022) --------------------------------------------
// k_morton counts the four 8-bit digit histograms of the codes as it writes them.  Each of the four
// passes is then ONE kernel: a block takes the next tile in launch order (an atomic counter, so every
// earlier tile belongs to a block that is already running), ranks its kSortTileKeys keys by digit
// (stable: warp chunks in key order, lanes in key order), publishes its per-digit counts, and finds
// how many keys of each digit precede it by decoupled look-back over the earlier tiles' published
// words, then scatters.  A status word is flag (bits 31:30) | count (bits 29:0): 0 = not yet
// published, kStatAgg = this tile's own count, kStatIncl = count over this and all earlier tiles.
// A look-back that finds a predecessor unpublished polls it a bounded number of times and then
// counts that tile's keys of the digit directly from the input, so no wait is unbounded and the
// result does not depend on the bound.
constexpr uint32_t kStatAgg = 1u << 30;
constexpr uint32_t kStatIncl = 2u << 30;
constexpr uint32_t kStatCount = (1u << 30) - 1u;

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// lanes of the warp with the same 8-bit digit: eight ballots (__match_any_sync takes 250 cycles of
// the SM's quarter, five times as long)
__device__ __forceinline__ uint32_t digit_peers(bool ok, uint32_t digit) {
    uint32_t peers = __ballot_sync(0xFFFFFFFFu, ok);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool one = (digit >> b) & 1u;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, one);
        peers &= one ? m : ~m;
    }
    return peers;
}

// exclusive prefix sum over the block's 256 threads (one value each); `warpSums` holds 8 words
__device__ __forceinline__ uint32_t block_exclusive_256(uint32_t v, uint32_t* warpSums) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) warpSums[w] = x;
    __syncthreads();
    uint32_t before = 0;
    for (int k = 0; k < w; ++k) before += warpSums[k];
    return before + x - v;
}

__global__ void __launch_bounds__(kSortThreads) k_sort_onesweep(const uint32_t* __restrict__ keysIn, const uint32_t* __restrict__ valsIn,
                                                                 uint32_t* __restrict__ keysOut, uint32_t* __restrict__ valsOut,
                                                                 uint32_t n, int pass, uint32_t* __restrict__ state, uint32_t nTiles,
                                                                 uint32_t spinLimit) {
    chain_wait();
    __shared__ uint32_t wc[kSortWarps][256];
    __shared__ uint32_t digitBase[256];
    __shared__ uint32_t warpSums[kSortWarps];
    __shared__ uint32_t tileShared;
    const int shift = 8 * pass;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) tileShared = atomicAdd(state + kSortTileCounters + pass, 1u);
    for (int i = threadIdx.x; i < kSortWarps * 256; i += kSortThreads) (&wc[0][0])[i] = 0;
    __syncthreads();
    const uint32_t tile = tileShared;
    const uint32_t ltmask = (1u << lane) - 1u;
    const uint32_t base = tile * kSortTileKeys + w * (kSortRounds * 32);
    uint32_t key[kSortRounds], val[kSortRounds], pos[kSortRounds];
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        uint32_t i = base + r * 32 + lane;
        bool ok = i < n;
        key[r] = ok ? keysIn[i] : 0u;
        val[r] = ok ? valsIn[i] : 0u;
        uint32_t digit = (key[r] >> shift) & 0xFFu;
        uint32_t peers = digit_peers(ok, digit);
        uint32_t before = wc[w][digit];
        __syncwarp();
        pos[r] = before + __popc(peers & ltmask);
        if (ok && (peers & ltmask) == 0) wc[w][digit] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // thread d: this tile's count of digit d, and each warp's exclusive offset within the tile
    const uint32_t d = threadIdx.x;
    uint32_t cnt = 0;
    for (int ww = 0; ww < kSortWarps; ++ww) {
        uint32_t t = wc[ww][d];
        wc[ww][d] = cnt;
        cnt += t;
    }
    uint32_t* status = state + kSortStatusOffset + (size_t)pass * nTiles * 256;
    st_relaxed(status + (size_t)tile * 256 + d, (tile == 0 ? kStatIncl : kStatAgg) | cnt);
    // keys of smaller digits in the whole input (this pass's histogram)
    const uint32_t globalBefore = block_exclusive_256(state[256 * pass + d], warpSums);
    // keys of digit d in earlier tiles
    uint32_t earlier = 0;
    for (int64_t t = (int64_t)tile - 1; t >= 0; --t) {
        const uint32_t* sp = status + (size_t)t * 256 + d;
        uint32_t v = ld_relaxed(sp);
        for (uint32_t spins = 0; (v >> 30) == 0 && spins < spinLimit; ++spins) {
            __nanosleep(100);
            v = ld_relaxed(sp);
        }
        if ((v >> 30) == 0) {  // still unpublished: count tile t's keys of digit d from the input
            uint32_t c = 0;
            const uint32_t b0 = (uint32_t)t * kSortTileKeys, b1 = min(n, b0 + kSortTileKeys);
            for (uint32_t i = b0; i < b1; ++i) c += ((keysIn[i] >> shift) & 0xFFu) == d;
            v = kStatAgg | c;
        }
        earlier += v & kStatCount;
        if ((v >> 30) == 2) break;
    }
    if (tile > 0) st_relaxed(status + (size_t)tile * 256 + d, kStatIncl | (earlier + cnt));
    digitBase[d] = globalBefore + earlier;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        uint32_t i = base + r * 32 + lane;
        if (i < n) {
            uint32_t dg = (key[r] >> shift) & 0xFFu;
            uint32_t dst = digitBase[dg] + wc[w][dg] + pos[r];
            if (dst < n) {  // always true: the counts are exact
                keysOut[dst] = key[r];
                valsOut[dst] = val[r];
            }
        }
    }
}

// ---- codes and sort of up to 65536 primitives in one launch ----------------------------------------
// As separate launches (bounds, codes, four onesweep passes) a build of this size is a chain of launches
// and of waits on words in L2, 8 us a pass for 0.1 us of traffic.  One thread-block cluster holds all of it
// in shared memory: every thread keeps ROUNDS keys in registers, the blocks exchange their centroid
// bounds and digit counts through distributed shared memory and scatter the (code, primitive) pairs
// straight into each other's (sorted by digit first: 1900 clocks a pass
// against 5500 in key order).  Stable: blocks, warps and rounds in key order, lanes in key order.  Two
// cluster barriers a pass.  As many blocks of 1024 threads as there are keys for, up to 16 (beyond
// the portable 8, which hold 32768 keys), so that a thread ranks few keys one after another.
// 50000 keys: 31 us, against 45 us in eight launches with their gaps.  (Ranking, 5000 clocks a pass, and
// the scatter, 1900, are what is left; lane masks by shared-memory atomics in place of the ballots:
// 2 % less for 32 KB more.)
constexpr int kClusterThreads = 1024;
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kClusterRounds = 4;  // keys a thread at most
struct ClusterSort {
    unsigned long long pair[kClusterThreads * kClusterRounds];    // code << 32 | primitive, from all blocks
    unsigned long long sorted[kClusterThreads * kClusterRounds];  // the block's pairs by digit
    uint32_t wc[kClusterWarps][256];  // counts by warp and digit, then offsets within a quarter of the warps
    uint32_t part[4][256];            // counts by quarter, then where a quarter's keys of a digit start in `sorted`
    uint32_t cnt[256];                // the block's counts: read by the other blocks
    uint32_t all[4][256], before[4][256];  // keys of a digit in all blocks, in earlier blocks (by quarter of the blocks)
    uint32_t shift[256];              // from a key's place in `sorted` to its place in the input's order
    uint32_t warpSums[2][8];
    float red[kClusterWarps][6];
    float bounds[6], total[6];        // centroid bounds: the block's (read by the others), the input's
};

template <int ROUNDS>
__global__ void __launch_bounds__(kClusterThreads) k_sort_cluster(const float* __restrict__ boxes, uint32_t n, uint32_t* morton,
                                                                  uint32_t* __restrict__ keysOut, uint32_t* order,
                                                                  uint32_t* __restrict__ arrivals, uint32_t* __restrict__ nodeBoxes) {
    chain_wait();
    extern __shared__ __align__(16) unsigned char smemRaw[];
    ClusterSort& S = *reinterpret_cast<ClusterSort*>(smemRaw);
    const cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), size = cluster.num_blocks();
    constexpr uint32_t kBlockKeys = kClusterThreads * ROUNDS;
    const uint32_t tid = threadIdx.x, w = tid >> 5, lane = tid & 31, ltmask = (1u << lane) - 1u;
    const uint32_t base = rank * kBlockKeys + w * (ROUNDS * 32) + lane;  // the thread's keys: base + 32 r
    uint32_t key[ROUNDS] = {}, val[ROUNDS] = {}, pos[ROUNDS];
    {
        float c[ROUNDS][3];
        float v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            const uint32_t p = base + 32 * r;
            if (p >= n) continue;
            centroid(boxes + 6 * (size_t)p, c[r]);
            for (int a = 0; a < 3; ++a) {
                v[a] = fminf(v[a], c[r][a]);
                v[3 + a] = fmaxf(v[3 + a], c[r][a]);
            }
        }
        auto reduce = [&]() {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    v[a] = fminf(v[a], __shfl_xor_sync(0xFFFFFFFFu, v[a], off));
                    v[3 + a] = fmaxf(v[3 + a], __shfl_xor_sync(0xFFFFFFFFu, v[3 + a], off));
                }
        };
        reduce();
        if (lane == 0)
            for (int a = 0; a < 6; ++a) S.red[w][a] = v[a];
        __syncthreads();
        if (w == 0) {
            for (int a = 0; a < 6; ++a) v[a] = S.red[lane][a];
            reduce();
            if (lane == 0)
                for (int a = 0; a < 6; ++a) S.bounds[a] = v[a];
        }
        // meanwhile: the hierarchy's words
        for (uint32_t i = rank * kClusterThreads + tid; i + 1 < n; i += size * kClusterThreads) arrivals[i] = 0u;
        for (uint32_t i = rank * kClusterThreads + tid; i < 6 * (n - 1); i += size * kClusterThreads) nodeBoxes[i] = kNoBox;
        cluster.sync();
        if (w == 0) {
            for (int a = 0; a < 6; ++a) v[a] = lane < size ? cluster.map_shared_rank(S.bounds, lane)[a] : a < 3 ? INFINITY : -INFINITY;
            reduce();
            if (lane == 0)
                for (int a = 0; a < 6; ++a) S.total[a] = v[a];
        }
        __syncthreads();
        // every axis is scaled by the largest centroid extent, as in k_morton; an axis without a
        // centroid (all NaN) has NaN bounds
        float lo[3], inv, emax = 0.0f;
        for (int a = 0; a < 3; ++a) {
            const bool any = S.total[a] <= S.total[3 + a];
            lo[a] = any ? S.total[a] : ord2f(0xFFFFFFFFu);
            emax = fmaxf(emax, __fsub_rn(any ? S.total[3 + a] : ord2f(0u), lo[a]));
        }
        inv = emax > 0.0f ? __fdiv_rn(1.0f, emax) : 0.0f;
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            const uint32_t p = base + 32 * r;
            if (p >= n) continue;
            const uint32_t x = quant10(c[r][0], lo[0], inv), y = quant10(c[r][1], lo[1], inv), z = quant10(c[r][2], lo[2], inv);
            key[r] = (expand10(x) << 2) | (expand10(y) << 1) | expand10(z);
            val[r] = p;
            morton[p] = key[r];
        }
    }
    const uint32_t held = min(kBlockKeys, n - min(n, rank * kBlockKeys));  // the block's keys
#pragma unroll 1
    for (int pass = 0; pass < 4; ++pass) {
        const int bits = 8 * pass;
        if (pass) {
#pragma unroll
            for (int r = 0; r < ROUNDS; ++r) {
                const unsigned long long kv = S.pair[w * (ROUNDS * 32) + 32 * r + lane];
                key[r] = (uint32_t)(kv >> 32);
                val[r] = (uint32_t)kv;
            }
        }
#pragma unroll
        for (int i = 0; i < kClusterWarps * 256 / kClusterThreads; ++i) (&S.wc[0][0])[tid + kClusterThreads * i] = 0;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            const bool ok = base + 32 * r < n;
            const uint32_t digit = (key[r] >> bits) & 0xFFu;
            const uint32_t peers = digit_peers(ok, digit);
            const uint32_t ahead = S.wc[w][digit];
            __syncwarp();
            pos[r] = ahead + __popc(peers & ltmask);
            if (ok && (peers & ltmask) == 0) S.wc[w][digit] = ahead + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        const uint32_t q = tid >> 8, d = tid & 255u;  // a quarter of the warps, then of the blocks; a digit
        {
            uint32_t c[kClusterWarps / 4], run = 0;
#pragma unroll
            for (int i = 0; i < kClusterWarps / 4; ++i) c[i] = S.wc[q * (kClusterWarps / 4) + i][d];
#pragma unroll
            for (int i = 0; i < kClusterWarps / 4; ++i) {
                S.wc[q * (kClusterWarps / 4) + i][d] = run;
                run += c[i];
            }
            S.part[q][d] = run;
        }
        __syncthreads();
        // exclusive prefix over the digits, 8 warps of it: within the warp here, the warps before by their sums
        auto prefix = [&](uint32_t v, uint32_t* sums) {
            uint32_t x = v;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
                if (lane >= (uint32_t)off) x += y;
            }
            if (lane == 31) sums[w] = x;
            return x - v;
        };
        uint32_t mineAt = 0;
        if (q == 0) {
            const uint32_t c = S.part[0][d] + S.part[1][d] + S.part[2][d] + S.part[3][d];
            S.cnt[d] = c;
            mineAt = prefix(c, S.warpSums[0]);
        }
        cluster.barrier_arrive();  // the counts are there
        __syncthreads();
        if (q == 0) {
            for (uint32_t k = 0; k < w; ++k) mineAt += S.warpSums[0][k];
            uint32_t at = mineAt;
            for (int i = 0; i < 4; ++i) {
                const uint32_t c = S.part[i][d];
                S.part[i][d] = at;
                at += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            if (base + 32 * r >= n) continue;
            const uint32_t dg = (key[r] >> bits) & 0xFFu;
            S.sorted[S.part[w / (kClusterWarps / 4)][dg] + S.wc[w][dg] + pos[r]] = (unsigned long long)key[r] << 32 | val[r];
        }
        cluster.barrier_wait();
        {
            uint32_t all = 0, before = 0;
#pragma unroll 4
            for (uint32_t b = q; b < size; b += 4) {
                const uint32_t c = cluster.map_shared_rank(S.cnt, b)[d];
                all += c;
                before += b < rank ? c : 0u;
            }
            S.all[q][d] = all;
            S.before[q][d] = before;
        }
        if (pass == 3) cluster.barrier_arrive();  // the last look into the other blocks' memory
        __syncthreads();
        uint32_t at = 0;
        if (q == 0)
            at = prefix(S.all[0][d] + S.all[1][d] + S.all[2][d] + S.all[3][d], S.warpSums[1]) + S.before[0][d] + S.before[1][d] +
                 S.before[2][d] + S.before[3][d];
        __syncthreads();
        if (q == 0) {
            for (uint32_t k = 0; k < w; ++k) at += S.warpSums[1][k];
            S.shift[d] = at - mineAt;
        }
        __syncthreads();
        // neighbours in `sorted` mostly stay neighbours: whole stretches go to a block
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            const uint32_t i = tid + kClusterThreads * r;
            if (i >= held) continue;
            const unsigned long long kv = S.sorted[i];
            const uint32_t dst = i + S.shift[(uint32_t)(kv >> (32 + bits)) & 0xFFu];
            if (pass < 3) {
                cluster.map_shared_rank(S.pair, dst / kBlockKeys)[dst % kBlockKeys] = kv;
            } else {
                keysOut[dst] = (uint32_t)(kv >> 32);
                order[dst] = (uint32_t)kv;
            }
        }
        if (pass < 3) cluster.sync();
    }
    cluster.barrier_wait();
}

// cluster size that this device schedules for k_sort_cluster: 16, 8, or 0 (none)
uint32_t cluster_limit() {
    constexpr int kDevices = 64;
    static std::atomic<int> known[kDevices];  // 0: not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 0;
    int v = known[dev].load(std::memory_order_acquire);
    if (!v) {
        v = -1;
        const void* fn[3] = {(const void*)k_sort_cluster<1>, (const void*)k_sort_cluster<2>, (const void*)k_sort_cluster<4>};
        bool ok = true;
        for (const void* f : fn)
            ok = ok && cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ClusterSort)) == cudaSuccess &&
                 cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        for (int size = 16; ok && v < 0 && size >= 8; size /= 2) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(size);
            cfg.blockDim = dim3(kClusterThreads);
            cfg.dynamicSmemBytes = sizeof(ClusterSort);
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim = {(unsigned)size, 1, 1};
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int clusters = 0;
            bool all = true;
            for (const void* f : fn) all = all && cudaOccupancyMaxActiveClusters(&clusters, f, &cfg) == cudaSuccess && clusters > 0;
            if (all) v = size;
        }
        if (v < 0) cudaGetLastError();  // a refused attribute is no error of the build
        known[dev].store(v, std::memory_order_release);
    }
    return v < 0 ? 0u : (uint32_t)v;
}

// TLAS leaf k: the instance at sorted position k with its inverse rows and its BLAS's root box
// and record pointers copied in
__global__ void k_inst_records(const uint32_t* __restrict__ order, uint32_t n, const DevInstance* __restrict__ inst,
                               const DevBlas* __restrict__ blas, InstRec* __restrict__ out) {
    chain_wait();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t ii = order[k];
    const DevInstance& d = inst[ii];
    InstRec r;
    r.inv[0] = d.inv[0];
    r.inv[1] = d.inv[1];
    r.inv[2] = d.inv[2];
    r.lo = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(0u));
    r.hi = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(ii));
    r.wide = nullptr;
    r.tris = nullptr;
    if (d.valid) {
        const DevBlas& b = blas[d.blas];
        r.lo = make_float4(b.root[0], b.root[1], b.root[2], __uint_as_float(b.n));
        r.hi = make_float4(b.root[3], b.root[4], b.root[5], __uint_as_float(ii));
        r.wide = b.wide;
        r.tris = b.tris;
    }
    out[k] = r;
}

// ---- hierarchy -----------------------------------------------------------------------------------
// The binary radix tree of the sorted codes (Karras 2012: its nodes and their numbering), built bottom
// up with the boxes (Apetrei 2014).  A node covers a range [l, r] of leaves and splits after leaf s; its
// parent splits where the range borders on the closer neighbour: after r if leaf r + 1 shares more bits
// with leaf r than leaf l - 1 with leaf l, else after l - 1.  The node is then its parent's left (right)
// child, and Karras' number for it is r (l); the root's is 0.  One thread per leaf climbs: of a
// split's two arrivals the first leaves its far end and stops, the second goes on with the union.
//
// The climb is a chain of dependent memory accesses, some 25 levels of it for 50000 leaves, so
//   - a block keeps the nodes whose range lies in its own kHierLeaves leaves in shared memory;
//   - of the others a level is ONE round trip: the arrival word carries the far end and the common bits
//     with the leaf beyond it (up to 2^25 leaves; more read them from the codes), no fence orders it
//     after the box, and the sibling's box is requested together with it.  Box words start as
//     kNoBox, which no union is, so a box still on its way is seen and asked for again; after
//     kHierPolls requests the box is taken from the leaves instead, so no wait is unbounded.
// 50000 leaves: 23 us (37 us with an acquire-release arrival and its box after it), against 12 us for
// the nodes and 36 us for the boxes as two kernels.
constexpr int kHierLeaves = 512;
constexpr int kHierPolls = 4096;

__device__ __forceinline__ int delta(uint32_t a, uint32_t b, uint32_t i, uint32_t j) {  // common leading bits of (code, position)
    return a == b ? 32 + __clz(i ^ j) : __clz(a ^ b);
}

__device__ __forceinline__ uint32_t swap_relaxed(uint32_t* p, uint32_t v) {
    uint32_t old;
    asm volatile("atom.exch.relaxed.gpu.global.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

__device__ __forceinline__ void load_box_relaxed(const float* p, uint32_t* b) {
#pragma unroll
    for (int a = 0; a < 6; ++a) b[a] = ld_relaxed(reinterpret_cast<const uint32_t*>(p) + a);
}
__device__ __forceinline__ bool box_there(const uint32_t* b) {
    bool there = true;
#pragma unroll
    for (int a = 0; a < 6; ++a) there = there && b[a] != kNoBox;
    return there;
}

// LEAVES: every box of another block's node is taken from the leaves (tests; a limit passed at run time cost 0.4 us)
template <bool LEAVES>
__global__ void __launch_bounds__(kHierLeaves) k_hierarchy(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ order,
                                                           const float* __restrict__ primBoxes, uint32_t n, uint32_t* __restrict__ left,
                                                           uint32_t* __restrict__ right, uint32_t* __restrict__ parents,
                                                           uint32_t* arrivals, float* nodeBoxes) {
    chain_wait();
    __shared__ uint32_t sKeys[kHierLeaves + 2];      // leaves first - 1 .. first + kHierLeaves
    __shared__ uint32_t sArrive[kHierLeaves];        // by split
    __shared__ float sLeaf[kHierLeaves][6], sNode[kHierLeaves][6];  // boxes by leaf and by node number
    const uint32_t first = blockIdx.x * kHierLeaves, k = first + threadIdx.x;
    const uint32_t end = min(n, first + kHierLeaves);  // one past the block's last leaf
    const bool packed = n < (1u << 25);
    float cur[6];
    if (k < n) {
        const float* b = primBoxes + 6 * (size_t)order[k];
#pragma unroll
        for (int a = 0; a < 6; ++a) sLeaf[threadIdx.x][a] = cur[a] = b[a];
        sKeys[threadIdx.x + 1] = keys[k];
        sArrive[threadIdx.x] = 0u;
    }
    if (threadIdx.x == 0) {
        sKeys[0] = first ? keys[first - 1] : 0u;
        sKeys[end - first + 1] = end < n ? keys[end] : 0u;
    }
    __syncthreads();
    if (k >= n) return;
    auto key = [&](uint32_t i) { return i + 1 >= first && i <= end ? sKeys[i + 1 - first] : keys[i]; };
    auto between = [&](uint32_t i, uint32_t j) { return delta(key(i), key(j), i, j); };
    uint32_t l = k, r = k, node = kLeaf | k;
    int dl = l > 0 ? between(l - 1, l) : -1, dr = r + 1 < n ? between(r, r + 1) : -1;
    // a radix tree has at most 62 levels; the bounds also hold for words that another build is writing
    for (int level = 0; level < 128; ++level) {
        if (dl < 0 && dr < 0) return;  // the root is done
        const bool isLeft = dr > dl;
        const uint32_t s = isLeft ? r : l - 1;  // the parent's split
        if (s >= n - 1u) return;                // never in a build that runs alone
        // the parent's range lies in the block if mine does and the sibling's does not reach past it
        const int ds = isLeft ? dr : dl;
        const bool local = l >= first && r < end &&
                           (isLeft ? r + 1 < end && !(end < n && between(r + 1, end) > ds)
                                   : l > first && !(first > 0 && between(first - 1, l - 1) > ds));
        const uint32_t mine = (isLeft ? l : r) + 1u + (packed ? (uint32_t)((isLeft ? dl : dr) + 1) << 25 : 0u);
        const uint32_t sibNode = isLeft ? s + 1 : s;  // the sibling's number if it is not a leaf
        uint32_t got, ob[6];
        if (local) {
            if (!(node & kLeaf)) {
#pragma unroll
                for (int a = 0; a < 6; ++a) sNode[node - first][a] = cur[a];
                __threadfence_block();
            }
            got = atomicExch(&sArrive[s - first], mine);
            __threadfence_block();
        } else {
            got = swap_relaxed(&arrivals[s], mine);
            load_box_relaxed(nodeBoxes + 6 * (size_t)min(sibNode, n - 2u), ob);
        }
        if (got == 0u) return;
        const uint32_t far = (packed ? got & 0x1FFFFFFu : got) - 1u;  // the other side's far end
        if (isLeft ? far <= s || far >= n : far > s) return;  // never in a build that runs alone
        const bool sibLeaf = far == sibNode;
        const uint32_t L = (isLeft ? l : far) == s ? (kLeaf | s) : s;
        const uint32_t R = (isLeft ? far : r) == s + 1 ? (kLeaf | (s + 1)) : s + 1;
        if (isLeft) {
            r = far;
            dr = packed ? (int)(got >> 25) - 1 : r + 1 < n ? between(r, r + 1) : -1;
        } else {
            l = far;
            dl = packed ? (int)(got >> 25) - 1 : l > 0 ? between(l - 1, l) : -1;
        }
        if (local) {
            const float* b = sibLeaf ? sLeaf[sibNode - first] : sNode[sibNode - first];
#pragma unroll
            for (int a = 0; a < 6; ++a) ob[a] = __float_as_uint(b[a]);
        } else if (sibLeaf) {
            const float* b = primBoxes + 6 * (size_t)order[sibNode];
#pragma unroll
            for (int a = 0; a < 6; ++a) ob[a] = __float_as_uint(b[a]);
        } else {
            for (int i = 0; !LEAVES && i < kHierPolls && !box_there(ob); ++i) load_box_relaxed(nodeBoxes + 6 * (size_t)sibNode, ob);
            if (LEAVES || !box_there(ob)) {
                const float none = __uint_as_float(0x7FFFFFFFu);  // passed over, and what a union of NaN boxes is
                float u[6] = {none, none, none, none, none, none};
                const uint32_t i0 = isLeft ? s + 1 : far, i1 = isLeft ? far : s;
                for (uint32_t i = i0; i <= i1; ++i) {
                    const float* b = primBoxes + 6 * (size_t)order[i];
                    for (int a = 0; a < 3; ++a) {
                        u[a] = fminf(u[a], b[a]);
                        u[3 + a] = fmaxf(u[3 + a], b[3 + a]);
                    }
                }
                for (int a = 0; a < 6; ++a) ob[a] = __float_as_uint(u[a]);
            }
        }
        node = dl < 0 && dr < 0 ? 0u : dr > dl ? r : l;
        if (node >= n - 1u) return;  // never in a build that runs alone
        float* o = nodeBoxes + 6 * (size_t)node;
        // the left child's box is the first operand
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float c0 = __uint_as_float(ob[a]), c1 = __uint_as_float(ob[3 + a]);
            cur[a] = isLeft ? fminf(cur[a], c0) : fminf(c0, cur[a]);
            cur[3 + a] = isLeft ? fmaxf(cur[3 + a], c1) : fmaxf(c1, cur[3 + a]);
        }
#pragma unroll
        for (int a = 0; a < 6; ++a) st_relaxed(reinterpret_cast<uint32_t*>(o) + a, __float_as_uint(cur[a]));
        left[node] = L;
        right[node] = R;
        parents[(L & kLeaf) ? (n - 1) + (L & ~kLeaf) : L] = node;
        parents[(R & kLeaf) ? (n - 1) + (R & ~kLeaf) : R] = node;
        if (dl < 0 && dr < 0) parents[0] = 0xFFFFFFFFu;
    }
}

// ---- refit ---------------------------------------------------------------------------------------
__device__ inline void load_box_cg(const float* p, float* b) {
    for (int a = 0; a < 6; ++a) b[a] = __ldcg(p + a);
}

__device__ __forceinline__ uint32_t arrive(uint32_t* flag) {  // release my box, acquire my sibling's
    uint32_t old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(flag) : "memory");
    return old;
}

// one thread per leaf climbs towards the root and writes each node's box as the union of its
// children's.  The climbing thread keeps the box of the child it comes from in registers and loads
// only its sibling's.  A leaf sibling's box is input data, so a node with a leaf child needs no
// arrival: the thread from its inner child (or, for two leaves, from its left leaf) goes on and the
// other stops at once.  A node with two inner children takes the arrival counter: the first
// arrival stops, the second (which then sees the first's box: release / acquire) goes on.
__global__ void k_bottom_up(const float* __restrict__ primBoxes, const uint32_t* __restrict__ order, uint32_t n,
                            const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                            const uint32_t* __restrict__ parents, uint32_t* flags, float* nodeBoxes) {
    chain_wait();
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    uint32_t node = parents[(n - 1) + k];
    uint32_t from = kLeaf | k;
    float cur[6];  // loaded once this thread knows that it goes on from its leaf
    // a finished tree has at most 64 levels and in-range parents; the bounds keep a tree that a
    // failed build left unfinished from sending the climb out of range or round in circles
    for (int level = 0; node < n - 1u && level < 128; ++level) {  // the root's parent is 0xFFFFFFFF
        const uint32_t L = left[node], R = right[node];
        const uint32_t other = L == from ? R : L;
        if ((other & kLeaf) ? (other & ~kLeaf) >= n : other >= n - 1u) break;  // in range in a finished tree
        if (other & kLeaf) {
            if ((from & kLeaf) && L != from) return;  // two leaves: the left one goes on
        } else if (from & kLeaf) {
            return;  // the thread from the inner child goes on
        } else if (arrive(&flags[node]) == 0) {
            return;  // two inner children: the second arrival goes on
        }
        if (level == 0) load_box_cg(primBoxes + 6 * (size_t)order[k], cur);
        float ob[6];
        if (other & kLeaf) load_box_cg(primBoxes + 6 * (size_t)order[other & ~kLeaf], ob);
        else load_box_cg(nodeBoxes + 6 * (size_t)other, ob);
        const float* bl = L == from ? cur : ob;
        const float* br = L == from ? ob : cur;
        float nb[6];
        for (int a = 0; a < 3; ++a) {
            nb[a] = fminf(bl[a], br[a]);
            nb[3 + a] = fmaxf(bl[3 + a], br[3 + a]);
        }
        float* o = nodeBoxes + 6 * (size_t)node;
        for (int a = 0; a < 6; ++a) {
            __stcg(o + a, nb[a]);
            cur[a] = nb[a];
        }
        from = node;
        node = parents[node];
    }
}

// ---- 4-wide records ----------------------------------------------------------------------------
__device__ inline void child_box(const float* __restrict__ primBoxes, const uint32_t* __restrict__ order, const float* nodeBoxes,
                                 uint32_t ref, float* b) {
    const float* p = (ref & kLeaf) ? primBoxes + 6 * (size_t)order[ref & ~kLeaf] : nodeBoxes + 6 * (size_t)ref;
    for (int a = 0; a < 6; ++a) b[a] = p[a];
}

__global__ void k_wide_records(const float* __restrict__ primBoxes, const uint32_t* __restrict__ order, uint32_t n,
                               const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                               const float* __restrict__ nodeBoxes, WideNode* __restrict__ out) {
    chain_wait();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i + 1 >= n) return;
    uint32_t refs[4];
    int k = 0;
    for (uint32_t c : {left[i], right[i]}) {
        if (c & kLeaf) {
            refs[k++] = c;
        } else {
            refs[k++] = left[c];
            refs[k++] = right[c];
        }
    }
    float lo[3][4], hi[3][4];
    uint32_t r[4];
    for (int j = 0; j < 4; ++j) {
        if (j < k) {
            float b[6];
            child_box(primBoxes, order, nodeBoxes, refs[j], b);
            for (int a = 0; a < 3; ++a) {
                lo[a][j] = b[a];
                hi[a][j] = b[3 + a];
            }
            r[j] = refs[j];
        } else {
            for (int a = 0; a < 3; ++a) {
                lo[a][j] = INFINITY;
                hi[a][j] = -INFINITY;
            }
            r[j] = kEmptySlot;
        }
    }
    WideNode w;
    w.lox = make_float4(lo[0][0], lo[0][1], lo[0][2], lo[0][3]);
    w.hix = make_float4(hi[0][0], hi[0][1], hi[0][2], hi[0][3]);
    w.loy = make_float4(lo[1][0], lo[1][1], lo[1][2], lo[1][3]);
    w.hiy = make_float4(hi[1][0], hi[1][1], hi[1][2], hi[1][3]);
    w.loz = make_float4(lo[2][0], lo[2][1], lo[2][2], lo[2][3]);
    w.hiz = make_float4(hi[2][0], hi[2][1], hi[2][2], hi[2][3]);
    w.ref = make_uint4(r[0], r[1], r[2], r[3]);
    out[i] = w;
}

// ---- binned-SAH BVH2 (TLAS, and BLASes up to kSahBlasMaxPrims triangles) ------------------------
// One CTA builds a BVH2 over the primitive boxes, top-down, level by level: each warp takes a node
// task (a range of the order array), reduces the range's box and centroid box, bins the centroids into
// 16 bins per axis (shared-memory atomics on order-preserving integer images of the bounds), evaluates
// the 45 surface-area-heuristic splits, partitions the range stably with ballots, and emits its
// children (single primitives become leaf refs, the rest next-level tasks).  Every split leaves both
// sides non-empty, so each level shortens every range.  From level medianLevel on, ranges are halved
// without binning, so no tree is deeper than medianLevel + ceil(log2 n) levels, whatever the centroid
// distribution (a surface-area split can peel one primitive off a range per level).
// A level's tasks are numbered after the previous levels' nodes, so a task is just its range; the nodes of
// the subtrees that single warps finish are numbered from the upper end.  The result has the LBVH's layout (order, left, right, nodeBoxes), so
// records, refits and traversal are shared.
constexpr int kSahBins = 16;
constexpr int kSahWarps = 32;
constexpr int kSahTaskWarps = 8;               // warps per block of k_sah_tasks
constexpr uint32_t kSahHandoff = 64;           // tasks of a level from which k_sah_tasks takes over
constexpr int kSahParallelLevels = 13;         // levels built by k_sah_level at most, one launch each
constexpr uint32_t kSahSmall = 4096;           // up to here one CTA holds the primitives of the top levels
// The level kernels run until a level's tasks hold some kSahTask primitives: a task of some hundreds costs a
// CTA 10 us and one warp of k_sah_tasks 20 us and more (61442 triangles: levels until 64, 128, 256, 512
// primitives 2.43, 2.47, 2.53, 2.68 ms for the whole scene load).  A small build's levels cost its CTA 6 us
// each, a level through k_sah_tasks' queue 9 us, so it hands over when its warps all have a task.
constexpr uint32_t kSahTask = 64;
constexpr uint32_t kSahSmallHandoff = 32;
// A subtree of m primitives on one warp takes m - 1 nodes one after another, 1.5 us each: 32 where the warps
// have enough of them, 16 in a small build, which has more warps than tasks.
constexpr uint32_t kSahSubtree = 32, kSahSubtreeSmall = 16;
constexpr uint32_t kSahWaitLimit = 1u << 22;   // polls of an unpublished task before k_sah_tasks gives up

__device__ __forceinline__ int ord_float(float f) {
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float unord_float(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }
__device__ __forceinline__ float half_area3(const float* lo, const float* hi) {
    const float dx = fmaxf(hi[0] - lo[0], 0.0f), dy = fmaxf(hi[1] - lo[1], 0.0f), dz = fmaxf(hi[2] - lo[2], 0.0f);
    return dx * dy + dy * dz + dz * dx;
}

// minimum and maximum over the warp (redux: one instruction each; as fminf a NaN is passed over)
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// The cheapest of the 3 x 15 surface-area splits of a task's bins (ties to the lowest candidate),
// found by the calling warp (all 32 lanes call it); -1 when no split leaves both sides non-empty.
// cnt(a, k), lo(a, k, c), hi(a, k, c) read bin k of axis a (bounds as ordered ints).  A half-warp takes
// an axis, a lane a bin: boxes and counts left and right of each split are prefix and suffix scans (four
// steps), a third of the instructions of a lane going over the 16 bins for its split.
template <class Cnt, class Lo, class Hi>
__device__ __forceinline__ int sah_best_split(const float* scale, int lane, Cnt cnt, Lo lo, Hi hi) {
    constexpr unsigned full = 0xFFFFFFFFu;
    float bestCost = INFINITY;
    int bestCand = -1;
    const int k = lane & 15;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int a = 2 * half + (lane >> 4);
        const float sc = a == 0 ? scale[0] : a == 1 ? scale[1] : a == 2 ? scale[2] : 0.0f;
        float L[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY}, R[6];
        int nl = sc > 0.0f ? cnt(a, k) : 0;
        if (nl)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                L[c] = fminf(L[c], unord_float(lo(a, k, c)));
                L[3 + c] = fmaxf(L[3 + c], unord_float(hi(a, k, c)));
            }
        int nr = nl;
#pragma unroll
        for (int c = 0; c < 6; ++c) R[c] = L[c];
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) {  // L, nl: bins 0 .. k; R, nr: bins k .. 15
            const int pn = __shfl_up_sync(full, nl, off, 16), sn = __shfl_down_sync(full, nr, off, 16);
            if (k >= off) nl += pn;
            if (k + off < 16) nr += sn;
#pragma unroll
            for (int c = 0; c < 3; ++c) {  // beyond the half-warp a lane gets its own value
                L[c] = fminf(L[c], __shfl_up_sync(full, L[c], off, 16));
                L[3 + c] = fmaxf(L[3 + c], __shfl_up_sync(full, L[3 + c], off, 16));
                R[c] = fminf(R[c], __shfl_down_sync(full, R[c], off, 16));
                R[3 + c] = fmaxf(R[3 + c], __shfl_down_sync(full, R[3 + c], off, 16));
            }
        }
        nr = __shfl_down_sync(full, nr, 1, 16);  // bins k + 1 .. 15
#pragma unroll
        for (int c = 0; c < 6; ++c) R[c] = __shfl_down_sync(full, R[c], 1, 16);
        const float cost = half_area3(L, L + 3) * (float)nl + half_area3(R, R + 3) * (float)nr;
        if (sc > 0.0f && k < kSahBins - 1 && nl && nr && cost < bestCost) {
            bestCost = cost;
            bestCand = a * (kSahBins - 1) + k;  // split before bin k + 1
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float oc = __shfl_xor_sync(full, bestCost, off);
        const int oi = __shfl_xor_sync(full, bestCand, off);
        if (oi >= 0 && (bestCand < 0 || oc < bestCost || (oc == bestCost && oi < bestCand))) {
            bestCost = oc;
            bestCand = oi;
        }
    }
    return bestCand;
}

// One primitive a lane into the bins of one axis (bins in shared memory, this warp's own).  The
// primitives of a range keep the mesh's order, so a warp's mostly fall into a few bins, and 32 atomics on
// one word take their turns: lanes of one bin are reduced first while the groups are large.
__device__ __forceinline__ void sah_bin(bool valid, int bin, const float* bx, int* cnt, int (*lo)[3], int (*hi)[3], int lane) {
    constexpr int kGroup = 8;
    unsigned todo = __ballot_sync(0xFFFFFFFFu, valid);
    while (__popc(todo) >= kGroup) {
        const int b0 = __shfl_sync(0xFFFFFFFFu, bin, __ffs(todo) - 1);
        const unsigned m = __ballot_sync(0xFFFFFFFFu, valid && bin == b0) & todo;
        if (__popc(m) < kGroup) break;
        if (m >> lane & 1u) {
            int l[3], h[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                l[c] = __reduce_min_sync(m, ord_float(bx[c]));
                h[c] = __reduce_max_sync(m, ord_float(bx[3 + c]));
            }
            if (lane == __ffs(m) - 1) {
                cnt[bin] += __popc(m);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    lo[bin][c] = min(lo[bin][c], l[c]);
                    hi[bin][c] = max(hi[bin][c], h[c]);
                }
            }
        }
        todo &= ~m;
        __syncwarp();
    }
    if (todo >> lane & 1u) {
        atomicAdd(&cnt[bin], 1);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            atomicMin(&lo[bin][c], ord_float(bx[c]));
            atomicMax(&hi[bin][c], ord_float(bx[3 + c]));
        }
    }
    __syncwarp();
}

// f(valid, primitive, box) for order[b, e), a lane each, the loads of four rounds in flight together
template <bool COHERENT, int kRounds, class F>
__device__ __forceinline__ void sah_each(const float* __restrict__ boxes, const uint32_t* order, uint32_t b, uint32_t e, int lane, F&& f) {
    for (uint32_t i0 = b; i0 < e; i0 += 32 * kRounds) {
        uint32_t prim[kRounds];
        float bx[kRounds][6];
#pragma unroll
        for (int j = 0; j < kRounds; ++j) {
            const uint32_t i = i0 + 32 * j + lane;
            prim[j] = i < e ? (COHERENT ? __ldcg(order + i) : order[i]) : 0u;
        }
#pragma unroll
        for (int j = 0; j < kRounds; ++j)
#pragma unroll
            for (int c = 0; c < 6; ++c) bx[j][c] = i0 + 32 * j + lane < e ? boxes[6 * (size_t)prim[j] + c] : 0.0f;
#pragma unroll
        for (int j = 0; j < kRounds; ++j)
            if (i0 + 32 * j < e) f(i0 + 32 * j + lane < e, prim[j], bx[j]);
    }
}

// a range's box (v[0..5]) and centroid box (v[6..11]), lane by lane; sah_bounds_warp: over the warp
__device__ __forceinline__ void sah_bounds_init(float* v) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        v[a] = v[6 + a] = INFINITY;
        v[3 + a] = v[9 + a] = -INFINITY;
    }
}
__device__ __forceinline__ void sah_bounds_add(float* v, const float* bx) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        v[a] = fminf(v[a], bx[a]);
        v[3 + a] = fmaxf(v[3 + a], bx[3 + a]);
        const float c = 0.5f * (bx[a] + bx[3 + a]);
        v[6 + a] = fminf(v[6 + a], c);
        v[9 + a] = fmaxf(v[9 + a], c);
    }
}
__device__ __forceinline__ void sah_bounds_warp(float* v) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        v[a] = warp_min(v[a]);
        v[3 + a] = warp_max(v[3 + a]);
        v[6 + a] = warp_min(v[6 + a]);
        v[9 + a] = warp_max(v[9 + a]);
    }
}
__device__ __forceinline__ float sah_scale(float clo, float chi) {
    const float ext = chi - clo;
    return ext > 0.0f ? (float)kSahBins / ext : 0.0f;
}
__device__ __forceinline__ int sah_bin_of(float lo, float hi, float origin, float scale) {
    const float c = 0.5f * (lo + hi);
    return max(0, min((int)((c - origin) * scale), kSahBins - 1));
}
__device__ __forceinline__ float pick3(const float* v, int a) { return a == 0 ? v[0] : a == 1 ? v[1] : v[2]; }
// a warp's bins cleared
__device__ __forceinline__ void sah_bins_clear(int (&lo)[3][kSahBins][3], int (&hi)[3][kSahBins][3], int (&cnt)[3][kSahBins], int lane) {
    for (int k = lane; k < 3 * kSahBins; k += 32) (&cnt[0][0])[k] = 0;
    for (int k = lane; k < 9 * kSahBins; k += 32) {
        (&lo[0][0][0])[k] = ord_float(INFINITY);
        (&hi[0][0][0])[k] = ord_float(-INFINITY);
    }
    __syncwarp();
}

// One level with fewer tasks than warps: G warps share a task (G * count <= 32, and about 64
// primitives of the largest task a warp at least), each taking a contiguous chunk of the task's range.
// The same computation as one warp per task -- bounds and bin contents are order-independent minima,
// maxima and counts, the split is chosen by the same rule, and the partition stays stable (each warp
// writes its chunk at the offsets of the chunks before it) -- so the tree is the same; the top levels
// just run on the whole CTA instead of a few warps.  1024 primitives in shared memory: 9 us a level, half
// of it instruction fetches of code that runs once (14 us and a launch with 32 warps a task and the
// group's bins and bounds merged by its first warp).
template <int kRounds>
__device__ __forceinline__ void sah_level_grouped(const float* __restrict__ boxes, uint32_t* __restrict__ order, uint32_t* __restrict__ tmp,
                                                  uint32_t* __restrict__ left, uint32_t* __restrict__ right, float* __restrict__ nodeBoxes,
                                                  const uint2* cur, uint2* nxt, uint32_t count, bool median, uint32_t baseCur,
                                                  uint32_t baseNext, uint32_t& nNext, int (*bLo)[3][kSahBins][3],
                                                  int (*bHi)[3][kSahBins][3], int (*bCnt)[3][kSahBins], float (*gPart)[12],
                                                  int* tBest, uint32_t* wLeft) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t largest = 0;
    if ((uint32_t)lane < count) {
        const uint2 tk = cur[lane];
        largest = tk.y - tk.x;
    }
    largest = __reduce_max_sync(0xFFFFFFFFu, largest);
    uint32_t G = kSahWarps;
    while (G > 1 && (G * count > (uint32_t)kSahWarps || (G - 1) * 64 >= largest)) G >>= 1;
    const uint32_t t = (uint32_t)warp / G, m = (uint32_t)warp % G;
    const bool has = t < count;  // warp-uniform
    const int lw = (int)(t * G);  // the task's leader warp (owner of its bins)
    uint32_t b = 0, e = 0, cb = 0, ce = 0, node = 0;
    if (has) {
        const uint2 tk = cur[t];
        b = tk.x;
        e = tk.y;
        node = baseCur + t;
        const uint32_t chunk = (e - b + G - 1) / G;
        cb = min(e, b + m * chunk);
        ce = min(e, cb + chunk);
    }
    // bounds and centroid bounds of the chunk, then of the task
    float v[12];
    sah_bounds_init(v);
    sah_each<false, kRounds>(boxes, order, cb, ce, lane, [&](bool valid, uint32_t, const float* bx) {
        if (valid) sah_bounds_add(v, bx);
    });
    sah_bounds_warp(v);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < 12; ++k) gPart[warp][k] = v[k];
    if (has && !median) sah_bins_clear(bLo[warp], bHi[warp], bCnt[warp], lane);
    __syncthreads();
    float tc[3] = {0.0f, 0.0f, 0.0f}, ts[3] = {0.0f, 0.0f, 0.0f};
    if (has) {  // every warp of the group: lane g takes the g-th chunk's
#pragma unroll
        for (int k = 0; k < 12; ++k) v[k] = gPart[lw + ((uint32_t)lane < G ? lane : 0)][k];
        sah_bounds_warp(v);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            tc[a] = v[6 + a];
            ts[a] = sah_scale(v[6 + a], v[9 + a]);
        }
        if (m == 0 && lane == 0)
#pragma unroll
            for (int k = 0; k < 6; ++k) nodeBoxes[6 * (size_t)node + k] = v[k];
        if (!median)  // every warp bins its chunk into its own bins (no atomics across warps)
            sah_each<false, kRounds>(boxes, order, cb, ce, lane, [&](bool valid, uint32_t, const float* bx) {
#pragma unroll 1
                for (int a = 0; a < 3; ++a)
                    if (pick3(ts, a) > 0.0f)
                        sah_bin(valid, sah_bin_of(pick3(bx, a), pick3(bx + 3, a), pick3(tc, a), pick3(ts, a)), bx, bCnt[warp][a],
                                bLo[warp][a], bHi[warp][a], lane);
            });
    }
    __syncthreads();
    if (has && !median && G > 1) {  // the group's bins into the leader's (counts add, bounds are minima and maxima: exact)
        constexpr int kWords = 3 * kSahBins;
#pragma unroll 1
        for (uint32_t k = m * 32 + lane; k < 7 * kWords; k += 32 * G) {
            if (k < kWords) {
                int r = 0;
                for (uint32_t g = 1; g < G; ++g) r += (&bCnt[lw + g][0][0])[k];
                (&bCnt[lw][0][0])[k] += r;
            } else if (k < 4 * kWords) {
                int r = (&bLo[lw][0][0][0])[k - kWords];
                for (uint32_t g = 1; g < G; ++g) r = min(r, (&bLo[lw + g][0][0][0])[k - kWords]);
                (&bLo[lw][0][0][0])[k - kWords] = r;
            } else {
                int r = (&bHi[lw][0][0][0])[k - 4 * kWords];
                for (uint32_t g = 1; g < G; ++g) r = max(r, (&bHi[lw + g][0][0][0])[k - 4 * kWords]);
                (&bHi[lw][0][0][0])[k - 4 * kWords] = r;
            }
        }
    }
    __syncthreads();
    if (has && m == 0) {  // the leader picks the split: cheapest surface-area cost, ties to the lowest candidate
        int bestCand = -1;
        if (!median)
            bestCand = sah_best_split(ts, lane, [&](int a, int k) { return bCnt[lw][a][k]; },
                                      [&](int a, int k, int c) { return bLo[lw][a][k][c]; },
                                      [&](int a, int k, int c) { return bHi[lw][a][k][c]; });
        if (lane == 0) tBest[t] = bestCand;
    }
    __syncthreads();
    const int best = has ? tBest[t] : -1;
    const int sa = best >= 0 ? best / (kSahBins - 1) : 0, sp = best >= 0 ? best % (kSahBins - 1) + 1 : 0;
    if (best >= 0) {  // left count of the chunk: its bins before the split (the leader's hold the task's)
        const int c = __reduce_add_sync(0xFFFFFFFFu, lane < sp ? bCnt[warp][sa][lane] : 0);
        if (lane == 0) wLeft[warp] = (uint32_t)c;
    }
    __syncthreads();
    uint32_t nlTotal = 0;
    if (best >= 0) {  // stable partition: this chunk's lefts after the lefts of the chunks before it, rights likewise
        const uint32_t c = (uint32_t)lane < G ? wLeft[lw + lane] : 0u;
        nlTotal = wLeft[lw];
        const uint32_t others = __reduce_add_sync(0xFFFFFFFFu, lane > 0 ? c : 0u);  // all chunks but the leader's
        const uint32_t ahead = __reduce_add_sync(0xFFFFFFFFu, lane > 0 && (uint32_t)lane < m ? c : 0u);
        const uint32_t before = m ? nlTotal - others + ahead : 0u;
        uint32_t lb = b + before, rb = b + nlTotal + ((cb - b) - before);
        sah_each<false, kRounds>(boxes, order, cb, ce, lane, [&](bool valid, uint32_t prim, const float* bx) {
            const bool isL = valid && sah_bin_of(pick3(bx, sa), pick3(bx + 3, sa), pick3(tc, sa), pick3(ts, sa)) < sp;
            const unsigned lm = __ballot_sync(0xFFFFFFFFu, isL), rm = __ballot_sync(0xFFFFFFFFu, valid && !isL);
            const unsigned below = (1u << lane) - 1u;
            if (isL) tmp[lb + __popc(lm & below)] = prim;
            else if (valid) tmp[rb + __popc(rm & below)] = prim;
            lb += __popc(lm);
            rb += __popc(rm);
        });
    }
    __syncthreads();
    if (best >= 0)
        for (uint32_t i = cb + lane; i < ce; i += 32) order[i] = tmp[i];
    if (has && m == 0 && lane == 0) {  // children: single primitives become leaf refs, the rest next-level tasks
        const uint32_t mid = best >= 0 ? b + nlTotal : b + (e - b) / 2;
        const uint32_t rb0[2] = {b, mid}, re0[2] = {mid, e};
        uint32_t ref[2];
        for (int c = 0; c < 2; ++c) {
            if (re0[c] - rb0[c] == 1) {
                ref[c] = kLeaf | rb0[c];
            } else {
                const uint32_t idx = atomicAdd(&nNext, 1u);
                nxt[idx] = make_uint2(rb0[c], re0[c]);
                ref[c] = baseNext + idx;
            }
        }
        left[node] = ref[0];
        right[node] = ref[1];
    }
}

// One node task on one warp: the range's box (written as the node's box) and centroid box, 16 bins
// per axis in this warp's shared-memory bins, the cheapest of the 45 surface-area splits (ties to
// the lowest candidate; no usable split or `median`: halve the range), a stable ballot partition of
// order[b, e) through tmp, then emit(mid) creates the children and writes the node's refs.
// COHERENT: order[] and tmp[] may have been written by other SMs (the task kernel), so they are read
// through L2.
template <bool COHERENT, int kRounds, class Emit>
__device__ __forceinline__ void sah_task_warp(const float* __restrict__ boxes, uint32_t* __restrict__ order, uint32_t* __restrict__ tmp,
                                              float* __restrict__ nodeBoxes, uint32_t b, uint32_t e, uint32_t node, bool median,
                                              int (&wLo)[3][kSahBins][3], int (&wHi)[3][kSahBins][3], int (&wCnt)[3][kSahBins],
                                              int lane, Emit&& emit) {
    float v[12];
    sah_bounds_init(v);
    sah_each<COHERENT, kRounds>(boxes, order, b, e, lane, [&](bool valid, uint32_t, const float* bx) {
        if (valid) sah_bounds_add(v, bx);
    });
    sah_bounds_warp(v);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < 6; ++k) nodeBoxes[6 * (size_t)node + k] = v[k];
    float clo[3], scale[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        clo[a] = v[6 + a];
        scale[a] = sah_scale(v[6 + a], v[9 + a]);
    }
    int bestCand = -1;
    if (!median) {
        sah_bins_clear(wLo, wHi, wCnt, lane);
        sah_each<COHERENT, kRounds>(boxes, order, b, e, lane, [&](bool valid, uint32_t, const float* bx) {
#pragma unroll
            for (int a = 0; a < 3; ++a)
                if (pick3(scale, a) > 0.0f)
                    sah_bin(valid, sah_bin_of(pick3(bx, a), pick3(bx + 3, a), pick3(clo, a), pick3(scale, a)), bx, wCnt[a], wLo[a], wHi[a],
                            lane);
        });
        bestCand = sah_best_split(scale, lane, [&](int a, int k) { return wCnt[a][k]; },
                                  [&](int a, int k, int c) { return wLo[a][k][c]; },
                                  [&](int a, int k, int c) { return wHi[a][k][c]; });
    }
    uint32_t mid = b + (e - b) / 2;  // no usable split (coincident centroids): halve the range
    if (bestCand >= 0) {
        const int a = bestCand / (kSahBins - 1), sp = bestCand % (kSahBins - 1) + 1;
        const uint32_t nl = (uint32_t)__reduce_add_sync(0xFFFFFFFFu, lane < sp ? wCnt[a][lane] : 0);
        uint32_t lb = 0, rb = 0;
        sah_each<COHERENT, kRounds>(boxes, order, b, e, lane, [&](bool valid, uint32_t prim, const float* bx) {
            const bool isL = valid && sah_bin_of(pick3(bx, a), pick3(bx + 3, a), pick3(clo, a), pick3(scale, a)) < sp;
            const unsigned lm = __ballot_sync(0xFFFFFFFFu, isL), rm = __ballot_sync(0xFFFFFFFFu, valid && !isL);
            const unsigned below = (1u << lane) - 1u;
            if (isL) tmp[b + lb + __popc(lm & below)] = prim;
            else if (valid) tmp[b + nl + rb + __popc(rm & below)] = prim;
            lb += __popc(lm);
            rb += __popc(rm);
        });
        __syncwarp();
        for (uint32_t i = b + lane; i < e; i += 32) order[i] = COHERENT ? __ldcg(tmp + i) : tmp[i];
        __syncwarp();
        mid = b + nl;
    }
    emit(mid);
    __syncwarp();
}

// The whole subtree of a task of at most 32 primitives on one warp, a primitive a lane: a node costs no
// access to memory but its own results.  Nodes are taken from a stack (lane i holds entry i); the
// lanes of a node's range are reordered by its partition.  Bounds, bins, costs, ties and partition as
// sah_task_warp's; two primitives need no bins: every split between them costs the same, so it is the
// first on the first axis that tells them apart.  Node ids: the root has its own, the others are
// first .. first + (e - b - 2) - 1.  Returns the level below the deepest node.
__device__ __forceinline__ uint32_t sah_subtree_warp(const float* __restrict__ boxes, uint32_t* __restrict__ order, uint32_t* __restrict__ left,
                                                     uint32_t* __restrict__ right, float* __restrict__ nodeBoxes, uint32_t b, uint32_t e,
                                                     uint32_t node, uint32_t first, uint32_t level, uint32_t medianLevel,
                                                     int (&wLo)[3][kSahBins][3], int (&wHi)[3][kSahBins][3], int (&wCnt)[3][kSahBins],
                                                     int lane) {
    constexpr unsigned full = 0xFFFFFFFFu;
    const int m = (int)(e - b);
    uint32_t prim = lane < m ? __ldcg(order + b + lane) : 0u;
    float bx[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) bx[c] = lane < m ? boxes[6 * (size_t)prim + c] : 0.0f;
    uint32_t stRange = (uint32_t)m << 8 | level << 16, stNode = node;  // entry 0: lanes 0 .. m - 1
    uint32_t deepest = 0;
    for (int sp = 1; sp > 0;) {
        --sp;
        const uint32_t rg = __shfl_sync(full, stRange, sp), nd = __shfl_sync(full, stNode, sp);
        const int lb = (int)(rg & 0xFFu), le = (int)(rg >> 8 & 0xFFu);
        const uint32_t lv = rg >> 16;
        const bool in = lane >= lb && lane < le;
        deepest = max(deepest, lv + 1);
        float v[12];
        sah_bounds_init(v);
        if (in) sah_bounds_add(v, bx);
        sah_bounds_warp(v);
        const float mineOut = lane == 0 ? v[0] : lane == 1 ? v[1] : lane == 2 ? v[2] : lane == 3 ? v[3] : lane == 4 ? v[4] : v[5];
        if (lane < 6) nodeBoxes[6 * (size_t)nd + lane] = mineOut;
        float scale[3];
        int bin[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            scale[a] = sah_scale(v[6 + a], v[9 + a]);
            bin[a] = sah_bin_of(bx[a], bx[3 + a], v[6 + a], scale[a]);
        }
        int axis = -1, before = 0;  // left: bin[axis] < before
        if (lv < medianLevel) {
            if (le - lb == 2) {
                float q[6];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    q[c] = fminf(INFINITY, bx[c]);
                    q[3 + c] = fmaxf(-INFINITY, bx[3 + c]);
                }
                const float area = half_area3(q, q + 3);
                const float cost = __shfl_sync(full, area, lb) + __shfl_sync(full, area, lb + 1);
                if (cost < INFINITY)
#pragma unroll
                    for (int a = 2; a >= 0; --a) {
                        const int b0 = __shfl_sync(full, bin[a], lb), b1 = __shfl_sync(full, bin[a], lb + 1);
                        if (scale[a] > 0.0f && b0 != b1) {
                            axis = a;
                            before = min(b0, b1) + 1;
                        }
                    }
            } else {
                sah_bins_clear(wLo, wHi, wCnt, lane);
                if (in)
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        if (pick3(scale, a) <= 0.0f) continue;
                        const int k = a == 0 ? bin[0] : a == 1 ? bin[1] : bin[2];
                        atomicAdd(&wCnt[a][k], 1);
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            atomicMin(&wLo[a][k][c], ord_float(bx[c]));
                            atomicMax(&wHi[a][k][c], ord_float(bx[3 + c]));
                        }
                    }
                __syncwarp();
                const int cand = sah_best_split(scale, lane, [&](int a, int k) { return wCnt[a][k]; },
                                                [&](int a, int k, int c) { return wLo[a][k][c]; },
                                                [&](int a, int k, int c) { return wHi[a][k][c]; });
                __syncwarp();
                if (cand >= 0) {
                    axis = cand / (kSahBins - 1);
                    before = cand % (kSahBins - 1) + 1;
                }
            }
        }
        int mid = lb + (le - lb) / 2;  // no usable split: halve the range
        if (axis >= 0) {
            const bool isL = in && (axis == 0 ? bin[0] : axis == 1 ? bin[1] : bin[2]) < before;
            const unsigned lm = __ballot_sync(full, isL), rm = __ballot_sync(full, in && !isL);
            mid = lb + __popc(lm);
            const unsigned below = (1u << lane) - 1u;
            int* perm = &wCnt[0][0];  // the bins are done with
            if (in) perm[isL ? lb + __popc(lm & below) : mid + __popc(rm & below)] = lane;
            __syncwarp();
            const int src = in ? perm[lane] : lane;
            __syncwarp();
            prim = __shfl_sync(full, prim, src);
#pragma unroll
            for (int c = 0; c < 6; ++c) bx[c] = __shfl_sync(full, bx[c], src);
        }
        uint32_t ref[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int r0 = c ? mid : lb, r1 = c ? le : mid;
            if (r1 - r0 == 1) {
                ref[c] = kLeaf | (b + (uint32_t)r0);
            } else {
                ref[c] = first++;
                if (lane == sp) {
                    stRange = (uint32_t)r0 | (uint32_t)r1 << 8 | (lv + 1) << 16;
                    stNode = ref[c];
                }
                ++sp;
            }
        }
        if (lane == 0) {
            left[nd] = ref[0];
            right[nd] = ref[1];
        }
    }
    if (lane < m) order[b + lane] = prim;
    return deepest;
}

// The first kSahParallelLevels levels, one launch per level: CTA t of level L splits task t of the
// level with all 32 of its warps (the grouped routine with one task), so the levels' tasks run on
// separate SMs.  Level L's tasks are the node ids from base_L = 1 + count_1 + ... + count_(L-1) on
// (count_0 = 1: the root), listed in tasksA for even L and tasksB for odd L; a child task takes the
// next slot of level L + 1 from the global counter lvCount[L + 1].  Level 0 also prepares order[]
// (identity) and the node refs (every node starts as (leaf 0, leaf 0), so a tree left unfinished by
// a task wait that gave up only refers to nodes and leaves in range).
__global__ void __launch_bounds__(kSahWarps * 32, 1) k_sah_level(const float* __restrict__ boxes, uint32_t n, uint32_t* __restrict__ order,
                                                                 uint32_t* __restrict__ tmp, uint32_t* __restrict__ left,
                                                                 uint32_t* __restrict__ right, float* __restrict__ nodeBoxes,
                                                                 uint2* __restrict__ tasksA, uint2* __restrict__ tasksB,
                                                                 uint32_t* __restrict__ lvCount, int level, uint32_t medianLevel) {
    chain_wait();
    __shared__ int bLo[kSahWarps][3][kSahBins][3], bHi[kSahWarps][3][kSahBins][3];
    __shared__ int bCnt[kSahWarps][3][kSahBins];
    __shared__ float gPart[kSahWarps][12];
    __shared__ int tBest[kSahWarps];
    __shared__ uint32_t wLeft[kSahWarps];
    uint2* cur = (level & 1) ? tasksB : tasksA;
    uint2* nxt = (level & 1) ? tasksA : tasksB;
    if (level == 0) {
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) order[i] = i;
        for (uint32_t i = threadIdx.x; i + 1 < n; i += blockDim.x) left[i] = right[i] = kLeaf;
        if (threadIdx.x == 0) cur[0] = make_uint2(0u, n);
        __syncthreads();
    }
    const uint32_t count = level == 0 ? 1u : lvCount[level];
    if (blockIdx.x >= count) return;
    uint32_t base = level == 0 ? 0u : 1u;
    for (int k = 1; k < level; ++k) base += lvCount[k];
    sah_level_grouped<4>(boxes, order, tmp, left, right, nodeBoxes, cur + blockIdx.x, nxt, 1u, (uint32_t)level >= medianLevel,
                      base + blockIdx.x, base + count, lvCount[level + 1], bLo, bHi, bCnt, gPart, tBest, wLeft);
}

// ---- one task over many CTAs (the top levels of large builds) -------------------------------------
// For builds of at least kSahSplitMin primitives, the first kSahSplitLevels levels split each task
// over kSplitCtas CTAs, in five launches per level, because one SM would otherwise bin a whole
// level's primitives.  CTA (t, m) takes chunk m of task t.
//   0 bounds: the chunk's box and centroid box          -> part[t][m]
//   1 bins:   the task's frame from all parts (minima and maxima: every CTA gets the same), the
//             chunk binned per warp, the warps merged    -> bins[t][m]
//   2 choose: all CTAs' bins merged (counts add, bounds are minima and maxima: exact), the split
//             chosen as the one-CTA builder chooses it (every CTA gets the same), the chunk's lefts
//             counted                                    -> left[t][m]; CTA m = 0: node box, best[t]
//   3 scatter: the chunk partitioned stably into tmp, its lefts after the lefts of the chunks (and
//             warps) before it
//   4 finish: tmp back into order; CTA m = 0 emits the children as k_sah_level does
// The tree is the one-CTA builder's: same bounds, bins, costs and candidate order, same stable
// partition.
constexpr int kSplitCtas = 32;
constexpr int kSahSplitLevels = 3;
constexpr uint32_t kSahSplitMin = 32768;
constexpr int kBinInts = 3 * kSahBins * 7;  // counts, then lo xyz, then hi xyz per (axis, bin)

struct SplitScratch {
    float* part;  // [4][kSplitCtas][12]
    int* bins;    // [4][kSplitCtas][kBinInts]
    uint32_t* left;  // [4][kSplitCtas]
    int* best;       // [4]
};

__device__ __forceinline__ int bin_slot_cnt(int a, int bn) { return a * kSahBins + bn; }
__device__ __forceinline__ int bin_slot_lo(int a, int bn, int c) { return 3 * kSahBins + (a * kSahBins + bn) * 3 + c; }
__device__ __forceinline__ int bin_slot_hi(int a, int bn, int c) { return 3 * kSahBins + 9 * kSahBins + (a * kSahBins + bn) * 3 + c; }

// the task's frame (box, centroid origin and bin scale) from the parts of all its CTAs, a part a lane
static_assert(kSplitCtas == 32, "a lane takes a part");
__device__ __forceinline__ void split_frame(const float* part, int lane, float* lo, float* hi, float* clo, float* scale) {
    float v[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) v[k] = part[12 * lane + k];
    sah_bounds_warp(v);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = v[a];
        hi[a] = v[3 + a];
        clo[a] = v[6 + a];
        scale[a] = sah_scale(v[6 + a], v[9 + a]);
    }
}

__global__ void __launch_bounds__(kSahWarps * 32, 1) k_sah_init(uint32_t n, uint32_t* __restrict__ order, uint32_t* __restrict__ left,
                                                                uint32_t* __restrict__ right, uint2* __restrict__ tasksA) {
    chain_wait();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        order[i] = i;
        if (i + 1 < n) left[i] = right[i] = kLeaf;  // every node starts as (leaf 0, leaf 0)
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) tasksA[0] = make_uint2(0u, n);
}

__global__ void __launch_bounds__(kSahWarps * 32, 1) k_sah_split(const float* __restrict__ boxes, uint32_t* __restrict__ order,
                                                                 uint32_t* __restrict__ tmp, uint32_t* __restrict__ left,
                                                                 uint32_t* __restrict__ right, float* __restrict__ nodeBoxes,
                                                                 uint2* __restrict__ tasksA, uint2* __restrict__ tasksB,
                                                                 uint32_t* __restrict__ lvCount, SplitScratch X, int level, int phase,
                                                                 uint32_t medianLevel) {
    chain_wait();
    __shared__ int sb[kSahWarps][kBinInts];  // per-warp bins; merged bins in sb[0]
    __shared__ float red[kSahWarps][12];
    __shared__ uint32_t wl[kSahWarps];
    __shared__ int sBest;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t t = blockIdx.x / kSplitCtas, m = blockIdx.x % kSplitCtas;
    const uint32_t count = level == 0 ? 1u : lvCount[level];
    if (t >= count) return;
    uint2* cur = (level & 1) ? tasksB : tasksA;
    uint2* nxt = (level & 1) ? tasksA : tasksB;
    uint32_t base = level == 0 ? 0u : 1u;
    for (int k = 1; k < level; ++k) base += lvCount[k];
    const uint2 tk = cur[t];
    const uint32_t b = tk.x, e = tk.y, node = base + t;
    const uint32_t chunk = (e - b + kSplitCtas - 1) / kSplitCtas;
    const uint32_t cb = min(e, b + m * chunk), ce = min(e, cb + chunk);
    float* part = X.part + (size_t)t * kSplitCtas * 12;
    int* binsT = X.bins + (size_t)t * kSplitCtas * kBinInts;
    uint32_t* leftT = X.left + (size_t)t * kSplitCtas;
    const bool median = (uint32_t)level >= medianLevel;
    if (phase == 0) {  // the chunk's box and centroid box
        float v[12];
        for (int a = 0; a < 3; ++a) {
            v[a] = v[6 + a] = INFINITY;
            v[3 + a] = v[9 + a] = -INFINITY;
        }
        for (uint32_t i = cb + threadIdx.x; i < ce; i += blockDim.x) {
            const float* bx = boxes + 6 * (size_t)order[i];
            for (int a = 0; a < 3; ++a) {
                v[a] = fminf(v[a], bx[a]);
                v[3 + a] = fmaxf(v[3 + a], bx[3 + a]);
                const float c = 0.5f * (bx[a] + bx[3 + a]);
                v[6 + a] = fminf(v[6 + a], c);
                v[9 + a] = fmaxf(v[9 + a], c);
            }
        }
        for (int off = 16; off > 0; off >>= 1)
            for (int k = 0; k < 12; ++k) {
                const float o = __shfl_xor_sync(0xFFFFFFFFu, v[k], off);
                v[k] = (k % 6) < 3 ? fminf(v[k], o) : fmaxf(v[k], o);
            }
        if (lane == 0)
            for (int k = 0; k < 12; ++k) red[warp][k] = v[k];
        __syncthreads();
        if (threadIdx.x < 12) {
            const int k = threadIdx.x;
            float r = red[0][k];
            for (int w = 1; w < kSahWarps; ++w) r = (k % 6) < 3 ? fminf(r, red[w][k]) : fmaxf(r, red[w][k]);
            part[12 * m + k] = r;
        }
        return;
    }
    float lo[3], hi[3], clo[3], scale[3];
    split_frame(part, lane, lo, hi, clo, scale);
    auto bin_of = [&](const float* bx, int a) {
        const float c = 0.5f * (bx[a] + bx[3 + a]);
        return max(0, min((int)((c - clo[a]) * scale[a]), kSahBins - 1));
    };
    if (phase == 1) {  // the chunk binned per warp, the warps merged into this CTA's bins
        if (median) return;
        for (int k = lane; k < 3 * kSahBins; k += 32) {
            const int a = k / kSahBins, bn = k % kSahBins;
            sb[warp][bin_slot_cnt(a, bn)] = 0;
            for (int c = 0; c < 3; ++c) {
                sb[warp][bin_slot_lo(a, bn, c)] = ord_float(INFINITY);
                sb[warp][bin_slot_hi(a, bn, c)] = ord_float(-INFINITY);
            }
        }
        __syncwarp();
        for (uint32_t i0 = cb + warp * 32; i0 < ce; i0 += blockDim.x) {
            const bool valid = i0 + lane < ce;
            float bx[6];
            const uint32_t prim = valid ? order[i0 + lane] : 0u;
            for (int c = 0; c < 6; ++c) bx[c] = valid ? boxes[6 * (size_t)prim + c] : 0.0f;
            for (int a = 0; a < 3; ++a)
                if (scale[a] > 0.0f)
                    sah_bin(valid, bin_of(bx, a), bx, &sb[warp][bin_slot_cnt(a, 0)], reinterpret_cast<int(*)[3]>(&sb[warp][bin_slot_lo(a, 0, 0)]),
                            reinterpret_cast<int(*)[3]>(&sb[warp][bin_slot_hi(a, 0, 0)]), lane);
        }
        __syncthreads();
        for (int k = threadIdx.x; k < kBinInts; k += blockDim.x) {
            int r = sb[0][k];
#pragma unroll 8
            for (int w = 1; w < kSahWarps; ++w)
                r = k < 3 * kSahBins ? r + sb[w][k] : (k < 3 * kSahBins + 9 * kSahBins ? min(r, sb[w][k]) : max(r, sb[w][k]));
            binsT[(size_t)m * kBinInts + k] = r;
        }
        return;
    }
    if (phase == 2) {  // every CTA's bins merged, the split chosen, the chunk's lefts counted
        if (!median)
            for (int k = threadIdx.x; k < kBinInts; k += blockDim.x) {
                int r = binsT[k];
#pragma unroll 8
                for (int c = 1; c < kSplitCtas; ++c) {
                    const int o = binsT[(size_t)c * kBinInts + k];
                    r = k < 3 * kSahBins ? r + o : (k < 3 * kSahBins + 9 * kSahBins ? min(r, o) : max(r, o));
                }
                sb[0][k] = r;
            }
        __syncthreads();
        if (warp == 0) {  // cheapest surface-area cost, ties to the lowest candidate
            int bestCand = -1;
            if (!median) {
                bestCand = sah_best_split(scale, lane, [&](int a, int k) { return sb[0][bin_slot_cnt(a, k)]; },
                                          [&](int a, int k, int c) { return sb[0][bin_slot_lo(a, k, c)]; },
                                          [&](int a, int k, int c) { return sb[0][bin_slot_hi(a, k, c)]; });
            }
            if (lane == 0) sBest = bestCand;
        }
        __syncthreads();
        const int best = sBest;
        if (m == 0 && threadIdx.x == 0) {
            X.best[t] = best;
            for (int a = 0; a < 3; ++a) {
                nodeBoxes[6 * (size_t)node + a] = lo[a];
                nodeBoxes[6 * (size_t)node + 3 + a] = hi[a];
            }
        }
        if (best < 0) return;
        const int sa = best / (kSahBins - 1), sp = best % (kSahBins - 1) + 1;
        uint32_t nl = 0;
        for (uint32_t i = cb + threadIdx.x; i < ce; i += blockDim.x) nl += bin_of(boxes + 6 * (size_t)order[i], sa) < sp;
        for (int off = 16; off > 0; off >>= 1) nl += __shfl_xor_sync(0xFFFFFFFFu, nl, off);
        if (lane == 0) wl[warp] = nl;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t s = 0;
            for (int w = 0; w < kSahWarps; ++w) s += wl[w];
            leftT[m] = s;
        }
        return;
    }
    const int best = X.best[t];
    if (phase == 3) {  // stable partition of the chunk: warp sub-chunks in order, lanes in order
        if (best < 0) return;
        const int sa = best / (kSahBins - 1), sp = best % (kSahBins - 1) + 1;
        uint32_t nlTotal = 0, before = 0;
        for (uint32_t c = 0; c < (uint32_t)kSplitCtas; ++c) {
            const uint32_t x = leftT[c];
            if (c < m) before += x;
            nlTotal += x;
        }
        const uint32_t sub = (ce - cb + kSahWarps - 1) / kSahWarps;
        const uint32_t wb = min(ce, cb + warp * sub), we = min(ce, wb + sub);
        uint32_t nl = 0;
        for (uint32_t i0 = wb; i0 < we; i0 += 32) {
            const uint32_t i = i0 + lane;
            nl += __popc(__ballot_sync(0xFFFFFFFFu, i < we && bin_of(boxes + 6 * (size_t)order[i], sa) < sp));
        }
        if (lane == 0) wl[warp] = nl;
        __syncthreads();
        uint32_t wBefore = 0;
        for (int w = 0; w < warp; ++w) wBefore += wl[w];
        const uint32_t lefts = before + wBefore;  // lefts ahead of this warp's sub-chunk in the task
        uint32_t lb = b + lefts, rb = b + nlTotal + ((wb - b) - lefts);
        for (uint32_t i0 = wb; i0 < we; i0 += 32) {
            const uint32_t i = i0 + lane;
            const bool valid = i < we;
            const uint32_t prim = valid ? order[i] : 0u;
            const bool isL = valid && bin_of(boxes + 6 * (size_t)prim, sa) < sp;
            const unsigned lm = __ballot_sync(0xFFFFFFFFu, isL), rm = __ballot_sync(0xFFFFFFFFu, valid && !isL);
            const unsigned below = (1u << lane) - 1u;
            if (isL) tmp[lb + __popc(lm & below)] = prim;
            else if (valid) tmp[rb + __popc(rm & below)] = prim;
            lb += __popc(lm);
            rb += __popc(rm);
        }
        return;
    }
    // phase 4: tmp back into order, the children
    if (best >= 0)
        for (uint32_t i = cb + threadIdx.x; i < ce; i += blockDim.x) order[i] = tmp[i];
    if (m == 0 && threadIdx.x == 0) {
        uint32_t nlTotal = 0;
        for (uint32_t c = 0; c < (uint32_t)kSplitCtas; ++c) nlTotal += leftT[c];
        const uint32_t mid = best >= 0 ? b + nlTotal : b + (e - b) / 2;
        const uint32_t rb0[2] = {b, mid}, re0[2] = {mid, e};
        uint32_t ref[2];
        for (int c = 0; c < 2; ++c) {
            if (re0[c] - rb0[c] == 1) {
                ref[c] = kLeaf | rb0[c];
            } else {
                const uint32_t idx = atomicAdd(&lvCount[level + 1], 1u);
                nxt[idx] = make_uint2(rb0[c], re0[c]);
                ref[c] = base + count + idx;
            }
        }
        left[node] = ref[0];
        right[node] = ref[1];
    }
}

// The rest of the top of the tree: one CTA, level by level from level kSahParallelLevels on (levels
// with fewer tasks than warps spread each task over a group of warps), until a level has `handoff`
// tasks or more.  That level's tasks go to the queue Q, whose slots are the node ids from baseCur
// on, and k_sah_tasks finishes the tree.
// SMALL: all levels from the root, for builds of up to kSahSmall primitives (a TLAS), whose boxes, order and
// partition buffer the CTA keeps in shared memory.
constexpr size_t kSahSmallSmem = kSahSmall * (24 + 4 + 4);
template <bool SMALL>
__global__ void __launch_bounds__(kSahWarps * 32, 1) k_sah_build(const float* __restrict__ boxesIn, uint32_t n, uint32_t* orderOut,
                                                                 uint32_t* tmpBuf, uint32_t* __restrict__ left,
                                                                 uint32_t* __restrict__ right, float* __restrict__ nodeBoxes,
                                                                 uint2* __restrict__ tasksA, uint2* __restrict__ tasksB,
                                                                 uint32_t firstLevel, uint32_t medianLevel, uint32_t handoff, SahQueue Q,
                                                                 const uint32_t* __restrict__ lvCount, uint32_t* __restrict__ levelsOut) {
    chain_wait();
    constexpr int kRounds = SMALL ? 1 : 4;
    extern __shared__ float sahSmem[];
    const float* boxes = SMALL ? sahSmem : boxesIn;
    uint32_t* order = SMALL ? reinterpret_cast<uint32_t*>(sahSmem) + 6 * kSahSmall : orderOut;
    uint32_t* tmp = SMALL ? reinterpret_cast<uint32_t*>(sahSmem) + 7 * kSahSmall : tmpBuf;
    __shared__ int bLo[kSahWarps][3][kSahBins][3], bHi[kSahWarps][3][kSahBins][3];
    __shared__ int bCnt[kSahWarps][3][kSahBins];
    __shared__ uint32_t nCur, nNext, baseCur, baseNext, levels;
    // levels with fewer tasks than warps: per-warp partial bounds, per-task centroid frame and split,
    // per-warp left counts
    __shared__ float gPart[kSahWarps][12];
    __shared__ int tBest[kSahWarps];
    __shared__ uint32_t wLeft[kSahWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {  // the state after the level kernels (their counts; level 0: the root)
        uint32_t base = 0, lv = 0;
        nCur = 1;
        while (lv < firstLevel && nCur) {
            base += nCur;
            nCur = lvCount[++lv];
        }
        nNext = 0;
        baseCur = base;          // node id of the current level's first task
        baseNext = base + nCur;  // node id of the next level's first task
        levels = lv;
    }
    __syncthreads();
    uint2* cur = (firstLevel & 1) ? tasksB : tasksA;
    uint2* nxt = (firstLevel & 1) ? tasksA : tasksB;
    if (SMALL) {  // no level kernels: the preparations of level 0
        for (uint32_t i = threadIdx.x; i < 6 * n; i += blockDim.x) sahSmem[i] = boxesIn[i];
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) order[i] = i;
        for (uint32_t i = threadIdx.x; i + 1 < n; i += blockDim.x) left[i] = right[i] = kLeaf;
        if (threadIdx.x == 0) cur[0] = make_uint2(0u, n);
        __syncthreads();
    }
    for (;;) {
        const uint32_t count = nCur;
        if (count == 0) break;
        if (count >= handoff) {  // the rest of the tree on every SM
            for (uint32_t t = threadIdx.x; t < count; t += blockDim.x) {
                const uint2 tk = cur[t];
                Q.tasks[t] = make_uint4(tk.x, tk.y, baseCur + t, levels);
                Q.ready[t] = 1u;  // the task kernel starts after this one
            }
            if (threadIdx.x == 0) {
                Q.ctr[1] = count;
                Q.ctr[2] = baseCur;
                Q.ctr[3] = n - 1 - baseCur;
                Q.ctr[4] = n - 1;           // ids from here down go to the subtrees
                Q.ctr[5] = n - 1 - baseCur;  // nodes not yet made
            }
            break;
        }
        const bool median = levels >= medianLevel;  // from here on ranges are halved: the depth stays bounded
        if (count < (uint32_t)kSahWarps) {
            sah_level_grouped<kRounds>(boxes, order, tmp, left, right, nodeBoxes, cur, nxt, count, median, baseCur, baseNext, nNext, bLo, bHi,
                              bCnt, gPart, tBest, wLeft);
        } else
        for (uint32_t t = warp; t < count; t += kSahWarps) {
            const uint2 tk = cur[t];
            const uint32_t b = tk.x, e = tk.y, node = baseCur + t;
            sah_task_warp<false, kRounds>(boxes, order, tmp, nodeBoxes, b, e, node, median, bLo[warp], bHi[warp], bCnt[warp], lane,
                                 [&](uint32_t mid) {  // single primitives become leaf refs, the rest next-level tasks
                                     if (lane != 0) return;
                                     const uint32_t rb0[2] = {b, mid}, re0[2] = {mid, e};
                                     uint32_t ref[2];
                                     for (int c = 0; c < 2; ++c) {
                                         if (re0[c] - rb0[c] == 1) {
                                             ref[c] = kLeaf | rb0[c];
                                         } else {
                                             const uint32_t idx = atomicAdd(&nNext, 1u);
                                             nxt[idx] = make_uint2(rb0[c], re0[c]);
                                             ref[c] = baseNext + idx;
                                         }
                                     }
                                     left[node] = ref[0];
                                     right[node] = ref[1];
                                 });
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            baseCur = baseNext;
            baseNext += nNext;
            nCur = nNext;
            nNext = 0;
            ++levels;
        }
        uint2* sw = cur;
        cur = nxt;
        nxt = sw;
        __syncthreads();
    }
    if (SMALL)
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) orderOut[i] = order[i];
    if (threadIdx.x == 0 && levelsOut) *levelsOut = levels;
}

// The rest of the tree on every SM: a warp claims the next queue slot, waits (bounded) until the
// slot's task is published, splits it as k_sah_build does, and publishes its children's tasks in
// the next free slots (node id = first node id of the queue + slot).  A task of at most `subtree` primitives is
// finished by its warp, whose node ids come from the upper end; a warp whose slot will not be
// used sees that every node is made, and is done.  A slot's task is published by the warp that split
// its parent, which claimed an earlier slot and runs, so every wait ends; a wait that still runs out
// sets *status to 2 and leaves that subtree as prepared (valid refs, unset boxes).
// A task costs its warp some 9 us of waits on L2 (claim, publication, order, boxes, children), which
// small ones would pay per node: 191 us for 61442 triangles (601 us with every node a task).
__global__ void __launch_bounds__(kSahTaskWarps * 32, 3) k_sah_tasks(const float* __restrict__ boxes, uint32_t* __restrict__ order,
                                                                  uint32_t* __restrict__ tmp, uint32_t* __restrict__ left,
                                                                  uint32_t* __restrict__ right, float* __restrict__ nodeBoxes,
                                                                  SahQueue Q, uint32_t medianLevel, uint32_t subtree, uint32_t* __restrict__ levelsOut,
                                                                  int* __restrict__ status, uint32_t waitLimit) {
    chain_wait();
    __shared__ int bLo[kSahTaskWarps][3][kSahBins][3], bHi[kSahTaskWarps][3][kSahBins][3];
    __shared__ int bCnt[kSahTaskWarps][3][kSahBins];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t total = Q.ctr[3], base = Q.ctr[2];  // written by k_sah_build
    uint32_t deepest = 0;
    for (;;) {
        uint32_t slot = 0, ok = 1;
        if (lane == 0) {
            slot = atomicAdd(Q.ctr, 1u);
            if (slot < total) {
                for (uint32_t spins = 0; ld_relaxed(Q.ready + slot) == 0; ++spins) {
                    if (ld_relaxed(Q.ctr + 5) == 0) {  // every node is made: no task is left for the slot
                        slot = total;
                        break;
                    }
                    if (spins >= waitLimit) {
                        ok = 0;
                        if (status) atomicExch(status, 2);
                        break;
                    }
                    __nanosleep(128);
                }
            }
        }
        slot = __shfl_sync(0xFFFFFFFFu, slot, 0);
        ok = __shfl_sync(0xFFFFFFFFu, ok, 0);
        if (slot >= total || !ok) break;
        __threadfence();  // after the publication: the task and its order[] range
        const uint4 tk = __ldcg(Q.tasks + slot);
        const uint32_t b = tk.x, e = tk.y, node = tk.z, level = tk.w;
        if (e - b <= subtree) {
            uint32_t first = 0;
            if (lane == 0 && e - b > 2) first = atomicSub(Q.ctr + 4, e - b - 2) - (e - b - 2);
            first = __shfl_sync(0xFFFFFFFFu, first, 0);
            deepest = max(deepest, sah_subtree_warp(boxes, order, left, right, nodeBoxes, b, e, node, first, level, medianLevel, bLo[warp],
                                                    bHi[warp], bCnt[warp], lane));
            if (lane == 0) atomicSub(Q.ctr + 5, e - b - 1);
            continue;
        }
        deepest = max(deepest, level + 1);
        sah_task_warp<true, 4>(boxes, order, tmp, nodeBoxes, b, e, node, level >= medianLevel, bLo[warp], bHi[warp], bCnt[warp], lane,
                            [&](uint32_t mid) {
                                const uint32_t rb0[2] = {b, mid}, re0[2] = {mid, e};
                                uint32_t ref[2] = {0u, 0u};
                                if (lane == 0) {
                                    const uint32_t inner = (mid - b > 1 ? 1u : 0u) + (e - mid > 1 ? 1u : 0u);
                                    uint32_t q = inner ? atomicAdd(Q.ctr + 1, inner) : 0u;
                                    for (int c = 0; c < 2; ++c) {
                                        if (re0[c] - rb0[c] == 1) {
                                            ref[c] = kLeaf | rb0[c];
                                        } else {
                                            ref[c] = base + q;
                                            Q.tasks[q] = make_uint4(rb0[c], re0[c], base + q, level + 1);
                                            ++q;
                                        }
                                    }
                                    left[node] = ref[0];
                                    right[node] = ref[1];
                                    atomicSub(Q.ctr + 5, 1u);
                                }
                                __threadfence();  // every lane's order[] writes and the new tasks, then the publication
                                __syncwarp();
                                if (lane == 0)
                                    for (int c = 0; c < 2; ++c)
                                        if (!(ref[c] & kLeaf)) st_relaxed(Q.ready + (ref[c] - base), 1u);
                            });
    }
    if (lane == 0 && levelsOut && deepest) atomicMax(levelsOut, deepest);
}

// parents of a BVH2 in the LBVH layout (internal node i at parents[i], the leaf at sorted position k
// at parents[n - 1 + k], the root's 0xFFFFFFFF), which the bottom-up refit walks
__global__ void k_parents(const uint32_t* __restrict__ left, const uint32_t* __restrict__ right, uint32_t n,
                          uint32_t* __restrict__ parents) {
    chain_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i + 1 >= n) return;
    const uint32_t L = left[i], R = right[i];
    for (const uint32_t c : {L, R}) {  // child refs of a finished tree are in range; anything else is skipped
        const uint32_t slot = (c & kLeaf) ? (n - 1) + (c & ~kLeaf) : c;
        if (((c & kLeaf) && (c & ~kLeaf) < n) || (!(c & kLeaf) && c > 0 && c + 1 < n)) parents[slot] = i;
    }
    if (i == 0) parents[0] = 0xFFFFFFFFu;
}

// ---- instances ----------------------------------------------------------------------------------
__global__ void k_instances(const rg_instance* __restrict__ in, uint32_t n, const DevBlas* __restrict__ blas, uint32_t nblas,
                            DevInstance* __restrict__ out, float* __restrict__ boxes, bool checkOffsets, uint32_t nm) {
    chain_wait();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    rg_instance I = in[i];
    const float* m = &I.transform[0][0];
    float a00 = m[0], a01 = m[1], a02 = m[2], t0 = m[3];
    float a10 = m[4], a11 = m[5], a12 = m[6], t1 = m[7];
    float a20 = m[8], a21 = m[9], a22 = m[10], t2 = m[11];
    float c00 = a11 * a22 - a12 * a21, c01 = a02 * a21 - a01 * a22, c02 = a01 * a12 - a02 * a11;
    float c10 = a12 * a20 - a10 * a22, c11 = a00 * a22 - a02 * a20, c12 = a02 * a10 - a00 * a12;
    float c20 = a10 * a21 - a11 * a20, c21 = a01 * a20 - a00 * a21, c22 = a00 * a11 - a01 * a10;
    float det = (a00 * c00 + a01 * c10) + a02 * c20;
    bool ok = (det != 0.0f) && isfinite(det) && I.blas < nblas && (I.mask & 0xFFu) != 0u;
    if (ok && checkOffsets && blas[I.blas].n > 0) {
        const DevBlas& B = blas[I.blas];
        ok = I.vertexBufferOffset == B.vOff && I.indexBufferOffset == B.iOff && (uint64_t)I.materialBufferOffset + B.maxMat < nm;
    }
    float id = ok ? 1.0f / det : 0.0f;
    float r[9] = {c00 * id, c01 * id, c02 * id, c10 * id, c11 * id, c12 * id, c20 * id, c21 * id, c22 * id};
    DevInstance d;
    for (int row = 0; row < 3; ++row) {
        float tr = -((r[3 * row + 0] * t0 + r[3 * row + 1] * t1) + r[3 * row + 2] * t2);
        d.inv[row] = make_float4(r[3 * row + 0], r[3 * row + 1], r[3 * row + 2], tr);
        d.m[row] = make_float4(m[4 * row + 0], m[4 * row + 1], m[4 * row + 2], m[4 * row + 3]);
    }
    d.blas = ok ? I.blas : 0u;
    d.valid = ok ? 1u : 0u;
    d.vOff = I.vertexBufferOffset;
    d.iOff = I.indexBufferOffset;
    d.mOff = I.materialBufferOffset;
    d.mask = I.mask;
    d.pad0 = d.pad1 = 0;
    out[i] = d;
    float* o = boxes + 6 * (size_t)i;
    if (ok && blas[I.blas].n > 0) {
        const float* rb = blas[I.blas].root;
        for (int row = 0; row < 3; ++row) {
            float lo = m[4 * row + 3], hi = m[4 * row + 3];
            for (int j = 0; j < 3; ++j) {
                float e = m[4 * row + j] * rb[j], f = m[4 * row + j] * rb[3 + j];
                lo = lo + fminf(e, f);
                hi = hi + fmaxf(e, f);
            }
            o[row] = lo;
            o[3 + row] = hi;
        }
    } else {
        o[0] = o[1] = o[2] = INFINITY;
        o[3] = o[4] = o[5] = -INFINITY;
    }
}

inline uint32_t blocks(uint32_t n, uint32_t t) { return (n + t - 1) / t; }

}  // namespace

cudaError_t tri_boxes(const rg_vertex* v, const uint32_t* idx, uint32_t vOff, uint32_t iOff, uint32_t n, float* boxes, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    launch_chain(k_tri_boxes, blocks(n, 256), 256, 0, s, v, idx, vOff, iOff, n, boxes);
    count_launch();
    return cudaGetLastError();
}

cudaError_t tri_records(const rg_vertex* v, const uint32_t* idx, uint32_t vOff, uint32_t iOff, const uint32_t* order, uint32_t n,
                        float4* tris, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    launch_chain(k_tri_records, blocks(n, 256), 256, 0, s, v, idx, vOff, iOff, order, n, tris);
    count_launch();
    return cudaGetLastError();
}

cudaError_t inst_records(const uint32_t* order, uint32_t n, const DevInstance* inst, const DevBlas* blas, InstRec* out,
                         cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    launch_chain(k_inst_records, blocks(n, 128), 128, 0, s, order, n, inst, blas, out);
    count_launch();
    return cudaGetLastError();
}

cudaError_t setup_instances(const rg_instance* in, uint32_t n, const DevBlas* blas, uint32_t nblas, DevInstance* out, float* boxes,
                            bool checkOffsets, uint32_t nm, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    launch_chain(k_instances, blocks(n, 128), 128, 0, s, in, n, blas, nblas, out, boxes, checkOffsets, nm);
    count_launch();
    return cudaGetLastError();
}

cudaError_t lbvh_refit(const LbvhBuffers& b, cudaStream_t s) {
    if (b.n <= 1) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(b.flags, 0, sizeof(uint32_t) * (b.n - 1), s);
    if (e != cudaSuccess) return e;
    launch_chain(k_bottom_up, blocks(b.n, 256), 256, 0, s, b.primBoxes, b.order, b.n, b.left, b.right, b.parents, b.flags, b.nodeBoxes);
    count_launch();
    return cudaGetLastError();
}

static int sah_task_grid() {  // persistent grid of k_sah_tasks (every resident block)
    // (per device and process; the shared memory of the small build is asked for on every device)
    if (cudaFuncSetAttribute((const void*)k_sah_build<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSahSmallSmem) != cudaSuccess)
        return 0;
    static std::atomic<int> grid{0};
    int g = grid.load(std::memory_order_acquire);
    if (g) return g;
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sah_tasks, kSahTaskWarps * 32, 0) != cudaSuccess)
        return 0;
    g = sms * max(per, 1);
    grid.store(g, std::memory_order_release);
    return g;
}

cudaError_t sah_build(const LbvhBuffers& b, bool parents, uint32_t* levels, cudaStream_t s) {
    if (b.n <= 1) return cudaSuccess;
    if (!b.sahQueue) return cudaErrorInvalidValue;
    const int grid = sah_task_grid();
    if (!grid) return cudaErrorUnknown;
    SahQueue Q;
    Q.tasks = reinterpret_cast<uint4*>(b.sahQueue);
    Q.ready = reinterpret_cast<uint32_t*>(b.sahQueue + 16 * (size_t)b.n);
    Q.ctr = Q.ready + b.n;
    uint32_t* lvCount = Q.ctr + 8;  // tasks per level of the level kernels
    cudaError_t e = cudaMemsetAsync(Q.ready, 0, 4 * (size_t)b.n + 96, s);  // ready words and counters
    if (e != cudaSuccess) return e;
    // scratch: the sort buffers (n words each); at most n / 2 tasks per level, 2 words each
    uint2* tasksA = reinterpret_cast<uint2*>(b.valsA);
    uint2* tasksB = reinterpret_cast<uint2*>(b.valsB);
    int lv0 = 0;
    if (b.n >= kSahSplitMin) {  // the first levels with each task over kSplitCtas CTAs
        SplitScratch X;  // in the queue's task records, which k_sah_build fills only later
        X.part = reinterpret_cast<float*>(Q.tasks);
        X.bins = reinterpret_cast<int*>(X.part + 4 * kSplitCtas * 12);
        X.left = reinterpret_cast<uint32_t*>(X.bins + 4 * kSplitCtas * kBinInts);
        X.best = reinterpret_cast<int*>(X.left + 4 * kSplitCtas);
        launch_chain(k_sah_init, 2 * kSplitCtas, kSahWarps * 32, 0, s, b.n, b.order, b.left, b.right, tasksA);
        count_launch();
        for (; lv0 < kSahSplitLevels; ++lv0)
            for (int ph = 0; ph < 5; ++ph) {
                launch_chain(k_sah_split, (1u << lv0) * kSplitCtas, kSahWarps * 32, 0, s, b.primBoxes, b.order, b.keysA, b.left, b.right,
                                                                                 b.nodeBoxes, tasksA, tasksB, lvCount, X, lv0, ph,
                                                                                 kSahMedianLevel);
                count_launch();
            }
    }
    const bool small = b.n <= kSahSmall;
    int levelKernels = 0;  // until a level's tasks hold some kSahTask primitives
    while (!small && levelKernels < kSahParallelLevels && (b.n >> levelKernels) > kSahTask) ++levelKernels;
    for (int lv = lv0; lv < levelKernels; ++lv)
        launch_chain(k_sah_level, 1u << lv, kSahWarps * 32, 0, s, b.primBoxes, b.n, b.order, b.keysA, b.left, b.right, b.nodeBoxes, tasksA,
                                                         tasksB, lvCount, lv, kSahMedianLevel);
    if (small)
        launch_chain(k_sah_build<true>, 1, kSahWarps * 32, kSahSmallSmem, s, b.primBoxes, b.n, b.order, b.keysA, b.left, b.right, b.nodeBoxes, tasksA,
                                                                   tasksB, 0u, kSahMedianLevel, kSahSmallHandoff, Q, lvCount, levels);
    else
        launch_chain(k_sah_build<false>, 1, kSahWarps * 32, 0, s, b.primBoxes, b.n, b.order, b.keysA, b.left, b.right, b.nodeBoxes, tasksA, tasksB,
                                                        (uint32_t)levelKernels, kSahMedianLevel, kSahHandoff, Q, lvCount, levels);
    // polls of an unpublished task before a warp gives up (RG_SAH_WAIT_LIMIT overrides; 0 makes
    // the first unpublished slot end the wait, which tests use to check the reported status)
    uint32_t waitLimit = kSahWaitLimit;
    if (const char* env = getenv("RG_SAH_WAIT_LIMIT")) waitLimit = (uint32_t)strtoul(env, nullptr, 10);
    launch_chain(k_sah_tasks, grid, kSahTaskWarps * 32, 0, s, b.primBoxes, b.order, b.keysA, b.left, b.right, b.nodeBoxes, Q, kSahMedianLevel,
                                                     small ? kSahSubtreeSmall : kSahSubtree, levels, b.status, waitLimit);
    count_launch(levelKernels - lv0 + 2);
    if (parents) {
        launch_chain(k_parents, blocks(b.n - 1, 256), 256, 0, s, b.left, b.right, b.n, b.parents);
        count_launch();
    }
    return cudaGetLastError();
}

cudaError_t wide_records(const LbvhBuffers& b, WideNode* out, cudaStream_t s) {
    if (b.n <= 1) return cudaSuccess;
    launch_chain(k_wide_records, blocks(b.n - 1, 256), 256, 0, s, b.primBoxes, b.order, b.n, b.left, b.right, b.nodeBoxes, out);
    count_launch();
    return cudaGetLastError();
}

cudaError_t lbvh_build(const LbvhBuffers& b, cudaStream_t s) {
    const uint32_t n = b.n;
    if (n == 0) return cudaSuccess;
    if (n > kStatCount) return cudaErrorInvalidValue;  // the sort's status words count in 30 bits
    const uint32_t limit = cluster_limit();
    if (n <= limit * kClusterThreads * kClusterRounds) {  // one cluster holds the keys
        // as many blocks as there are keys for, so that a thread ranks few keys one after another
        uint32_t size = 1, rounds = 1;
        while (size < limit && size * kClusterThreads < n) size *= 2;
        while (size * kClusterThreads * rounds < n) rounds *= 2;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(size);
        cfg.blockDim = dim3(kClusterThreads);
        cfg.dynamicSmemBytes = sizeof(ClusterSort);
        cfg.stream = s;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim = {size, 1, 1};
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_chain
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 2;
        const auto kernel = rounds == 1 ? k_sort_cluster<1> : rounds == 2 ? k_sort_cluster<2> : k_sort_cluster<4>;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, (const float*)b.primBoxes, n, b.morton, b.keysA, b.order, b.flags,
                                                 reinterpret_cast<uint32_t*>(b.nodeBoxes));
        if (e != cudaSuccess) return e;
        count_launch();
    } else {
        const uint32_t nTiles = (uint32_t)sort_tiles(n);
        cudaError_t e = cudaMemsetAsync(b.sortState, 0, 4 * sort_state_words(n), s);
        if (e != cudaSuccess) return e;
        uint32_t* bounds = b.sortState + kSortBounds;
        uint32_t gb = min(blocks(n, 256), 1024u);
        launch_chain(k_centroid_bounds, gb, 256, 0, s, b.primBoxes, n, bounds);
        launch_chain(k_morton, min(blocks(n, 256), kMortonMaxBlocks), 256, 0, s, b.primBoxes, n, bounds, b.morton, b.keysA, b.valsA, b.valsB, b.order,
                                                                       b.flags, reinterpret_cast<uint32_t*>(b.nodeBoxes), b.sortState);
        count_launch(2);
        // polls of an unpublished predecessor tile before a look-back counts that tile itself
        // (RG_SORT_SPIN_LIMIT overrides; 0 makes every such look-back count, which tests use)
        uint32_t spinLimit = 1u << 16;
        if (const char* env = getenv("RG_SORT_SPIN_LIMIT")) spinLimit = (uint32_t)strtoul(env, nullptr, 10);
        const uint32_t *kin = b.keysA, *vin = b.valsA;  // keys A -> B -> A -> B -> A, values A -> B -> A -> B -> order
        uint32_t* kout[4] = {b.keysB, b.keysA, b.keysB, b.keysA};
        uint32_t* vout[4] = {b.valsB, b.valsA, b.valsB, b.order};
        for (int pass = 0; pass < 4; ++pass) {
            launch_chain(k_sort_onesweep, nTiles, kSortThreads, 0, s, kin, vin, kout[pass], vout[pass], n, pass, b.sortState, nTiles, spinLimit);
            count_launch();
            kin = kout[pass];
            vin = vout[pass];
        }
    }
    if (n == 1) return cudaGetLastError();
    // (RG_HIER_POLL_LIMIT=0: no sibling's box is waited for, which tests use)
    const char* env = getenv("RG_HIER_POLL_LIMIT");
    launch_chain(env && strtoul(env, nullptr, 10) == 0 ? k_hierarchy<true> : k_hierarchy<false>, blocks(n, kHierLeaves), kHierLeaves, 0, s, b.keysA,
                 b.order, b.primBoxes, n, b.left, b.right, b.parents, b.flags, b.nodeBoxes);
    count_launch();
    return cudaGetLastError();
}

}  // namespace rg
