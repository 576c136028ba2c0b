// filter.cu -- the learned roughness filter on the 5th-generation tensor cores.
//
// A 5-layer 3x3 convolutional network stands in for the screen-space roughness approximation
// (rough_prepare.comp + 10 x rough_blur_h/v, raytracer.cpp:112-122): from the frame's G-buffers it
// predicts the rough-reflection radiance that the composite (postprocess.comp:28-50) mixes in.
//   layers: 16(12 used) -> 32 -> 64 -> 64 -> 32 -> 16(3 used), ReLU after layers 1-4, the output of
//   layer 1 added to the input of layer 5 (skip), every layer at full resolution.
// Activations are BF16 NHWC, accumulation FP32 in tensor memory.  Each convolution is an implicit
// GEMM over strips of 128 pixels (M): input rows of 130 pixels lie in shared memory as the TMA writes
// them, pixel after pixel, swizzled over a pixel's channels, and a tap's A descriptor starts at the tap's
// pixel: no im2col copy.  Rows in boxes of 16 bytes (8 channels, one plane a box) took 1.3 - 1.5 times as
// long to copy: 0.57 us against 0.40 us a row of 64 channels and SM, and 470 us against 433 us for the
// network at 1080p.  The data
// gradient is the same kernel on transposed, flipped weights; the weight gradient is a GEMM over
// pixels with both operands MN-major (channels contiguous), accumulated in tensor memory per CTA and
// reduced across CTAs in a fixed order (deterministic).
//
// Descriptor conventions (no swizzle): core matrix = 8 rows x 16 bytes; the leading-byte offset is
// the stride between core matrices along K, the stride-byte offset the stride along M / N.
#include <algorithm>
#include <atomic>

#include <cuda.h>
#include <cuda_bf16.h>

#include "rg_internal.cuh"
#include "rg_tma.cuh"

namespace rg {

namespace {

using bf16 = __nv_bfloat16;

// ---- tcgen05 / mbarrier helpers ----------------------------------------------------------------
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// the same with a swizzle whose span is a row of C BF16 channels (32, 64 or 128 bytes), as the TMA writes
// rows of pixels: the 16-byte chunks of a row are permuted by the row's address, so an operand may start
// at any pixel of a row (its start address carries the pixel) and at any 32-byte step inside it.
// K-major (channels are K): sbo = 8 pixels, lbo unused.  MN-major (pixels are K): sbo = 8 pixels, lbo = the
// next C channels.
template <int C>
__device__ __forceinline__ uint64_t umma_desc_rows(uint32_t addr, uint32_t lbo) {
    static_assert(C == 16 || C == 32 || C == 64, "swizzle spans");
    return umma_desc(addr, lbo, 8 * C * 2) | ((uint64_t)(C == 64 ? 2 : C == 32 ? 4 : 6) << 61);
}

// instruction descriptor of tcgen05.mma kind::f16: D F32, A and B BF16, M x N, operand majors
__host__ __device__ constexpr uint32_t umma_idesc(int m, int n, bool aMN, bool bMN) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (aMN ? 1u << 15 : 0u) | (bMN ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols));
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void umma_commit(uint64_t* mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Row-streaming convolution.  A work item is a strip of 128 output pixels x a segment of rows of
// one image; a CTA walks its items down the rows, three output rows (a group) at a time.  Input rows
// (130 pixels: the strip and a 1-pixel halo, zero outside the image) stream through a ring of
// shared-memory slots, each row loaded once per item.  Input row i feeds output rows i+1, i, i-1 through the kernel rows dy = 0, 1, 2, so a group's accumulator is
// a window of three adjacent TMEM blocks and each of its five input rows r-1 .. r+3 feeds it with ONE
// tcgen05.mma per column tap dx and 16-channel step (M = 128 pixels, N = COUT, 2 COUT, 3 COUT, 2 COUT,
// COUT), the B operand stacking the kernel rows' weights.  62 MMAs instead of 108 per 3 rows of a
// 64-channel layer, each issued from fully unrolled code with constant offsets: one issuing thread
// must keep the tensor core fed, so the issue path carries no arithmetic beyond descriptor adds.
// Warp roles (320 threads):
//   warp 0     TMA producer: refills a slot once the MMAs of the last group reading its row completed;
//   warp 1     MMA issuer: group by group into alternating accumulator windows;
//   warps 2-9  epilogue, two warps per TMEM lane quarter (half the channels each): drain a completed
//              window, hand it back, then bias, ReLU, skip add, mask; a lane writes 16 channels of its
//              pixel with one 32-byte store, a whole sector (through a swizzled shared-memory stage and
//              16-byte stores the epilogue took 70 - 90 % of the time of the layers into 32 and 64 channels).
constexpr int kStripPx = 128, kRowW = kStripPx + 2;
// bytes of a ring slot: `pixels` pixels of C channels, rounded up to the period of the widest swizzle
constexpr int slot_bytes(int pixels, int C) { return (pixels * C * 2 + 1023) / 1024 * 1024; }
constexpr int kEpiWarps = 8;
constexpr int kConvThreads = 32 * (2 + kEpiWarps);
constexpr int kGroupRows = 3;

template <int CIN, int COUT>
struct ConvShape {
    static constexpr int CC = CIN / 8;
    static constexpr int kRing = 8;                               // input row slots
    static constexpr int kWin = 3 * COUT;                         // TMEM columns of one group's window
    static constexpr int kWindows = 3 * COUT * 4 <= 512 ? 4 : 2;  // accumulator windows (groups in flight)
    static constexpr int kRowBytes = slot_bytes(kRowW, CIN);      // one slot
    static constexpr uint32_t kRowTx = kRowW * CIN * 2;           // bytes the TMA writes per row
    static constexpr int kWeightBytes = 9 * CIN * COUT * 2;       // [dx][ci/8][kernel row 2, 1, 0][co][8]
    static constexpr int kSmem = kWeightBytes + kRing * kRowBytes + 1024;
    static constexpr uint32_t kCols = kWindows * kWin <= 32 ? 32 : (kWindows * kWin <= 64 ? 64 : (kWindows * kWin <= 128 ? 128 : (kWindows * kWin <= 256 ? 256 : 512)));
    static_assert(CIN % 16 == 0 && COUT % 16 == 0 && kWin <= 256 && kWindows * kWin <= 512, "shape");
    static_assert(kWeightBytes % 1024 == 0, "ring slots aligned to the swizzle period");
};

// bounded wait that also gives up when another role has given up (abort flag in shared memory)
__device__ __forceinline__ bool mbar_wait_or_abort(uint64_t* mbar, uint32_t phase, volatile int* abort, int* status) {
    for (int spin = 0; spin < (1 << 22); ++spin) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(smem_u32(mbar)), "r"(phase)
            : "memory");
        if (done) return true;
        if ((spin & 255) == 255 && *abort) return false;
    }
    *abort = 1;
    if (status) atomicExch(status, 3);  // 3: a wait of the learned filter gave up
    return false;
}
// The producer and MMA warps run their loops as whole warps, on values that are the same in all lanes --
// the warp number through a shuffle, wait results through a vote -- and elect one lane only around the
// copies and MMAs.  Descriptors and coordinates then live in uniform registers, where those
// instructions take them; under a branch on the lane number each MMA took about 120 clocks to issue,
// most of it moving its operands there.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ bool warp_wait_or_abort(uint64_t* mbar, uint32_t phase, volatile int* abort, int* status) {
    return __all_sync(0xFFFFFFFFu, mbar_wait_or_abort(mbar, phase, abort, status));
}
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0); }
__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// 8 consecutive FP32 columns of this thread's TMEM lane, without waiting (tmem_wait_ld before use)
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

// N consecutive BF16 channels of one pixel (N = 8 or 16: one 16- or 32-byte access, a whole sector)
template <int N>
struct Chan {
    uint32_t r[N / 2];
};
template <int N>
__device__ __forceinline__ Chan<N> load_chan(const bf16* p) {
    Chan<N> c;
    if constexpr (N == 16)
        asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(c.r[0]), "=r"(c.r[1]), "=r"(c.r[2]), "=r"(c.r[3]), "=r"(c.r[4]), "=r"(c.r[5]), "=r"(c.r[6]), "=r"(c.r[7])
                     : "l"(p));
    else
        asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(c.r[0]), "=r"(c.r[1]), "=r"(c.r[2]), "=r"(c.r[3]) : "l"(p));
    return c;
}
template <int N>
__device__ __forceinline__ void store_chan(bf16* p, const Chan<N>& c) {
    if constexpr (N == 16)
        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(c.r[0]), "r"(c.r[1]), "r"(c.r[2]), "r"(c.r[3]), "r"(c.r[4]),
                     "r"(c.r[5]), "r"(c.r[6]), "r"(c.r[7])
                     : "memory");
    else
        asm volatile("st.global.v4.b32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(c.r[0]), "r"(c.r[1]), "r"(c.r[2]), "r"(c.r[3]) : "memory");
}
__device__ __forceinline__ float2 chan_pair(uint32_t r) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r)); }
__device__ __forceinline__ uint32_t pack_pair(float x, float y) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&v);
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(kConvThreads, 1) k_filter_conv(const __grid_constant__ CUtensorMap tmapX, const FilterConvArgs a,
                                                                 int segRows) {
    chain_wait();
    using S = ConvShape<CIN, COUT>;
    using bf16 = __nv_bfloat16;
    constexpr int CC = S::CC, NW = S::kWindows, KK = CIN / 16;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* wsm = smem;
    uint8_t* ring = smem + S::kWeightBytes;
    __shared__ uint32_t tmem_base;
    __shared__ __align__(8) uint64_t full[S::kRing], empty[S::kRing], accFull[NW], accEmpty[NW], drain;
    __shared__ int abortFlag, issuedRows, consumedRows;
    __shared__ __align__(16) float biasSm[COUT];
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    // weights: packed [tap = dy * 3 + dx][ci/8][co][8] -> [dx][ci/8][kernel row 2, 1, 0][co][8]
    for (int i = tid; i < S::kWeightBytes / 16; i += blockDim.x) {
        const int co = i % COUT, dyr = (i / COUT) % 3, cc = (i / (3 * COUT)) % CC, dx = i / (3 * COUT * CC);
        const int tap = (2 - dyr) * 3 + dx;
        reinterpret_cast<uint4*>(wsm)[i] = reinterpret_cast<const uint4*>(a.w)[((size_t)tap * CC + cc) * COUT + co];
    }
    for (int i = tid; i < COUT; i += blockDim.x) biasSm[i] = a.bias ? a.bias[i] : 0.0f;
    if (tid == 0) {
        for (int k = 0; k < S::kRing; ++k) {
            mbar_init(&full[k], 1);
            mbar_init(&empty[k], 1);
        }
        for (int k = 0; k < NW; ++k) {
            mbar_init(&accFull[k], 1);
            mbar_init(&accEmpty[k], kEpiWarps);
        }
        mbar_init(&drain, 1);
        abortFlag = 0;
        issuedRows = consumedRows = 0;
        mbar_init_fence();
    }
    async_proxy_fence();  // the weights are read by the tensor core
    if (warp == 1) tmem_alloc(&tmem_base, S::kCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    volatile int* abort = &abortFlag;
    // segRows is a multiple of 3; a segment's last group may run past the image (zero input rows,
    // results not stored)
    const int strips = (a.W + kStripPx - 1) / kStripPx, segs = (a.H + segRows - 1) / segRows;
    const int items = a.B * strips * segs;
    auto item_of = [&](int item, int& b, int& x0, int& ys, int& ng) {
        b = item / (strips * segs);
        const int rem = item % (strips * segs);
        x0 = (rem / segs) * kStripPx;
        ys = (rem % segs) * segRows;
        ng = (min(ys + segRows, a.H) - ys + kGroupRows - 1) / kGroupRows;
    };
    if (warp == 0) {  // producer: input rows ys - 1 .. ys + 3 ng of each item
        int seq = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
            int b, x0, ys, ng;
            item_of(item, b, x0, ys, ng);
            for (int k = 0; k < kGroupRows * ng + 2; ++k, ++seq) {
                const int slot = seq % S::kRing, fill = seq / S::kRing;
                ok = fill == 0 || warp_wait_or_abort(&empty[slot], (uint32_t)((fill - 1) & 1), abort, a.status);
                if (!ok) break;
                if (elect_one()) {
                    mbar_expect_tx(&full[slot], S::kRowTx);
                    tma_load_4d(ring + slot * S::kRowBytes, &tmapX, 0, x0 - 1, ys - 1 + k, b, &full[slot]);
                    issuedRows = seq + 1;
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {  // MMA issuer
        // descriptors: the start address sits in the low 14 bits (address / 16) and every operand lies
        // below 256 KB, so offsets add to it without a carry
        const uint64_t adesc0 = umma_desc_rows<CIN>(smem_u32(ring), 16), bdesc0 = umma_desc(smem_u32(wsm), 3 * COUT * 16, 128);
        constexpr uint32_t id1 = umma_idesc(128, COUT, false, false), id2 = umma_idesc(128, 2 * COUT, false, false),
                           id3 = umma_idesc(128, 3 * COUT, false, false);
        int base = 0, waited = 0, g = 0;  // first input row of the item, input rows waited for, groups issued
        bool ok = true;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
            int b, x0, ys, ng;
            item_of(item, b, x0, ys, ng);
            for (int j = 0; j < ng; ++j, ++g) {
                const int w = g % NW;
                ok = g < NW || warp_wait_or_abort(&accEmpty[w], (uint32_t)((g / NW - 1) & 1), abort, a.status);
                const int first = base + kGroupRows * j;  // input row r - 1 of this group
                for (; waited < first + 5 && ok; ++waited)
                    ok = warp_wait_or_abort(&full[waited % S::kRing], (uint32_t)((waited / S::kRing) & 1), abort, a.status);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    consumedRows = waited;
                    uint64_t arow[5];
#pragma unroll
                    for (int p = 0; p < 5; ++p) arow[p] = adesc0 + (uint64_t)((((first + p) % S::kRing) * S::kRowBytes) >> 4);
                    const uint32_t d0 = tmem + (uint32_t)(w * S::kWin);
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
                        for (int kk = 0; kk < KK; ++kk) {
                            const uint64_t aoff = (uint64_t)((kk * 32 + dx * CIN * 2) >> 4);
                            const uint64_t bk = bdesc0 + (uint64_t)((dx * CC + 2 * kk) * 3 * COUT);
                            const bool f = dx == 0 && kk == 0;  // the step where rows r+1 and r+2 start
                            // input r - 1: row r (kernel row 0)
                            umma(d0, arow[0] + aoff, bk + 2 * COUT, id1, f ? 0u : 1u);
                            // input r: rows r, r + 1 (kernel rows 1, 0)
                            if (f) {
                                umma(d0, arow[1] + aoff, bk + COUT, id1, 1u);
                                umma(d0 + COUT, arow[1] + aoff, bk + 2 * COUT, id1, 0u);
                            } else {
                                umma(d0, arow[1] + aoff, bk + COUT, id2, 1u);
                            }
                            // input r + 1: rows r .. r + 2 (kernel rows 2, 1, 0)
                            if (f) {
                                umma(d0, arow[2] + aoff, bk, id2, 1u);
                                umma(d0 + 2 * COUT, arow[2] + aoff, bk + 2 * COUT, id1, 0u);
                            } else {
                                umma(d0, arow[2] + aoff, bk, id3, 1u);
                            }
                            // input r + 2: rows r + 1, r + 2 (kernel rows 2, 1); input r + 3: row r + 2
                            umma(d0 + COUT, arow[3] + aoff, bk, id2, 1u);
                            umma(d0 + 2 * COUT, arow[4] + aoff, bk, id1, 1u);
                        }
                    umma_commit(&accFull[w]);
                    // input rows no later group of the item reads
                    umma_commit(&empty[first % S::kRing]);
                    umma_commit(&empty[(first + 1) % S::kRing]);
                    umma_commit(&empty[(first + 2) % S::kRing]);
                    if (j == ng - 1) {
                        umma_commit(&empty[(first + 3) % S::kRing]);
                        umma_commit(&empty[(first + 4) % S::kRing]);
                    }
                }
                __syncwarp();
            }
            base += kGroupRows * ng + 2;
        }
        if (elect_one()) umma_commit(&drain);  // completes when every MMA issued above has
        __syncwarp();
        mbar_wait(&drain, 0u, nullptr);
    } else {  // epilogue: TMEM lane quarter warp % 4 = pixels 32 (warp % 4) .. + 31; channel half h
        constexpr int CH = COUT / 2, N = CH >= 16 ? 16 : 8, NC = CH / N;
        const int q = warp & 3, h = (warp - 2) >> 2, cbase = h * CH;
        int g = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
            int b, x0, ys, ng;
            item_of(item, b, x0, ys, ng);
            const int ye = min(ys + segRows, a.H);
            const int xx = x0 + q * 32 + lane;
            const size_t rowStep = (size_t)a.W * COUT;
            size_t at = (((size_t)b * a.H + ys) * a.W + xx) * COUT + cbase;  // this lane's channels in the group's first row
            for (int j = 0; j < ng; ++j, ++g, at += kGroupRows * rowStep) {
                const int w = g % NW, y0 = ys + kGroupRows * j;
                auto live = [&](int r) { return y0 + r < ye && xx < a.W; };
                // narrow layers fetch the skip input of the group's rows before waiting for the
                // accumulators (registers allow it); 64-channel layers and masks load in place
                constexpr bool kPre = CH <= 16;
                Chan<N> addPre[kPre ? kGroupRows : 1][kPre ? NC : 1];
                if constexpr (kPre)
                    if (a.add)
#pragma unroll
                        for (int r = 0; r < kGroupRows; ++r)
#pragma unroll
                            for (int c = 0; c < NC; ++c)
                                if (live(r)) addPre[r][c] = load_chan<N>(a.add + at + r * rowStep + c * N);
                if (!mbar_wait_or_abort(&accFull[w], (uint32_t)((g / NW) & 1), abort, a.status)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                uint32_t raw[kGroupRows][CH];
#pragma unroll
                for (int r = 0; r < kGroupRows; ++r)
#pragma unroll
                    for (int c = 0; c < CH; c += 8)
                        tmem_ld8_nowait(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(w * S::kWin + r * COUT + cbase + c), raw[r] + c);
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&accEmpty[w]);  // the window goes back before the math and stores
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    float bias[N];
#pragma unroll
                    for (int e = 0; e < N; e += 4) *reinterpret_cast<float4*>(bias + e) = *reinterpret_cast<const float4*>(biasSm + cbase + c * N + e);
#pragma unroll
                    for (int r = 0; r < kGroupRows; ++r) {
                        if (!live(r)) continue;
                        const size_t o = at + r * rowStep + c * N;
                        float v[N];
#pragma unroll
                        for (int e = 0; e < N; ++e) {
                            v[e] = __uint_as_float(raw[r][c * N + e]) + bias[e];
                            if (a.relu) v[e] = fmaxf(v[e], 0.0f);
                        }
                        auto packed = [&] {
                            Chan<N> p;
#pragma unroll
                            for (int e = 0; e < N / 2; ++e) p.r[e] = pack_pair(v[2 * e], v[2 * e + 1]);
                            return p;
                        };
                        if (a.y) store_chan<N>(a.y + o, packed());
                        if (a.add) {
                            // forward skip (a.ya): the sum of the stored BF16 activations, x5 = bf16(bf16(y4) + y1);
                            // backward (the skip gradient into layer 1's): FP32 sum, rounded once on the way out
                            const bool storedSum = a.ya != nullptr;
                            const Chan<N> av = kPre ? addPre[kPre ? r : 0][kPre ? c : 0] : load_chan<N>(a.add + o);
#pragma unroll
                            for (int e = 0; e < N / 2; ++e) {
                                const float2 ad = chan_pair(av.r[e]), own = storedSum ? chan_pair(pack_pair(v[2 * e], v[2 * e + 1]))
                                                                                      : make_float2(v[2 * e], v[2 * e + 1]);
                                v[2 * e] = own.x + ad.x;
                                v[2 * e + 1] = own.y + ad.y;
                            }
                        }
                        if (a.ya) store_chan<N>(a.ya + o, packed());
                        if (a.yf && c == 0 && cbase == 0)
                            reinterpret_cast<float4*>(a.yf)[((size_t)b * a.H + y0 + r) * a.W + xx] = make_float4(v[0], v[1], v[2], v[3]);
                        if (a.ym) {
                            const Chan<N> mk = load_chan<N>(a.mask + o);
#pragma unroll
                            for (int e = 0; e < N / 2; ++e) {
                                const float2 m = chan_pair(mk.r[e]);
                                v[2 * e] = m.x > 0.0f ? v[2 * e] : 0.0f;
                                v[2 * e + 1] = m.y > 0.0f ? v[2 * e + 1] : 0.0f;
                            }
                            store_chan<N>(a.ym + o, packed());
                        }
                    }
                }
            }
        }
    }
    __syncthreads();
    // an abandoned pipeline may still have row copies in flight: wait for them (bounded) before the
    // shared memory goes away; the MMA issuer already waited for its MMAs
    if (tid == 0 && abortFlag)
        for (int k = consumedRows; k < issuedRows; ++k) mbar_wait(&full[k % S::kRing], (uint32_t)((k / S::kRing) & 1), nullptr);
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, S::kCols);
}

// ---- weight and bias gradients: dW[co][tap][ci] = sum_p g[p][co] * x[p + tap][ci], db[co] = sum_p g[p][co]
// D (M = 128 rows: output channels) x (N = CIN per tap) over K = pixels, both operands MN-major: A = a
// row of g, B = a row of x from the tap's pixel on, both as the TMA writes them.  The bias sum is one more product, with a tile of ones as B.
// A CTA takes an equal run of the (image, strip of 128 pixels, row) list, so all CTAs end together, and
// streams it: each row of g once, each row of x once (plus two rows where a run starts or enters the next
// strip), through rings of shared-memory slots filled by TMA, while one thread issues the MMAs with
// constant descriptor offsets; everything accumulates in tensor memory.  The three x rows that an output
// row needs lie one after another in the ring, so one MMA (M = 128, N = 3 CIN, K = 16) takes the three
// taps of a kernel column: 24 MMAs a row instead of 72.  Where the ring wraps inside the three rows, two
// MMAs share them.  Rows of A beyond COUT repeat its channels; their results are not read.  With 64 input channels the nine taps (576 columns) exceed tensor
// memory: half of the CTAs take columns 0 and 1 of the kernel, the others column 2.
// 32 crops of 128 x 128, 64 -> 64: 410 us with one tile staged, multiplied and waited for at a time by one warp
// quartet, 96 us now, bias sum (113 us in a kernel of its own) included.
template <int CIN, int COUT>
struct DwShape {
    static constexpr int kGroups = CIN == 64 ? 2 : 1;
    static constexpr int kCols0 = CIN == 64 ? 2 : 3;  // kernel columns of the first group
    static constexpr int kGBytes = slot_bytes(kStripPx, COUT), kXBytes = slot_bytes(kRowW, CIN);
    static constexpr int kGRing = 4, kXRing = 8;
    static constexpr uint32_t kGTx = kStripPx * COUT * 2, kXTx = kRowW * CIN * 2;
    static constexpr int kOnes = 2 * 256;  // B tile of ones: [2 chunks][16 pixels][8]
    static constexpr int kUsed = kGRing * kGBytes + kXRing * kXBytes + kOnes;
    // at least 120 KB: one CTA holds an SM (and its tensor memory) at a time
    static constexpr int kSmem = kUsed + 1024 > 120 * 1024 ? kUsed + 1024 : 120 * 1024;
    static constexpr int kBiasCol = kCols0 * 3 * CIN;  // tensor-memory column of the bias sums
    static constexpr uint32_t kCols = kBiasCol + 16 <= 256 ? 256 : 512;
    static_assert(kBiasCol + 16 <= 512 && 3 * CIN <= 256 && kSmem <= 227 * 1024, "shape");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(128, 1) k_filter_dw(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapG, int B,
                                                      int H, int W, int ctas0, float* __restrict__ partial, float* __restrict__ biasPartial,
                                                      int* status) {
    chain_wait();
    using S = DwShape<CIN, COUT>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *gring = smem, *xring = smem + S::kGRing * S::kGBytes, *ones = xring + S::kXRing * S::kXBytes;
    __shared__ uint32_t tmem_base;
    __shared__ __align__(8) uint64_t xFull[S::kXRing], xEmpty[S::kXRing], gFull[S::kGRing], gEmpty[S::kGRing], drain;
    __shared__ int abortFlag, issuedX, issuedG, consumedX, consumedG;
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    // group 0 (CTAs 0 .. ctas0 - 1): kernel columns 0 .. kCols0 - 1 and the bias; group 1: the last column
    const bool second = S::kGroups > 1 && (int)blockIdx.x >= ctas0;
    const int cta = second ? (int)blockIdx.x - ctas0 : (int)blockIdx.x, ctas = second ? (int)gridDim.x - ctas0 : ctas0;
    for (int i = tid; i < S::kOnes / 2; i += blockDim.x) reinterpret_cast<bf16*>(ones)[i] = __float2bfloat16(1.0f);
    if (tid == 0) {
        for (int k = 0; k < S::kXRing; ++k) {
            mbar_init(&xFull[k], 1);
            mbar_init(&xEmpty[k], 1);
        }
        for (int k = 0; k < S::kGRing; ++k) {
            mbar_init(&gFull[k], 1);
            mbar_init(&gEmpty[k], 1);
        }
        mbar_init(&drain, 1);
        abortFlag = 0;
        issuedX = issuedG = consumedX = consumedG = 0;
        mbar_init_fence();
    }
    async_proxy_fence();  // the ones are read by the tensor core
    if (warp == 0) tmem_alloc(&tmem_base, S::kCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    volatile int* abort = &abortFlag;
    const int strips = (W + kStripPx - 1) / kStripPx;
    const long long rows = (long long)B * strips * H, r0 = rows * cta / ctas, r1 = rows * (cta + 1) / ctas;
    // the run of rows from r on that lie in one strip of one image: its image, first pixel, first row, length
    auto run_at = [&](long long r, int& b, int& x0, int& y0) {
        const long long bs = r / H;
        b = (int)(bs / strips);
        x0 = (int)(bs % strips) * kStripPx;
        y0 = (int)(r % H);
        return (int)min((long long)(H - y0), r1 - r);
    };
    if (warp == 0) {  // copies: x rows y0 - 1 .. y0 + n, g rows y0 .. y0 + n - 1 of each run
        int sx = 0, sg = 0;
        bool ok = true;
        for (long long r = r0; r < r1 && ok;) {
            int b, x0, y0;
            const int n = run_at(r, b, x0, y0);
            for (int k = 0; k < n + 2; ++k) {
                const int xs = sx % S::kXRing;
                ok = sx < S::kXRing || warp_wait_or_abort(&xEmpty[xs], (uint32_t)((sx / S::kXRing - 1) & 1), abort, status);
                if (!ok) break;
                ++sx;
                if (elect_one()) {
                    mbar_expect_tx(&xFull[xs], S::kXTx);
                    tma_load_4d(xring + xs * S::kXBytes, &mapX, 0, x0 - 1, y0 - 1 + k, b, &xFull[xs]);
                    issuedX = sx;
                }
                __syncwarp();
                if (k >= n) continue;
                const int gs = sg % S::kGRing;
                ok = sg < S::kGRing || warp_wait_or_abort(&gEmpty[gs], (uint32_t)((sg / S::kGRing - 1) & 1), abort, status);
                if (!ok) break;
                ++sg;
                if (elect_one()) {
                    mbar_expect_tx(&gFull[gs], S::kGTx);
                    tma_load_4d(gring + gs * S::kGBytes, &mapG, 0, x0, y0 + k, b, &gFull[gs]);
                    issuedG = sg;
                }
                __syncwarp();
            }
            r += n;
        }
    } else if (warp == 1) {  // MMA issuer: output row j of a run takes x rows j, j + 1, j + 2 of the run
        // A: COUT channels, repeated over the 128 rows (lbo 0); B: CIN channels of consecutive slots
        const uint64_t a0 = umma_desc_rows<COUT>(smem_u32(gring), 0), b0 = umma_desc_rows<CIN>(smem_u32(xring), S::kXBytes),
                       one = umma_desc(smem_u32(ones), 128, 256);
        constexpr uint32_t id1 = umma_idesc(128, CIN, true, true), id2 = umma_idesc(128, 2 * CIN, true, true),
                           id3 = umma_idesc(128, 3 * CIN, true, true), idOne = umma_idesc(128, 16, true, true);
        int sx = 0, sg = 0, seen = 0;  // first x row of the run, g row, x rows waited for
        uint32_t acc = 0;
        bool ok = true;
        for (long long r = r0; r < r1 && ok;) {
            int b, x0, y0;
            const int n = run_at(r, b, x0, y0);
            for (int j = 0; j < n; ++j, ++sg) {
                for (; seen < sx + j + 3 && ok; ++seen)
                    ok = warp_wait_or_abort(&xFull[seen % S::kXRing], (uint32_t)((seen / S::kXRing) & 1), abort, status);
                ok = ok && warp_wait_or_abort(&gFull[sg % S::kGRing], (uint32_t)((sg / S::kGRing) & 1), abort, status);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    consumedX = seen;
                    consumedG = sg + 1;
                    const uint64_t ad = a0 + (uint64_t)(((sg % S::kGRing) * S::kGBytes) >> 4);
                    const int slot = (sx + j) % S::kXRing, ahead = S::kXRing - slot;  // slots before the ring wraps
                    const uint64_t bd = b0 + (uint64_t)((slot * S::kXBytes) >> 4);
                    // columns c .. of the kernel from the first one of this group on
                    auto column = [&](int c, int dx) {
#pragma unroll
                        for (int kk = 0; kk < kStripPx / 16; ++kk) {
                            const uint64_t ak = ad + (uint64_t)(2 * COUT * kk), off = (uint64_t)((16 * kk + dx) * CIN / 8);
                            const uint32_t d = tmem + (uint32_t)(c * 3 * CIN), go = kk == 0 ? acc : 1u;
                            if (ahead >= 3) {
                                umma(d, ak, bd + off, id3, go);
                            } else if (ahead == 2) {
                                umma(d, ak, bd + off, id2, go);
                                umma(d + 2 * CIN, ak, b0 + off, id1, go);
                            } else {
                                umma(d, ak, bd + off, id1, go);
                                umma(d + CIN, ak, b0 + off, id2, go);
                            }
                        }
                    };
                    if (second) {
                        column(0, S::kCols0);
                    } else {
#pragma unroll
                        for (int c = 0; c < S::kCols0; ++c) column(c, c);
#pragma unroll
                        for (int kk = 0; kk < kStripPx / 16; ++kk)
                            umma(tmem + (uint32_t)S::kBiasCol, ad + (uint64_t)(2 * COUT * kk), one, idOne, kk == 0 ? acc : 1u);
                    }
                    umma_commit(&gEmpty[sg % S::kGRing]);
                    umma_commit(&xEmpty[(sx + j) % S::kXRing]);
                    if (j == n - 1) {
                        umma_commit(&xEmpty[(sx + n) % S::kXRing]);
                        umma_commit(&xEmpty[(sx + n + 1) % S::kXRing]);
                    }
                }
                __syncwarp();
                acc = 1u;
            }
            sx += n + 2;
            r += n;
        }
        if (elect_one()) umma_commit(&drain);  // completes when every MMA issued above has
        __syncwarp();
        mbar_wait(&drain, 0u, nullptr);
    }
    __syncthreads();
    // an abandoned pipeline may still have copies in flight: wait for them (bounded) before the shared
    // memory goes away
    if (tid == 0 && abortFlag) {
        for (int k = consumedX; k < issuedX; ++k) mbar_wait(&xFull[k % S::kXRing], (uint32_t)((k / S::kXRing) & 1), nullptr);
        for (int k = consumedG; k < issuedG; ++k) mbar_wait(&gFull[k % S::kGRing], (uint32_t)((k / S::kGRing) & 1), nullptr);
    }
    __syncthreads();
    tc_fence_after();
    // partial[cta][co][tap][ci] for this CTA's taps (zero when it had no row)
    const int co = warp * 32 + lane;
    const bool some = r1 > r0 && !abortFlag;
    float* out = partial + (size_t)cta * COUT * 9 * CIN;
    if (warp * 32 < COUT) {
        const uint32_t row = tmem + ((uint32_t)(warp * 32) << 16);
        float v[16];
        const int cols = second ? 3 - S::kCols0 : S::kCols0, dx0 = second ? S::kCols0 : 0;
#pragma unroll 1
        for (int t = 0; t < 3 * cols; ++t)
#pragma unroll 1
            for (int c0 = 0; c0 < CIN; c0 += 16) {
                tmem_ld16(row + (uint32_t)(t * CIN + c0), v);
                if (co < COUT)
#pragma unroll
                    for (int q = 0; q < 16; ++q) out[((size_t)co * 9 + (t % 3) * 3 + dx0 + t / 3) * CIN + c0 + q] = some ? v[q] : 0.0f;
            }
        if (!second) {
            tmem_ld16(row + (uint32_t)S::kBiasCol, v);
            if (co < COUT) biasPartial[(size_t)cta * COUT + co] = some ? v[0] : 0.0f;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, S::kCols);
}

// ---- small kernels -------------------------------------------------------------------------------
// packs layer weights W[co][ci][3][3] (FP32, real sizes) into the B-operand layout [tap][ci/8][co][8]
// of the padded shape; transposed: the data-gradient weights W'[ci][co][8 - tap] with roles swapped
__global__ void k_filter_pack(const float* __restrict__ W, int coutReal, int cinReal, int cin, int cout, int transposed,
                              bf16* __restrict__ out) {
    const int n = 9 * cin * cout;  // in the packed (possibly transposed) shape: K = 9 * cin, N = cout
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int e = i % 8, row = (i / 8) % cout, kc = i / (8 * cout);
        const int tap = kc / (cin / 8), ci = (kc % (cin / 8)) * 8 + e;  // K index = tap * cin + ci
        float v = 0.0f;
        if (!transposed) {
            if (row < coutReal && ci < cinReal) v = W[((size_t)row * cinReal + ci) * 9 + tap];
        } else {  // packed cin = layer's cout, packed cout (row) = layer's cin
            const int lco = ci, lci = row;
            if (lco < coutReal && lci < cinReal) v = W[((size_t)lco * cinReal + lci) * 9 + (8 - tap)];
        }
        out[i] = __float2bfloat16(v);
    }
}

// The end of a training step, all layers in one launch: gradients = sums of the CTAs' partials, Adam
// (Kingma & Ba 2015) on the FP32 master parameters, and the packed BF16 weights of the new parameters.
// A block takes 64 parameters, in the partials' order so that its loads are whole sectors; four threads
// sum a quarter of the CTAs each (in a fixed order: a step is deterministic).  lr = 0: gradients only.
// The five reductions of 152 partials took 244 us one thread a parameter; all of this takes 17 us.
__global__ void __launch_bounds__(256) k_filter_finish(const FilterFinish f) {
    chain_wait();
    __shared__ float part[4][64];
    const int j = threadIdx.x & 63, q = threadIdx.x >> 6;
    int l = 0;
    while (l + 1 < 5 && (int)blockIdx.x >= f.layer[l + 1].block0) ++l;
    const FilterFinish::Layer& L = f.layer[l];
    const int nW = L.coutReal * 9 * L.cinReal, i = ((int)blockIdx.x - L.block0) * 64 + j;
    const bool weight = i < nW, valid = i < nW + L.coutReal;
    const int ci = weight ? i % L.cinReal : 0, tap = weight ? i / L.cinReal % 9 : 0, co = weight ? i / (9 * L.cinReal) : i - nW;
    float s = 0.0f;
    if (valid) {
        const size_t stride = weight ? (size_t)L.cout * 9 * L.cin : (size_t)L.cout;
        const float* p = weight ? L.partial + ((size_t)co * 9 + tap) * L.cin + ci : L.biasPartial + co;
#pragma unroll 8
        for (int c = q, n = weight && tap % 3 == 2 ? L.ctas[1] : L.ctas[0]; c < n; c += 4) s += p[stride * c];
    }
    part[q][j] = s;
    __syncthreads();
    if (q || !valid) return;
    const float gi = (part[0][j] + part[1][j]) + (part[2][j] + part[3][j]);
    const int k = weight ? L.offW + (co * L.cinReal + ci) * 9 + tap : L.offB + co;
    f.grad[k] = gi;
    if (!(f.lr > 0.0f)) return;
    const float mi = f.b1 * f.m[k] + (1.0f - f.b1) * gi, vi = f.b2 * f.v[k] + (1.0f - f.b2) * gi * gi;
    f.m[k] = mi;
    f.v[k] = vi;
    const float w = f.w[k] - f.lr * (mi / f.c1) / (sqrtf(vi / f.c2) + f.eps);
    f.w[k] = w;
    if (!weight) {
        L.bias[co] = w;
        return;
    }
    // as k_filter_pack lays them out
    const bf16 b = __float2bfloat16(w);
    L.packed[((size_t)(tap * (L.cin / 8) + ci / 8) * L.cout + co) * 8 + ci % 8] = b;
    if (L.packedT) L.packedT[((size_t)((8 - tap) * (L.cout / 8) + co / 8) * L.cin + ci) * 8 + co % 8] = b;
}

// mean-squared error over the 3 predicted channels; g = d(loss)/d(out) into channels 0..2 of [P][16]
__global__ void __launch_bounds__(256) k_filter_loss(const float4* __restrict__ out, const float4* __restrict__ target, size_t P,
                                                     float scale, bf16* __restrict__ g, float* __restrict__ partial) {
    chain_wait();
    __shared__ float red[256];
    float s = 0.0f;
    for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (size_t)gridDim.x * blockDim.x) {
        const float4 o = out[p], t = target[p];
        const float d0 = o.x - t.x, d1 = o.y - t.y, d2 = o.z - t.z;
        s += d0 * d0 + d1 * d1 + d2 * d2;
        __align__(16) bf16 v[16];
        v[0] = __float2bfloat16(2.0f * scale * d0);
        v[1] = __float2bfloat16(2.0f * scale * d1);
        v[2] = __float2bfloat16(2.0f * scale * d2);
        for (int j = 3; j < 16; ++j) v[j] = __float2bfloat16(0.0f);
        uint4* dst = reinterpret_cast<uint4*>(g + p * 16);
        dst[0] = reinterpret_cast<uint4*>(v)[0];
        dst[1] = reinterpret_cast<uint4*>(v)[1];
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int off = 128; off > 0; off >>= 1) {
        if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

__device__ __forceinline__ float4 unpack_half4(uint2 u) {
    const __half2 a = *reinterpret_cast<const __half2*>(&u.x), b = *reinterpret_cast<const __half2*>(&u.y);
    const float2 fa = __half22float2(a), fb = __half22float2(b);
    return make_float4(fa.x, fa.y, fb.x, fb.y);
}

// the 16-channel filter input of one frame from its RGBA16F G-buffers (channels 12..15 zero):
//   0-2 rough RGB (reflection / refraction radiance), 3-5 normal, 6 log-scaled linear depth,
//   7 roughness term (rough.a), 8-10 base colour, 11 reflect contribution
__global__ void k_filter_gbuffer(const uint2* __restrict__ base, const uint2* __restrict__ normal, const uint2* __restrict__ rough, size_t P,
                                 float samples, bf16* __restrict__ out) {
    chain_wait();
    for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (size_t)gridDim.x * blockDim.x) {
        const float4 b = unpack_half4(base[p]), n = unpack_half4(normal[p]), r = unpack_half4(rough[p]);
        // normal.w = log(sum of sample depths) * 0.25 / S  ->  mean depth
        const float depth = expf(n.w * 4.0f * samples) / samples;
        const float ld = log1pf(fmaxf(depth, 0.0f)) * 0.108574f;  // / log(10001)
        const float c[12] = {r.x, r.y, r.z, n.x, n.y, n.z, ld, r.w, b.x, b.y, b.z, b.w};
        __align__(16) bf16 v[16];
#pragma unroll
        for (int j = 0; j < 12; ++j) v[j] = __float2bfloat16(c[j]);
#pragma unroll
        for (int j = 12; j < 16; ++j) v[j] = __float2bfloat16(0.0f);
        uint4* dst = reinterpret_cast<uint4*>(out + p * 16);
        dst[0] = reinterpret_cast<uint4*>(v)[0];
        dst[1] = reinterpret_cast<uint4*>(v)[1];
    }
}

// postprocess.comp:28-50 with the filter's prediction in place of roughColorsA
__global__ void k_filter_composite(const uint2* __restrict__ base, const float4* __restrict__ pred, size_t P, float4 fade, int showAlpha,
                                   uint2* __restrict__ finalImg) {
    chain_wait();
    for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (size_t)gridDim.x * blockDim.x) {
        const float4 b = unpack_half4(base[p]), r = pred[p];
        float cr = fminf(fmaxf(b.x * (1.0f - b.w) + r.x * b.w, 0.0f), 1.0f);
        float cg = fminf(fmaxf(b.y * (1.0f - b.w) + r.y * b.w, 0.0f), 1.0f);
        float cb = fminf(fmaxf(b.z * (1.0f - b.w) + r.z * b.w, 0.0f), 1.0f);
        const float luma = (cr * 0.299f + cg * 0.587f) + cb * 0.114f;
        cr = cr * (1.0f - fade.w) + fade.x * fade.w;
        cg = cg * (1.0f - fade.w) + fade.y * fade.w;
        cb = cb * (1.0f - fade.w) + fade.z * fade.w;
        if (showAlpha) cr = cg = cb = luma;  // postprocess.comp:41-49 debug view
        const __half2 lo = __floats2half2_rn(cr, cg), hi = __floats2half2_rn(cb, luma);
        uint2 o;
        o.x = *reinterpret_cast<const uint32_t*>(&lo);
        o.y = *reinterpret_cast<const uint32_t*>(&hi);
        finalImg[p] = o;
    }
}

// RGBA16F rough image of a (glossy) reference render -> FP32 RGBx targets
__global__ void k_filter_target(const uint2* __restrict__ rough, size_t P, float4* __restrict__ out) {
    for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (size_t)gridDim.x * blockDim.x) {
        const float4 r = unpack_half4(rough[p]);
        out[p] = make_float4(r.x, r.y, r.z, 0.0f);
    }
}


// tensor map of an NHWC BF16 activation [B][H][W][C]: boxes of one row of `pixels` pixels, all channels,
// swizzled over a pixel's channels
cudaError_t row_map(CUtensorMap* map, const void* x, int B, int H, int W, int C, int pixels) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return cudaErrorNotSupported;
    if ((reinterpret_cast<uintptr_t>(x) & 15u) != 0) return cudaErrorMisalignedAddress;
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)B};
    const cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2};
    const cuuint32_t box[4] = {(cuuint32_t)C, (cuuint32_t)pixels, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUtensorMapSwizzle swizzle = C == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : C == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(x), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// CTAs per SM of a persistent kernel: shared memory, registers and TMEM columns (512 per SM)
template <class K>
int ctas_per_sm(K kernel, int smem, uint32_t tmemCols, int threads) {
    int dev = 0, smemSm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smemSm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) return 1;
    int per = smemSm / (smem + 1024);
    per = std::min(per, 65536 / std::max(1, fa.numRegs * threads));
    per = std::min(per, (int)(512 / tmemCols));
    per = std::min(per, 16);
    return std::max(per, 1);
}

template <int CIN, int COUT>
cudaError_t conv_launch(const FilterConvArgs& a, cudaStream_t s) {
    using S = ConvShape<CIN, COUT>;
    static std::atomic<int> gridCache{0};
    int grid = gridCache.load(std::memory_order_acquire);
    if (!grid) {
        cudaError_t e = cudaFuncSetAttribute(k_filter_conv<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem);
        if (e != cudaSuccess) return e;
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        grid = sms * ctas_per_sm(k_filter_conv<CIN, COUT>, S::kSmem, S::kCols, kConvThreads);
        gridCache.store(grid, std::memory_order_release);
    }
    if (a.B <= 0 || a.H <= 0 || a.W <= 0) return cudaSuccess;
    CUtensorMap map;
    cudaError_t e = row_map(&map, a.x, a.B, a.H, a.W, CIN, kRowW);
    if (e != cudaSuccess) return e;
    // segments of rows (a multiple of 3): about two items per CTA, at least 9 rows (each item re-reads
    // 2 halo rows)
    const long long strips = (a.W + kStripPx - 1) / kStripPx, rowsTotal = (long long)a.B * strips * a.H;
    int segRows = (int)std::min<long long>(a.H, std::max<long long>(9, (rowsTotal + 2LL * grid - 1) / (2LL * grid)));
    segRows = (segRows + kGroupRows - 1) / kGroupRows * kGroupRows;
    const long long items = (long long)a.B * strips * ((a.H + segRows - 1) / segRows);
    launch_chain(k_filter_conv<CIN, COUT>, (int)std::min<long long>(items, grid), kConvThreads, S::kSmem, s, map, a, segRows);
    count_launch();
    return cudaGetLastError();
}

template <int CIN, int COUT>
cudaError_t dw_launch(const bf16* x, const bf16* g, int B, int H, int W, float* partial, float* biasPartial, int* ctas, int* status,
                      cudaStream_t s) {
    using S = DwShape<CIN, COUT>;
    static std::atomic<bool> attr{false};
    if (!attr.load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(k_filter_dw<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem);
        if (e != cudaSuccess) return e;
        attr.store(true, std::memory_order_release);
    }
    CUtensorMap mx, mg;
    cudaError_t e = row_map(&mx, x, B, H, W, CIN, kRowW);
    if (e == cudaSuccess) e = row_map(&mg, g, B, H, W, COUT, kStripPx);
    if (e != cudaSuccess) return e;
    // one CTA per SM; two groups take half each: both copy every row, which bounds them (two thirds for the
    // two columns: 106 us for 64 -> 64 on 32 crops against 96)
    const int all = filter_dw_ctas();
    ctas[0] = S::kGroups == 1 ? all : std::max(1, all / 2);
    ctas[1] = S::kGroups == 1 ? all : std::max(1, all - ctas[0]);
    const int grid = S::kGroups == 1 ? all : ctas[0] + ctas[1];
    launch_chain(k_filter_dw<CIN, COUT>, grid, 128, S::kSmem, s, mx, mg, B, H, W, ctas[0], partial, biasPartial, status);
    count_launch();
    return cudaGetLastError();
}

}  // namespace

// ---- launchers (rg_internal.cuh) ---------------------------------------------------------------------
cudaError_t filter_conv(int cin, int cout, const FilterConvArgs& a, cudaStream_t s) {
    if (cin == 16 && cout == 32) return conv_launch<16, 32>(a, s);
    if (cin == 32 && cout == 64) return conv_launch<32, 64>(a, s);
    if (cin == 64 && cout == 64) return conv_launch<64, 64>(a, s);
    if (cin == 64 && cout == 32) return conv_launch<64, 32>(a, s);
    if (cin == 32 && cout == 16) return conv_launch<32, 16>(a, s);
    return cudaErrorInvalidValue;
}

int filter_dw_ctas() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

cudaError_t filter_dw(int cin, int cout, const void* x, const void* g, int B, int H, int W, float* partial, float* biasPartial, int* ctas,
                      int* status, cudaStream_t s) {
    const bf16 *X = static_cast<const bf16*>(x), *G = static_cast<const bf16*>(g);
    if (cin == 16 && cout == 32) return dw_launch<16, 32>(X, G, B, H, W, partial, biasPartial, ctas, status, s);
    if (cin == 32 && cout == 64) return dw_launch<32, 64>(X, G, B, H, W, partial, biasPartial, ctas, status, s);
    if (cin == 64 && cout == 64) return dw_launch<64, 64>(X, G, B, H, W, partial, biasPartial, ctas, status, s);
    if (cin == 64 && cout == 32) return dw_launch<64, 32>(X, G, B, H, W, partial, biasPartial, ctas, status, s);
    if (cin == 32 && cout == 16) return dw_launch<32, 16>(X, G, B, H, W, partial, biasPartial, ctas, status, s);
    return cudaErrorInvalidValue;
}

cudaError_t filter_pack(const float* W, int coutReal, int cinReal, int cin, int cout, int transposed, void* out, cudaStream_t s) {
    k_filter_pack<<<64, 256, 0, s>>>(W, coutReal, cinReal, cin, cout, transposed, static_cast<bf16*>(out));
    count_launch();
    return cudaGetLastError();
}

cudaError_t filter_finish(FilterFinish& f, cudaStream_t s) {
    int blocks = 0;
    for (FilterFinish::Layer& l : f.layer) {
        l.block0 = blocks;
        blocks += (l.coutReal * (9 * l.cinReal + 1) + 63) / 64;
    }
    launch_chain(k_filter_finish, blocks, 256, 0, s, f);
    count_launch();
    return cudaGetLastError();
}

cudaError_t filter_loss(const float4* out, const float4* target, size_t P, float scale, void* g, float* partial, int blocks, cudaStream_t s) {
    launch_chain(k_filter_loss, blocks, 256, 0, s, out, target, P, scale, static_cast<bf16*>(g), partial);
    count_launch();
    return cudaGetLastError();
}

cudaError_t filter_gbuffer(const uint2* base, const uint2* normal, const uint2* rough, size_t P, float samples, void* out, cudaStream_t s) {
    launch_chain(k_filter_gbuffer, (unsigned)((P + 255) / 256 < 4096 ? (P + 255) / 256 : 4096), 256, 0, s, base, normal, rough, P, samples,
                                                                                                 static_cast<bf16*>(out));
    count_launch();
    return cudaGetLastError();
}

cudaError_t filter_composite(const uint2* base, const float4* pred, size_t P, const float fade[4], int showAlpha, uint2* finalImg,
                             cudaStream_t s) {
    launch_chain(k_filter_composite, (unsigned)((P + 255) / 256 < 4096 ? (P + 255) / 256 : 4096), 256, 0, s, 
        base, pred, P, make_float4(fade[0], fade[1], fade[2], fade[3]), showAlpha, finalImg);
    count_launch();
    return cudaGetLastError();
}

namespace {
__global__ void k_filter_bias_pad(const float* __restrict__ b, int cReal, int c, float* __restrict__ out) {
    const int i = threadIdx.x;
    if (i < c) out[i] = i < cReal ? b[i] : 0.0f;
}
}  // namespace

cudaError_t filter_bias_pad(const float* b, int cReal, int c, float* out, cudaStream_t s) {
    k_filter_bias_pad<<<1, 64, 0, s>>>(b, cReal, c, out);
    count_launch();
    return cudaGetLastError();
}

cudaError_t filter_target(const uint2* rough, size_t P, float4* out, cudaStream_t s) {
    k_filter_target<<<(unsigned)((P + 255) / 256 < 4096 ? (P + 255) / 256 : 4096), 256, 0, s>>>(rough, P, out);
    count_launch();
    return cudaGetLastError();
}

}  // namespace rg
