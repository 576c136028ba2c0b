// rg_internal.cuh -- device-side layouts and helpers shared by the rgcuda kernels.
//
// All translation units are compiled with -fmad=false: every + - * / below is one IEEE operation,
// so the ray geometry (Morton codes, traversal, intersection, secondary ray set-up) reproduces the
// same bits as a plain C++ evaluation of the same expressions.  Fused multiply-adds are written
// out as fmaf() where they are wanted.
#pragma once

#include <utility>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/rgcuda.h"
#include "tree_plan.h"

namespace rg {

constexpr uint32_t kLeaf = 0x80000000u;
#ifndef RG_STACK_DEPTH
#define RG_STACK_DEPTH 48
#endif
constexpr int kTraversalStack = RG_STACK_DEPTH;
constexpr int kMaxFrames = 10;  // maxRecursions (<= 8 supported) + primary + masked-miss leaf


// 4-wide record of BVH2 node i: the boxes and refs of i's grandchildren (a leaf child stands in
// for its own slot).  Traversal visits records only, so it skips every other BVH2 level; the
// BVH2 itself stays the built and checked structure.  Empty slots have ref kEmptySlot and an
// inverted box.  112 B = seven 16-byte loads.
constexpr uint32_t kEmptySlot = 0xFFFFFFFEu;
struct __align__(16) WideNode {
    float4 lox, hix, loy, hiy, loz, hiz;  // per slot
    uint4 ref;
};
static_assert(sizeof(WideNode) == 112, "wide node");

struct Box {
    float lo[3], hi[3];
};

// per-BLAS record read by the traversal kernel
struct DevBlas {
    const WideNode* wide;
    const float4* tris;  // 3 float4 per sorted leaf: v0 (w = primitive id bits), v1, v2
    uint32_t n;          // triangle count
    uint32_t maxMat;     // largest matIndex of the vertices its triangles reference
    float root[6];       // root box (lo xyz, hi xyz)
    uint32_t vOff, iOff; // vertex and index offsets it was built from (range-checked on the host)
    uint32_t pad0, pad1;
};
static_assert(sizeof(DevBlas) == 64, "BLAS table entry");

// per-instance record read by the traversal and shading code
struct __align__(16) DevInstance {
    float4 inv[3];  // world -> object rows
    float4 m[3];    // object -> world rows
    uint32_t blas, valid, vOff, iOff;
    uint32_t mOff, mask, pad0, pad1;
};
static_assert(sizeof(DevInstance) == 128, "instance");

// TLAS leaf record, in leaf (sorted) order: what the traversal needs to enter an instance, in one
// fetch of six independent 16-byte loads
struct __align__(16) InstRec {
    float4 inv[3];           // world -> object rows
    float4 lo;               // BLAS root box lo xyz; w = BLAS triangle count bits (0: invalid or empty)
    float4 hi;               // BLAS root box hi xyz; w = instance index bits
    const WideNode* wide;    // the BLAS's 4-wide records
    const float4* tris;      // its leaf-ordered triangles
};
static_assert(sizeof(InstRec) == 96, "instance record");

struct DevScene {
    const DevBlas* blas;
    const DevInstance* inst;
    const WideNode* tlasWide;
    const InstRec* tlasLeaves;  // sorted position -> instance record
    uint32_t tlasN;
    uint32_t pad;
    const float* tlasRoot;      // root box (lo xyz, hi xyz), device memory
    const rg_vertex* vertices;
    const uint32_t* indices;
    const rg_material* materials;
};

// ---- explicit-rounding helpers ------------------------------------------------------------------
__host__ __device__ inline uint32_t expand10(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

__device__ inline uint32_t quant10(float c, float lo, float inv) {
    float d = __fsub_rn(c, lo);
    float q = __fmul_rn(d, inv);
    float s = __fmul_rn(q, 1024.0f);
    s = fminf(fmaxf(s, 0.0f), 1023.0f);
    return (uint32_t)s;
}

// order-preserving float <-> uint mapping for atomic min/max
__device__ inline uint32_t f2ord(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ inline float ord2f(uint32_t u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u); }

__host__ __device__ inline float3 f3(float x, float y, float z) { return make_float3(x, y, z); }

}  // namespace rg

// internal launchers implemented in the .cu files
namespace rg {

// kernels launched by this library in this process (rg_launch_count)
extern std::atomic<uint64_t> g_launches;
inline void count_launch(uint64_t n = 1) { g_launches.fetch_add(n, std::memory_order_relaxed); }

// A chain of short launches: each is set up while the one before it still runs (its blocks are placed as soon as
// that one's have ended) and waits for that one's memory itself, first thing, with chain_wait.  1.5 us
// less between two launches, of which a frame has 20 to 50 and a scene load 60: 160x90 frame 10 % shorter,
// 640x360 spheres 7.6 %, 1080p game frame 1 %.  Letting the next blocks in earlier (launch_dependents) costs more
// than it gives, 2 % of the game frame: they hold places of blocks still working.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// kernel: one that starts with chain_wait
template <class... P, class... A>
cudaError_t launch_chain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

struct LbvhBuffers {  // scratch + outputs of one LBVH build, sized by the caller (n primitives)
    uint32_t n;
    // inputs
    float* primBoxes;      // n x 6, primitive order
    // outputs
    uint32_t* morton;      // n, primitive order
    uint32_t* order;       // n, sorted position -> primitive
    uint32_t* left;        // n-1
    uint32_t* right;       // n-1
    float* nodeBoxes;      // (n-1) x 6
    // scratch
    uint32_t* keysA; uint32_t* keysB; uint32_t* valsA; uint32_t* valsB;
    uint32_t* sortState;   // sort_state_words(n): digit histograms, tile counters, centroid bounds, look-back words
    uint32_t* parents;     // 2n (internal n-1 then leaves n)
    uint32_t* flags;       // n-1
    // binned-SAH builds: the task queue of k_sah_tasks (sah_queue_bytes(n), 16-byte aligned) and a
    // status word set to 2 when one of its waits gave up (nullable)
    unsigned char* sahQueue = nullptr;
    int* status = nullptr;
};

// task queue of the SAH builder's task kernel: n task records (range, node id, level), n ready
// words, 8 counters (claims, pushes, first node id, nodes in total, end of the node ids that are left,
// nodes not yet made), 16 per-level task counts of its level kernels
struct SahQueue {
    uint4* tasks;
    uint32_t* ready;
    uint32_t* ctr;
};
constexpr size_t sah_queue_bytes(size_t n) { return 20 * n + 96; }

// onesweep radix sort of the Morton codes: keys per tile, and the layout of its state words (zeroed
// by each build): 4 passes x 256 digit counts, 4 tile counters, then per pass one status word per
// (tile, digit)
constexpr uint32_t kSortTileKeys = 2048;
constexpr uint32_t kSortTileCounters = 4 * 256;
constexpr uint32_t kSortBounds = kSortTileCounters + 8;  // the centroid bounds (6 words)
constexpr uint32_t kSortStatusOffset = kSortTileCounters + 32;
constexpr size_t sort_tiles(size_t n) { return (n + kSortTileKeys - 1) / kSortTileKeys; }
constexpr size_t sort_state_words(size_t n) { return kSortStatusOffset + 4 * 256 * sort_tiles(n); }
cudaError_t lbvh_build(const LbvhBuffers& b, cudaStream_t s);
cudaError_t lbvh_refit(const LbvhBuffers& b, cudaStream_t s);  // topology kept, primBoxes changed
cudaError_t wide_records(const LbvhBuffers& b, WideNode* out, cudaStream_t s);  // after build / refit
// binned-SAH BVH2 over b.primBoxes in the LBVH's layout (order, left, right, nodeBoxes), one CTA;
// parents (for refits) on request.  *levels (device word, nullable) receives the number of levels.
// From level kSahMedianLevel on, ranges are halved without binning, so a tree has at most
// kSahMedianLevel + ceil(log2 n) levels.  The TLAS uses it up to kSahMaxPrims instances (it is
// rebuilt every frame), BLASes up to kSahBlasMaxPrims triangles (built once per scene load), the
// LBVH otherwise.
constexpr uint32_t kSahMaxPrims = 8192;
constexpr uint32_t kSahBlasMaxPrims = 1u << 18;
constexpr uint32_t kSahMedianLevel = 32;
cudaError_t sah_build(const LbvhBuffers& b, bool parents, uint32_t* levels, cudaStream_t s);
cudaError_t tri_boxes(const rg_vertex* v, const uint32_t* idx, uint32_t vOff, uint32_t iOff, uint32_t n, float* boxes,
                      cudaStream_t s);
cudaError_t tri_records(const rg_vertex* v, const uint32_t* idx, uint32_t vOff, uint32_t iOff, const uint32_t* order, uint32_t n,
                        float4* tris, cudaStream_t s);
// world boxes and shading records of n instances.  checkOffsets (instances from device memory, which
// the host never saw): an instance is also invalid -- never hit -- unless its vertex and index offsets
// are its BLAS's own and its material offset keeps the BLAS's materials below nm.
cudaError_t setup_instances(const rg_instance* in, uint32_t n, const DevBlas* blas, uint32_t nblas, DevInstance* out,
                            float* boxes, bool checkOffsets, uint32_t nm, cudaStream_t s);
// the TLAS leaf records (after the TLAS build; again after a BLAS refit, which moves root boxes)
cudaError_t inst_records(const uint32_t* order, uint32_t n, const DevInstance* inst, const DevBlas* blas, InstRec* out,
                         cudaStream_t s);

// words of the traversal kernel: its work counter, and one a ray for the lists of rays whose short stack overflowed
struct TraceWork {
    uint32_t* fetch;
    uint32_t* overflow;
};

// Ray trees (trace.cu): one node per traced ray.  The roots, one per sample of the chunk, are nodes
// 0 .. treeRoots - 1 (their rays and states are recomputed, not stored).
struct RayTree {
    float4* rayO;       // origin, tmin; once composed: colour, payload depth
    float4* rayD;       // direction, tmax
    uint4* state;       // curIOR bits, recDepth | rayType << 4 | job << 6, parent and flags, refDepth bits
    float4* hitTUV;     // t, u, v, primitive bits
    uint32_t* hitInst;  // instance or 0xFFFFFFFF (miss)
    float4* surf;       // of a hit: world normal, material index bits
    uint4* link;        // of a hit: its shadow, reflection and refraction node
    uint32_t* overflow; // links of the lists of rays whose short traversal stack overflowed
    uint32_t* cand[2];  // nodes whose assumptions k_tree_check verifies (the list in use: treeCand)
    uint32_t* ctl;      // kTreeCtlWords words
    uint32_t capacity;  // nodes, at most kTreePoolMax
};
// words of RayTree::ctl: nodes appended after the roots; rays that the last check changed, 16 minus the
// least recursion depth of the rays replaced since the last round, nodes traced when the last check ran;
// the traversal kernel's work counter; lengths of the candidate lists; then the first node of every round, and a
// batch's words
enum : int { kTreeAlloc = 0, kTreeChanges = 1, kTreeLevels = 2, kTreeTraced = 3, kTreeFetch = 4, kTreeCand = 5, kTreeBounds = 7 };
constexpr uint32_t kTreeMaxNodes = 1u << 29;
// room for the rounds' bounds (a chunk that needs more goes again in parts, as one that filled the pool)
constexpr int kTreeMaxRounds = 512 * 9;
// of a batch: more rounds are needed, the chunk filled the pool, rounds run, a chunk is set up (polled together);
// the chunk's roots and first work item, the candidate list in use, the round to trace next and the one
// traced last, samples a chunk, whether any chunk filled the pool, chunks done, their nodes (float); kept from launch to
// launch: the chunks of the last one (as many as there is room for; their samples), its nodes, and the batch's samples, the
// pool's nodes and the slots that they hold for
enum : int {
    kTreeMore = kTreeBounds + kTreeMaxRounds + 1, kTreeFull, kTreeTop, kTreeLive, kTreeRoots, kTreeBase, kTreeCandList, kTreeRound,
    kTreeTracedRound, kTreeChunk, kTreeWasFull, kTreeDone, kTreeNodes, kTreeFollow, kTreePlanned, kTreePlanNodes, kTreePlanOf,
    kTreePlan = kTreePlanOf + 3, kTreeCtlWords = kTreePlan + 16
};
constexpr int kTreeComposeRun = 4;  // rounds composed per run of that loop
// loops of a batch's graph: their conditions; words: runs of the loops on this chunk (at most maxRuns), sticky limit
// flag (graph form), kernels launched in total, rounds in this launch; kernels of a chunk, a run of rounds, a run of compositions
struct TreeLoop {
    bool graph;
    cudaGraphConditionalHandle chunks, rounds, composes;
    uint32_t* words;
    uint32_t maxRuns, chunkKernels, roundKernels, composeKernels;
};
// Pool size: nodes per sample.  The benchmark scenes trace 2.5 to 4 rays a sample; a chunk of samples
// that fills the pool goes again in smaller chunks, and the next pool is larger, up to kTreeNodesMax a sample (no more
// than the paths of one ray at a time took, 1.6 KB a sample).  Without a memory budget a pool of up to kTreeGrowNodes
// (1.9 GB) grows to kTreeNodesMost a sample: a chunk more costs a small frame as much as all of its samples.
constexpr uint32_t kTreeNodesMin = 7, kTreeNodesMax = 13, kTreeNodesMost = 64;
constexpr size_t kTreeGrowNodes = 1u << 24;
// a batch of more samples than slots takes kTreeNodesMax a slot at once up to here (1.5 GB): its chunks are fewer
constexpr uint32_t kTreeFewSlots = 1u << 20;
constexpr size_t kTreePoolMin = 4608;  // nodes of any pool: four times a sample's tree at 8 recursions without replaced rays
constexpr size_t kTreePoolMax = kTreeMaxNodes - 4;  // links keep 29 bits for a node, three of their values for no node
// nodes of the pool for `roots` samples; a pool at its bound holds fewer samples a chunk
constexpr size_t tree_pool_nodes(size_t roots, size_t perRoot, size_t least) {
    const size_t n = roots > kTreePoolMax / perRoot ? kTreePoolMax : roots * perRoot;
    return n < least ? (least < kTreePoolMax ? least : kTreePoolMax) : n;
}

// one render job of a batch: a scene, its UBO and its image size.  Work items of the batch are
// numbered job after job; job j owns [workBase, workBase + workCount) and writes its per-sample
// payload sums to samples[sampleBase + (y * W + x) * S + s].
struct JobDesc {
    DevScene scene;
    rg_ubo ubo;
    uint32_t W, H, S, tilesX;
    uint32_t workBase;    // first work item (work items: 8x4 pixel tiles x 32 pixels x S samples)
    uint32_t workCount;
    uint32_t sampleBase;  // first per-sample slot in TraceParams::samples
    uint32_t pad;
};

struct TraceParams {
    DevScene scene;
    rg_ubo ubo;
    uint32_t W, H;
    uint2* base;    // RGBA16F images (8 B per pixel)
    uint2* normal;
    uint2* rough;
    unsigned long long* counters;  // 8 per frame + 8 cumulative
    float4* samples;               // W*H*S*3 per-sample payload sums (k_trace -> k_resolve)
    uint32_t* workCounter;         // work-item counter of the persistent kernel
    int countVisits;
    TraceWork wf;
    // batch (launch_trace_batch): the job table in device memory, the batch's work items, samples a chunk at
    // most, and the rounds every chunk runs (1 + the largest recursion limit)
    const JobDesc* jobs;
    uint32_t njobs;
    uint32_t totalWork;
    uint32_t slots;
    int batchRounds;
    const uint32_t* perm;  // nullable: order in which the trace kernel takes the round's rays
    uint32_t glossySeed;   // 0: the reference's mirror shading; else glossy reference shading (seed)
    // ray trees: the first round computes the camera rays of the roots itself
    int firstRound;
    // ray trees: node pool; the current chunk of samples (work items treeBase + k, k < treeRoots), the
    // candidate list in use
    RayTree tree;
    uint32_t treeBase, treeRoots, treeCand;
    // ray query (rg_trace_rays_device): queryCount rays read from the caller's buffer (origin, tmin,
    // direction, tmax: two float4 per ray) and hits written in rg_trace_rays' layout, so the query
    // needs neither a queue copy before the traversal nor a read-out pass after it
    const float4* queryRays;
    float* queryTuv;
    uint32_t* queryIds;
    uint32_t queryCount;
};
cudaError_t launch_trace(const TraceParams& p, cudaStream_t s);
// Work items of a frame: W x H pixels padded to whole 8 x 4 tiles, times S samples (more than W * H * S when W or H is
// not a multiple of the tile).  Each is the root of a ray tree, those outside the image an idle one.
constexpr int kTileW = 8, kTileH = 4;
inline size_t frame_work_items(uint32_t W, uint32_t H, uint32_t S) {
    return (size_t)((W + kTileW - 1) / kTileW) * ((H + kTileH - 1) / kTileH) * (kTileW * kTileH) * S;
}
// kernelEvents (nullable): callback that returns a (start, end) event pair to record around each
// traversal launch
typedef bool (*EventPairFn)(void* user, cudaEvent_t* start, cudaEvent_t* end);
// what a frame's second lane of chunks runs with: an idle stream, events that tie it to the frame's stream, control
// words and pinned words of its own
struct TreeLane {
    cudaStream_t stream;
    cudaEvent_t fork, join;
    uint32_t *ctl, *hostWords;
};
// a frame through ray trees, and its resolve.  hostWords: four pinned words polled after each check;
// iterations: rounds run; load: of the last frame, then of this one; mayGrow: a frame of one chunk that fills the
// pool is left undone (load->again)
cudaError_t launch_trace_tree(const TraceParams& p, cudaStream_t s, const TreeLane& second, uint32_t* hostWords, int* iterations, TreeLoad* load,
                              bool mayGrow, EventPairFn kernelEvents = nullptr, void* user = nullptr);
// traversal launch shape of the batch loop: block size {64,128,256}, stack entries {16,24,32,48},
// ray-sort key applied to each round but the first before it is traced
struct TraceTune {
    int threads = 128, depth = 48, sortKey = RG_SORT_NONE;
};
bool tune_supported(const TraceTune& t);
// scratch of the ray sort (keys and permutation: a word a node of the pool; hist: 4096 bucket counts, zero between
// rounds, and 4096 offsets)
struct SortScratch {
    uint32_t *keysA, *valsA, *hist;
};
// every job of p.jobs through ray trees, the loops on the host; hostWords: four pinned words polled after each check
// and chunk; loopWords as below; cudaErrorLaunchTimeout when the loops gave up
cudaError_t launch_trace_batch(const TraceParams& p, const TraceTune& tune, const SortScratch& sort, uint32_t* loopWords, cudaStream_t s,
                               uint32_t* hostWords, int* iterations, bool* poolFull, EventPairFn kernelEvents = nullptr, void* user = nullptr);
// graph form, enqueued on stream s while it captures; the loops run on the device (bodies captured on the idle stream s2).
// loopWords: TreeLoop::words, the sticky flag and the kernel count zeroed by the caller once.
cudaError_t capture_trace_batch(const TraceParams& p, const TraceTune& tune, const SortScratch& sort, cudaStream_t s,
                                cudaStream_t s2, uint32_t* loopWords);
// raygen.rgen:36-38 for one job of a batch: average its samples into RGBA16F G-buffers
cudaError_t launch_resolve_job(const float4* samples, const JobDesc& hostJob, uint2* base, uint2* normal, uint2* rough,
                               cudaStream_t s);
// closest hits of n rays (8 floats each, device memory, 16-byte aligned) by one launch of the frame
// loop's traversal kernel (k_wf_trace in its query form): the kernel takes the rays straight from
// `rays` and writes the hits in rg_trace_rays' layout; stack of `depth` (16, 24, 32 or 48) entries,
// 48 when p.countVisits
cudaError_t launch_trace_queue(const TraceParams& p, const float* rays, uint32_t n, float* tuv, uint32_t* ids, int depth,
                               cudaStream_t s);

// ---- learned roughness filter (filter.cu) ----
// one 3x3 convolution of NHWC BF16 activations (x 16-byte aligned): v = conv(x, w) + bias, then
// ReLU (relu), y = v, v += add, ya = v, ym = v where mask > 0 else 0, yf = v[0..3] in FP32
struct FilterConvArgs {
    const __nv_bfloat16* x;     // [B][H][W][CIN]
    const __nv_bfloat16* w;     // packed [9][CIN/8][COUT][8] (K = tap * CIN + ci, rows = output channels)
    const float* bias;          // nullable [COUT]
    const __nv_bfloat16* add;   // nullable [B][H][W][COUT]
    const __nv_bfloat16* mask;  // nullable [B][H][W][COUT] (required with ym)
    __nv_bfloat16* y;           // nullable [B][H][W][COUT]
    __nv_bfloat16* ya;          // nullable [B][H][W][COUT]
    __nv_bfloat16* ym;          // nullable [B][H][W][COUT]
    float* yf;                  // nullable [B][H][W][4]
    int B, H, W, relu;
    int* status;                // set when a tensor-core or copy completion wait gave up
};
cudaError_t filter_conv(int cin, int cout, const FilterConvArgs& a, cudaStream_t s);
int filter_dw_ctas();  // most CTAs whose partials a weight gradient leaves
// partial[cta][cout][9][cin] and biasPartial[cta][cout] of ctas[0] CTAs, ctas[1] for kernel column 2 (x, g
// 16-byte aligned)
cudaError_t filter_dw(int cin, int cout, const void* x, const void* g, int B, int H, int W, float* partial, float* biasPartial, int* ctas,
                      int* status, cudaStream_t s);
cudaError_t filter_pack(const float* W, int coutReal, int cinReal, int cin, int cout, int transposed, void* out, cudaStream_t s);
// the end of a training step: gradients from the partials of all layers, Adam, packed weights
struct FilterFinish {
    struct Layer {
        const float *partial, *biasPartial;
        __nv_bfloat16 *packed, *packedT;  // packedT nullable (the first layer has no data gradient)
        float* bias;                      // padded bias
        int cout, cin, coutReal, cinReal, offW, offB;
        int ctas[2];                      // CTAs with partials: kernel columns 0 and 1, column 2
        int block0;                       // set by filter_finish
    } layer[5];
    float *w, *grad, *m, *v;
    float lr, b1, b2, eps, c1, c2;
};
cudaError_t filter_finish(FilterFinish& f, cudaStream_t s);
cudaError_t filter_loss(const float4* out, const float4* target, size_t P, float scale, void* g, float* partial, int blocks, cudaStream_t s);
cudaError_t filter_gbuffer(const uint2* base, const uint2* normal, const uint2* rough, size_t P, float samples, void* out, cudaStream_t s);
cudaError_t filter_composite(const uint2* base, const float4* pred, size_t P, const float fade[4], int showAlpha, uint2* finalImg,
                             cudaStream_t s);
cudaError_t filter_target(const uint2* rough, size_t P, float4* out, cudaStream_t s);
cudaError_t filter_bias_pad(const float* b, int cReal, int c, float* out, cudaStream_t s);
// the filter on one frame (G-buffers -> input -> network -> composite into finalImg); filter_api.cu.
// status: the rendering context's device-wait status word (3 when a wait of the filter gave up)
cudaError_t filter_frame(rg_filter* f, const uint2* base, const uint2* normal, const uint2* rough, uint32_t W, uint32_t H, float samples,
                         const float fade[4], int showAlpha, uint2* finalImg, int* status, cudaStream_t s);
const float4* filter_prediction(const rg_filter* f);  // [P] of the last frame: RGB, w unused

struct PostParams {
    uint32_t W, H;
    const uint2* base;     // half4 images (8 B per pixel)
    const uint2* normal;
    const uint2* rough;
    uint2* finalImg;       // half4, postprocess output (FXAA input)
    uint2* fxaaOut;        // half4, FXAA output (becomes the final image)
    float4* framebuffer;   // RGBA32F output
    // debug outputs (nullable)
    float* dbgTransition;  // W*H floats
    uint2* dbgA;           // half4
    uint2* dbgB;           // half4
    float fade[4];
    int showAlpha;
    int fxaa;
    int* status;           // nullable: set to 1 when a staged copy of the roughness pass never landed
    uint32_t waitLimit;    // polls of a staged copy before the pass gives up (see post_wait_limit)
};
cudaError_t launch_rough_post(const PostParams& p, cudaStream_t s);
cudaError_t launch_fxaa(const PostParams& p, cudaStream_t s);
cudaError_t f32_to_h16(const float4* in, uint2* out, size_t n, cudaStream_t s);
cudaError_t h16_to_f32(const uint2* in, float4* out, size_t n, cudaStream_t s);
cudaError_t r32_to_rgba(const float* in, float4* out, size_t n, cudaStream_t s);

}  // namespace rg
