// trace.cu -- per-pixel ray generation, two-level BVH traversal and closest-hit / miss shading.
//
// Replaces traceRaysKHR with the raygen / closest-hit / miss / shadow-miss programs
// (render/raytracer.cpp:99-100; resources/shaders/raygen.h:69-115, raygen.rgen:30-39,
// closesthit.rchit:74-268, miss.rmiss:38-83, shadowMiss.rmiss:30-34).
//
// GB300 has no RT cores, so traversal is software: 4-wide records derived from the BVH2 (one
// 112-byte record = six 16-byte plane loads plus the refs tests four children), nearest-child-first
// stack traversal, TLAS leaves switch to the instance's BLAS with the ray moved into object space, and
// a watertight ray/triangle test (Woop, Benthin, Wald 2013).  Closest-hit ties (equal t) resolve to
// the smaller (instance, primitive).  Box tests only ever accept more than the exact test would (see
// the ray set-up below), so the hit found does not depend on the tree: it is the brute-force answer.
//
// Frames and batches run the reference's recursion (nested traceRayEXT calls sharing ONE payload,
// payload.h:29-43) as ray trees, described at k_tree_expand.  The megakernel runs it as written, by an
// explicit state machine per thread: a paused closest-hit invocation is a Frame on a
// small per-thread stack with a resume code, and every trace (of any depth) happens in the same
// outer loop so the threads of a warp traverse together.  Payload fields that the reference leaves
// stale (depth, rayType, curIOR, refDepth) leak exactly as in the reference.
//
// GLSL-undefined cases follow fixed policies: r/(tr+r) with tr+r == 0 -> 0; pow(x, n) with
// integer n -> repeated multiply; a zero direction (refract at total internal reflection) -> no
// traversal, miss shader; clamp/min/max treat a NaN operand as absent (fminf/fmaxf).
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "rg_internal.cuh"

namespace rg {
namespace {

// ---------------------------------------------------------------------------------------------
// ray set-up and primitive tests
//
// Box tests use one fused multiply-add per plane: t = l * j + C with j = 1/d and C = -o/d.  C is a
// rounded product, so it is kept as a bracket [cl, ch] around -o*j, and the products-sums are rounded
// down for entry planes and up for exit planes: every computed entry is at or below the exact one and
// every exit at or above, and the remaining rounding of 1/d itself is covered by the kInflate margin
// (Ize 2013).  |j| is clamped to [2^-60, 2^64] so that nothing overflows.  Past 2^64 (a zero or tiny
// direction component) the entry plane's t stays a lower bound where it is positive.  The exit
// plane's t is raised by the ray's current far bound tfar (ch = -o*j + tfar, rounded up): an exit
// plane ahead of the origin then lies at or beyond tfar and never rejects the box, while one behind
// the origin still does (its exact t is at or below the clamped one, so raising it stays an upper
// bound).  tfar only shrinks during a traversal, so terms set with an earlier tfar stay valid.
// Below 2^-60 the exit plane's t stays an upper bound where it is positive and the entry plane is
// dropped (cl = -inf).  Boxes are therefore never rejected when the exact test accepts them,
// including rays that start on a plane with a zero direction component.  Which of a box's two
// planes is the entry one follows from the sign of j (the ray's octant).
struct Ray {
    float ox, oy, oz;              // origin of the current level (world, or the instance's object space)
    float dx, dy, dz;              // WORLD direction (kept while inside a BLAS: only instance entry reads it)
    float jx, jy, jz;              // 1/d of the current level, magnitude clamped to [2^-60, 2^64]
    float clx, cly, clz;           // -o*j rounded down (-inf: entry planes dropped)
    float chx, chy, chz;           // -o*j rounded up (plus the far bound where |j| = 2^64)
    float Sx, Sy, Sz;              // shear of the watertight triangle test (BLAS level; kNoShear: the direction)
    uint32_t bits;                 // kx | ky << 2 | kz << 4 (triangle test axes) | octant << 6 | kNoShear
};

__device__ __forceinline__ float comp(float x, float y, float z, int k) { return k == 0 ? x : (k == 1 ? y : z); }

// j, cl, ch from the origin, 1/d and the ray's current far bound tfar
__device__ __forceinline__ void box_terms(float o, float inv, float tfar, float& j, float& cl, float& ch) {
    const float ai = fabsf(inv);
    j = copysignf(fminf(fmaxf(ai, 0x1p-60f), 0x1p64f), inv);
    const float c = -(o * j);
    const float err = fabsf(c) * 0x1p-22f;  // |c - (-o j)| <= 2^-24 |c| (one rounding)
    // the clamp rules read j alone (so that a saved j restores valid terms); at exactly 2^64 or
    // 2^-60 they only accept more
    cl = fabsf(j) > 0x1p-60f ? __fsub_rd(c, err) : -INFINITY;
    ch = fabsf(j) < 0x1p64f ? __fadd_ru(c, err) : __fadd_ru(__fadd_ru(c, err), tfar);
}

__device__ __forceinline__ uint32_t octant(float jx, float jy, float jz) {
    return (jx < 0.0f ? 1u : 0u) | (jy < 0.0f ? 2u : 0u) | (jz < 0.0f ? 4u : 0u);
}

__device__ __forceinline__ void set_box_terms(Ray& r, float ix, float iy, float iz, float tfar) {
    box_terms(r.ox, ix, tfar, r.jx, r.clx, r.chx);
    box_terms(r.oy, iy, tfar, r.jy, r.cly, r.chy);
    box_terms(r.oz, iz, tfar, r.jz, r.clz, r.chz);
    r.bits = (r.bits & 63u) | octant(r.jx, r.jy, r.jz) << 6;
}

// 1/d for the box terms alone: 2^-23 relative (2 ulp of slack with the rounding of -o*j is in
// kInflate), a zero or subnormal d gives an infinity, which box_terms clamps like any 1/d above 2^64.
// Correctly rounded divisions take some ten instructions each, three at every instance entry.
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The triangle test's axes and shear, from the object-space direction that ray_pre left in S; run
// before the first triangle of a BLAS (kNoShear), since most instance entries of a crowded scene
// leave the BLAS again from inner nodes.
constexpr uint32_t kNoShear = 512u;
__device__ __forceinline__ void ray_shear(Ray& r) {
    const float dx = r.Sx, dy = r.Sy, dz = r.Sz;
    float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
    int kz = 0;
    if (ay > ax) kz = 1;
    if (az > (kz == 0 ? ax : ay)) kz = 2;
    int kx = kz + 1 == 3 ? 0 : kz + 1;
    int ky = kx + 1 == 3 ? 0 : kx + 1;
    float dkz = comp(dx, dy, dz, kz);
    if (dkz < 0.0f) { int t = kx; kx = ky; ky = t; }
    r.bits = (r.bits & ~(63u | kNoShear)) | (uint32_t)kx | (uint32_t)ky << 2 | (uint32_t)kz << 4;
    r.Sx = comp(dx, dy, dz, kx) / dkz;
    r.Sy = comp(dx, dy, dz, ky) / dkz;
    r.Sz = 1.0f / dkz;
}

// object-space ray at instance entry: origin, box terms, the direction for ray_shear; the world
// direction in r stays untouched
__device__ __forceinline__ void ray_pre(Ray& r, float ox, float oy, float oz, float dx, float dy, float dz, float tfar) {
    r.ox = ox; r.oy = oy; r.oz = oz;
    r.Sx = dx; r.Sy = dy; r.Sz = dz;
    r.bits = 0u;
    set_box_terms(r, rcp(dx), rcp(dy), rcp(dz), tfar);
    r.bits |= kNoShear;
}

// the world-space ray at the TLAS level (no triangle is tested there)
__device__ __forceinline__ void ray_pre_world(Ray& r, float ox, float oy, float oz, float dx, float dy, float dz, float tfar) {
    r.ox = ox; r.oy = oy; r.oz = oz;
    r.dx = dx; r.dy = dy; r.dz = dz;
    r.bits = 0u;
    set_box_terms(r, rcp(dx), rcp(dy), rcp(dz), tfar);
}

// The box's entry and exit t carry the error of j alone (the products and sums are rounded outwards):
// 2^-23 each, against an exact triangle test; 1 + 2*gamma_3 (Ize 2013) for a correctly rounded j
// was 1.0000004, the bound here is 1 + 2^-20 with room for both.
constexpr float kInflate = 1.000001f;

// one instruction each; as fmaxf/fminf a NaN operand is passed over
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// entry and exit t of one box given its entry planes (n) and exit planes (f)
__device__ __forceinline__ float box_test(const Ray& r, float nx, float ny, float nz, float fx, float fy, float fz, float tmin,
                                          float tbest) {
    const float tn = fmaxf(max3(__fmaf_rd(nx, r.jx, r.clx), __fmaf_rd(ny, r.jy, r.cly), __fmaf_rd(nz, r.jz, r.clz)), tmin);
    const float tf = fminf(min3(__fmaf_ru(fx, r.jx, r.chx), __fmaf_ru(fy, r.jy, r.chy), __fmaf_ru(fz, r.jz, r.chz)), tbest);
    return tn <= tf * kInflate ? tn : INFINITY;
}

// a box given as lo xyz, hi xyz
__device__ __forceinline__ float box_test6(const Ray& r, const float* lo, const float* hi, float tmin, float tbest) {
    const uint32_t o = r.bits >> 6;
    return box_test(r, (o & 1) ? hi[0] : lo[0], (o & 2) ? hi[1] : lo[1], (o & 4) ? hi[2] : lo[2],
                    (o & 1) ? lo[0] : hi[0], (o & 2) ? lo[1] : hi[1], (o & 4) ? lo[2] : hi[2], tmin, tbest);
}

struct Hit {
    float t, u, v;
    uint32_t inst, prim;
    bool hit;
};

__device__ __forceinline__ bool accept(float t, float tmin, uint32_t inst, uint32_t prim, const Hit& h) {
    if (!(t >= tmin)) return false;
    if (!h.hit) return t <= h.t;
    if (t < h.t) return true;
    if (t == h.t) return inst < h.inst || (inst == h.inst && prim < h.prim);
    return false;
}

__device__ __forceinline__ void tri_test(const Ray& r, float4 a, float4 b, float4 c, float tmin, uint32_t inst, Hit& h) {
    const int kx = (int)(r.bits & 3u), ky = (int)((r.bits >> 2) & 3u), kz = (int)((r.bits >> 4) & 3u);
    float A0 = a.x - r.ox, A1 = a.y - r.oy, A2 = a.z - r.oz;
    float B0 = b.x - r.ox, B1 = b.y - r.oy, B2 = b.z - r.oz;
    float C0 = c.x - r.ox, C1 = c.y - r.oy, C2 = c.z - r.oz;
    float Akz = comp(A0, A1, A2, kz), Bkz = comp(B0, B1, B2, kz), Ckz = comp(C0, C1, C2, kz);
    float Ax = comp(A0, A1, A2, kx) - r.Sx * Akz, Ay = comp(A0, A1, A2, ky) - r.Sy * Akz;
    float Bx = comp(B0, B1, B2, kx) - r.Sx * Bkz, By = comp(B0, B1, B2, ky) - r.Sy * Bkz;
    float Cx = comp(C0, C1, C2, kx) - r.Sx * Ckz, Cy = comp(C0, C1, C2, ky) - r.Sy * Ckz;
    float U = Cx * By - Cy * Bx;
    float V = Ax * Cy - Ay * Cx;
    float W = Bx * Ay - By * Ax;
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
        V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
        W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return;
    float det = (U + V) + W;
    if (det == 0.0f) return;
    float Az = r.Sz * Akz, Bz = r.Sz * Bkz, Cz = r.Sz * Ckz;
    float T = (U * Az + V * Bz) + W * Cz;
    float rc = 1.0f / det;
    float t = T * rc;
    uint32_t prim = __float_as_uint(a.w);
    if (!accept(t, tmin, inst, prim, h)) return;
    h.t = t;
    h.u = V * rc;
    h.v = W * rc;
    h.inst = inst;
    h.prim = prim;
    h.hit = true;
}

constexpr uint32_t kMarker = 0xFFFFFFFFu;  // stack entry: leave the BLAS, back to the TLAS

struct VisitCounts {
    unsigned long long nodes, tris, overflow;
};

constexpr int kTraceThreads = 128;
#ifndef RG_TRACE_MIN_BLOCKS
#define RG_TRACE_MIN_BLOCKS 4
#endif

// per-thread traversal stack in shared memory, laid out [depth][thread] so that the 32 lanes of a
// warp touching the same depth hit 32 different banks.  THREADS = block size, DEPTH = entries.
// Beside it, six floats per thread keep the world-space ray's origin and clamped inverse direction
// while the ray is inside a BLAS (the world direction itself stays in registers), so leaving the BLAS
// restores them instead of dividing again.
// The last of the DEPTH words flags an overflow in bit 0 (a push that found the other DEPTH - 1 entries
// full), so the flag costs the traversal loop neither a register nor shared memory beyond the stack.  Its other
// bits are the kernel's (k_wf_trace: the lane's overflowed rays).  Who starts a ray finds the flag clear: a kernel
// starts the word at zero and clears the flag when it is done with a ray that set it.
template <int THREADS, int DEPTH>
struct SmemStackT {
    static constexpr int kDepth = DEPTH - 1;
    uint32_t* base;  // &stack[0][threadIdx.x]
    float* saved;    // &world[0][threadIdx.x]
    __device__ __forceinline__ uint32_t& operator[](int i) const { return base[i * THREADS]; }
    __device__ __forceinline__ float& w(int i) const { return saved[i * THREADS]; }
    __device__ __forceinline__ uint32_t& over() const { return base[(DEPTH - 1) * THREADS]; }
    static constexpr int kStride = THREADS;  // words from one entry to the next
};
// the same stack in (L1-cached) local memory
#ifndef RG_STACK_SMEM
#define RG_STACK_SMEM 1
#endif
template <int DEPTH>
struct LocalStackT {
    static constexpr int kDepth = DEPTH - 1;
    uint32_t* base;
    float* saved;
    __device__ __forceinline__ uint32_t& operator[](int i) const { return base[i]; }
    __device__ __forceinline__ float& w(int i) const { return saved[i]; }
    __device__ __forceinline__ uint32_t& over() const { return base[DEPTH - 1]; }
};
#define RG_DECLARE_SMEM_STACK(name, THREADS, DEPTH)      \
    __shared__ uint32_t name##_mem[DEPTH][THREADS];      \
    __shared__ float name##_world[6][THREADS];           \
    const SmemStackT<THREADS, DEPTH> name{&name##_mem[0][threadIdx.x], &name##_world[0][threadIdx.x]}
#if RG_STACK_SMEM
#define RG_DECLARE_STACK(name) RG_DECLARE_SMEM_STACK(name, kTraceThreads, kTraversalStack)
using TravStack = SmemStackT<kTraceThreads, kTraversalStack>;
#else
#define RG_DECLARE_STACK(name)                 \
    uint32_t name##_mem[kTraversalStack];      \
    float name##_world[6];                     \
    const LocalStackT<kTraversalStack> name{name##_mem, name##_world}
using TravStack = LocalStackT<kTraversalStack>;
#endif
#ifndef RG_WF_MIN_BLOCKS
#define RG_WF_MIN_BLOCKS 7
#endif

// Resumable traversal of one ray: trav_begin sets it up, each trav_step processes one record or one
// leaf (a record tests four children and descends into the nearest hit; a TLAS leaf moves
// the ray into the instance's object space and descends into its BLAS behind a marker entry; a BLAS
// leaf runs the triangle test).  The kernel interleaves trav_step with shading so that a lane whose
// ray finished does not idle.
struct Trav {
    float tmin;
    Ray r;  // the ray of the current level (world or object space); its shear terms are used in BLASes only
    Hit h;
    const WideNode* nodes;
    const float4* tris;
    uint32_t ref, inst;
    int sp;
    bool inBlas, active;
    // shared rays only (see drain): first stack word not given away; whether the stack holds the marker
    // of the instance the lane is in (a lane that was given a BLAS node has none)
    int sb;
    bool marker;
};

template <class STACK>
__device__ __forceinline__ void trav_begin(Trav& T, const DevScene& sc, float ox, float oy, float oz, float dx, float dy, float dz,
                                           float tmin, float tmax, const STACK& stack) {
    T.h.hit = false;
    T.h.t = tmax;
    T.h.u = T.h.v = 0.0f;
    T.h.inst = T.h.prim = 0xFFFFFFFFu;
    T.active = false;
    if ((dx == 0.0f && dy == 0.0f && dz == 0.0f) || sc.tlasN == 0) return;
    T.tmin = tmin;
    ray_pre_world(T.r, ox, oy, oz, dx, dy, dz, tmax);
    if (sc.tlasN > 1 && box_test6(T.r, sc.tlasRoot, sc.tlasRoot + 3, tmin, T.h.t) == INFINITY) return;
    T.sp = 0;
    T.nodes = sc.tlasWide;
    T.tris = nullptr;
    T.inBlas = false;
    T.inst = 0;
    T.ref = sc.tlasN == 1 ? kLeaf : 0u;
    T.active = true;
}

// One record: an inner node's four boxes, a triangle, an instance, or the way back to the TLAS.  The
// loop is bound by instruction issue (71 % of the slots) and by the latency of the record behind it, so
// what counts is instructions a step.  Approximate 1/d, the shear set up at the first triangle, min
// and max of three, no tests for empty slots and pushes without a branch took 4.5 % of the 1920x1080 game
// frame and 1M secondary rays from 538 to 482 us.  Records with each plane pair
// stored both ways round (256-bit loads) gave 1 % more for twice the memory, smaller records with
// selects lost 2 %, stack entries with their t (culled when popped) lost 0.5 %.
template <bool COUNT, bool SHARED = false, class STACK>
__device__ __forceinline__ void trav_step(Trav& T, const DevScene& sc, const STACK& stack, VisitCounts& vc) {
    const uint32_t ref = T.ref;
    const float tmin = T.tmin;
    if (!(ref & kLeaf)) {
        if (COUNT) vc.nodes++;
        const WideNode* nd = T.nodes + ref;
        // entry and exit plane vectors of the ray's octant (lox, hix, loy, hiy, loz, hiz in order)
        const float4* pl = &nd->lox;
        const uint32_t o = T.r.bits >> 6;
        const uint32_t ox = o & 1u, oy = (o >> 1) & 1u, oz = (o >> 2) & 1u;
        const float4 nx = __ldg(pl + ox), fx = __ldg(pl + (ox ^ 1u));
        const float4 ny = __ldg(pl + 2 + oy), fy = __ldg(pl + 2 + (oy ^ 1u));
        const float4 nz = __ldg(pl + 4 + oz), fz = __ldg(pl + 4 + (oz ^ 1u));
        const uint4 rf = __ldg(&nd->ref);
        float t[4];
        uint32_t r[4] = {rf.x, rf.y, rf.z, rf.w};
        t[0] = box_test(T.r, nx.x, ny.x, nz.x, fx.x, fy.x, fz.x, tmin, T.h.t);
        t[1] = box_test(T.r, nx.y, ny.y, nz.y, fx.y, fy.y, fz.y, tmin, T.h.t);
        t[2] = box_test(T.r, nx.z, ny.z, nz.z, fx.z, fy.z, fz.z, tmin, T.h.t);
        t[3] = box_test(T.r, nx.w, ny.w, nz.w, fx.w, fy.w, fz.w, tmin, T.h.t);
        // nearest first: 5 compare-exchanges sort the four (t, ref) pairs
#define RG_CSWAP(a, b)                                           \
        if (t[b] < t[a]) {                                       \
            float tt = t[a]; t[a] = t[b]; t[b] = tt;             \
            uint32_t rr = r[a]; r[a] = r[b]; r[b] = rr;          \
        }
        RG_CSWAP(0, 1) RG_CSWAP(2, 3) RG_CSWAP(0, 2) RG_CSWAP(1, 3) RG_CSWAP(1, 2)
#undef RG_CSWAP
        if (t[0] != INFINITY) {
            // with room for three, each is stored and kept by advancing: no branch per child
            if (T.sp + 3 <= STACK::kDepth) {
#pragma unroll
                for (int j = 3; j >= 1; --j) {
                    stack[T.sp] = r[j];
                    T.sp += t[j] != INFINITY ? 1 : 0;
                }
            } else {
#pragma unroll 1
                for (int j = 3; j >= 1; --j) {
                    const float tj = j == 3 ? t[3] : j == 2 ? t[2] : t[1];
                    const uint32_t rj = j == 3 ? r[3] : j == 2 ? r[2] : r[1];
                    if (tj == INFINITY) continue;
                    if (T.sp < STACK::kDepth) stack[T.sp++] = rj;
                    else stack.over() |= 1u;
                }
            }
            T.ref = r[0];
            return;
        }
    } else if (ref == kEmptySlot) {
        // an empty slot's box is inverted: only a ray whose box terms hold a NaN takes it
    } else if (T.inBlas) {
        if (COUNT) vc.tris++;
        const float4* tp = T.tris + 3 * (size_t)(ref & ~kLeaf);
        if (T.r.bits & kNoShear) ray_shear(T.r);
        tri_test(T.r, __ldg(tp), __ldg(tp + 1), __ldg(tp + 2), tmin, T.inst, T.h);
    } else {
        const InstRec* ir = sc.tlasLeaves + (ref & ~kLeaf);
        const float4 i0 = __ldg(&ir->inv[0]), i1 = __ldg(&ir->inv[1]), i2 = __ldg(&ir->inv[2]);
        const float4 lo = __ldg(&ir->lo), hi = __ldg(&ir->hi);
        const uint32_t bn = __float_as_uint(lo.w);
        if (bn > 0) {
            const float ox = T.r.ox, oy = T.r.oy, oz = T.r.oz, dx = T.r.dx, dy = T.r.dy, dz = T.r.dz;  // world ray (TLAS level)
            float qx = ((i0.x * ox + i0.y * oy) + i0.z * oz) + i0.w;
            float qy = ((i1.x * ox + i1.y * oy) + i1.z * oz) + i1.w;
            float qz = ((i2.x * ox + i2.y * oy) + i2.z * oz) + i2.w;
            float ex = (i0.x * dx + i0.y * dy) + i0.z * dz;
            float ey = (i1.x * dx + i1.y * dy) + i1.z * dz;
            float ez = (i2.x * dx + i2.y * dy) + i2.z * dz;
            if (!(ex == 0.0f && ey == 0.0f && ez == 0.0f)) {
                Ray orr;
                orr.dx = dx; orr.dy = dy; orr.dz = dz;  // the world direction stays in the ray
                ray_pre(orr, qx, qy, qz, ex, ey, ez, T.h.t);
                const float blo[3] = {lo.x, lo.y, lo.z}, bhi[3] = {hi.x, hi.y, hi.z};
                if (box_test6(orr, blo, bhi, tmin, T.h.t) != INFINITY) {
                    if (T.sp < STACK::kDepth) {
                        const ulonglong2 pp = __ldg(reinterpret_cast<const ulonglong2*>(&ir->wide));
                        stack.w(0) = ox; stack.w(1) = oy; stack.w(2) = oz;
                        stack.w(3) = T.r.jx; stack.w(4) = T.r.jy; stack.w(5) = T.r.jz;
                        stack[T.sp++] = kMarker;
                        T.r = orr;
                        T.nodes = reinterpret_cast<const WideNode*>(pp.x);
                        T.tris = reinterpret_cast<const float4*>(pp.y);
                        T.inst = __float_as_uint(hi.w);
                        T.inBlas = true;
                        if (SHARED) T.marker = true;
                        T.ref = bn == 1 ? kLeaf : 0u;
                        return;
                    }
                    stack.over() |= 1u;
                }
            }
        }
    }
    // pop (a marker leaves the BLAS: back to the world-space ray and the TLAS)
    for (;;) {
        if (T.sp == (SHARED ? T.sb : 0)) {
            T.active = false;
            return;
        }
        uint32_t nr = stack[--T.sp];
        if (nr != kMarker) {
            T.ref = nr;
            return;
        }
        T.inBlas = false;
        T.nodes = sc.tlasWide;
        T.r.ox = stack.w(0); T.r.oy = stack.w(1); T.r.oz = stack.w(2);
        box_terms(T.r.ox, stack.w(3), T.h.t, T.r.jx, T.r.clx, T.r.chx);
        box_terms(T.r.oy, stack.w(4), T.h.t, T.r.jy, T.r.cly, T.r.chy);
        box_terms(T.r.oz, stack.w(5), T.h.t, T.r.jz, T.r.clz, T.r.chz);
        T.r.bits = octant(T.r.jx, T.r.jy, T.r.jz) << 6;
        }
}

// Deep re-trace.  The short stack of the kernels (kTraversalStack entries in shared memory, or the
// batch tuner's depth) holds the far children of the records on the ray's current path: up to 3 per
// 4-wide record level, plus one marker while the ray is inside a BLAS.  Deep trees whose boxes the
// ray hits many at a time can need more.  A push that finds the short stack full sets Trav::over
// instead, and when that ray's traversal ends it is traced again from the start with this stack of
// kDeepStack entries in local memory, so its result is complete.  Every tree this library builds has
// at most 64 BVH2 levels (LBVH: 30 code bits plus at most 32 index bits of tie-break, one level per
// bit; binned SAH: kSahMedianLevel + 18), i.e. at most 32 record levels, so a TLAS path, a marker and
// a BLAS path take at most 3 * 32 + 1 + 3 * 32 = 193 entries.  Should a push still find it full, the
// ray is counted in counters[7] (rg_stats.deep_overflows), never silently.
constexpr int kDeepStack = 196;  // 195 entries and the overflow flag
__device__ __forceinline__ Hit deep_hit(const DevScene& sc, float4 o, float4 d, const LocalStackT<kDeepStack>& st, unsigned long long* counters) {
    VisitCounts vc = {0, 0, 0};
    Trav T;
    st.over() = 0u;
    trav_begin(T, sc, o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w, st);
    while (T.active) trav_step<false>(T, sc, st, vc);
    if (st.over() && counters) {
        atomicAdd(counters + 7, 1ull);
        atomicAdd(counters + 15, 1ull);
    }
    return T.h;
}
__device__ __noinline__ void retrace_deep(const DevScene* sc, float4 o, float4 d, Hit* out, unsigned long long* counters) {
    uint32_t mem[kDeepStack];
    float world[6];
    *out = deep_hit(*sc, o, d, LocalStackT<kDeepStack>{mem, world}, counters);
}

// ---------------------------------------------------------------------------------------------
// GLSL helpers with the oracle's operation order
struct V3 {
    float x, y, z;
};
__device__ __forceinline__ V3 v3(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ V3 v3s(float s) { return {s, s, s}; }
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 operator*(V3 a, V3 b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ V3 operator*(V3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ V3 operator-(V3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ float dot(V3 a, V3 b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }
__device__ __forceinline__ float clampf(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }
__device__ __forceinline__ V3 normalize(V3 v) {
    float l = sqrtf(dot(v, v));
    return {v.x / l, v.y / l, v.z / l};
}
__device__ __forceinline__ float mixs(float x, float y, float a) { return x * (1.0f - a) + y * a; }
__device__ __forceinline__ V3 mix(V3 x, V3 y, float a) { return {mixs(x.x, y.x, a), mixs(x.y, y.y, a), mixs(x.z, y.z, a)}; }
__device__ __forceinline__ V3 reflect(V3 I, V3 N) {
    float k = 2.0f * dot(N, I);
    return I - N * k;
}
__device__ __forceinline__ V3 refract(V3 I, V3 N, float eta) {
    float d = dot(N, I);
    float k = 1.0f - eta * eta * (1.0f - d * d);
    if (k < 0.0f) return v3s(0.0f);
    float s = eta * d + sqrtf(k);
    return I * eta - N * s;
}
__device__ __forceinline__ float glsl_mod(float x, float y) { return x - y * floorf(x / y); }
__device__ __forceinline__ float len(V3 v) { return sqrtf(dot(v, v)); }
__device__ __forceinline__ bool is_zero(V3 v) { return v.x == 0.0f && v.y == 0.0f && v.z == 0.0f; }

enum : int { RT_GENERIC = 0, RT_SHADOW_TRACE = 1, RT_SHADOW_INTERNAL = 2 };

struct Payload {  // payload.h:29-39
    V3 hitValue;
    float reflectContribution;
    V3 normal;
    V3 roughRGB;
    float roughA;
    float depth, curIOR, refDepth;
    int rayType, recDepth;
    uint32_t seed;  // glossy reference shading: per-sample random seed (0: mirror shading); not in payload.h
};

// resume codes of a paused closest-hit invocation
enum : int {
    R_G_SHADOW = 0,    // GENERIC, after the shadow ray (closesthit.rchit:193)
    R_G_REFLECT = 1,   // GENERIC, after the reflection ray (:215)
    R_G_REFR_F = 2,    // GENERIC, after the front-face refraction ray (:232)
    R_G_REFR_B = 3,    // GENERIC, after the back-face refraction ray (:244)
    R_SI_A = 4,        // SHADOW_INTERNAL, after the shadow-trace ray (:133)
    R_SI_B = 5,        // SHADOW_INTERNAL, after the mask-0 trace (:144)
    R_ST_C = 6         // SHADOW_TRACE, after the shadow-internal ray (:158)
};

struct __align__(16) Frame {
    int kind, front, rayConsumption, pad;
    V3 origin, D, n;
    float t;
    V3 diffuse, specular;
    float transparency, reflectivity, roughness, ior, emission;
    V3 base;          // GENERIC: baseColor; SHADOW_INTERNAL: shadowCol
    V3 shadow;        // GENERIC: shadowColor
    V3 reflectColor;  // GENERIC
    float reflectDepth;
    float pad1;
};
static_assert(sizeof(Frame) == 144, "frame");

// miss.rmiss:38-83
__device__ void sky(Payload& p, V3 D, V3 L) {
    const V3 sunTone = v3(1.0f, 0.6f, 0.05f), skyTone = v3(0.2f, 0.4f, 0.8f), scatterTone = v3(1.0f, 0.3f, 0.0f);
    const float scatterFactor = 1.3f, powFactor = 80.0f;
    V3 rayDir = normalize(D);
    float y = fabsf(D.y + 1.5f) / 3.0f;
    float sun = 1.0f - len(rayDir - normalize(-L));
    sun = clampf(sun, 0.0f, 2.0f);
    float glow = sun;
    glow = clampf(glow, 0.0f, 1.0f);
    sun = powf(sun, powFactor);
    sun = sun * 1000.0f;
    sun = clampf(sun, 0.0f, 16.0f);
    glow = glow * glow * glow * glow * glow * glow * 1.0f;
    glow = powf(glow, y);
    glow = clampf(glow, 0.0f, 1.0f);
    sun = sun * powf(y * y, 1.0f / 1.65f);
    glow = glow * powf(y * y, 1.0f / 2.0f);
    sun = sun + glow;
    V3 sunColor = sunTone * sun;
    float atmosphere = sqrtf(1.0f - y);
    float scatter = powf(4.0f - L.y, 1.0f / 15.0f);
    scatter = 1.0f - clampf(scatter, 0.8f, 1.0f);
    V3 scatterColor = mix(v3s(1.0f), scatterTone * 1.5f, scatter);
    V3 skyScatter = mix(skyTone, scatterColor, atmosphere / scatterFactor);
    V3 res = sunColor + skyScatter;
    p.hitValue = res;
    p.roughRGB = res;
    p.roughA = 0.0f;
    p.depth = 10000.0f;
}

__device__ __forceinline__ uint2 pack_half4(float a, float b, float c, float d) {
    __half2 lo = __floats2half2_rn(a, b), hi = __floats2half2_rn(c, d);
    return make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}

__constant__ float kAA[9][8][2] = {
    {{0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
    {{0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
    {{0.25f, 0.25f}, {-0.25f, -0.25f}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
    {{-0.125f, -0.375f}, {0.375f, -0.125f}, {-0.375f, 0.125f}, {0.125f, 0.375f}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
    {{-0.125f, -0.375f}, {0.375f, -0.125f}, {-0.375f, 0.125f}, {0.125f, 0.375f}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
    {{0.0625f, -0.1875f}, {-0.0625f, 0.1875f}, {0.3125f, 0.0625f}, {-0.1875f, -0.3125f}, {-0.3125f, 0.3125f}, {-0.4375f, -0.0625f}, {0.1875f, 0.4375f}, {0.4375f, -0.4375f}},
    {{0.0625f, -0.1875f}, {-0.0625f, 0.1875f}, {0.3125f, 0.0625f}, {-0.1875f, -0.3125f}, {-0.3125f, 0.3125f}, {-0.4375f, -0.0625f}, {0.1875f, 0.4375f}, {0.4375f, -0.4375f}},
    {{0.0625f, -0.1875f}, {-0.0625f, 0.1875f}, {0.3125f, 0.0625f}, {-0.1875f, -0.3125f}, {-0.3125f, 0.3125f}, {-0.4375f, -0.0625f}, {0.1875f, 0.4375f}, {0.4375f, -0.4375f}},
    {{0.0625f, -0.1875f}, {-0.0625f, 0.1875f}, {0.3125f, 0.0625f}, {-0.1875f, -0.3125f}, {-0.3125f, 0.3125f}, {-0.4375f, -0.0625f}, {0.1875f, 0.4375f}, {0.4375f, -0.4375f}},
};

// column-major mat4 * vec4 with the oracle's summation order
__device__ __forceinline__ void mul4(const float* m, float v0, float v1, float v2, float v3, float* o) {
#pragma unroll
    for (int r = 0; r < 4; ++r) o[r] = ((m[r] * v0 + m[4 + r] * v1) + m[8 + r] * v2) + m[12 + r] * v3;
}

enum : int { PH_HIT, PH_G_REFLECT, PH_G_REFRACT, PH_G_COMPOSE, PH_RETURN };

struct RayReq {
    V3 o, d;
    float tmin, tmax;
    int missIndex;
    bool masked;
};

struct RayCounts {  // per thread (flushed as 64-bit sums)
    uint32_t primary, shadow, secondary, masked;
};

__device__ __forceinline__ uint32_t pcg_hash(uint32_t v) {  // PCG-RXS-M-XS (O'Neill 2014) output permutation
    const uint32_t st = v * 747796405u + 2891336453u;
    const uint32_t w = ((st >> ((st >> 28u) + 4u)) ^ st) * 277803737u;
    return (w >> 22u) ^ w;
}

// Glossy reference shading: a GGX microfacet normal (Walter et al. 2007, alpha = roughness^2) drawn
// around n from two uniforms of the sample's seed and stream k
__device__ __forceinline__ V3 ggx_normal(V3 n, float roughness, uint32_t seed, uint32_t k) {
    const uint32_t h1 = pcg_hash(seed * 2654435761u + k), h2 = pcg_hash(h1 ^ 0x9E3779B9u);
    const float u1 = (float)(h1 >> 8) * (1.0f / 16777216.0f), u2 = (float)(h2 >> 8) * (1.0f / 16777216.0f);
    const float a = roughness * roughness;
    const float tan2 = a * a * u1 / fmaxf(1.0f - u1, 1e-7f);
    const float cosT = rsqrtf(1.0f + tan2), sinT = sqrtf(fmaxf(0.0f, 1.0f - cosT * cosT));
    const float phi = 6.28318530718f * u2;
    // orthonormal basis around n (Duff et al. 2017)
    const float sg = copysignf(1.0f, n.z), aa = -1.0f / (sg + n.z), bb = n.x * n.y * aa;
    const V3 t = v3(1.0f + sg * n.x * n.x * aa, sg * bb, -sg * n.x), b = v3(bb, sg + n.y * n.y * aa, -n.y);
    return normalize(t * (sinT * cosf(phi)) + b * (sinT * sinf(phi)) + n * cosT);
}

__device__ __forceinline__ void load_material(const rg_material* M, Frame& cur) {
    cur.diffuse = v3(__ldg(&M->diffuse[0]), __ldg(&M->diffuse[1]), __ldg(&M->diffuse[2]));
    cur.specular = v3(__ldg(&M->specular[0]), __ldg(&M->specular[1]), __ldg(&M->specular[2]));
    cur.transparency = __ldg(&M->transparency);
    cur.reflectivity = __ldg(&M->reflectivity);
    cur.roughness = __ldg(&M->roughness);
    cur.ior = __ldg(&M->ior);
    cur.emission = __ldg(&M->emission);
    cur.rayConsumption = (int)__ldg(&M->rayConsumption);
}

// gridEffect, closesthit.rchit:74-91
__device__ __forceinline__ void grid_effect(V3 pos, float refDepth, float hitT, Frame& cur) {
    float aa = ((refDepth + hitT) + 8.0f) / 30.0f;
    float aa2 = aa / 2.0f;
    float minmod = fminf(fabsf(glsl_mod((pos.x + 1000.0f) * 10.0f + aa2, 20.0f) - aa2),
                         fabsf(glsl_mod((pos.z + 1000.0f) * 10.0f + aa2, 20.0f) - aa2));
    if (minmod < aa2) {
        float aa_sq = aa * aa;
        minmod = minmod - (aa2 - aa_sq / 3.0f);
        minmod = minmod * (3.0f / aa_sq);
        float f = mixs(aa / 10.0f, 1.0f, minmod);
        cur.diffuse = cur.diffuse * f;
        cur.specular = cur.specular * f;
        cur.reflectivity = cur.reflectivity * f;
    }
    if (glsl_mod((pos.x + 1000.0f) * 5.0f, 20.0f) < 10.0f && glsl_mod((pos.z + 1000.0f) * 5.0f, 20.0f) < 10.0f)
        cur.reflectivity = cur.reflectivity * 1.5f;
}

// Whether the sign of the grid effect's factor f can depend on refDepth at pos.  With D the distance to
// the nearest line (in tenths of a unit) and a = (refDepth + t + 8) / 30, f <= 0 needs D <=
// a (1.5 - 1.15 a) / (3 - 0.3 a), which is at most 0.175 and negative from a = 1.305 on; refDepth only
// grows while siblings run.  The margins cover the rounding of pos * 10.
__device__ __forceinline__ bool grid_sign_varies(V3 pos, float refDepth, float hitT) {
    if (((refDepth + hitT) + 8.0f) / 30.0f > 1.32f) return false;
    const float wx = glsl_mod((pos.x + 1000.0f) * 10.0f, 20.0f), wz = glsl_mod((pos.z + 1000.0f) * 10.0f, 20.0f);
    const float d = fminf(fminf(wx, 20.0f - wx), fminf(wz, 20.0f - wz));
    return !(d > 0.25f);
}

// closesthit.rchit:95-122 of hit h of `ray`: attribute fetch, world position, world normal and grid
// effect (returned: whether the material has it); matId: the material's index
__device__ __forceinline__ bool closest_hit_surface(const DevScene& sc, const Hit& h, const RayReq& ray, float refDepth, Frame& cur,
                                                    uint32_t& matId) {
    const DevInstance* in = sc.inst + h.inst;
    const uint32_t vOff = __ldg(&in->vOff), iOff = __ldg(&in->iOff), mOff = __ldg(&in->mOff);
    const float4 m0 = __ldg(&in->m[0]), m1 = __ldg(&in->m[1]), m2 = __ldg(&in->m[2]);
    const float bx = (1.0f - h.u) - h.v, by = h.u, bz = h.v;
    const uint32_t ib = iOff + 3 * h.prim;
    const rg_vertex* v0 = sc.vertices + vOff + __ldg(sc.indices + ib);
    const rg_vertex* v1 = sc.vertices + vOff + __ldg(sc.indices + ib + 1);
    const rg_vertex* v2 = sc.vertices + vOff + __ldg(sc.indices + ib + 2);
    V3 n0 = v3(__ldg(&v0->normal[0]), __ldg(&v0->normal[1]), __ldg(&v0->normal[2]));
    V3 n1 = v3(__ldg(&v1->normal[0]), __ldg(&v1->normal[1]), __ldg(&v1->normal[2]));
    V3 n2 = v3(__ldg(&v2->normal[0]), __ldg(&v2->normal[1]), __ldg(&v2->normal[2]));
    matId = mOff + __ldg(&v0->matIndex);
    const rg_material* M = sc.materials + matId;
    load_material(M, cur);
    cur.origin = ray.o + ray.d * h.t;
    cur.D = ray.d;
    cur.t = h.t;
    V3 vn = (n0 * bx + n1 * by) + n2 * bz;
    V3 wn = v3((m0.x * vn.x + m0.y * vn.y) + m0.z * vn.z, (m1.x * vn.x + m1.y * vn.y) + m1.z * vn.z,
               (m2.x * vn.x + m2.y * vn.y) + m2.z * vn.z);
    cur.n = normalize(wn);
    const bool effect = __ldg(&M->effectId) == 1;
    if (effect) grid_effect(cur.origin, refDepth, h.t, cur);
    return effect;
}

// what a SHADOW_TRACE invocation reads of its hit: position and material
__device__ __forceinline__ void shadow_hit_surface(const DevScene& sc, const Hit& h, const RayReq& ray, Frame& cur, uint32_t& matId) {
    const DevInstance* in = sc.inst + h.inst;
    const rg_vertex* v0 = sc.vertices + __ldg(&in->vOff) + __ldg(sc.indices + __ldg(&in->iOff) + 3 * h.prim);
    matId = __ldg(&in->mOff) + __ldg(&v0->matIndex);
    cur.transparency = __ldg(&sc.materials[matId].transparency);
    cur.origin = ray.o + ray.d * h.t;
    cur.D = ray.d;
    cur.n = v3s(0.0f);
}

// the reflection and refraction directions of a GENERIC hit (closesthit.rchit:206-251), eta given; with
// glossy reference shading (a seed, at the sample's primary hit) through a sampled microfacet
template <bool GLOSSY>
__device__ __forceinline__ V3 reflect_dir(const Frame& cur, uint32_t seed, int recDepth) {
    V3 dir = reflect(cur.D, cur.n);
    if (GLOSSY && seed && recDepth == 0 && cur.roughness > 0.0f) {
        const V3 g = reflect(cur.D, ggx_normal(cur.n, cur.roughness, seed, 1u));
        if (dot(g, cur.n) > 0.0f) dir = g;
    }
    return dir;
}
template <bool GLOSSY>
__device__ __forceinline__ V3 refract_dir(const Frame& cur, float eta, uint32_t seed, int recDepth) {
    V3 dir = refract(cur.D, cur.n, eta);
    if (GLOSSY && seed && recDepth == 0 && cur.roughness > 0.0f) {
        const V3 g = refract(cur.D, ggx_normal(cur.n, cur.roughness, seed, 2u), eta);
        if (!is_zero(g)) dir = g;
    }
    return dir;
}

// One step of the closest-hit / miss state machine: consume the result `h` of the pending trace and
// run the paused invocations on the frame stack until the next trace is needed (returns true, `ray`
// set) or the sample's primary trace has returned (returns false).
template <bool GLOSSY = true>
__device__ __forceinline__ bool shade_step(const DevScene& sc, const V3 L, const int maxRec, const Hit& h, Payload& p, RayReq& ray,
                                           Frame* frames, int& fsp, Frame& cur, RayCounts& cnt) {
    int ph;
    if (!h.hit) {
        if (ray.missIndex == 0) sky(p, ray.d, L);
        else p.hitValue = v3s(1.0f);  // shadowMiss.rmiss:30-34
        ph = PH_RETURN;
    } else {
        ph = PH_HIT;
    }
    bool newRay = false;
    V3 refractColor = v3s(1.0f);
    while (!newRay) {
        if (ph == PH_HIT) {
            uint32_t matId;
            closest_hit_surface(sc, h, ray, p.refDepth, cur, matId);
            const float hitT = h.t;
            if (p.rayType == RT_SHADOW_INTERNAL) {  // :125-152
                float thick = clampf(hitT * (1.0f - cur.transparency) * 10.0f, 0.0f, 1.0f);
                V3 shadowCol = p.hitValue - mix(v3s(0.0f), normalize(v3s(1.1f) - cur.diffuse) + v3s(0.1f), thick);
                if (p.recDepth < maxRec) {
                    p.rayType = RT_SHADOW_TRACE;
                    p.recDepth++;
                    cnt.shadow++;
                    cur.base = shadowCol;
                    cur.kind = R_SI_A;
                    frames[fsp++] = cur;
                    ray.o = cur.origin; ray.d = cur.D; ray.tmin = 0.01f; ray.tmax = 1000.0f; ray.missIndex = 0; ray.masked = false;
                    newRay = true;
                } else {
                    p.hitValue = shadowCol * 0.4f;
                    ph = PH_RETURN;
                }
            } else if (p.rayType == RT_SHADOW_TRACE) {  // :153-166
                if (cur.transparency > 0.0f) {
                    if (p.recDepth < maxRec) {
                        p.rayType = RT_SHADOW_INTERNAL;
                        p.recDepth++;
                        cnt.shadow++;
                        cur.kind = R_ST_C;
                        frames[fsp++] = cur;
                        ray.o = cur.origin; ray.d = cur.D; ray.tmin = 0.01f; ray.tmax = 1000.0f; ray.missIndex = 1; ray.masked = false;
                        newRay = true;
                    } else {
                        ph = PH_RETURN;
                    }
                } else {
                    float f = mixs(0.4f, 0.8f, clampf(logf(hitT) / 8.0f, 0.0f, 1.0f));
                    p.hitValue = p.hitValue * f;
                    ph = PH_RETURN;
                }
            } else {  // GENERIC, :168-204
                cur.front = dot(-cur.D, cur.n) > 0.0f;
                if (!cur.front) cur.n = normalize(-cur.n);
                float ndl = dot(-L, cur.n);
                float dp = fmaxf(ndl, 0.2f);
                cur.base = cur.diffuse * dp;
                cur.reflectColor = v3s(1.0f);
                cur.reflectDepth = 0.0f;
                if (ndl > 0.07f) {
                    if (p.recDepth < maxRec) {
                        p.hitValue = v3s(1.0f);
                        p.rayType = RT_SHADOW_TRACE;
                        p.recDepth++;
                        cnt.shadow++;
                        cur.kind = R_G_SHADOW;
                        frames[fsp++] = cur;
                        ray.o = cur.origin; ray.d = -L; ray.tmin = 0.01f * 10.0f; ray.tmax = 1000.0f; ray.missIndex = 1; ray.masked = false;
                        newRay = true;
                    } else {
                        cur.shadow = v3s(1.0f);
                        ph = PH_G_REFLECT;
                    }
                } else {
                    float tr = cur.transparency;
                    float sm = tr * tr;
                    cur.shadow = tr < 1.0f ? mix(v3s(1.0f), cur.diffuse * sm, tr) : v3s(0.4f);
                    ph = PH_G_REFLECT;
                }
            }
        } else if (ph == PH_G_REFLECT) {  // :206-221
            if (p.recDepth < maxRec && cur.reflectivity > 0.0f) {
                const V3 dir = reflect_dir<GLOSSY>(cur, p.seed, p.recDepth);
                p.recDepth += cur.rayConsumption;
                p.refDepth = p.refDepth + cur.t;
                cnt.secondary++;
                cur.kind = R_G_REFLECT;
                frames[fsp++] = cur;
                ray.o = cur.origin; ray.d = dir; ray.tmin = 0.01f; ray.tmax = 1000.0f; ray.missIndex = 0; ray.masked = false;
                newRay = true;
            } else {
                ph = PH_G_REFRACT;
            }
        } else if (ph == PH_G_REFRACT) {  // :223-251
            if (p.recDepth < maxRec && cur.transparency > 0.0f) {
                const V3 dir = refract_dir<GLOSSY>(cur, cur.front ? p.curIOR / cur.ior : cur.ior / 1.0f, p.seed, p.recDepth);
                p.curIOR = cur.front ? cur.ior : 1.0f;
                cur.kind = cur.front ? R_G_REFR_F : R_G_REFR_B;
                p.recDepth++;
                if (!is_zero(dir)) cnt.secondary++;  // only rays that traverse
                frames[fsp++] = cur;
                ray.o = cur.origin; ray.d = dir; ray.tmin = 0.01f; ray.tmax = 1000.0f; ray.missIndex = 0; ray.masked = false;
                newRay = true;
            } else {
                refractColor = v3s(1.0f);
                ph = PH_G_COMPOSE;
            }
        } else if (ph == PH_G_COMPOSE) {  // :253-267
            V3 baseColor = cur.base * cur.shadow;
            baseColor = baseColor + cur.diffuse * cur.emission;
            float total = fmaxf(cur.transparency, cur.reflectivity);
            float den = cur.transparency + cur.reflectivity;
            float w = den == 0.0f ? 0.0f : cur.reflectivity / den;
            V3 roughCol = mix(refractColor, cur.reflectColor, w);
            p.hitValue = mix(baseColor, roughCol, total);
            if (p.recDepth == 0) {
                p.hitValue = baseColor;
                p.normal = cur.n;
                p.roughRGB = roughCol;
                p.roughA = fminf((cur.reflectDepth / 50.0f) * cur.roughness, cur.roughness / 2.1f);
                p.reflectContribution = total;
            }
            p.depth = cur.t;
            ph = PH_RETURN;
        } else {  // PH_RETURN: resume the paused invocation
            if (fsp == 0) break;
            cur = frames[--fsp];
            switch (cur.kind) {
                case R_G_SHADOW:
                    p.recDepth--;
                    cur.shadow = p.hitValue;
                    p.rayType = RT_GENERIC;
                    ph = PH_G_REFLECT;
                    break;
                case R_G_REFLECT:
                    p.recDepth -= cur.rayConsumption;
                    cur.reflectColor = p.hitValue * cur.specular;
                    cur.reflectDepth = p.depth;
                    ph = PH_G_REFRACT;
                    break;
                case R_G_REFR_F:
                    p.recDepth--;
                    refractColor = p.hitValue;
                    ph = PH_G_COMPOSE;
                    break;
                case R_G_REFR_B:
                    p.recDepth--;
                    refractColor = mix(v3s(1.0f), cur.diffuse, logf(1.0f + cur.t)) * p.hitValue;
                    ph = PH_G_COMPOSE;
                    break;
                case R_SI_A:
                    p.recDepth--;
                    if (p.depth < 1000.0f) {
                        p.hitValue = p.hitValue * cur.base;
                        ph = PH_RETURN;
                    } else {
                        float eta = cur.ior / 1.0f;
                        V3 dir = refract(cur.D, cur.n, eta);
                        float x = dot(L, dir);
                        float dp = x * x * x * x * x + 0.75f;
                        cur.base = cur.base * dp;
                        cur.kind = R_SI_B;
                        frames[fsp++] = cur;
                        cnt.masked++;
                        ray.o = cur.origin; ray.d = -dir; ray.tmin = 0.01f; ray.tmax = 1000.0f; ray.missIndex = 0; ray.masked = true;
                        newRay = true;
                    }
                    break;
                case R_SI_B:
                    p.hitValue = cur.base + p.hitValue * 0.1f;
                    ph = PH_RETURN;
                    break;
                default:  // R_ST_C
                    p.recDepth--;
                    ph = PH_RETURN;
                    break;
            }
        }
    }
    return newRay;
}

// raygen.h:84-102: camera ray of one sample and the payload initialisation
__device__ __forceinline__ void start_sample(const rg_ubo& U, const V3 camO, uint32_t px, uint32_t py, uint32_t W, uint32_t H,
                                             int sample, int aaRow, Payload& p, RayReq& ray, uint32_t glossySeed = 0u) {
    float pcx = ((float)px + 0.5f) + kAA[aaRow][sample & 7][0];
    float pcy = ((float)py + 0.5f) + kAA[aaRow][sample & 7][1];
    float ux = pcx / (float)W, uy = pcy / (float)H;
    float dx = ux * 2.0f - 1.0f, dy = uy * 2.0f - 1.0f;
    float tg[4], dw[4];
    mul4(U.projInverse, dx, dy, 1.0f, 1.0f, tg);
    V3 tn = normalize(v3(tg[0], tg[1], tg[2]));
    mul4(U.viewInverse, tn.x, tn.y, tn.z, 0.0f, dw);
    ray.o = camO;
    ray.d = v3(dw[0], dw[1], dw[2]);
    ray.tmin = 0.001f;
    ray.tmax = 10000.0f;
    ray.missIndex = 0;
    ray.masked = false;
    p.hitValue = v3s(0.0f);
    p.normal = v3s(0.0f);
    p.roughRGB = v3s(0.0f);
    p.roughA = 0.0f;
    p.depth = 0.0f;
    p.refDepth = 0.0f;
    p.curIOR = 1.0f;
    p.rayType = RT_GENERIC;
    p.recDepth = 0;
    p.reflectContribution = 0.0f;
    p.seed = glossySeed ? ((pcg_hash(glossySeed ^ pcg_hash(px + pcg_hash(py + pcg_hash((uint32_t)sample)))) & 0xFFFFFFu) | 1u) : 0u;
}

#ifndef RG_TRACE_STEPS
#define RG_TRACE_STEPS 4
#endif
#ifndef RG_SHADE_THRESHOLD
#define RG_SHADE_THRESHOLD 16
#endif
enum : int { kIdle = 0, kTraverse = 1, kResult = 2 };

// starts the traversal of the pending trace; mask-0 traces and zero directions need none
template <class STACK>
__device__ __forceinline__ int begin_ray(Trav& T, const DevScene& sc, const RayReq& ray, const STACK& stack) {
    stack.over() = 0u;
    if (ray.masked) {
        T.h.hit = false;
        T.active = false;
        return kResult;
    }
    trav_begin(T, sc, ray.o.x, ray.o.y, ray.o.z, ray.d.x, ray.d.y, ray.d.z, ray.tmin, ray.tmax, stack);
    return T.active ? kTraverse : kResult;
}

// (kTileW x kTileH, the 32 pixels of one work tile, are declared in rg_internal.cuh)

// Persistent kernel: each lane takes (pixel, sample) work items from a global counter -- in
// warp-aggregated batches -- and runs the sample's whole depth-first trace sequence.  Traversal is
// resumable: every loop iteration advances each lane's ray by up to RG_TRACE_STEPS nodes, and a
// lane whose ray finished shades it and starts its next ray (or takes the next work item) while
// the other lanes keep traversing, so no lane idles behind the longest ray of its warp.  Work items
// enumerate 8x4 pixel tiles, then pixels, then samples, so consecutive items are coherent.
// Each sample's payload sums go to `samples` (12 floats); k_resolve averages them in sample order.
template <bool COUNT>
__global__ void __launch_bounds__(kTraceThreads, RG_TRACE_MIN_BLOCKS) k_trace(const __grid_constant__ TraceParams P) {
    RG_DECLARE_STACK(stk);
    const DevScene& sc = P.scene;
    const rg_ubo& U = P.ubo;
    const V3 L = v3(U.lightDir[0], U.lightDir[1], U.lightDir[2]);
    const int maxRec = U.maxRecursions;
    const uint32_t S = (uint32_t)U.numSamples;
    const int aaRow = S < 8 ? (int)S : 8;
    const uint32_t tilesX = (P.W + kTileW - 1) / kTileW, tilesY = (P.H + kTileH - 1) / kTileH;
    const uint32_t total = tilesX * tilesY * (kTileW * kTileH) * S;
    const unsigned lane = threadIdx.x & 31;
    const unsigned ltmask = (1u << lane) - 1u;

    float org[4];
    mul4(U.viewInverse, 0.0f, 0.0f, 0.0f, 1.0f, org);
    const V3 camO = v3(org[0], org[1], org[2]);

    RayCounts cnt = {0, 0, 0, 0};
    VisitCounts vc = {0, 0, 0};
    Frame frames[kMaxFrames];
    int fsp = 0;
    Payload p;
    RayReq ray;
    Frame cur;
    Trav T;
    T.active = false;
    bool alive = true;
    int state = kIdle;
    uint32_t px = 0, py = 0, sample = 0;

    for (;;) {
        // A shading round runs when at least RG_SHADE_THRESHOLD lanes of the warp wait (finished ray
        // or no work) or no lane is traversing: the waiting lanes shade together, idle lanes take new
        // work items (one atomic per warp), then every lane with a ray continues traversing.
        const unsigned travMask = __ballot_sync(0xFFFFFFFFu, state == kTraverse);
        const unsigned waitMask = __ballot_sync(0xFFFFFFFFu, state == kResult || (alive && state == kIdle));
        if (travMask == 0 || __popc(waitMask) >= RG_SHADE_THRESHOLD) {
            if (state == kResult) {
                // closest-hit / miss shading of the finished trace, up to the next trace
                if (shade_step(sc, L, maxRec, T.h, p, ray, frames, fsp, cur, cnt)) {
                    state = begin_ray(T, sc, ray, stk);
                } else {
                    float4* o = P.samples + 3 * ((size_t)(py * P.W + px) * S + sample);
                    o[0] = make_float4(p.hitValue.x, p.hitValue.y, p.hitValue.z, p.reflectContribution);
                    o[1] = make_float4(p.normal.x, p.normal.y, p.normal.z, p.depth);
                    o[2] = make_float4(p.roughRGB.x, p.roughRGB.y, p.roughRGB.z, p.roughA);
                    state = kIdle;
                }
            }
            const bool need = alive && state == kIdle;
            const unsigned needMask = __ballot_sync(0xFFFFFFFFu, need);
            if (needMask) {
                const int leader = __ffs(needMask) - 1;
                uint32_t base = 0;
                if ((int)lane == leader) base = atomicAdd(P.workCounter, (uint32_t)__popc(needMask));
                base = __shfl_sync(0xFFFFFFFFu, base, leader);
                if (need) {
                    const uint32_t id = base + (uint32_t)__popc(needMask & ltmask);
                    if (id >= total) {
                        alive = false;
                    } else {
                        sample = id % S;
                        const uint32_t pid = id / S, tile = pid / (kTileW * kTileH), within = pid % (kTileW * kTileH);
                        px = (tile % tilesX) * kTileW + within % kTileW;
                        py = (tile / tilesX) * kTileH + within / kTileW;
                        if (px < P.W && py < P.H) {
                            start_sample(U, camO, px, py, P.W, P.H, (int)sample, aaRow, p, ray, P.glossySeed);
                            cnt.primary++;
                            fsp = 0;
                            state = begin_ray(T, sc, ray, stk);
                        }
                    }
                }
            }
            if (!__any_sync(0xFFFFFFFFu, alive)) break;
        }
        if (state == kTraverse) {
#pragma unroll 1
            for (int k = 0; k < RG_TRACE_STEPS; ++k) {
                trav_step<COUNT>(T, sc, stk, vc);
                if (!T.active) {
                    if (stk.over()) {
                        vc.overflow++;
                        retrace_deep(&sc, make_float4(ray.o.x, ray.o.y, ray.o.z, ray.tmin), make_float4(ray.d.x, ray.d.y, ray.d.z, ray.tmax),
                                     &T.h, P.counters);
                    }
                    state = kResult;
                    break;
                }
            }
        }
    }

    // ray statistics: warp reduction then one atomic per warp (all lanes are here)
    unsigned long long c[7] = {cnt.primary, cnt.shadow, cnt.secondary, cnt.masked, vc.nodes, vc.tris, vc.overflow};
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        unsigned long long v = c[k];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
        if (lane == 0 && v) {
            atomicAdd(P.counters + k, v);
            atomicAdd(P.counters + 8 + k, v);
        }
    }
}

// raygen.h:116 + raygen.rgen:36-38: average one pixel's S samples (in sample order) into the three
// RGBA16F G-buffer images; normal.w = log(sum of depths) * 0.25 / S
__device__ __forceinline__ void resolve_pixel(const float4* s, uint32_t S, size_t pix, uint2* base, uint2* normal, uint2* rough) {
    float4 a = s[0], b = s[1], c = s[2];
    for (uint32_t k = 1; k < S; ++k) {
        const float4 a2 = s[3 * k], b2 = s[3 * k + 1], c2 = s[3 * k + 2];
        a.x = a.x + a2.x; a.y = a.y + a2.y; a.z = a.z + a2.z; a.w = a.w + a2.w;
        b.x = b.x + b2.x; b.y = b.y + b2.y; b.z = b.z + b2.z; b.w = b.w + b2.w;
        c.x = c.x + c2.x; c.y = c.y + c2.y; c.z = c.z + c2.z; c.w = c.w + c2.w;
    }
    const float fs = (float)S;
    base[pix] = pack_half4(a.x / fs, a.y / fs, a.z / fs, a.w / fs);
    normal[pix] = pack_half4(b.x / fs, b.y / fs, b.z / fs, (logf(b.w) * 0.25f) / fs);
    rough[pix] = pack_half4(c.x / fs, c.y / fs, c.z / fs, c.w / fs);
}

__global__ void k_resolve(const TraceParams P) {
    chain_wait();
    const uint32_t x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (x >= P.W || y >= P.H) return;
    const uint32_t S = (uint32_t)P.ubo.numSamples;
    const size_t pix = (size_t)y * P.W + x;
    resolve_pixel(P.samples + 3 * pix * S, S, pix, P.base, P.normal, P.rough);
}

// samples: the job's first sample (samples + 3 * sampleBase)
__global__ void k_resolve_job(const float4* __restrict__ samples, uint32_t W, uint32_t H, uint32_t S, uint2* base, uint2* normal,
                              uint2* rough) {
    const uint32_t x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (x >= W || y >= H) return;
    const size_t pix = (size_t)y * W + x;
    resolve_pixel(samples + 3 * pix * S, S, pix, base, normal, rough);
}

// ---------------------------------------------------------------------------------------------
// Frames and batches: rays traced by launches of one traversal kernel, between them what the hits need.

__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, bool want) {
    const unsigned mask = __ballot_sync(0xFFFFFFFFu, want);
    if (!mask) return 0;
    const unsigned lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if ((int)lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    return base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}

__device__ __forceinline__ void flush_counts(const TraceParams& P, unsigned long long* c, int n) {
    const unsigned lane = threadIdx.x & 31;
    for (int k = 0; k < n; ++k) {
        unsigned long long v = c[k];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
        c[k] = v;
    }
    if (lane == 0)
        for (int k = 0; k < n; ++k)
            if (c[k]) {
                atomicAdd(P.counters + k, c[k]);
                atomicAdd(P.counters + 8 + k, c[k]);
            }
}

// work item -> pixel and sample: work items enumerate 8x4 pixel tiles (row-major over the tile
// grid), then the 32 pixels of a tile (row-major), then the samples of a pixel
__device__ __forceinline__ bool decode_work(uint32_t id, uint32_t W, uint32_t H, uint32_t S, uint32_t tilesX, uint32_t& px,
                                            uint32_t& py, uint32_t& sample) {
    sample = id % S;
    const uint32_t pid = id / S, tile = pid / (kTileW * kTileH), within = pid % (kTileW * kTileH);
    px = (tile % tilesX) * kTileW + within % kTileW;
    py = (tile / tilesX) * kTileH + within / kTileW;
    return px < W && py < H;
}

// the job owning work item `id`: the last job whose workBase <= id (jobs are in work order)
__device__ __forceinline__ uint32_t find_job(const JobDesc* __restrict__ jobs, uint32_t n, uint32_t id) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (jobs[mid].workBase <= id) lo = mid;
        else hi = mid;
    }
    return lo;
}

// camera ray and fresh payload of work item `id` of a batch (raygen.h:84-102 with the job's UBO);
// false when the item's pixel lies outside its image
__device__ __forceinline__ bool batch_primary(const TraceParams& P, uint32_t id, uint32_t& job, uint32_t& sampleIdx, Payload& p,
                                              RayReq& ray) {
    job = find_job(P.jobs, P.njobs, id);
    const JobDesc& J = P.jobs[job];
    uint32_t px, py, s;
    if (!decode_work(id - J.workBase, J.W, J.H, J.S, J.tilesX, px, py, s)) return false;
    float org[4];
    mul4(J.ubo.viewInverse, 0.0f, 0.0f, 0.0f, 1.0f, org);
    const int aaRow = J.S < 8 ? (int)J.S : 8;
    start_sample(J.ubo, v3(org[0], org[1], org[2]), px, py, J.W, J.H, (int)s, aaRow, p, ray, P.glossySeed);
    sampleIdx = J.sampleBase + (py * J.W + px) * J.S + s;
    return true;
}

__device__ __forceinline__ void store_sample(float4* so, const Payload& p) {
    so[0] = make_float4(p.hitValue.x, p.hitValue.y, p.hitValue.z, p.reflectContribution);
    so[1] = make_float4(p.normal.x, p.normal.y, p.normal.z, p.depth);
    so[2] = make_float4(p.roughRGB.x, p.roughRGB.y, p.roughRGB.z, p.roughA);
}

// work items of a frame: one per (pixel, sample) in 8x4-tile order; path = (py * W + px) * S + sample
// camera ray and initial payload of work item id (raygen.h:84-102); false outside the image
__device__ __forceinline__ bool frame_work_item(const TraceParams& P, uint32_t id, uint32_t& path, Payload& p, RayReq& ray) {
    const rg_ubo& U = P.ubo;
    const uint32_t S = (uint32_t)U.numSamples;
    const uint32_t tilesX = (P.W + kTileW - 1) / kTileW;
    uint32_t px = 0, py = 0, sample = 0;
    if (!decode_work(id, P.W, P.H, S, tilesX, px, py, sample)) return false;
    float org[4];
    mul4(U.viewInverse, 0.0f, 0.0f, 0.0f, 1.0f, org);
    start_sample(U, v3(org[0], org[1], org[2]), px, py, P.W, P.H, (int)sample, S < 8 ? (int)S : 8, p, ray, P.glossySeed);
    path = (py * P.W + px) * S + sample;
    return true;
}

// The chunk of samples whose trees are grown: its roots, its first work item and the candidate list in use.
// A frame's host loop passes them; a batch's chunks are set up on the device (k_tree_next).
template <bool BATCH>
__device__ __forceinline__ uint32_t tree_roots(const TraceParams& P) { return BATCH ? P.tree.ctl[kTreeRoots] : P.treeRoots; }
template <bool BATCH>
__device__ __forceinline__ uint32_t tree_base(const TraceParams& P) { return BATCH ? P.tree.ctl[kTreeBase] : P.treeBase; }
template <bool BATCH>
__device__ __forceinline__ uint32_t tree_cand(const TraceParams& P) { return BATCH ? P.tree.ctl[kTreeCandList] : P.treeCand; }

// the camera ray of root k of the chunk, its fresh payload and its sample index; false outside the image
template <bool BATCH>
__device__ __forceinline__ bool tree_root(const TraceParams& P, uint32_t k, uint32_t& job, uint32_t& sample, Payload& p, RayReq& ray) {
    job = 0;
    if (BATCH) return batch_primary(P, tree_base<BATCH>(P) + k, job, sample, p, ray);
    return frame_work_item(P, tree_base<BATCH>(P) + k, sample, p, ray);
}
#ifndef RG_DRAIN_LANES
#define RG_DRAIN_LANES 8
#endif
#ifndef RG_DRAIN_ROUNDS
#define RG_DRAIN_ROUNDS 2
#endif
// The end of a launch of few rays: it lasts as long as its longest ray, whose record steps (up to 90 on
// the sphere scene, 200 on the game frame) wait for memory one after another while the other lanes of
// its warp idle.  The closest hit does not depend on the order in which subtrees are visited, so the
// warp's idle lanes take them over: each live lane gives the bottom entry of its stack (the largest
// subtree left) to an idle lane, with the ray at that entry's level.  Lanes of one ray share the best t as
// hits are found; a lane that finishes hands its hit to another lane of the same ray, and the last one
// writes it.  Ties go to the smaller (instance, primitive) as everywhere, so the hit is the one the ray's
// own lane would have found.  One game-frame ray of 153 records: 43 us against 57; the 1280x720 game frame
// with the filter: 2.20 ms against 2.25 ms without.  From RG_DRAIN_LANES live lanes on only: with 16 and
// 32 the sphere frame is 1 % and 7 % slower.
template <bool COUNT, class STACK, class SceneOf, class HitOut>
__device__ __forceinline__ void drain(Trav& T, uint32_t& slot, const DevScene*& scp, const STACK& stk, VisitCounts& vc, SceneOf&& sceneOf,
                                      HitOut&& hitOut) {
    const unsigned lane = threadIdx.x & 31, full = 0xFFFFFFFFu, below = (1u << lane) - 1u;
    T.sb = 0;
    T.marker = T.inBlas;
    for (;;) {
        const unsigned live = __ballot_sync(full, T.active);
        if (!live) break;
        // what the lane can give: TLAS entry (bottom of a stack at TLAS level or below the marker), or
        // a BLAS entry (just above the marker, or the bottom of a stack without one)
        const int held = T.active ? T.sp - T.sb : 0;
        const bool atMarker = held > 0 && T.inBlas && T.marker && stk[T.sb] == kMarker;
        const unsigned givers = __ballot_sync(full, held > (atMarker ? 1 : 0));
        if (givers && live != full) {
            const unsigned idle = ~live;
            const int pairs = min(__popc(givers), __popc(idle));
            const bool gives = (givers >> lane & 1u) && __popc(givers & below) < pairs;
            const bool takes = (idle >> lane & 1u) && __popc(idle & below) < pairs;
            const bool blasLevel = T.inBlas && (atMarker || !T.marker);
            uint32_t entry = 0;
            if (gives) {
                entry = stk[T.sb + (atMarker ? 1 : 0)];
                if (atMarker) stk[T.sb + 1] = kMarker;
                ++T.sb;
                if (!T.inBlas) {  // the taker reads the world ray where a ray inside a BLAS has parked it
                    stk.w(0) = T.r.ox; stk.w(1) = T.r.oy; stk.w(2) = T.r.oz;
                    stk.w(3) = T.r.jx; stk.w(4) = T.r.jy; stk.w(5) = T.r.jz;
                }
            }
            __syncwarp();
            unsigned from = lane;
            if (takes) {  // the giver of the same rank
                unsigned m = givers;
                for (int r = __popc(idle & below); r > 0; --r) m &= m - 1u;
                from = (unsigned)__ffs(m) - 1u;
            }
            Trav N;
            N.tmin = __shfl_sync(full, T.tmin, from);
            N.h.t = __shfl_sync(full, T.h.t, from);
            N.ref = __shfl_sync(full, entry, from);
            N.inst = __shfl_sync(full, T.inst, from);
            N.inBlas = __shfl_sync(full, (int)blasLevel, from) != 0;
            N.nodes = reinterpret_cast<const WideNode*>(__shfl_sync(full, reinterpret_cast<unsigned long long>(T.nodes), from));
            N.tris = reinterpret_cast<const float4*>(__shfl_sync(full, reinterpret_cast<unsigned long long>(T.tris), from));
            N.r.ox = __shfl_sync(full, T.r.ox, from); N.r.oy = __shfl_sync(full, T.r.oy, from); N.r.oz = __shfl_sync(full, T.r.oz, from);
            N.r.dx = __shfl_sync(full, T.r.dx, from); N.r.dy = __shfl_sync(full, T.r.dy, from); N.r.dz = __shfl_sync(full, T.r.dz, from);
            N.r.jx = __shfl_sync(full, T.r.jx, from); N.r.jy = __shfl_sync(full, T.r.jy, from); N.r.jz = __shfl_sync(full, T.r.jz, from);
            N.r.clx = __shfl_sync(full, T.r.clx, from); N.r.cly = __shfl_sync(full, T.r.cly, from); N.r.clz = __shfl_sync(full, T.r.clz, from);
            N.r.chx = __shfl_sync(full, T.r.chx, from); N.r.chy = __shfl_sync(full, T.r.chy, from); N.r.chz = __shfl_sync(full, T.r.chz, from);
            N.r.Sx = __shfl_sync(full, T.r.Sx, from); N.r.Sy = __shfl_sync(full, T.r.Sy, from); N.r.Sz = __shfl_sync(full, T.r.Sz, from);
            N.r.bits = __shfl_sync(full, T.r.bits, from);
            const uint32_t slotN = __shfl_sync(full, slot, from);
            const DevScene* scN = reinterpret_cast<const DevScene*>(__shfl_sync(full, reinterpret_cast<unsigned long long>(scp), from));
            if (takes) {
                slot = slotN;
                scp = scN;
                N.h.hit = false;
                N.h.u = N.h.v = 0.0f;
                N.h.inst = N.h.prim = 0xFFFFFFFFu;
                N.sp = N.sb = 0;
                N.marker = false;
                N.active = true;
                if (!N.inBlas) {
                    const float* w = stk.saved + ((int)from - (int)lane);
                    N.r.ox = w[0]; N.r.oy = w[STACK::kStride]; N.r.oz = w[2 * STACK::kStride];
                    box_terms(N.r.ox, w[3 * STACK::kStride], N.h.t, N.r.jx, N.r.clx, N.r.chx);
                    box_terms(N.r.oy, w[4 * STACK::kStride], N.h.t, N.r.jy, N.r.cly, N.r.chy);
                    box_terms(N.r.oz, w[5 * STACK::kStride], N.h.t, N.r.jz, N.r.clz, N.r.chz);
                    N.r.bits = octant(N.r.jx, N.r.jy, N.r.jz) << 6;
                    N.nodes = sceneOf(scN).tlasWide;
                    N.tris = nullptr;
                }
                T = N;
            }
            __syncwarp();
        }
        const bool was = T.active;
        const float before = T.h.t;
#pragma unroll 1
        for (int j = 0; j < RG_DRAIN_ROUNDS; ++j) {
            const bool inner = T.active && !(T.ref & kLeaf);
            if (!__any_sync(full, inner)) break;
            if (inner) trav_step<COUNT, true>(T, sceneOf(scp), stk, vc);
        }
        if (T.active && (T.ref & kLeaf)) trav_step<COUNT, true>(T, sceneOf(scp), stk, vc);
        // a closer hit shortens the ray for its other lanes
        for (unsigned m = __ballot_sync(full, T.h.t < before && T.h.hit); m; m &= m - 1u) {
            const int f = __ffs(m) - 1;
            const float t = __shfl_sync(full, T.h.t, f);
            if (__shfl_sync(full, slot, f) == slot && T.h.t > t) {
                T.h.t = t;
                T.h.hit = false;
            }
        }
        for (unsigned m = __ballot_sync(full, was && !T.active); m;) {
            const int f = __ffs(m) - 1;
            m &= m - 1u;
            const uint32_t sf = __shfl_sync(full, slot, f);
            const unsigned peers = __ballot_sync(full, (T.active || (m >> lane & 1u)) && slot == sf);
            if (!peers) {
                if ((int)lane == f) hitOut();
                continue;
            }
            Hit h;
            h.t = __shfl_sync(full, T.h.t, f);
            h.u = __shfl_sync(full, T.h.u, f);
            h.v = __shfl_sync(full, T.h.v, f);
            h.inst = __shfl_sync(full, T.h.inst, f);
            h.prim = __shfl_sync(full, T.h.prim, f);
            h.hit = __shfl_sync(full, (int)T.h.hit, f) != 0;
            const uint32_t over = __shfl_sync(full, stk.over() & 1u, f);
            if ((int)lane == __ffs(peers) - 1) {
                if (h.hit && accept(h.t, h.t, h.inst, h.prim, T.h)) T.h = h;
                stk.over() |= over;
            } else if ((int)lane == f) {
                stk.over() &= ~1u;
            }
        }
    }
}

// closest hit of every ray of a set.  Lanes whose ray finished take new rays (one atomic per warp) as
// soon as RG_FETCH_THRESHOLD lanes of the warp are idle, so a warp does not wait for its longest ray;
// between fetches every lane advances its ray by RG_WF_STEPS steps.  Its forms:
//   kFormTree   the nodes of one round of a frame's ray trees (q: the round); the first round computes
//               the camera rays of the roots itself;
//   kFormBatch  the same for a batch; the ray's scene is its job's scene, and P.perm (nullable) gives the
//               order the rays are taken in;
//   kFormQuery  rg_trace_rays_device: rays and hits in the caller's buffers.
enum TraceForm : int { kFormTree, kFormBatch, kFormQuery };
#ifndef RG_FETCH_THRESHOLD
#define RG_FETCH_THRESHOLD 8
#endif
#ifndef RG_WF_STEPS
#define RG_WF_STEPS 6
#endif
#ifndef RG_INNER_ROUNDS
#define RG_INNER_ROUNDS 3
#endif
// Shared memory: the stack (DEPTH words) and the parked world ray (6 words) per thread, nothing else:
// at 128 threads x 48 words that is 27,648 B, and 7 blocks (plus the 1 KB the driver reserves per
// block) fill the 196 KB shared-memory carve-out exactly.  One more byte per block moves the SM to
// the 228 KB carve-out and halves the L1 left for BVH records (measured: trace stage +5 %).
// a finished ray's hit: the frame loop's hit record (t, u, v, primitive; instance or 0xFFFFFFFF), or
// for a ray query rg_trace_rays' layout in the caller's buffers (t, u, v and (instance, primitive);
// zeros and 0xFFFFFFFF for a miss)
template <TraceForm FORM>
__device__ __forceinline__ void put_hit(const TraceParams& P, uint32_t slot, const Hit& h, bool hit) {
    if (FORM == kFormQuery) {
        float* t = P.queryTuv + 3 * (size_t)slot;
        uint32_t* id = P.queryIds + 2 * (size_t)slot;
        t[0] = hit ? h.t : 0.0f;
        t[1] = hit ? h.u : 0.0f;
        t[2] = hit ? h.v : 0.0f;
        id[0] = hit ? h.inst : 0xFFFFFFFFu;
        id[1] = hit ? h.prim : 0xFFFFFFFFu;
    } else {
        P.tree.hitTUV[slot] = make_float4(h.t, h.u, h.v, __uint_as_float(h.prim));
        P.tree.hitInst[slot] = hit ? h.inst : 0xFFFFFFFFu;
    }
}

// lanes of a warp that take rays in a launch of `count`, and blocks that have rays
__device__ __forceinline__ uint32_t trace_width(uint32_t count, uint32_t threads) {
    const uint32_t warps = gridDim.x * (threads / 32);
    return min(32u, max(1u, (count + warps - 1u) / warps));
}
__device__ __forceinline__ uint32_t trace_workers(uint32_t count, uint32_t threads) {
    const uint32_t perBlock = trace_width(count, threads) * (threads / 32);
    return min(gridDim.x, (count + perBlock - 1u) / perBlock);
}

template <bool COUNT, TraceForm FORM, int THREADS, int DEPTH>
__global__ void __launch_bounds__(THREADS, (RG_WF_MIN_BLOCKS * 128) / THREADS) k_wf_trace(const __grid_constant__ TraceParams P, int q) {
    chain_wait();
    RG_DECLARE_SMEM_STACK(stk, THREADS, DEPTH);
    stk.over() = 0u;
    const TraceWork& wf = P.wf;
    constexpr bool BATCH = FORM == kFormBatch, QUERY = FORM == kFormQuery, TREE = !QUERY;
    const bool first = TREE && P.firstRound;
    uint32_t node0 = 0, count;  // TREE: the round's first node
    if (BATCH && q < 0) q = (int)P.tree.ctl[kTreeRound];
    if (TREE) {
        node0 = first ? 0u : P.tree.ctl[kTreeBounds + q];
        const uint32_t roots = tree_roots<BATCH>(P);
        const uint32_t end = first ? roots : min(roots + *(volatile uint32_t*)(P.tree.ctl + kTreeAlloc), P.tree.capacity);
        count = end - node0;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            P.tree.ctl[kTreeBounds + q + 1] = end;  // the next round's first node
            P.tree.ctl[kTreeChanges] = P.tree.ctl[kTreeLevels] = P.tree.ctl[kTreeCand + (tree_cand<BATCH>(P) ^ 1u)] = 0;  // k_tree_check's
            if (BATCH) P.tree.ctl[kTreeTracedRound] = (uint32_t)q;
        }
    } else {
        count = P.queryCount;
    }
    const unsigned lane = threadIdx.x & 31;
    const unsigned ltmask = (1u << lane) - 1u;
    VisitCounts vc = {0, 0, 0};
    Trav T;
    T.active = false;
    uint32_t slot = 0;
    const DevScene* scp = nullptr;  // BATCH: scene of the lane's ray
#define RG_SC (BATCH ? *scp : P.scene)
    // a finished ray's hit record; a ray whose short stack overflowed also joins the lane's list (its first ray, plus 1,
    // beside the flag; the next one's in the overflow words by ray), which the lane traces again at the end
#define RG_WF_HIT_OUT()                                                                      \
    do {                                                                                     \
        if (stk.over() & 1u) {                                                               \
            wf.overflow[slot] = stk.over() >> 1;                                             \
            stk.over() = (slot + 1u) << 1;                                                   \
        }                                                                                    \
        put_hit<FORM>(P, slot, T.h, T.h.hit);                                                \
    } while (0)
    // starts ray k of the launch
    auto begin = [&](uint32_t k) {
        if (first) {  // camera ray of root k, computed here
            slot = k;
            uint32_t sample, job;
            Payload p0;
            RayReq r0;
            if (tree_root<BATCH>(P, k, job, sample, p0, r0)) {
                if (BATCH) scp = &P.jobs[job].scene;
                trav_begin(T, RG_SC, r0.o.x, r0.o.y, r0.o.z, r0.d.x, r0.d.y, r0.d.z, r0.tmin, r0.tmax, stk);
                if (!T.active) put_hit<FORM>(P, slot, T.h, false);
            }
        } else if (TREE) {
            slot = node0 + (BATCH && P.perm ? P.perm[k] : k);
            if (BATCH) scp = &P.jobs[P.tree.state[slot].y >> 6].scene;
            const float4 o = P.tree.rayO[slot], d = P.tree.rayD[slot];
            trav_begin(T, RG_SC, o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w, stk);
            if (!T.active) put_hit<FORM>(P, slot, T.h, false);
        } else {
            slot = k;
            const float4 o = P.queryRays[2 * (size_t)slot], d = P.queryRays[2 * (size_t)slot + 1];
            trav_begin(T, P.scene, o.x, o.y, o.z, d.x, d.y, d.z, o.w, d.w, stk);
            if (!T.active) put_hit<FORM>(P, slot, T.h, false);  // zero direction or the scene box missed
        }
    };
    // while-while: lanes on inner nodes descend together (the others wait), then every lane at a
    // leaf processes it, so each pass runs one kind of step across most of the warp
    auto passes = [&]() {
#pragma unroll 1
        for (int k = 0; k < RG_WF_STEPS; ++k) {
#pragma unroll 1
            for (int j = 0; j < RG_INNER_ROUNDS; ++j) {
                const bool inner = T.active && !(T.ref & kLeaf);
                if (!__any_sync(0xFFFFFFFFu, inner)) break;
                if (inner) {
                    trav_step<COUNT>(T, RG_SC, stk, vc);
                    if (!T.active) RG_WF_HIT_OUT();
                }
            }
            if (T.active && (T.ref & kLeaf)) {
                trav_step<COUNT>(T, RG_SC, stk, vc);
                if (!T.active) RG_WF_HIT_OUT();
            }
        }
    };
    const uint32_t workers = trace_workers(count, THREADS);
    if (blockIdx.x >= workers) return;
    if (workers < gridDim.x || trace_width(count, THREADS) < 32u) {
        // Fewer rays than lanes: spread over all warps, whose other lanes join in.  Warp w takes rays
        // w * width .. + width - 1 without the fetch counter, and blocks without a ray are done.
        const uint32_t width = trace_width(count, THREADS), k = (blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5)) * width + lane;
        if (lane < width && k < count) begin(k);
        while (__popc(__ballot_sync(0xFFFFFFFFu, T.active)) > RG_DRAIN_LANES) passes();
        drain<COUNT>(T, slot, scp, stk, vc, [&](const DevScene* sc) -> const DevScene& { return BATCH ? *sc : P.scene; }, [&] { RG_WF_HIT_OUT(); });
    } else {
        bool exhausted = false;
        for (;;) {
            const unsigned idle = __ballot_sync(0xFFFFFFFFu, !T.active);
            if (__popc(idle) >= RG_FETCH_THRESHOLD || idle == 0xFFFFFFFFu) {
                const bool need = !T.active && !exhausted;
                const unsigned needMask = __ballot_sync(0xFFFFFFFFu, need);
                if (needMask) {
                    const int leader = __ffs(needMask) - 1;
                    uint32_t base = 0;
                    if ((int)lane == leader) base = atomicAdd(wf.fetch, (uint32_t)__popc(needMask));
                    base = __shfl_sync(0xFFFFFFFFu, base, leader);
                    if (need) {
                        const uint32_t k = base + (uint32_t)__popc(needMask & ltmask);
                        if (k >= count) exhausted = true;
                        else begin(k);
                    }
                }
                if (!__any_sync(0xFFFFFFFFu, T.active || !exhausted)) break;
            }
            passes();
        }
    }
#undef RG_WF_HIT_OUT
#undef RG_SC
    // The lane's rays whose short stack overflowed, from the start with the deep stack.  (The last block to finish
    // did this for the whole launch: 4097 rays that all overflow a 16-word stack took 104 ms.)
    for (uint32_t next = stk.over() >> 1; next;) {
        const uint32_t s = next - 1u;
        next = wf.overflow[s];
        vc.overflow++;
        float4 o, d;
        const DevScene* sc = &P.scene;
        if (first) {  // root s's camera ray, as the first round computed it
            uint32_t sample, job;
            Payload p0;
            RayReq r0;
            tree_root<BATCH>(P, s, job, sample, p0, r0);
            if (BATCH) sc = &P.jobs[job].scene;
            o = make_float4(r0.o.x, r0.o.y, r0.o.z, r0.tmin);
            d = make_float4(r0.d.x, r0.d.y, r0.d.z, r0.tmax);
        } else if (TREE) {
            o = P.tree.rayO[s];
            d = P.tree.rayD[s];
            if (BATCH) sc = &P.jobs[P.tree.state[s].y >> 6].scene;
        } else {
            o = P.queryRays[2 * (size_t)s];
            d = P.queryRays[2 * (size_t)s + 1];
        }
        Hit h;
        retrace_deep(sc, o, d, &h, P.counters);
        put_hit<FORM>(P, s, h, h.hit);
    }
    unsigned long long c[3] = {vc.nodes, vc.tris, vc.overflow};
    for (int k = 0; k < 3; ++k) {
        unsigned long long v = c[k];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
        if (lane == 0 && v) {
            atomicAdd(P.counters + 4 + k, v);
            atomicAdd(P.counters + 12 + k, v);
        }
    }
}

// ---- ray trees -------------------------------------------------------------------------------------
// The reference's recursion is depth-first on one payload, so a path traced as the shaders run it has
// one ray in flight at a time: up to 70 rays in sequence, and a frame as many rounds.  But which rays a
// hit issues follows from the hit, its recursion depth and its ray type; of the payload's state that
// earlier siblings leave behind, only curIOR (the direction of a front-face refraction) and refDepth (a
// grid material's colour and reflectivity) matter.  So every sample's rays are a tree of nodes:
//   rounds    k_wf_trace and k_tree_expand grow all trees breadth first, one recursion level a round:
//             the shadow, reflection and refraction rays of a level's hits are traced by one launch,
//             curIOR and refDepth taken as if no sibling had changed them.  Every nested trace is at
//             least one recursion level deeper, so maxRecursions + 1 rounds finish the trees.
//             A refraction in a reflection's subtree that changes the curIOR of the refraction after
//             it (0.07 - 0.6 % of the samples on the benchmark scenes) replaces that ray at once, and
//             one or two more rounds grow the replacements.
//   check     k_tree_check compares what the finished subtrees leave in curIOR and refDepth with what
//             was assumed.  A refraction ray that still comes out different, or a reflection ray that
//             must or must not be there, is replaced, its new subtree grown by further rounds, and the
//             check repeated until nothing changes.
//   compose   k_tree_compose evaluates the hits bottom-up, a round at a time from the last: a hit's
//             colour is a function of its surface, its shadow chain and its children's colours.
// All of it evaluates the shaders' expressions on the shaders' operands, in their order, so the images
// are the depth-first ones bit for bit.
//
// A node: ray (origin, tmin; direction, tmax), state (curIOR and refDepth on entry, recursion depth,
// ray type, job, parent), hit, surface of the hit (world normal -- flipped toward the ray for GENERIC
// hits --, material), links to its shadow / reflection / refraction node.  Roots (nodes 0 ..
// treeRoots - 1, one per sample of the chunk) have no stored ray and state: both are recomputed.
constexpr uint32_t kNodeMask = kTreeMaxNodes - 1u;  // links: node ids below kTreeMaxNodes, or
constexpr uint32_t kNoNode = kNodeMask;             //   no ray issued
constexpr uint32_t kZeroFront = kNodeMask - 1u;     //   a front-face refraction of zero direction: misses,
constexpr uint32_t kZeroBack = kNodeMask - 2u;      //   leaves curIOR = ior; a back-face one: leaves 1
static_assert(kTreePoolMax <= kZeroBack, "a node of a pool is never one of the links' values for none");
constexpr uint32_t kFrontBit = 0x80000000u;         // links.x: the ray hit the front face
constexpr uint32_t kOffBit = 0x40000000u;           // state.z: a sibling may have changed refDepth
constexpr uint32_t kDeadBit = 0x80000000u;          // state.z: below a ray that was replaced
__device__ __forceinline__ bool is_node(uint32_t link) { return link < kZeroBack; }

struct NodeState {
    float curIOR, refDepth;
    uint32_t rec, type, job, parent;  // parent: with kOffBit / kDeadBit
};
template <bool BATCH>
__device__ __forceinline__ NodeState node_state(const TraceParams& P, uint32_t i) {
    if (i < tree_roots<BATCH>(P)) return {1.0f, 0.0f, 0u, (uint32_t)RT_GENERIC, 0u, kNodeMask};
    const uint4 s = P.tree.state[i];
    return {__uint_as_float(s.x), __uint_as_float(s.w), s.y & 15u, (s.y >> 4) & 3u, s.y >> 6, s.z};
}
__device__ __forceinline__ uint4 pack_state(float curIOR, uint32_t rec, uint32_t type, uint32_t job, uint32_t parent, float refDepth) {
    return make_uint4(__float_as_uint(curIOR), rec | type << 4 | job << 6, parent, __float_as_uint(refDepth));
}

template <bool BATCH>
__device__ __forceinline__ const DevScene& tree_scene(const TraceParams& P, uint32_t job) { return BATCH ? P.jobs[job].scene : P.scene; }
template <bool BATCH>
__device__ __forceinline__ const rg_ubo& tree_ubo(const TraceParams& P, uint32_t job) { return BATCH ? P.jobs[job].ubo : P.ubo; }
__device__ __forceinline__ V3 light_of(const rg_ubo& u) { return v3(u.lightDir[0], u.lightDir[1], u.lightDir[2]); }

__device__ __forceinline__ bool node_hit(const RayTree& t, uint32_t i) { return t.hitInst[i] != 0xFFFFFFFFu; }

// marks the GENERIC nodes from y down as replaced (what nodes from `fresh` on issued or will issue
// learns it from its parent)
__device__ void bury(const RayTree& t, uint32_t y, uint32_t fresh) {
    uint32_t st[2 * kMaxFrames];
    int n = 0;
    st[n++] = y;
    while (n) {
        y = st[--n];
        atomicOr(&t.state[y].z, kDeadBit);
        if (y >= fresh || !node_hit(t, y)) continue;
        const uint4 c = t.link[y];
        if (is_node(c.y)) st[n++] = c.y;
        if (is_node(c.z)) st[n++] = c.z;
    }
}

// GENERIC node x's ray and hit, for rays it issues anew
template <bool BATCH>
__device__ __forceinline__ void reissue_frame(const TraceParams& P, uint32_t x, NodeState& st, uint32_t& seed, Frame& cur) {
    const RayTree& t = P.tree;
    RayReq ray;
    seed = 0;
    if (x < tree_roots<BATCH>(P)) {
        Payload p;
        uint32_t sample;
        tree_root<BATCH>(P, x, st.job, sample, p, ray);
        seed = p.seed;
    } else {
        const float4 o = t.rayO[x], d = t.rayD[x];
        ray.o = v3(o.x, o.y, o.z);
        ray.d = v3(d.x, d.y, d.z);
    }
    const float4 sf = t.surf[x];
    cur.t = t.hitTUV[x].x;
    cur.D = ray.d;
    cur.n = v3(sf.x, sf.y, sf.z);
    cur.origin = ray.o + ray.d * cur.t;
    load_material(tree_scene<BATCH>(P, st.job).materials + __float_as_uint(sf.w), cur);
}

// a new GENERIC node for a ray of direction dir from cur; kNoNode when the pool is full
template <bool BATCH>
__device__ __forceinline__ uint32_t append_ray(const TraceParams& P, const Frame& cur, V3 dir, float ior, uint32_t rec, uint32_t job,
                                               uint32_t parent, float refDepth) {
    const RayTree& t = P.tree;
    const uint32_t at = tree_roots<BATCH>(P) + atomicAdd(t.ctl + kTreeAlloc, 1u);
    if (at >= t.capacity) return kNoNode;
    t.rayO[at] = make_float4(cur.origin.x, cur.origin.y, cur.origin.z, 0.01f);
    t.rayD[at] = make_float4(dir.x, dir.y, dir.z, 1000.0f);
    t.state[at] = pack_state(ior, rec, RT_GENERIC, job, parent, refDepth);
    atomicMax(t.ctl + kTreeLevels, 16u - rec);
    __threadfence();  // before the link to it: whoever replaces it finds its state
    return at;
}

// front-face hit x (cur) refracts with curIOR = ior; refDepth: v before its reflection ray
template <bool BATCH, bool GLOSSY>
__device__ __forceinline__ void replace_refraction(const TraceParams& P, uint32_t x, const NodeState& st, uint32_t seed, const Frame& cur,
                                                   float ior, float v, uint32_t fresh) {
    const RayTree& t = P.tree;
    const V3 dir = refract_dir<GLOSSY>(cur, ior / cur.ior, seed, (int)st.rec);
    const uint32_t to = is_zero(dir) ? kZeroFront
                                     : append_ray<BATCH>(P, cur, dir, cur.ior, st.rec + 1u, st.job, x | kOffBit, is_node(t.link[x].y) ? v + cur.t : v);
    // the refraction link and the curIOR it was issued with, in one exchange
    const unsigned long long pair = (unsigned long long)__float_as_uint(ior) << 32 | to;
    const uint32_t old = (uint32_t)atomicExch(reinterpret_cast<unsigned long long*>(&t.link[x].z), pair);
    if (is_node(old)) bury(t, old, fresh);
}

// GENERIC node y refracts and leaves curIOR = ior (as far as is known yet): the refraction that runs next
// in depth-first order outside y's subtree is that of the nearest ancestor whose reflection subtree y is
// the last refraction of.  `fresh`: first node of the current round.
template <bool BATCH, bool GLOSSY>
__device__ __forceinline__ void refraction_left(const TraceParams& P, uint32_t y, float ior, uint32_t fresh) {
    const RayTree& t = P.tree;
    while (y >= tree_roots<BATCH>(P)) {
        const uint32_t x = t.state[y].z & kNodeMask;
        const uint4 c = t.link[x];
        if (c.y == y && c.z != kNoNode) {
            if (!(c.x & kFrontBit) || c.w == __float_as_uint(ior)) return;
            NodeState st = node_state<BATCH>(P, x);
            if (x >= tree_roots<BATCH>(P) && (st.parent & kDeadBit)) return;
            uint32_t seed;
            Frame cur;
            reissue_frame<BATCH>(P, x, st, seed, cur);
            replace_refraction<BATCH, GLOSSY>(P, x, st, seed, cur, ior, st.refDepth, fresh);
            return;
        }
        if (c.y != y && c.z != y) return;  // y was replaced
        y = x;
    }
}

// Surfaces and child rays of one round's hits.  A warp appends its shadow rays, then its reflection,
// then its refraction rays, with one atomic: 32 hits of a few surfaces give runs of similar rays.
// (A batch's 80 registers would leave 6 blocks an SM; 8, with spills, make the mixed batch 1.4 % faster.  A frame's 71
// registers leave 7; 8 are 0.4 % faster and slower by scene, 10 cost 1 to 2 %.)
template <bool BATCH, bool GLOSSY>
__global__ void __launch_bounds__(128, BATCH ? 8 : 7) k_tree_expand(const __grid_constant__ TraceParams P, int round) {
    chain_wait();
    const RayTree& t = P.tree;
    const bool first = P.firstRound != 0, counted = BATCH && round < 0;
    if (counted) round = (int)t.ctl[kTreeTracedRound];
    const uint32_t begin = first ? 0u : t.ctl[kTreeBounds + round], end = t.ctl[kTreeBounds + round + 1];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        t.ctl[kTreeFetch] = 0;  // the next trace launch's work counter
        if (BATCH) t.ctl[kTreeRound] = (uint32_t)round + (counted && begin == end ? 0u : 1u);  // a round without rays is not counted
    }
    const unsigned lane = threadIdx.x & 31, below = (1u << lane) - 1u;
    for (uint32_t base = begin + blockIdx.x * blockDim.x; base < end; base += gridDim.x * blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        bool want[3] = {false, false, false}, candidate = false;
        V3 dir[3];
        float depthC = 0.0f, iorT = 0.0f, tminS = 0.01f;
        uint32_t recR = 0, typeS = RT_SHADOW_TRACE, link[3] = {kNoNode, kNoNode, kNoNode}, off = 0, offT = 0, matId = 0;
        Frame cur;
        NodeState st = {1.0f, 0.0f, 0u, (uint32_t)RT_GENERIC, 0u, 0u};
        const uint32_t inst = i < end ? t.hitInst[i] : 0xFFFFFFFFu;
        bool live = inst != 0xFFFFFFFFu;
        if (live) {
            RayReq ray;
            uint32_t seed = 0;
            if (first) {
                uint32_t sample;
                Payload p;
                live = tree_root<BATCH>(P, i, st.job, sample, p, ray);
                seed = p.seed;
            } else {
                st = node_state<BATCH>(P, i);
                if (round > 1 && (st.parent & kNodeMask) >= tree_roots<BATCH>(P) && (t.state[st.parent & kNodeMask].z & kDeadBit)) {  // its parent was replaced
                    st.parent |= kDeadBit;
                    t.state[i].z = st.parent;
                }
                live = !(st.parent & kDeadBit);
                const float4 o = t.rayO[i], d = t.rayD[i];
                ray.o = v3(o.x, o.y, o.z);
                ray.d = v3(d.x, d.y, d.z);
            }
            if (live) {
                const float4 ht = t.hitTUV[i];
                const Hit h = {ht.x, ht.y, ht.z, inst, __float_as_uint(ht.w), true};
                const DevScene& sc = tree_scene<BATCH>(P, st.job);
                bool effect = false;
                if (st.type == RT_SHADOW_TRACE) shadow_hit_surface(sc, h, ray, cur, matId);
                else effect = closest_hit_surface(sc, h, ray, st.refDepth, cur, matId);
                const rg_ubo& u = tree_ubo<BATCH>(P, st.job);
                const bool deeper = (int)st.rec < u.maxRecursions;
                off = st.parent & kOffBit;
                if (st.type == RT_SHADOW_INTERNAL) {
                    want[0] = deeper;
                    dir[0] = cur.D;
                } else if (st.type == RT_SHADOW_TRACE) {
                    want[0] = deeper && cur.transparency > 0.0f;
                    dir[0] = cur.D;
                    typeS = RT_SHADOW_INTERNAL;
                } else {
                    cur.front = dot(-cur.D, cur.n) > 0.0f;
                    if (!cur.front) cur.n = normalize(-cur.n);
                    const V3 L = light_of(u);
                    if (deeper && dot(-L, cur.n) > 0.07f) {
                        want[0] = true;
                        dir[0] = -L;
                        tminS = 0.01f * 10.0f;
                    }
                    depthC = st.refDepth;
                    offT = off;
                    if (deeper && cur.reflectivity > 0.0f) {
                        want[1] = true;
                        dir[1] = reflect_dir<GLOSSY>(cur, seed, (int)st.rec);
                        recR = st.rec + (uint32_t)cur.rayConsumption;
                        depthC = st.refDepth + cur.t;
                        offT = kOffBit;
                    }
                    if (deeper && cur.transparency > 0.0f) {
                        dir[2] = refract_dir<GLOSSY>(cur, cur.front ? st.curIOR / cur.ior : cur.ior / 1.0f, seed, (int)st.rec);
                        iorT = cur.front ? cur.ior : 1.0f;
                        want[2] = !is_zero(dir[2]);
                        if (!want[2]) link[2] = cur.front ? kZeroFront : kZeroBack;
                    }
                    candidate = deeper && ((cur.front && want[1] && cur.transparency > 0.0f) ||
                                            (effect && off && grid_sign_varies(cur.origin, st.refDepth, cur.t)));
                }
            }
        }
        const unsigned m0 = __ballot_sync(0xFFFFFFFFu, want[0]), m1 = __ballot_sync(0xFFFFFFFFu, want[1]),
                       m2 = __ballot_sync(0xFFFFFFFFu, want[2]);
        const uint32_t n0 = (uint32_t)__popc(m0), n1 = (uint32_t)__popc(m1), n2 = (uint32_t)__popc(m2);
        uint32_t at = 0;
        if (n0 + n1 + n2) {
            if (lane == 0) at = atomicAdd(t.ctl + kTreeAlloc, n0 + n1 + n2);
            at = tree_roots<BATCH>(P) + __shfl_sync(0xFFFFFFFFu, at, 0);
        }
        const uint32_t cp = warp_append(t.ctl + kTreeCand + tree_cand<BATCH>(P), candidate);
        if (candidate && cp < t.capacity) t.cand[tree_cand<BATCH>(P)][cp] = i;
        if (!live && inst != 0xFFFFFFFFu && !first) t.link[i] = make_uint4(kNoNode, kNoNode, kNoNode, 0u);
        if (live) {
            const uint32_t c[3] = {at + (uint32_t)__popc(m0 & below), at + n0 + (uint32_t)__popc(m1 & below),
                                   at + n0 + n1 + (uint32_t)__popc(m2 & below)};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (!want[k] || c[k] >= t.capacity) continue;  // a full pool discards the whole chunk (launch_trace_tree)
                link[k] = c[k];
                t.rayO[c[k]] = make_float4(cur.origin.x, cur.origin.y, cur.origin.z, k == 0 ? tminS : 0.01f);
                t.rayD[c[k]] = make_float4(dir[k].x, dir[k].y, dir[k].z, 1000.0f);
                t.state[c[k]] = k == 0 ? pack_state(st.curIOR, st.rec + 1u, typeS, st.job, i, st.refDepth)
                              : k == 1 ? pack_state(st.curIOR, recR, RT_GENERIC, st.job, i | off, depthC)
                                       : pack_state(iorT, st.rec + 1u, RT_GENERIC, st.job, i | offT, depthC);
            }
            const bool front = cur.front && st.type == RT_GENERIC;
            t.link[i] = make_uint4(link[0] | (front ? kFrontBit : 0u), link[1], link[2], __float_as_uint(st.curIOR));
            t.surf[i] = make_float4(cur.n.x, cur.n.y, cur.n.z, __uint_as_float(matId));
            // a refraction behind some ancestor's reflection sets the curIOR of that ancestor's refraction.
            // A front-face one is expected to leave the object again (curIOR 1) unless the recursion
            // limit stops it inside.
            if (link[2] != kNoNode && !first) {
                const bool stays = front && (link[2] == kZeroFront || (int)st.rec + 1 >= tree_ubo<BATCH>(P, st.job).maxRecursions);
                refraction_left<BATCH, GLOSSY>(P, i, stays ? cur.ior : 1.0f, begin);
            }
        }
    }
}

// refDepth after the shaders ran the invocation at node y and everything below it, from value v before
// it: every reflection ray adds the t of the hit that issued it, in depth-first order.  Nodes from
// `fresh` on are not traced yet and count as misses.
__device__ float fold_ref_depth(const RayTree& t, uint32_t y, float v, uint32_t fresh) {
    uint32_t st[2 * kMaxFrames];
    int n = 0;
    st[n++] = y;
    while (n) {
        y = st[--n];
        if (y >= fresh) continue;
        const bool hit = node_hit(t, y);
        const uint4 c = t.link[y];
        const float ht = t.hitTUV[y].x;
        if (!hit) continue;
        if (is_node(c.z)) st[n++] = c.z;
        if (is_node(c.y)) {
            v = v + ht;
            st[n++] = c.y;
        }
    }
    return v;
}

// refDepth on entry of GENERIC node x as the depth-first order leaves it.  These walks are 40 % of the
// composition's time, each step a wait for memory, so what a level or a node needs is requested together
// (1920x1080 game frame: composition 3.09 -> 2.80 ms).  Marking the subtrees that add nothing while they grow
// saves no more here than it costs there.
template <bool BATCH>
__device__ float exact_ref_depth(const TraceParams& P, uint32_t x, uint32_t fresh) {
    const RayTree& t = P.tree;
    const uint32_t roots = tree_roots<BATCH>(P);
    uint32_t sibling[kMaxFrames];  // of the levels passed: the reflection ray before it (kZeroFront: x itself or above it), or kNoNode
    float add[kMaxFrames];
    int n = 0;
    NodeState s = node_state<BATCH>(P, x);
    while (x >= roots && (s.parent & kOffBit) && n < kMaxFrames) {
        const uint32_t p = s.parent & kNodeMask;
        const uint4 c = t.link[p];
        add[n] = t.hitTUV[p].x;
        s = node_state<BATCH>(P, p);
        sibling[n++] = !is_node(c.y) ? kNoNode : c.y != x ? c.y : kZeroFront;
        x = p;
    }
    float v = s.refDepth;  // no sibling changed it here
    while (n) {
        const uint32_t y = sibling[--n];
        if (y == kNoNode) continue;
        v = v + add[n];
        if (is_node(y)) v = fold_ref_depth(t, y, v, fresh);
    }
    return v;
}

// The candidates -- front-face hits with a reflection and a refraction ray, and grid-effect hits whose
// refDepth a sibling may have changed -- against the finished subtrees (nodes below `fresh`).  What a
// subtree leaves in curIOR is set by its last refraction: the end of the walk along refraction links,
// or along the reflection link where an invocation refracts nothing.  Replaced rays are appended for the
// next rounds; candidates whose subtree could still change stay in the other list.
template <bool BATCH, bool GLOSSY>
__global__ void __launch_bounds__(128) k_tree_check(const __grid_constant__ TraceParams P, int round) {
    chain_wait();
    const RayTree& t = P.tree;
    if (BATCH) round = (int)t.ctl[kTreeRound];
    const uint32_t n = min(t.ctl[kTreeCand + tree_cand<BATCH>(P)], t.capacity), fresh = t.ctl[kTreeBounds + round];
    if (blockIdx.x == 0 && threadIdx.x == 0) t.ctl[kTreeTraced] = fresh;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const uint32_t k = base + threadIdx.x;
        bool keep = false;
        uint32_t x = 0;
        if (k < n) {
            x = t.cand[tree_cand<BATCH>(P)][k];
            NodeState st = node_state<BATCH>(P, x);
            if (x < tree_roots<BATCH>(P)) st.parent = 0u;
            uint4 c = t.link[x];
            const bool sibling = is_node(c.y) && c.y < fresh && node_hit(t, c.y);  // a reflection ray with a subtree
            if (!(st.parent & kDeadBit) && is_node(c.y) && c.y >= fresh) keep = true;
            else if (!(st.parent & kDeadBit) && (sibling || (st.parent & kOffBit))) {
                uint32_t seed;
                Frame cur;
                reissue_frame<BATCH>(P, x, st, seed, cur);
                const rg_material* materials = tree_scene<BATCH>(P, st.job).materials;
                const bool grid = __ldg(&materials[__float_as_uint(t.surf[x].w)].effectId) == 1 && (st.parent & kOffBit) &&
                                  grid_sign_varies(cur.origin, st.refDepth, cur.t);
                uint32_t changes = 0;
                float v = st.refDepth;
                if (grid) {
                    v = exact_ref_depth<BATCH>(P, x, fresh);
                    grid_effect(cur.origin, v, cur.t, cur);
                    const bool reflects = cur.reflectivity > 0.0f;
                    if (reflects && !is_node(c.y)) {
                        c.y = append_ray<BATCH>(P, cur, reflect_dir<GLOSSY>(cur, seed, (int)st.rec), st.curIOR,
                                         st.rec + (uint32_t)cur.rayConsumption, st.job, x | kOffBit, v + cur.t);
                        t.link[x].y = c.y;
                        ++changes;
                    } else if (!reflects && is_node(c.y)) {
                        bury(t, c.y, fresh);
                        t.link[x].y = c.y = kNoNode;
                        ++changes;
                    }
                }
                if ((c.x & kFrontBit) && cur.transparency > 0.0f) {
                    float ior = st.curIOR;
                    for (uint32_t y = c.y; is_node(y) && y < fresh && node_hit(t, y);) {
                        const uint4 cy = t.link[y];
                        if (is_node(cy.z)) {
                            ior = __uint_as_float(t.state[cy.z].x);
                            y = cy.z;
                        } else if (cy.z == kNoNode) {
                            y = cy.y;
                        } else {
                            ior = cy.z == kZeroBack ? 1.0f : __ldg(&materials[__float_as_uint(t.surf[y].w)].ior);
                            break;
                        }
                    }
                    if (c.w != __float_as_uint(ior)) {
                        replace_refraction<BATCH, GLOSSY>(P, x, st, seed, cur, ior, v, fresh);
                        ++changes;
                    }
                }
                if (changes) atomicAdd(t.ctl + kTreeChanges, changes);
                if (sibling) {
                    const uint4 cy = t.link[c.y < fresh ? c.y : x];
                    keep = cy.y != kNoNode || cy.z != kNoNode || (st.parent & kOffBit);  // (off: c.y may yet reflect)
                }
                keep = keep || grid || changes;
            }
        }
        const uint32_t pos = warp_append(t.ctl + kTreeCand + (tree_cand<BATCH>(P) ^ 1u), keep);
        if (keep && pos < t.capacity) t.cand[tree_cand<BATCH>(P) ^ 1u][pos] = x;
    }
}

// Whether the shadow chain of GENERIC node x ends in the sky: its last ray goes on behind a
// SHADOW_INTERNAL hit (closesthit.rchit:133) and misses.
__device__ bool chain_meets_sky(const TraceParams& P, uint32_t x) {
    const RayTree& t = P.tree;
    uint32_t s = t.link[x].x & kNodeMask;
    for (bool behind = false;; behind = true) {
        if (!is_node(s)) return false;
        const bool hit = node_hit(t, s);
        const uint32_t j = t.link[s].x & kNodeMask;  // SHADOW_INTERNAL (none at an opaque hit)
        if (!hit) return behind;
        if (!is_node(j)) return false;
        const bool inside = node_hit(t, j);
        s = t.link[j].x & kNodeMask;
        if (!inside) return false;
    }
}

// payload.depth < 1000 on entry of GENERIC node x: the last GENERIC hit or sky miss that the
// depth-first order finished before it (0 before any)
template <bool BATCH>
__device__ bool depth_is_near(const TraceParams& P, uint32_t x) {
    const RayTree& t = P.tree;
    while (x >= tree_roots<BATCH>(P)) {
        const uint32_t p = t.state[x].z & kNodeMask;
        const uint4 c = t.link[p];
        if (c.z == x && is_node(c.y)) return node_hit(t, c.y) && t.hitTUV[c.y].x < 1000.0f;
        if (chain_meets_sky(P, p)) return false;
        x = p;
    }
    return true;
}

// shadowCol of SHADOW_INTERNAL hit j (closesthit.rchit:126-128); every such hit finds hitValue at 1
__device__ __forceinline__ V3 internal_shadow(const RayTree& t, uint32_t j, const Frame& m) {
    const float thick = clampf(t.hitTUV[j].x * (1.0f - m.transparency) * 10.0f, 0.0f, 1.0f);
    return v3s(1.0f) - mix(v3s(0.0f), normalize(v3s(1.1f) - m.diffuse) + v3s(0.1f), thick);
}

// hitValue that the shadow ray s of GENERIC node x returns with (closesthit.rchit:125-166, 193): the
// chain SHADOW_TRACE, SHADOW_INTERNAL, SHADOW_TRACE, ... walked to its end and unwound
template <bool BATCH>
__device__ V3 shadow_chain(const TraceParams& P, const DevScene& sc, const V3 L, uint32_t x, uint32_t s, RayCounts& cnt) {
    const RayTree& t = P.tree;
    uint32_t inner[kMaxFrames];  // SHADOW_INTERNAL hits passed
    int n = 0;
    V3 value = v3s(1.0f);
    bool far = false;
    Frame m;
    auto surface = [&](uint32_t k) {
        const uint32_t id = __float_as_uint(t.surf[k].w);
        load_material(sc.materials + id, m);
        if (__ldg(&sc.materials[id].effectId) == 1) {  // the chain's rays carry x's refDepth
            const NodeState sk = node_state<BATCH>(P, x);
            const float4 o = t.rayO[k], d = t.rayD[k];
            const float ht = t.hitTUV[k].x;
            grid_effect(v3(o.x, o.y, o.z) + v3(d.x, d.y, d.z) * ht, (sk.parent & kOffBit) && x >= tree_roots<BATCH>(P) ? exact_ref_depth<BATCH>(P, x, kNodeMask) : sk.refDepth, ht, m);
        }
    };
    for (;;) {
        cnt.shadow++;
        // requested together, whether the ray hit or not: a hop of the chain is one way to memory
        const bool hit = node_hit(t, s);
        const uint32_t j = t.link[s].x & kNodeMask, id = __float_as_uint(t.surf[s].w);
        const float tS = t.hitTUV[s].x;
        if (!hit) {
            if (n) {  // behind a SHADOW_INTERNAL hit: miss shader 0
                const float4 d = t.rayD[s];
                Payload p;
                sky(p, v3(d.x, d.y, d.z), L);
                value = p.hitValue;
                far = true;
            }
            break;
        }
        const float transparency = __ldg(&sc.materials[id].transparency);
        if (!(transparency > 0.0f)) {
            value = value * mixs(0.4f, 0.8f, clampf(logf(tS) / 8.0f, 0.0f, 1.0f));
            break;
        }
        if (!is_node(j)) break;  // recursion limit
        cnt.shadow++;
        const bool inside = node_hit(t, j);
        const uint32_t a = t.link[j].x & kNodeMask;
        if (!inside) break;  // shadow miss: 1
        if (!is_node(a)) {  // recursion limit
            surface(j);
            value = internal_shadow(t, j, m) * 0.4f;
            break;
        }
        inner[n++] = j;
        s = a;
    }
    if (n && !far) far = !depth_is_near<BATCH>(P, x);
    while (n) {
        const uint32_t j = inner[--n];
        surface(j);
        V3 col = internal_shadow(t, j, m);
        if (!far) {
            value = value * col;
            continue;
        }
        const float4 d = t.rayD[j], sf = t.surf[j];
        const V3 dir = refract(v3(d.x, d.y, d.z), v3(sf.x, sf.y, sf.z), m.ior / 1.0f);
        const float q = dot(L, dir);
        col = col * (q * q * q * q * q + 0.75f);
        cnt.masked++;
        Payload p;
        sky(p, -dir, L);
        value = col + p.hitValue * 0.1f;
    }
    return value;
}

// Colours of one round's GENERIC nodes from their children's (rayO of a child: colour; its ray is no
// longer needed once its own colour is known); roots write their sample's payload sums.
template <bool BATCH>
__global__ void __launch_bounds__(128) k_tree_compose(const __grid_constant__ TraceParams P, int round) {
    chain_wait();
    const RayTree& t = P.tree;
    if (BATCH) {  // round < 0: counted from the last round down, rounds before P.batchRounds have launches of their own
        if (t.ctl[kTreeFull]) return;
        if (round < 0 && (round += (int)t.ctl[kTreeTop]) < P.batchRounds) return;
    }
    const bool roots = round == 0;
    const uint32_t begin = roots ? 0u : t.ctl[kTreeBounds + round], end = t.ctl[kTreeBounds + round + 1];
    RayCounts cnt = {0, 0, 0, 0};
    for (uint32_t i = begin + blockIdx.x * blockDim.x + threadIdx.x; i < end; i += gridDim.x * blockDim.x) {
        uint32_t sample = 0;
        Payload p;
        RayReq ray;
        NodeState st = {1.0f, 0.0f, 0u, (uint32_t)RT_GENERIC, 0u, 0u};
        if (roots) {
            if (!tree_root<BATCH>(P, i, st.job, sample, p, ray)) continue;
            cnt.primary++;
        } else {
            st = node_state<BATCH>(P, i);
            if (st.type != RT_GENERIC || (st.parent & kDeadBit)) continue;
            const float4 d = t.rayD[i];
            ray.d = v3(d.x, d.y, d.z);
        }
        const rg_ubo& u = tree_ubo<BATCH>(P, st.job);
        const V3 L = light_of(u);
        if (!node_hit(t, i)) {
            sky(p, ray.d, L);
        } else {
            const DevScene& sc = tree_scene<BATCH>(P, st.job);
            const float4 sf = t.surf[i];
            const uint4 c = t.link[i];
            Frame cur;
            cur.t = t.hitTUV[i].x;
            cur.n = v3(sf.x, sf.y, sf.z);
            const rg_material* M = sc.materials + __float_as_uint(sf.w);
            load_material(M, cur);
            if (__ldg(&M->effectId) == 1) {
                if (!roots) {
                    const float4 o = t.rayO[i];
                    ray.o = v3(o.x, o.y, o.z);
                }
                grid_effect(ray.o + ray.d * cur.t, (st.parent & kOffBit) ? exact_ref_depth<BATCH>(P, i, kNodeMask) : st.refDepth, cur.t, cur);
            }
            // closesthit.rchit:168-204
            const bool deeper = (int)st.rec < u.maxRecursions;
            const float ndl = dot(-L, cur.n);
            V3 base = cur.diffuse * fmaxf(ndl, 0.2f), shadow = v3s(1.0f);
            if (ndl > 0.07f) {
                if (deeper) shadow = shadow_chain<BATCH>(P, sc, L, i, c.x & kNodeMask, cnt);
            } else {
                const float tr = cur.transparency, sm = tr * tr;
                shadow = tr < 1.0f ? mix(v3s(1.0f), cur.diffuse * sm, tr) : v3s(0.4f);
            }
            // :206-221
            V3 reflectColor = v3s(1.0f), refractColor = v3s(1.0f);
            float reflectDepth = 0.0f;
            if (is_node(c.y)) {
                cnt.secondary++;
                const float4 r = t.rayO[c.y];
                reflectColor = v3(r.x, r.y, r.z) * cur.specular;
                reflectDepth = r.w;
            }
            // :223-251
            if (c.z != kNoNode) {
                V3 value;
                if (is_node(c.z)) {
                    cnt.secondary++;
                    const float4 r = t.rayO[c.z];
                    value = v3(r.x, r.y, r.z);
                } else {
                    Payload q;
                    sky(q, v3s(0.0f), L);
                    value = q.hitValue;
                }
                refractColor = (c.x & kFrontBit) ? value : mix(v3s(1.0f), cur.diffuse, logf(1.0f + cur.t)) * value;
            }
            // :253-267
            base = base * shadow;
            base = base + cur.diffuse * cur.emission;
            const float total = fmaxf(cur.transparency, cur.reflectivity), den = cur.transparency + cur.reflectivity;
            const V3 roughCol = mix(refractColor, reflectColor, den == 0.0f ? 0.0f : cur.reflectivity / den);
            p.hitValue = mix(base, roughCol, total);
            p.depth = cur.t;
            if (roots) {
                p.hitValue = base;
                p.normal = cur.n;
                p.roughRGB = roughCol;
                p.roughA = fminf((reflectDepth / 50.0f) * cur.roughness, cur.roughness / 2.1f);
                p.reflectContribution = total;
            }
        }
        if (roots) store_sample(P.samples + 3 * (size_t)sample, p);
        else t.rayO[i] = make_float4(p.hitValue.x, p.hitValue.y, p.hitValue.z, p.depth);
    }
    __syncwarp();
    unsigned long long c[4] = {cnt.primary, cnt.shadow, cnt.secondary, cnt.masked};
    flush_counts(P, c, 4);
}

// The sample of root k depth first on one thread, as the megakernel runs it.  A chunk that fills the pool goes again in
// parts, down to single samples; a sample whose tree, replaced rays included, exceeds the pool even then is
// rendered this way, so no bound on the size of a tree has to hold.  (1013 nodes at 8 recursions without replacements; how
// many nodes replacements can leave behind depends on the scene.)  Frames and stack lie in shared memory: local
// memory is reserved for every thread that the chip can hold.
struct DepthFirstMem {
    Frame frames[kMaxFrames];
    uint32_t stack[kDeepStack];
    float world[6];
};
template <bool BATCH>
__device__ __forceinline__ void sample_depth_first(const TraceParams& P, uint32_t k, DepthFirstMem& m) {
    uint32_t job, sample;
    Payload p;
    RayReq ray;
    if (!tree_root<BATCH>(P, k, job, sample, p, ray)) return;
    const DevScene& sc = tree_scene<BATCH>(P, job);
    const rg_ubo& u = tree_ubo<BATCH>(P, job);
    RayCounts cnt = {1, 0, 0, 0};
    Frame cur;
    int fsp = 0;
    Hit h;
    do {
        h.hit = false;  // a mask-0 trace meets nothing
        if (!ray.masked)
            h = deep_hit(sc, make_float4(ray.o.x, ray.o.y, ray.o.z, ray.tmin), make_float4(ray.d.x, ray.d.y, ray.d.z, ray.tmax),
                         LocalStackT<kDeepStack>{m.stack, m.world}, P.counters);
    } while (shade_step(sc, light_of(u), u.maxRecursions, h, p, ray, m.frames, fsp, cur, cnt));
    store_sample(P.samples + 3 * (size_t)sample, p);
    const uint32_t c[4] = {cnt.primary, cnt.shadow, cnt.secondary, cnt.masked};
    for (int i = 0; i < 4; ++i) {
        atomicAdd(P.counters + i, (unsigned long long)c[i]);
        atomicAdd(P.counters + 8 + i, (unsigned long long)c[i]);
    }
}
// the one sample of a frame's chunk
__global__ void k_sample_depth_first(const __grid_constant__ TraceParams P) {
    __shared__ DepthFirstMem m;
    sample_depth_first<false>(P, 0, m);
}

// ---- chunks and loops of a batch, on the device -----------------------------------------------------
// A batch goes through the same trees as a frame, its samples numbered job after job, in chunks that share
// the node pool.  Its launches are captured once in a graph whose loops run on the device: over the chunks,
// over the rounds that the check asks for, and over the composition of those rounds.  One thread between them
// decides (the host loop of launch_trace_batch runs the same kernels and polls the words).
// Loop runs cost 20 us each, so the rounds that every chunk needs (batchRounds) are launched without a loop,
// and a run holds the rounds that replaced rays can need at most; rounds without rays end in 3 us.
// Six scenes, 10 M samples: half the time of a loop of one ray a path and round (3.8 against 7.1 ms), whose rounds
// dragged on for the longest path (16 of them, then 1 ms of single threads finishing paths).

// after a check: whether rays are still to be traced or checked, as launch_trace_tree decides
__global__ void k_tree_step(const __grid_constant__ TraceParams P, const TreeLoop loop) {
    uint32_t* c = P.tree.ctl;
    const uint32_t rounds = c[kTreeRound], nodes = c[kTreeRoots] + c[kTreeAlloc];
    bool full = nodes > P.tree.capacity;
    bool more = !full && (nodes > c[kTreeTraced] || c[kTreeChanges]);
    loop.words[0] += 1u;
    if (more && loop.words[0] >= loop.maxRuns) {
        if (loop.graph) loop.words[1] = 1u;
        more = false;
        full = true;  // the chunk is not composed,
        c[kTreeRoots] = 0u;  // and no other follows
    }
    if (more && rounds + (uint32_t)P.batchRounds >= (uint32_t)kTreeMaxRounds) {  // no room for the rounds' bounds: as a full pool
        more = false;
        full = true;
    }
    if (more) c[kTreeCandList] ^= 1u;
    else loop.words[3] += rounds;
    const bool extra = !more && !full && rounds > (uint32_t)P.batchRounds;
    c[kTreeMore] = more;
    c[kTreeFull] = full;
    c[kTreeTop] = rounds;
    if (loop.graph) {
        loop.words[2] += (more ? loop.roundKernels : 0u) + (extra ? loop.composeKernels : 0u);
        cudaGraphSetConditional(loop.rounds, more);
        cudaGraphSetConditional(loop.composes, extra);
    }
}

// after kTreeComposeRun rounds beyond the first P.batchRounds were composed
__global__ void k_tree_composed(const __grid_constant__ TraceParams P, const TreeLoop loop) {
    uint32_t* c = P.tree.ctl;
    const uint32_t top = c[kTreeTop] - min(c[kTreeTop], (uint32_t)kTreeComposeRun);
    const bool more = top > (uint32_t)P.batchRounds;
    c[kTreeTop] = top;
    loop.words[2] += more ? loop.composeKernels : 0u;
    cudaGraphSetConditional(loop.composes, more);
}

// The next chunk (first: of a launch).  One that filled the pool goes again in halves (a single sample: depth first).
// A chunk has a fixed cost (its launches and loop runs, 0.1 to 0.8 ms), so with fewer slots than samples the next one holds
// as many as the last one's nodes a sample let expect, at most twice as many as it: 4.1 M samples at 1024
// slots 165 ms against 1873 ms with chunks of `slots` samples that stayed at an eighth after a full one, 10 M mixed ones at
// 4096 slots 118 against 1158 ms.  A launch of few chunks leaves their sizes to the next one of the same batch size,
// which then fills no pool in vain.  kTreeLive: a chunk is set up (1), none is left (0), or the loops gave up (2)
__global__ void k_tree_next(const __grid_constant__ TraceParams P, const TreeLoop loop, bool first) {
    __shared__ DepthFirstMem m;
    constexpr uint32_t kPlan = kTreeCtlWords - kTreePlan;
    uint32_t* c = P.tree.ctl;
    const uint32_t whole = min(min(P.totalWork, P.slots), max(1u, P.tree.capacity / kTreeNodesMin));
    if (first) {
        loop.words[0] = loop.words[3] = 0u;
        c[kTreeBase] = c[kTreeRoots] = c[kTreeFull] = c[kTreeWasFull] = c[kTreeDone] = c[kTreeNodes] = 0u;
        const bool follow = c[kTreePlanned] && c[kTreePlanOf] == P.totalWork && c[kTreePlanOf + 1] == P.tree.capacity && c[kTreePlanOf + 2] == P.slots;
        c[kTreeFollow] = follow;
        if (!follow) c[kTreePlanned] = 0u;
        c[kTreeChunk] = follow ? c[kTreePlan] : whole;
    }
    bool stop = false;
    const bool full = c[kTreeFull] != 0u;
    const uint32_t roots = c[kTreeRoots];
    if (full && roots <= whole) c[kTreeWasFull] = 1u;  // (more samples than the pool is meant for: no larger pool)
    if (full && roots != 1u) {
        stop = roots == 0u;  // the check gave up
        c[kTreeChunk] = (roots + 1u) / 2u;
        c[kTreeFollow] = c[kTreePlanned] = 0u;
    } else if (roots) {
        const uint32_t nodes = roots + c[kTreeAlloc], done = c[kTreeDone] + 1u;
        const float all = __uint_as_float(c[kTreeNodes]) + (float)nodes;
        if (full) {
            sample_depth_first<true>(P, 0, m);
            c[kTreeChunk] = whole;
        } else {  // samples that fill 7/8 of the pool if they are like these
            const unsigned long long fit = (unsigned long long)(P.tree.capacity - P.tree.capacity / 8u) * roots / nodes;
            c[kTreeChunk] = (uint32_t)max(1ull, min(fit, 2ull * roots));
        }
        if (done <= kPlan) c[kTreePlan + done - 1u] = roots;  // (that place of the last plan is done with)
        if (c[kTreeFollow] && done < c[kTreePlanned]) c[kTreeChunk] = c[kTreePlan + done];
        c[kTreeBase] += roots;
        c[kTreeDone] = done;
        c[kTreeNodes] = __float_as_uint(all);
        if (c[kTreeBase] >= P.totalWork) {  // the plan of the next launch, unless the rays got far fewer under it
            const bool fewer = c[kTreeFollow] && all < 0.5f * __uint_as_float(c[kTreePlanNodes]);
            if (!c[kTreeFollow]) c[kTreePlanNodes] = __float_as_uint(all);
            c[kTreePlanned] = done <= kPlan && !fewer ? done : 0u;
            c[kTreePlanOf] = P.totalWork;
            c[kTreePlanOf + 1] = P.tree.capacity;
            c[kTreePlanOf + 2] = P.slots;
        }
    }
    bool more = !stop && c[kTreeBase] < P.totalWork;
    if (!first) {
        loop.words[0] += 1u;
        if (more && loop.words[0] >= loop.maxRuns) {
            stop = true;
            more = false;
        }
        // every chunk has the limit's runs for itself (a batch of many small chunks is no endless loop); the parts of a
        // chunk that filled the pool share them until one is done
        if (!full || roots == 1u) loop.words[0] = 0u;
    }
    c[kTreeRoots] = more ? min(min(c[kTreeChunk], P.tree.capacity), P.totalWork - c[kTreeBase]) : 0u;
    c[kTreeAlloc] = c[kTreeChanges] = c[kTreeLevels] = c[kTreeTraced] = c[kTreeFetch] = c[kTreeCand] = c[kTreeCand + 1] = 0u;
    c[kTreeCandList] = c[kTreeRound] = c[kTreeFull] = 0u;
    c[kTreeLive] = more ? 1u : stop ? 2u : 0u;
    if (loop.graph) {
        if (stop) loop.words[1] = 1u;
        loop.words[2] += (first ? 1u : 0u) + (more ? loop.chunkKernels : 0u);
        if (!first) cudaGraphSetConditional(loop.chunks, more);
    }
}

// ---- ray sort of a round (batch, optional) ------------------------------------------------
// Bucket keys: direction octant (8 buckets) or the Morton code of the origin quantised to 16 cells
// per axis of the scene's root box (4096 buckets).  The order within a bucket is arbitrary: every
// ray's result is a function of the ray alone, so the sort changes which lane traces a ray, not
// what it returns.
template <int KEY>
struct SortBuckets {
    static constexpr int n = KEY == RG_SORT_OCTANT ? 8 : 4096;
};

template <int KEY>
__device__ __forceinline__ uint32_t ray_sort_key(const TraceParams& P, uint32_t node) {
    const float4 o = P.tree.rayO[node], d = P.tree.rayD[node];
    if (KEY == RG_SORT_OCTANT) return (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
    const DevScene& sc = P.jobs[P.tree.state[node].y >> 6].scene;
    if (sc.tlasN == 0) return 0u;
    const float* b = sc.tlasRoot;
    const float x = fminf(fmaxf((o.x - b[0]) / (b[3] - b[0]) * 16.0f, 0.0f), 15.0f);
    const float y = fminf(fmaxf((o.y - b[1]) / (b[4] - b[1]) * 16.0f, 0.0f), 15.0f);
    const float z = fminf(fmaxf((o.z - b[2]) / (b[5] - b[2]) * 16.0f, 0.0f), 15.0f);
    return (expand10((uint32_t)x) << 2) | (expand10((uint32_t)y) << 1) | expand10((uint32_t)z);
}

// nodes that the traversal launch of round q (negative: the current one) will trace
__device__ __forceinline__ uint2 round_nodes(const TraceParams& P, int q) {
    const RayTree& t = P.tree;
    const uint32_t begin = t.ctl[kTreeBounds + (q < 0 ? t.ctl[kTreeRound] : (uint32_t)q)];
    return make_uint2(begin, min(tree_roots<true>(P) + t.ctl[kTreeAlloc], t.capacity) - begin);
}

// per block: histogram of the round's keys in shared memory, added to the global bucket counts
template <int KEY>
__global__ void __launch_bounds__(256) k_sort_count(const TraceParams P, int q, uint32_t* __restrict__ keys,
                                                     uint32_t* __restrict__ buckets) {
    constexpr int NB = SortBuckets<KEY>::n;
    __shared__ uint32_t h[NB];
    for (int i = threadIdx.x; i < NB; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const uint2 nodes = round_nodes(P, q);
    const uint32_t count = nodes.y;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const uint32_t k = ray_sort_key<KEY>(P, nodes.x + i);
        keys[i] = k;
        atomicAdd(&h[k], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < NB; i += blockDim.x)
        if (h[i]) atomicAdd(&buckets[i], h[i]);
}

// exclusive scan of the bucket counts into offsets (one block of 1024 threads); clears the counts
template <int NB>
__global__ void __launch_bounds__(1024) k_sort_offsets(uint32_t* __restrict__ buckets, uint32_t* __restrict__ offsets) {
    constexpr int PER = (NB + 1023) / 1024;
    __shared__ uint32_t part[1024];
    uint32_t v[PER], sum = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int b = threadIdx.x * PER + k;
        v[k] = b < NB ? buckets[b] : 0u;
        sum += v[k];
    }
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const uint32_t t = threadIdx.x >= (unsigned)off ? part[threadIdx.x - off] : 0u;
        __syncthreads();
        part[threadIdx.x] += t;
        __syncthreads();
    }
    uint32_t run = part[threadIdx.x] - sum;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int b = threadIdx.x * PER + k;
        if (b < NB) {
            offsets[b] = run;
            buckets[b] = 0u;
        }
        run += v[k];
    }
}

// perm[offsets[key]++] = ray: each block reserves one range per bucket, then fills it
template <int KEY>
__global__ void __launch_bounds__(256) k_sort_scatter(const TraceParams P, int q, const uint32_t* __restrict__ keys,
                                                       uint32_t* __restrict__ offsets, uint32_t* __restrict__ perm) {
    constexpr int NB = SortBuckets<KEY>::n;
    __shared__ uint32_t h[NB], start[NB];
    for (int i = threadIdx.x; i < NB; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const uint32_t count = round_nodes(P, q).y;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) atomicAdd(&h[keys[i]], 1u);
    __syncthreads();
    for (int i = threadIdx.x; i < NB; i += blockDim.x) {
        start[i] = h[i] ? atomicAdd(&offsets[i], h[i]) : 0u;
        h[i] = 0;
    }
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const uint32_t k = keys[i];
        perm[start[k] + atomicAdd(&h[k], 1u)] = i;
    }
}

}  // namespace

cudaError_t launch_trace(const TraceParams& p, cudaStream_t s) {
    static std::atomic<int> gridBlocks[2];  // zero-initialised (static storage); first use computes them
    const int c = p.countVisits ? 1 : 0;
    if (!gridBlocks[c].load(std::memory_order_acquire)) {
        int dev = 0, sms = 0, perSm = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = c ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, k_trace<true>, kTraceThreads, 0)
                  : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, k_trace<false>, kTraceThreads, 0);
        if (e != cudaSuccess) return e;
        gridBlocks[c].store(sms * (perSm > 0 ? perSm : 1), std::memory_order_release);
    }
    const int gBlocks = gridBlocks[c].load(std::memory_order_acquire);
    cudaError_t e = cudaMemsetAsync(p.workCounter, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    if (p.countVisits) k_trace<true><<<gBlocks, kTraceThreads, 0, s>>>(p);
    else k_trace<false><<<gBlocks, kTraceThreads, 0, s>>>(p);
    count_launch();
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    dim3 grid((p.W + 31) / 32, (p.H + 7) / 8);
    launch_chain(k_resolve, grid, 256, 0, s, p);
    count_launch();
    return cudaGetLastError();
}

static int persistent_grid(const void* fn, int threads, int smem) {
    int dev = 0, sms = 0, perSm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, fn, threads, smem) != cudaSuccess) return 0;
    return sms * (perSm > 0 ? perSm : 1);
}

// persistent grid sizes, one per kernel (computed on first use; contexts on several host threads
// share the table)
static int grid_of(const void* fn, int threads) {
    static std::mutex mu;
    static const void* fns[64];
    static int grids[64];
    static int n = 0;
    std::lock_guard<std::mutex> lock(mu);
    for (int k = 0; k < n; ++k)
        if (fns[k] == fn) return grids[k];
    const int g = persistent_grid(fn, threads, 0);
    if (g && n < 64) {
        fns[n] = fn;
        grids[n] = g;
        ++n;
    }
    return g;
}

typedef void (*TraceKernel)(const TraceParams, int);

// the traversal kernel of one launch shape
static TraceKernel trace_kernel(bool batch, bool count, int threads, int depth) {
    if (count) return batch ? k_wf_trace<true, kFormBatch, kTraceThreads, kTraversalStack> : k_wf_trace<true, kFormTree, kTraceThreads, kTraversalStack>;
    if (!batch) return k_wf_trace<false, kFormTree, kTraceThreads, kTraversalStack>;
#define RG_TK(T, D) \
    if (threads == T && depth == D) return k_wf_trace<false, kFormBatch, T, D>;
    RG_TK(64, 16) RG_TK(64, 24) RG_TK(64, 32) RG_TK(64, 48)
    RG_TK(128, 16) RG_TK(128, 24) RG_TK(128, 32) RG_TK(128, 48)
    RG_TK(256, 16) RG_TK(256, 24) RG_TK(256, 32)  // 256 x 48 exceeds the 48 KB of static shared memory
#undef RG_TK
    return nullptr;
}

bool tune_supported(const TraceTune& t) {
    return trace_kernel(true, false, t.threads, t.depth) != nullptr && t.sortKey >= RG_SORT_NONE && t.sortKey <= RG_SORT_MORTON;
}

// the query form of the traversal kernel for a stack depth (visit counting: the default depth only)
static TraceKernel query_kernel(bool count, int depth) {
    if (count) return k_wf_trace<true, kFormQuery, kTraceThreads, kTraversalStack>;
    switch (depth) {
        case 16: return k_wf_trace<false, kFormQuery, kTraceThreads, 16>;
        case 24: return k_wf_trace<false, kFormQuery, kTraceThreads, 24>;
        case 32: return k_wf_trace<false, kFormQuery, kTraceThreads, 32>;
        case 48: return k_wf_trace<false, kFormQuery, kTraceThreads, 48>;
        default: return nullptr;
    }
}

cudaError_t launch_trace_queue(const TraceParams& p, const float* rays, uint32_t n, float* tuv, uint32_t* ids, int depth,
                               cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    if (reinterpret_cast<uintptr_t>(rays) & 15u) return cudaErrorInvalidValue;  // read as float4
    const TraceKernel trace = query_kernel(p.countVisits != 0, depth);
    if (!trace) return cudaErrorInvalidValue;
    const int g = grid_of((const void*)trace, kTraceThreads);
    if (!g) return cudaErrorUnknown;
    TraceParams q = p;
    q.firstRound = 0;
    q.perm = nullptr;
    constexpr uint32_t kPart = 1u << 30;  // rays of a launch: the lists of overflowed rays keep 31 bits for one
    for (uint32_t at = 0; at < n; at += std::min(n - at, kPart)) {
        q.queryRays = reinterpret_cast<const float4*>(rays) + 2 * (size_t)at;
        q.queryTuv = tuv + 3 * (size_t)at;
        q.queryIds = ids + 2 * (size_t)at;
        q.queryCount = std::min(n - at, kPart);
        const cudaError_t e = cudaMemsetAsync(q.wf.fetch, 0, sizeof(uint32_t), s);
        if (e != cudaSuccess) return e;
        trace<<<g, kTraceThreads, 0, s>>>(q, 0);
        count_launch();
    }
    return cudaGetLastError();
}

// one lane of a frame: chunks of its samples, one after another in a stream, in a part of the node pool
struct FrameLane {
    TraceParams p;
    cudaStream_t s = nullptr;
    uint32_t* hostWords = nullptr;
    int k = 0, levels = 0;
    bool busy = false;
};

// nodes [at, at + n) of a pool, with control words of its own
static RayTree tree_part(const RayTree& t, size_t at, uint32_t n, uint32_t* ctl) {
    RayTree r = t;
    r.rayO += at; r.rayD += at; r.state += at; r.hitTUV += at; r.hitInst += at; r.surf += at; r.link += at; r.overflow += at;
    r.cand[0] += at; r.cand[1] += at;
    r.ctl = ctl;
    r.capacity = n;
    return r;
}

// Samples from which a frame runs as two lanes, each with half of the samples and of the pool in a stream of its own:
// every round ends with its longest rays and walks, and the host polls after every check; meanwhile the other
// lane has the chip.  2.75 M samples (1279x717, 3 a pixel) 6 % shorter, 8.3 M 1.7 %, 0.92 M 0, 0.23 M 3 % longer (its
// rounds no longer fill the chip).
constexpr uint32_t kTwoLanes = 1u << 20;
cudaError_t launch_trace_tree(const TraceParams& p0, cudaStream_t s, const TreeLane& second, uint32_t* hostWords, int* iterations, TreeLoad* load,
                              bool mayGrow, EventPairFn kernelEvents, void* user) {
    const TraceKernel trace = trace_kernel(false, p0.countVisits != 0, kTraceThreads, kTraversalStack);
    // glossy reference shading has kernels of its own; the reference's shading keeps the lean ones
    const auto expand = p0.glossySeed ? k_tree_expand<false, true> : k_tree_expand<false, false>;
    const auto check = p0.glossySeed ? k_tree_check<false, true> : k_tree_check<false, false>;
    const int gTrace = grid_of((const void*)trace, kTraceThreads), gExpand = grid_of((const void*)expand, 128),
              gCheck = grid_of((const void*)check, 128), gCompose = grid_of((const void*)k_tree_compose<false>, 128);
    if (!gTrace || !gExpand || !gCheck || !gCompose) return cudaErrorUnknown;
    const int maxRec = p0.ubo.maxRecursions;
    const uint32_t work = (uint32_t)frame_work_items(p0.W, p0.H, (uint32_t)p0.ubo.numSamples), cap = p0.tree.capacity;
    int it = 0;
    const int lanes = work >= kTwoLanes && !kernelEvents ? 2 : 1;
    FrameLane lane[2];
    for (int l = 0; l < lanes; ++l) {
        FrameLane& L = lane[l];
        L.p = p0;
        L.s = l ? second.stream : s;
        L.hostWords = l ? second.hostWords : hostWords;
        if (lanes == 2) L.p.tree = tree_part(p0.tree, (size_t)l * (cap / 2), cap / 2, l ? second.ctl : p0.tree.ctl);
        L.p.wf = {L.p.tree.ctl + kTreeFetch, L.p.tree.overflow};
    }
    const uint32_t pool = lane[0].p.tree.capacity;
    ChunkPlan plan(work, (uint32_t)lanes, pool, pool / kTreeNodesMin, std::move(*load));
    *load = TreeLoad();
    bool again = false;
    // rounds of a lane, its check and the words that decide what comes next
    auto rounds = [&](FrameLane& L) -> cudaError_t {
        cudaError_t e;
        for (int l = 0; l < L.levels; ++l, ++L.k, ++it) {
            L.p.firstRound = L.k == 0;
            cudaEvent_t e0 = nullptr, e1 = nullptr;
            if (kernelEvents && !kernelEvents(user, &e0, &e1)) e0 = e1 = nullptr;
            if (e0) cudaEventRecord(e0, L.s);
            if ((e = launch_chain(trace, gTrace, kTraceThreads, 0, L.s, L.p, L.k)) != cudaSuccess) return e;
            if (e1) cudaEventRecord(e1, L.s);
            if ((e = launch_chain(expand, gExpand, 128, 0, L.s, L.p, L.k)) != cudaSuccess) return e;
            count_launch(2);
        }
        if (maxRec == 0) return cudaSuccess;  // no hit issues a ray
        if ((e = launch_chain(check, gCheck, 128, 0, L.s, L.p, L.k)) != cudaSuccess) return e;
        count_launch();
        return cudaMemcpyAsync(L.hostWords, L.p.tree.ctl, 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, L.s);
    };
    auto start = [&](FrameLane& L) -> cudaError_t {  // the next chunk
        L.busy = plan.next(L.p.treeBase, L.p.treeRoots);
        if (!L.busy) return cudaSuccess;
        L.p.treeCand = 0;
        L.k = 0;
        L.levels = maxRec + 1;
        const cudaError_t e = cudaMemsetAsync(L.p.tree.ctl, 0, kTreeBounds * sizeof(uint32_t), L.s);
        return e != cudaSuccess ? e : rounds(L);
    };
    // what follows a lane's check
    auto advance = [&](FrameLane& L) -> cudaError_t {
        cudaError_t e;
        if (maxRec > 0) {
            if ((e = cudaStreamSynchronize(L.s)) != cudaSuccess) return e;
            const uint32_t* h = L.hostWords;
            const uint32_t nodes = L.p.treeRoots + h[kTreeAlloc];
            const bool pending = nodes > h[kTreeTraced], more = pending || h[kTreeChanges];
            // from the shallowest new ray down
            L.levels = pending && h[kTreeLevels] ? std::max(1, maxRec + 1 - (16 - (int)h[kTreeLevels])) : 1;
            if (nodes > L.p.tree.capacity || (more && L.k + L.levels >= kTreeMaxRounds)) {
                if (mayGrow && L.p.treeRoots == work) {  // nothing is composed yet
                    again = true;
                    L.busy = false;
                    return cudaSuccess;
                }
                if (L.p.treeRoots > 1) {  // in parts
                    plan.filled(L.p.treeBase, L.p.treeRoots);
                } else {
                    plan.done(L.p.treeBase, 1u, nodes);
                    k_sample_depth_first<<<1, 1, 0, L.s>>>(L.p);
                    count_launch();
                    if ((e = cudaGetLastError()) != cudaSuccess) return e;
                }
                return start(L);
            }
            if (more) {
                L.p.treeCand ^= 1u;
                return rounds(L);
            }
            plan.done(L.p.treeBase, L.p.treeRoots, nodes);
        }
        count_launch(L.k);
        while (L.k--)
            if ((e = launch_chain(k_tree_compose<false>, gCompose, 128, 0, L.s, L.p, L.k)) != cudaSuccess) return e;
        return start(L);
    };
    auto run = [&]() -> cudaError_t {
        cudaError_t e;
        if (lanes == 2) {
            if ((e = cudaEventRecord(second.fork, s)) != cudaSuccess) return e;
            if ((e = cudaStreamWaitEvent(second.stream, second.fork, 0)) != cudaSuccess) return e;
        }
        for (int l = 0; l < lanes; ++l)
            if ((e = start(lane[l])) != cudaSuccess) return e;
        while (lane[0].busy || lane[1].busy)
            for (int l = 0; l < lanes; ++l)
                if (lane[l].busy && (e = advance(lane[l])) != cudaSuccess) return e;
        if (lanes == 2) {
            if ((e = cudaEventRecord(second.join, second.stream)) != cudaSuccess) return e;
            return cudaStreamWaitEvent(s, second.join, 0);
        }
        return cudaSuccess;
    };
    const cudaError_t e = run();
    if (e != cudaSuccess) {
        if (lanes == 2) cudaStreamSynchronize(second.stream);  // nothing of the frame runs on behind its stream's back
        return e;
    }
    if (again) {
        load->full = load->again = true;
        return cudaSuccess;
    }
    if (iterations) *iterations = it;
    *load = plan.load();
    dim3 grid((p0.W + 31) / 32, (p0.H + 7) / 8);
    launch_chain(k_resolve, grid, 256, 0, s, p0);
    count_launch();
    return cudaGetLastError();
}

// sort of queue q by the tune's key into p.perm (the scratch's valsA)
static cudaError_t enqueue_sort(const TraceParams& p, int key, const SortScratch& sc, int grid, int q, cudaStream_t s) {
    if (key == RG_SORT_OCTANT) {
        k_sort_count<RG_SORT_OCTANT><<<grid, 256, 0, s>>>(p, q, sc.keysA, sc.hist);
        k_sort_offsets<SortBuckets<RG_SORT_OCTANT>::n><<<1, 1024, 0, s>>>(sc.hist, sc.hist + 4096);
        k_sort_scatter<RG_SORT_OCTANT><<<grid, 256, 0, s>>>(p, q, sc.keysA, sc.hist + 4096, sc.valsA);
    } else {
        k_sort_count<RG_SORT_MORTON><<<grid, 256, 0, s>>>(p, q, sc.keysA, sc.hist);
        k_sort_offsets<SortBuckets<RG_SORT_MORTON>::n><<<1, 1024, 0, s>>>(sc.hist, sc.hist + 4096);
        k_sort_scatter<RG_SORT_MORTON><<<grid, 256, 0, s>>>(p, q, sc.keysA, sc.hist + 4096, sc.valsA);
    }
    count_launch(3);
    return cudaGetLastError();
}

// a batch's launches: the kernels, their grids, and one round of them
struct BatchLaunch {
    TraceKernel trace = nullptr;
    int threads = 0, gTrace = 0, gExpand = 0, gCheck = 0, gCompose = 0, gSort = 0, sortKey = RG_SORT_NONE;
    SortScratch sort{};
    bool init(const TraceParams& p, const TraceTune& tune, const SortScratch& sc) {
        const bool c = p.countVisits != 0;
        threads = c ? kTraceThreads : tune.threads;
        trace = trace_kernel(true, c, threads, c ? kTraversalStack : tune.depth);
        sortKey = tune.sortKey;
        sort = sc;
        if (!trace || !tune_supported(tune)) return false;
        gTrace = grid_of((const void*)trace, threads);
        gExpand = grid_of((const void*)k_tree_expand<true, false>, 128);
        gCheck = grid_of((const void*)k_tree_check<true, false>, 128);
        gCompose = grid_of((const void*)k_tree_compose<true>, 128);
        gSort = grid_of((const void*)k_sort_scatter<RG_SORT_MORTON>, 256);
        return gTrace && gExpand && gCheck && gCompose && gSort;
    }
    // the bucket counts start at zero; each round's k_sort_offsets leaves them at zero again
    cudaError_t begin(cudaStream_t s) const {
        return sortKey == RG_SORT_NONE ? cudaSuccess : cudaMemsetAsync(sort.hist, 0, SortBuckets<RG_SORT_MORTON>::n * sizeof(uint32_t), s);
    }
    int perRound() const { return 2 + (sortKey != RG_SORT_NONE ? 3 : 0); }
    // round k (negative: the current one)
    cudaError_t round(TraceParams p, int k, cudaStream_t s, cudaEvent_t e0 = nullptr, cudaEvent_t e1 = nullptr) const {
        p.firstRound = k == 0;
        p.perm = nullptr;
        if (sortKey != RG_SORT_NONE && k != 0) {  // camera rays are coherent as they come
            p.perm = sort.valsA;
            const cudaError_t e = enqueue_sort(p, sortKey, sort, gSort, k, s);
            if (e != cudaSuccess) return e;
        }
        if (e0) cudaEventRecord(e0, s);
        trace<<<gTrace, threads, 0, s>>>(p, k);
        if (e1) cudaEventRecord(e1, s);
        k_tree_expand<true, false><<<gExpand, 128, 0, s>>>(p, k);
        count_launch(2);
        return cudaGetLastError();
    }
    void check(const TraceParams& p, cudaStream_t s) const {
        k_tree_check<true, false><<<gCheck, 128, 0, s>>>(p, -1);
        count_launch();
    }
    void compose(const TraceParams& p, int k, cudaStream_t s) const {
        k_tree_compose<true><<<gCompose, 128, 0, s>>>(p, k);
        count_launch();
    }
};

static TraceParams batch_params(const TraceParams& p0) {
    TraceParams p = p0;
    p.wf = {p.tree.ctl + kTreeFetch, p.tree.overflow};
    return p;
}

// runs of the loops on a chunk before a batch gives up (RG_BATCH_LOOP_LIMIT overrides, read when a graph is
// captured and at every batch of the host loop; tests use a small limit to check the reported error)
static uint32_t loop_limit() {
    const char* env = getenv("RG_BATCH_LOOP_LIMIT");
    return env ? (uint32_t)strtoul(env, nullptr, 10) : 50000u;
}

cudaError_t launch_trace_batch(const TraceParams& p0, const TraceTune& tune, const SortScratch& sort, uint32_t* loopWords, cudaStream_t s,
                               uint32_t* hostWords, int* iterations, bool* poolFull, EventPairFn kernelEvents, void* user) {
    const TraceParams p = batch_params(p0);
    BatchLaunch B;
    if (!B.init(p, tune, sort)) return cudaErrorInvalidValue;
    const TreeLoop loop = {false, 0, 0, 0, loopWords, loop_limit(), 0, 0, 0};
    auto poll = [&]() {
        cudaError_t e = cudaMemcpyAsync(hostWords, p.tree.ctl + kTreeMore, 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        return e;
    };
    auto round = [&](int k) {
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        if (kernelEvents && !kernelEvents(user, &e0, &e1)) e0 = e1 = nullptr;
        return B.round(p, k, s, e0, e1);
    };
    cudaError_t e;
    *iterations = 0;
    *poolFull = false;
    if ((e = B.begin(s)) != cudaSuccess) return e;
    k_tree_next<<<1, 1, 0, s>>>(p, loop, true);
    count_launch();
    for (;;) {
        for (int k = 0; k < p.batchRounds; ++k)
            if ((e = round(k)) != cudaSuccess) return e;
        for (;;) {
            B.check(p, s);
            k_tree_step<<<1, 1, 0, s>>>(p, loop);
            count_launch();
            if ((e = poll()) != cudaSuccess) return e;
            if (!hostWords[0]) break;
            for (int k = 0; k < std::max(1, p.batchRounds - 1); ++k)
                if ((e = round(-1)) != cudaSuccess) return e;
        }
        *iterations += (int)hostWords[2];
        if (hostWords[1]) *poolFull = true;
        else
            for (int k = (int)hostWords[2] - 1; k >= 0; --k) B.compose(p, k, s);
        k_tree_next<<<1, 1, 0, s>>>(p, loop, false);
        count_launch();
        if ((e = poll()) != cudaSuccess) return e;
        if (hostWords[3] == 2u) return cudaErrorLaunchTimeout;  // the loops gave up: samples are missing
        if (!hostWords[3]) break;
    }
    return cudaGetLastError();
}

// a while node after what stream s has captured so far; *body is its empty body graph
static cudaError_t add_while(cudaStream_t s, cudaGraphConditionalHandle* h, bool startTrue, cudaGraphNode_t* node, cudaGraph_t* body) {
    cudaStreamCaptureStatus st;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    cudaError_t e = cudaStreamGetCaptureInfo(s, &st, nullptr, &g, &deps, nullptr, &nd);
    if (e != cudaSuccess) return e;
    if (st != cudaStreamCaptureStatusActive) return cudaErrorStreamCaptureInvalidated;
    if (startTrue && (e = cudaGraphConditionalHandleCreate(h, g, 1u, cudaGraphCondAssignDefault)) != cudaSuccess) return e;
    cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
    cp.conditional.handle = *h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    if ((e = cudaGraphAddNode(node, g, deps, nullptr, nd, &cp)) != cudaSuccess) return e;
    *body = cp.conditional.phGraph_out[0];
    return cudaStreamUpdateCaptureDependencies(s, node, nullptr, 1, cudaStreamSetCaptureDependencies);
}

cudaError_t capture_trace_batch(const TraceParams& p0, const TraceTune& tune, const SortScratch& sort, cudaStream_t s,
                                cudaStream_t s2, uint32_t* loopWords) {
    const TraceParams p = batch_params(p0);
    if (p.countVisits) return cudaErrorInvalidValue;  // the visit-counting build runs the host loop
    BatchLaunch B;
    if (!B.init(p, tune, sort)) return cudaErrorInvalidValue;
    const int R = p.batchRounds, more = std::max(1, R - 1);
    TreeLoop loop = {true, 0, 0, 0, loopWords, loop_limit(), (uint32_t)(R * B.perRound() + 2 + R + 1), (uint32_t)(more * B.perRound() + 2),
                     (uint32_t)kTreeComposeRun + 1u};
    cudaStream_t s3 = nullptr;  // captures the inner loops' bodies
    cudaError_t e = cudaStreamCreateWithFlags(&s3, cudaStreamNonBlocking);
    if (e != cudaSuccess) return e;
    auto capture = [&]() -> cudaError_t {
        cudaError_t e;
        cudaGraphNode_t node;
        cudaGraph_t chunk = nullptr, body = nullptr, done = nullptr;
        if ((e = B.begin(s)) != cudaSuccess) return e;
        k_tree_next<<<1, 1, 0, s>>>(p, loop, true);
        if ((e = add_while(s, &loop.chunks, true, &node, &chunk)) != cudaSuccess) return e;
        if ((e = cudaStreamBeginCaptureToGraph(s2, chunk, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed)) != cudaSuccess) return e;
        auto inner = [&]() -> cudaError_t {
            cudaError_t e;
            cudaGraphNode_t n1;
            // both handles are set by k_tree_step before their nodes are reached
            if ((e = cudaGraphConditionalHandleCreate(&loop.rounds, chunk, 0u, 0)) != cudaSuccess) return e;
            if ((e = cudaGraphConditionalHandleCreate(&loop.composes, chunk, 0u, 0)) != cudaSuccess) return e;
            for (int k = 0; k < R; ++k)
                if ((e = B.round(p, k, s2)) != cudaSuccess) return e;
            B.check(p, s2);
            k_tree_step<<<1, 1, 0, s2>>>(p, loop);
            if ((e = add_while(s2, &loop.rounds, false, &n1, &body)) != cudaSuccess) return e;
            if ((e = cudaStreamBeginCaptureToGraph(s3, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed)) != cudaSuccess) return e;
            for (int k = 0; k < more && e == cudaSuccess; ++k) e = B.round(p, -1, s3);
            B.check(p, s3);
            k_tree_step<<<1, 1, 0, s3>>>(p, loop);
            cudaError_t e2 = cudaStreamEndCapture(s3, &done);
            if (e != cudaSuccess || e2 != cudaSuccess) return e != cudaSuccess ? e : e2;
            if ((e = add_while(s2, &loop.composes, false, &n1, &body)) != cudaSuccess) return e;
            if ((e = cudaStreamBeginCaptureToGraph(s3, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed)) != cudaSuccess) return e;
            for (int k = 1; k <= kTreeComposeRun; ++k) B.compose(p, -k, s3);
            k_tree_composed<<<1, 1, 0, s3>>>(p, loop);
            if ((e = cudaStreamEndCapture(s3, &done)) != cudaSuccess) return e;
            for (int k = R - 1; k >= 0; --k) B.compose(p, k, s2);
            k_tree_next<<<1, 1, 0, s2>>>(p, loop, false);
            return cudaGetLastError();
        };
        e = inner();
        const cudaError_t e2 = cudaStreamEndCapture(s2, &done);
        return e != cudaSuccess ? e : e2;
    };
    e = capture();
    cudaStreamDestroy(s3);
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_resolve_job(const float4* samples, const JobDesc& j, uint2* base, uint2* normal, uint2* rough, cudaStream_t s) {
    dim3 grid((j.W + 31) / 32, (j.H + 7) / 8);
    k_resolve_job<<<grid, 256, 0, s>>>(samples + 3 * (size_t)j.sampleBase, j.W, j.H, j.S, base, normal, rough);
    count_launch();
    return cudaGetLastError();
}

}  // namespace rg
