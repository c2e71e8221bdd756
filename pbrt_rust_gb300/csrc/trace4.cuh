// trace4.cuh - traversal over the 4-wide layout (layout.h: QuadNode).
//
// Each node holds the four grandchildren of one binary node N of the
// reference tree.  A visit tests the four child boxes and takes the ones that
// pass in the order in which BVHAccelerator::intersect
// (src/primitive/aggregates/bvh.rs:390-417) would: N's children in
// dir_is_neg[axis(N)] order, and inside each, that child's children in
// dir_is_neg order of its own axis.
//
// Why the results are the reference's bit for bit although the boxes here are
// rounded.  The reference tests a leaf's primitives iff the leaf's own box
// and every box above it pass against the maxt of the moment.  A box contains
// its children's boxes, its planes are among theirs or beyond them, and f32
// subtraction and multiplication are monotone, so whenever a leaf's box
// passes, the boxes above it do (they are tested earlier, against a maxt at
// least as large): the leaf's own box alone decides.  So a walk is exact if
// it reaches, in the reference's order, every leaf whose box passes, and
// lets a leaf's hits count only if the leaf's exact box passes.  Testing a
// primitive changes nothing unless it is hit, so a leaf of one primitive has
// its exact box tested only then (with the reference's operations,
// trace.cuh: slab).  The boxes on the way need only never be smaller than
// the exact ones:
//  * the stored planes are rounded outwards;
//  * a plane's distance is one fused multiply-add, t = code * (scale / d) +
//    (org - o) / d, where the reference computes (plane - o) * (1 / d).  Both
//    subtractions are exact but for one rounding of their result, so what
//    matters is how far the tree is from the ray's origin, not how far either
//    is from the coordinates' zero.  With u = 2^-24, i = |1 / d|, c the middle
//    of the tree's box on the axis, h half its extent and a few units in the
//    last place of its coordinates (tree_margins), a node has |org - o| <=
//    |c - o| + 2.1 h and code * scale <= 4.1 h, and the rounding of the two
//    forms adds up to at most u i (5 |c - o| + 27 h); the near planes are
//    moved towards the ray's start and the far planes away from it by
//    e = u i (6 |c - o| + 32 h);
//  * an axis with d = 0 has 1 / d replaced by kZeroInv, so large that e, here
//    of all three axes' sums, is beyond every other distance: a plane at the
//    origin or within e / i of it never culls, one farther off does.  The
//    exact test has +-inf there, as the reference.
// One box may pass where a box above it does not: with d = -0 the reference
// rejects an origin on the boundary of a box, unless the box is flat there.  A
// triangle of such a flat leaf is not hit (its determinant is 0); an analytic
// shape or an instance in one may be, so a walk that comes to them there gives
// up and the ray takes the exact walk described below.
// The deferred children are pushed with their entry distance and re-checked
// against maxt when popped.
//
// All of this needs finite numbers of moderate size.  Trees beyond 2^40 have
// no 4-wide layout (HostBVH::wide), and a ray that is not `clean` (NaN or
// infinite components, |c - o| above 2^41, |d| or 1 / d above 2^60, tmin below
// -2^60) is walked over the binary layout in the exact mode of trace.cuh
// instead (exact_hit / exact_any), as is a ray that accepted a hit at
// distance NaN, after which the reference's box tests ignore maxt, and a ray
// from so far away (DevBVH4::mid.w) that its margins would have it visit most
// of the tree.  Kernels
// with one thread per ray do that after the walk; the persistent ones mark
// the ray for a replay kernel queued behind them, because the call inside
// their loop costs the walk its registers (2^22 incoherent rays into a
// terrain of a million triangles: 586 us with the calls, 529 without).
//
// The stack: ROWS 8-byte entries per thread in shared memory ([entry][thread],
// so a warp's accesses hit distinct banks), the oldest entries going to an
// array in local memory when they run out.  The tree's bound
// (HostBVH::stack4_bound) counts the children that exist.  An empty slot's
// planes lie the wrong way round, but in a node smaller than the margins it
// passes all the same and takes entries beyond the bound, so a walk may find
// its stack full; it then gives up and the ray takes the exact walk, whose
// entries (one per level at most) the bound does cover.  The bottom entry is a
// word that ends the walk, so a pop needs no test for an empty stack.  A visit
// stores
// all four children without branches: a 128-word table in shared memory,
// indexed by the node's visiting order for the ray's octant and the mask of
// passing children, gives each child's place above the top (children that
// fail go to the place above the last one), and the first child is then
// popped like any other, so the lanes of a warp run the same instructions
// whether they hit children or not.  Against ordering the children by
// compare-and-swap and branching per push, a visit is about 110 instructions
// instead of 210 (2^20 rays into 4096 random triangles: 524 -> 405 us).
// Registers are what the walk is short of (64 at 8 blocks per SM): a thread's
// rows follow from the top's address, and a ray that has to give up is one
// whose maxt is NaN.
// INST: the tree may hold instance records (kernels take it only for scenes
// that have instances).
#pragma once
#include <stdint.h>

#include "layout.h"
#include "trace.cuh"

namespace pbrt {

// A tree in both layouts.
struct DevBVH4 {
    DevBVH pair;            // the binary layout, primitives and analytic records
    const QuadNode* nodes;
    const LeafBox* boxes;
    uint32_t root_ref;      // the root's child word
    float4 mid, half, spread;  // HostBVH::middle (w: far), ::half, ::spread
};

// Stack words that are not children (leaf words stay below: HostBVH::wide
// bounds the primitives).
constexpr uint32_t kWalkDone = 0xfffffffdu;  // the bottom of the stack
constexpr uint32_t kExitInst = 0xfffffffeu;  // ends the walk of an instance definition

constexpr float kInvMax = 1.152921504606846976e18f;     // 2^60, for |d| too
constexpr float kZeroInv = 1.9342813113834067e25f;      // 2^84, in place of 1 / 0

// An instance definition's 4-wide stack bound is at most 96 (checked at
// creation) and a binary walk defers no more entries than the 4-wide one.
constexpr int kInstStack = 104;

template <bool ANY>
__device__ __noinline__ TraceResult instance_test(const DevBVH4* insts, const SphereRec* s, float ox, float oy,
                                                  float oz, float dx, float dy, float dz, float tmin, float maxt) {
    float o[3], d[3];
    xf_point(s->w2o, ox, oy, oz, o);  // transform.rs:230-237: o as a point, d as a vector
    xf_vector(s->w2o, dx, dy, dz, d);
    DRay ri = make_dray(make_float4(o[0], o[1], o[2], tmin), make_float4(d[0], d[1], d[2], maxt));
    const DevBVH& B = insts[s->instance].pair;
    TraceResult res;
    int st = 0;
    bool nan_hit = false;
    traverse<kInstStack, ANY>(B, ri, &res, &st, &nan_hit);
    if (!ANY && nan_hit) traverse<kInstStack, false, false, true>(B, ri, &res, &st);  // replay
    return res;
}

// One ray over the binary layout in exact mode: the closest hit's record /
// whether anything is hit.  `ray`: its two float4.  Out of line: few rays
// need them.
template <int STACK, bool INST>
static __device__ __noinline__ float4 exact_hit(const DevBVH& bvh, const float4* ray, int* status) {
    const DRay r = make_dray(__ldg(ray), __ldg(ray + 1));
    TraceResult res;
    int st = 0;
    traverse<STACK, false, INST, true>(bvh, r, &res, &st);
    if (st) atomicMax(status, st);
    return make_float4(__int_as_float(res.prim), res.t, res.b1, res.b2);
}
template <int STACK, bool INST>
static __device__ __noinline__ bool exact_any(const DevBVH& bvh, const float4* ray, int* status) {
    const DRay r = make_dray(__ldg(ray), __ldg(ray + 1));
    TraceResult res;
    int st = 0;
    const bool found = traverse<STACK, true, INST>(bvh, r, &res, &st);
    if (st) atomicMax(status, st);
    return found;
}

// Two f32 values in one 64-bit register; sm_103a multiplies and adds both in
// one instruction, each rounded on its own.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

struct Words8 {
    uint32_t w[8];
};
__device__ __forceinline__ Words8 ld_words8(const void* p) {  // 32 bytes in one load
    Words8 q;
    asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(q.w[0]), "=r"(q.w[1]), "=r"(q.w[2]), "=r"(q.w[3]), "=r"(q.w[4]), "=r"(q.w[5]), "=r"(q.w[6]),
                   "=r"(q.w[7])
                 : "l"(p));
    return q;
}

// Byte k of a plane word as the plane's grid coordinate (layout.h).
__device__ __forceinline__ float plane(uint32_t w, int k) {
    return __uint_as_float(__byte_perm(w, 0x43000000u, 0x7044u | ((uint32_t)k << 8)));
}

// Stack entries by 32-bit shared-memory address.
__device__ __forceinline__ void st_entry(uint32_t addr, uint32_t ref, float t) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(ref), "f"(t) : "memory");
}
__device__ __forceinline__ void ld_entry(uint32_t addr, uint32_t& ref, float& t) {
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(ref), "=f"(t) : "r"(addr) : "memory");
}

// The push table: entry [code][fails], byte k = rows above the top at which
// child k goes (the child visited first on top; children whose box failed,
// bit 3 - k of `fails`, above them all).  code: bit 0 / 1 = the first / second
// pair's children swap places, bit 2 = the pairs do.
constexpr int kPushTable = 128;
__device__ __forceinline__ uint32_t push_entry(uint32_t i) {
    const uint32_t code = i >> 4, mask = (__brev(i) >> 28) ^ 15u;  // bit k: child k passed
    auto place = [&](uint32_t k) {  // of child k among the four
        const uint32_t pair = k >> 1;
        return ((pair ^ (code >> 2)) << 1) | ((k & 1u) ^ ((code >> pair) & 1u));
    };
    uint32_t e = 0;
    for (uint32_t k = 0; k < 4; ++k) {
        uint32_t row = 0;
        for (uint32_t j = 0; j < 4; ++j)
            if ((mask >> j) & 1u) row += ((mask >> k) & 1u) ? (place(j) > place(k) ? 1u : 0u) : 1u;
        e |= row << (8 * k);
    }
    return e;
}
// The rows that stay on the stack.
__device__ __forceinline__ uint32_t push_rows(uint32_t i) { return 4u - (uint32_t)__popc(i & 15u); }

// Shared memory of a block of 4-wide walks: the stacks, the push table and,
// with instances, the world rays of the lanes that are inside one.
template <int BLOCK, int ROWS, bool INST>
struct alignas(16) WalkShared {
    uint2 stack[ROWS][BLOCK];
    uint2 push[kPushTable];  // the places; by how much the top moves
    float world[INST ? 12 : 1][INST ? BLOCK : 1];
    // every thread of the block; __syncthreads() inside
    __device__ __forceinline__ void init() {
        if (threadIdx.x < kPushTable)
            push[threadIdx.x] = make_uint2(push_entry(threadIdx.x), push_rows(threadIdx.x) * (BLOCK * 8u));
        __syncthreads();
    }
};

// INST walks' extra state: the tree being walked (-1: the scene's, else the
// definition) with its arrays, and the instance's first id (0 outside).
template <bool INST>
struct InstWalk {
    const QuadNode* nodes_;
    const PrimRec* prims_;
    int32_t def_;
    uint32_t base_;
};
template <>
struct InstWalk<false> {};

enum { kStartMiss = 0, kStartWalk = 1, kStartExact = 2 };

// The oldest entries of a walk's stack, in local memory.  A kernel declares
// it beside the walk: inside it, its variable indexing would keep the whole
// walk out of registers.
template <int OVF>
struct Overflow {
    uint2 e[OVF];
};

// The walk of one ray.  `cur` is the next node (non-negative as an integer),
// the next leaf, or one of the stack words above; node() and leaf() move it
// on.  OVF: entries of the overflow (64 or 256, as the tree's stack bound
// asks).
template <int BLOCK, int ROWS, int OVF, bool ANY, bool INST = false>
struct Walk4 : InstWalk<INST> {
    static constexpr uint32_t kRow = BLOCK * 8u;
    static constexpr int kSpill = ROWS - 8;  // rows moved to the overflow at a time
    using Shared = WalkShared<BLOCK, ROWS, INST>;
    using Ovf = Overflow<OVF>;

    float ox, oy, oz, tmin;
    float dx, dy, dz, maxt;
    float ix, iy, iz;  // 1 / d (kZeroInv for d = 0)
    float ex, ey, ez;  // margins of a plane's distance
    uint32_t oct3;     // 3 * the ray's octant
    uint32_t cur;
    uint32_t top;      // shared-memory address of the first free row
    int spilled;       // entries in the overflow
    int32_t prim;      // -1: none yet
    float b1, b2;
    uint32_t base, push_tab;  // shared-memory addresses, the same for all threads

    __device__ __forceinline__ void bind(Shared& sh) {
        base = (uint32_t)__cvta_generic_to_shared(sh.stack);
        push_tab = (uint32_t)__cvta_generic_to_shared(sh.push);
        top = base + threadIdx.x * 8u;
        st_entry(top, kWalkDone, __int_as_float(0xff800000));  // -inf: always taken
        cur = kWalkDone;
    }

    // Row i of this thread, from the top's address, which is in one of its rows.
    __device__ __forceinline__ uint32_t row(int i) const {
        return base + ((top - base) & (kRow - 1u)) + (uint32_t)i * kRow;
    }

    // 1 / d, octant and margins of the ray (o, d) in a tree; false if the ray
    // is not clean or too far away (see above).  (One margin for all axes
    // inside instances, which reads less of the definition's record, makes
    // entries 1 % cheaper and lets far rays visit up to three times as much: 2^20
    // rays from 3000 extents into 64 instances 570 -> 726 us.)
    __device__ __forceinline__ bool aim(const DevBVH4& tree) {
        const bool zx = dx == 0.0f, zy = dy == 0.0f, zz = dz == 0.0f;
        ix = 1.0f / dx;
        iy = 1.0f / dy;
        iz = 1.0f / dz;
        // a sum, so that a NaN component fails the comparison
        const float sd = fabsf(dx) + fabsf(dy) + fabsf(dz);
        bool ok = sd <= kInvMax && sd > 0.0f && tmin >= -kInvMax && maxt == maxt &&
                  max3f(zx ? 0.0f : fabsf(ix), zy ? 0.0f : fabsf(iy), zz ? 0.0f : fabsf(iz)) <= kInvMax;
        if (zx) ix = copysignf(kZeroInv, dx);
        if (zy) iy = copysignf(kZeroInv, dy);
        if (zz) iz = copysignf(kZeroInv, dz);
        octant();
        return margins(tree, zx, zy, zz) && ok;
    }
    __device__ __forceinline__ void octant() {
        oct3 = 3u * ((__float_as_uint(ix) >> 31) | ((__float_as_uint(iy) >> 31) << 1) |
                     ((__float_as_uint(iz) >> 31) << 2));
    }
    // false: too far away, or a NaN in the origin.
    __device__ __forceinline__ bool margins(const DevBVH4& tree, bool zx, bool zy, bool zz) {
        const float4 mid = tree.mid, spread = tree.spread;
        const float mx = __fmaf_rn(kFarMargin, fabsf(mid.x - ox), spread.x),
                    my = __fmaf_rn(kFarMargin, fabsf(mid.y - oy), spread.y),
                    mz = __fmaf_rn(kFarMargin, fabsf(mid.z - oz), spread.z), all = mx + my + mz;
        ex = (zx ? all : mx) * fabsf(ix);
        ey = (zy ? all : my) * fabsf(iy);
        ez = (zz ? all : mz) * fabsf(iz);
        return all <= mid.w;
    }
    // The ray with the reference's 1 / d, for the exact tests.
    __device__ __forceinline__ DRay ray() const {
        DRay r;
        r.ox = ox;
        r.oy = oy;
        r.oz = oz;
        r.tmin = tmin;
        r.dx = dx;
        r.dy = dy;
        r.dz = dz;
        r.tmax = maxt;
        auto inv = [](float i) { return fabsf(i) == kZeroInv ? copysignf(__int_as_float(0x7f800000), i) : i; };
        r.ix = inv(ix);
        r.iy = inv(iy);
        r.iz = inv(iz);
        r.neg = 0;
        return r;
    }

    __device__ __forceinline__ int start(const DevBVH4& bvh, float4 a, float4 b) {
        ox = a.x;
        oy = a.y;
        oz = a.z;
        tmin = a.w == 0.0f ? -0.0f : a.w;  // node(): an entry at +0 would fail against an exit at -0
        dx = b.x;
        dy = b.y;
        dz = b.z;
        maxt = b.w;
        prim = -1;
        b1 = 0.0f;
        b2 = 0.0f;
        spilled = 0;
        top = row(1);
        if constexpr (INST) {
            this->nodes_ = bvh.nodes;
            this->prims_ = bvh.pair.prims;
            this->def_ = -1;
            this->base_ = 0;
        }
        if (bvh.pair.empty) return kStartMiss;
        if (!aim(bvh)) return kStartExact;
        // the root's box, from its middle, with the same margins (this form's
        // rounding: u i (5 |c - o| + 4 h) against the reference's)
        const float tx = (bvh.mid.x - ox) * ix, rx = __fmaf_rn(bvh.half.x, fabsf(ix), ex);
        const float ty = (bvh.mid.y - oy) * iy, ry = __fmaf_rn(bvh.half.y, fabsf(iy), ey);
        const float tz = (bvh.mid.z - oz) * iz, rz = __fmaf_rn(bvh.half.z, fabsf(iz), ez);
        const float t0 = max3f(tx - rx, ty - ry, fmaxf(tz - rz, tmin));
        const float t1 = min3f(tx + rx, ty + ry, fminf(tz + rz, maxt));
        if (t0 > t1) return kStartMiss;
        cur = bvh.root_ref;
        return kStartWalk;
    }

    // Moves the oldest rows to the overflow when fewer than four are free; a
    // walk whose overflow is full gives up.
    __device__ __forceinline__ void make_room(Ovf& ov) {
        if (top < base + (ROWS - 3) * kRow) return;
        if (spilled + kSpill > OVF) return give_up();
        for (int i = 0; i < kSpill; ++i) {
            uint32_t ref;
            float t;
            ld_entry(row(1 + i), ref, t);
            ov.e[spilled + i] = make_uint2(ref, __float_as_uint(t));
        }
        spilled += kSpill;
        for (uint32_t a = row(1 + kSpill); a < top; a += kRow) {
            uint32_t ref;
            float t;
            ld_entry(a, ref, t);
            st_entry(a - kSpill * kRow, ref, t);
        }
        top -= kSpill * kRow;
    }
    // An any-hit walk's maxt does not change, so its entries still pass.
    __device__ __forceinline__ void pop() {
        float t;
        do {
            top -= kRow;
            ld_entry(top, cur, t);
        } while (!ANY && t > maxt);
    }
    // cur == kWalkDone: brings spilled rows back and goes on; false when the
    // walk is over.
    __device__ __forceinline__ bool resume(Ovf& ov) {
        if (spilled == 0) return false;
        spilled -= kSpill;
        for (int i = 0; i < kSpill; ++i)
            st_entry(row(1 + i), ov.e[spilled + i].x, __uint_as_float(ov.e[spilled + i].y));
        top = row(1 + kSpill);
        pop();
        return true;
    }

    // Visits inner node `cur`.  The integer pipe is the busiest (69 % with
    // issue at 77 % on camera rays of a terrain frame; the byte permutes,
    // minima and selects run there), so a child's failing is the sign bit of
    // exit - entry, shifted into the table index (the sign is wrong only for
    // an exit at -0, a hit's or the ray's maxt, and an entry at +0, which
    // cannot be: tmin is not +0 and a near plane at +0 less the margin is
    // beyond -0 without it), and its row's address one
    // 16-bit dot product, which the multiply pipe does; the table also holds
    // how far the top moves (a population count otherwise).  Against
    // compares, a mask, permutes and multiplies: terrain frame's camera /
    // shadow rays 1945 / 2692 -> 1899 / 2594 us, shadow rays at 56 registers
    // (9 blocks per SM) 2553.
    __device__ __forceinline__ void node(const DevBVH4& bvh, Ovf& ov) {
        const QuadNode* nodes;
        if constexpr (INST)
            nodes = this->nodes_;
        else
            nodes = bvh.nodes;
        const char* p = reinterpret_cast<const char*>(nodes + cur);
        const Words8 q0 = ld_words8(p), q1 = ld_words8(p + 32);
        const bool px = ix < 0.0f, py = iy < 0.0f, pz = iz < 0.0f;
        const uint32_t nx = px ? q0.w[7] : q0.w[6], fx = px ? q0.w[6] : q0.w[7];
        const uint32_t ny = py ? q1.w[1] : q1.w[0], fy = py ? q1.w[0] : q1.w[1];
        const uint32_t nz = pz ? q1.w[3] : q1.w[2], fz = pz ? q1.w[2] : q1.w[3];
        const float gx = __uint_as_float(q0.w[0]) - ox, gy = __uint_as_float(q0.w[1]) - oy,
                    gz = __uint_as_float(q0.w[2]) - oz;
        const float ax = __uint_as_float(q0.w[3]) * ix, ay = __uint_as_float(q0.w[3] << 16) * iy,
                    az = __uint_as_float(q0.w[4]) * iz;
        const uint64_t bx = pack2(__fmaf_rn(gx, ix, -ex), __fmaf_rn(gx, ix, ex));
        const uint64_t by = pack2(__fmaf_rn(gy, iy, -ey), __fmaf_rn(gy, iy, ey));
        const uint64_t bz = pack2(__fmaf_rn(gz, iz, -ez), __fmaf_rn(gz, iz, ez));
        const uint64_t ax2 = pack2(ax, ax), ay2 = pack2(ay, ay), az2 = pack2(az, az);
        float t[4];
        uint32_t index = q0.w[5] >> oct3;  // the visiting order, then a bit per child: not passed
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float n0, f0, n1, f1, n2, f2;
            unpack2(fma2(pack2(plane(nx, k), plane(fx, k)), ax2, bx), n0, f0);
            unpack2(fma2(pack2(plane(ny, k), plane(fy, k)), ay2, by), n1, f1);
            unpack2(fma2(pack2(plane(nz, k), plane(fz, k)), az2, bz), n2, f2);
            t[k] = max3f(n0, n1, fmaxf(n2, tmin));
            const float t1 = min3f(f0, f1, fminf(f2, maxt));
            index = __funnelshift_l(__float_as_uint(t1 - t[k]), index, 1);
        }
        uint32_t e, up;
        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(e), "=r"(up) : "r"(push_tab + (index & 127u) * 8u));
        st_entry(__dp2a_lo(kRow, e, top), q1.w[4], t[0]);
        st_entry(__dp2a_lo(kRow << 16, e, top), q1.w[5], t[1]);
        st_entry(__dp2a_hi(kRow, e, top), q1.w[6], t[2]);
        st_entry(__dp2a_hi(kRow << 16, e, top), q1.w[7], t[3]);
        top += up;
        make_room(ov);
        pop();
    }

    // Hit at t of primitive word `id`.
    __device__ __forceinline__ void accept(uint32_t id, float t, float u, float v) {
        maxt = ANY || maxt == maxt ? t : maxt;  // NaN stays: gave_up()
        if constexpr (INST)
            prim = (int32_t)(this->base_ + (id & ~kSphereBit));
        else
            prim = (int32_t)(id & ~kSphereBit);
        b1 = u;
        b2 = v;
    }
    // An any-hit walk is over.
    __device__ __forceinline__ void stop() {
        cur = kWalkDone;
        spilled = 0;
    }
    // The ray takes the exact walk; this one is over, also after a pop.
    __device__ __forceinline__ void give_up() {
        maxt = __int_as_float(0x7fc00000);  // gave_up()
        top = row(1);
        stop();
    }

    // Whether a leaf's box, which the ray passes, is flat where the ray's
    // direction (of reciprocals i) is -0: a box above it need not pass then.
    __device__ __forceinline__ static bool beside(const LeafBox* box, float i_x, float i_y, float i_z) {
        if (min3f(i_x, i_y, i_z) != -kZeroInv) return false;
        const float4 lo = ldg4(box->lo), hi = ldg4(box->hi);
        return (i_x == -kZeroInv && lo.x == hi.x) || (i_y == -kZeroInv && lo.y == hi.y) ||
               (i_z == -kZeroInv && lo.z == hi.z);
    }

    // INST: the instance record S (first id `first`) of the scene's tree;
    // `rest` is the leaf word of the rest of its leaf (0: none), `box` the
    // leaf's.  1 when its walk was entered (`cur` set), 0 when the ray misses
    // it, 2 when the primitive-space ray is not clean or the leaf's box flat
    // beside it: the whole ray then takes the exact walk.  TransformedPrimitive::intersect
    // (transformed.rs:35-56): the primitive-space ray is w2p(ray) - o as a
    // point, d as a vector, mint and the current maxt kept.  If it passes the
    // definition's root box, the walk pushes the rest of the leaf and an exit
    // word (both with entry distance -inf, so they are always taken) and
    // continues in the definition's tree with that ray; popping the exit word
    // restores the world ray and the scene's tree.  The definition is thus
    // searched completely, in the reference's order, before the leaf's next
    // primitive, and the shared maxt is the reference's ray.set_maxt.
    __device__ __forceinline__ int enter(const DevBVH4& bvh, Shared& sh, const SphereRec* S, uint32_t first,
                                         uint32_t rest, const LeafBox* box) {
        const DevBVH4& D = bvh.pair.insts[S->instance];
        if (D.pair.empty) return 0;
        float o[3], d[3];
        xf_point(S->w2o, ox, oy, oz, o);  // transform.rs:230-237
        xf_vector(S->w2o, dx, dy, dz, d);
        float* w = &sh.world[0][threadIdx.x];
        const float keep[12] = {ox, oy, oz, dx, dy, dz, ix, iy, iz, ex, ey, ez};
#pragma unroll
        for (int k = 0; k < 12; ++k) w[k * BLOCK] = keep[k];
        ox = o[0];
        oy = o[1];
        oz = o[2];
        dx = d[0];
        dy = d[1];
        dz = d[2];
        const ChildRec& R = D.pair.root;
        float tr;
        if (!aim(D)) return 2;
        if (!slab(R.lo_x, R.lo_y, R.lo_z, R.hi_x, R.hi_y, R.hi_z, ray(), maxt, &tr)) {
            restore(bvh, sh);
            return 0;
        }
        if (beside(box, w[6 * BLOCK], w[7 * BLOCK], w[8 * BLOCK])) return 2;
        if (rest) {
            st_entry(top, rest, __int_as_float(0xff800000));
            top += kRow;
        }
        st_entry(top, kExitInst, __int_as_float(0xff800000));
        top += kRow;
        if constexpr (INST) {
            this->nodes_ = D.nodes;
            this->prims_ = D.pair.prims;
            this->def_ = (int32_t)S->instance;
            this->base_ = first;
        }
        cur = D.root_ref;
        return 1;
    }
    // Back to the scene's tree and the world ray.
    __device__ __forceinline__ void restore(const DevBVH4& bvh, Shared& sh) {
        const float* w = &sh.world[0][threadIdx.x];
        ox = w[0];
        oy = w[BLOCK];
        oz = w[2 * BLOCK];
        dx = w[3 * BLOCK];
        dy = w[4 * BLOCK];
        dz = w[5 * BLOCK];
        ix = w[6 * BLOCK];
        iy = w[7 * BLOCK];
        iz = w[8 * BLOCK];
        ex = w[9 * BLOCK];
        ey = w[10 * BLOCK];
        ez = w[11 * BLOCK];
        octant();
        if constexpr (INST) {
            this->nodes_ = bvh.nodes;
            this->prims_ = bvh.pair.prims;
            this->def_ = -1;
            this->base_ = 0;
        }
    }

    // `cur` is a leaf (or INST: the exit word): tests its primitives in order
    // and goes on.
    __device__ __forceinline__ void leaf(const DevBVH4& bvh, Shared& sh, Ovf& ov) {
        const PrimRec* prims;
        const SphereRec* spheres;
        const LeafBox* boxes;
        if constexpr (INST) {
            if (cur == kExitInst) {
                restore(bvh, sh);
                pop();
                return;
            }
            prims = this->prims_;
            const DevBVH4& B = this->def_ < 0 ? bvh : bvh.pair.insts[this->def_];
            spheres = B.pair.spheres;
            boxes = B.boxes;
        } else {
            prims = bvh.pair.prims;
            spheres = bvh.pair.spheres;
            boxes = bvh.boxes;
        }
        uint32_t off = cur & ~kNode4Leaf;
        for (;;) {
            const PrimRec* pr = prims + off;
            const float4 r0 = ldg4(pr->r0), r1 = ldg4(pr->r1), r2 = ldg4(pr->r2);
            const uint32_t id = __float_as_uint(r0.w), flags = __float_as_uint(r2.w);
            auto table_box = [&]() {
                const LeafBox* b = boxes + (flags >> kPrimBoxShift);
                const float4 lo = ldg4(b->lo), hi = ldg4(b->hi);
                float tr;
                return slab(lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, ray(), maxt, &tr);
            };
            if ((flags & kPrimBoxEntry) && !table_box()) break;
            float t, u = 0.0f, v = 0.0f;
            bool hit;
            if (id & kSphereBit) {
                const uint32_t si = __float_as_uint(r1.w);
                if constexpr (INST) {
                    const SphereRec* S = spheres + si;
                    if (S->kind == kQuadInstance) {  // only in the scene's tree: definitions hold none
                        const int e = enter(bvh, sh, S, id & ~kSphereBit,
                                            (flags & kPrimLastBit) ? 0u : (kNode4Leaf | (off + 1)),
                                            boxes + (flags >> kPrimBoxShift));
                        if (e == 1) return make_room(ov);
                        if (e == 2) return give_up();
                        if (flags & kPrimLastBit) break;
                        ++off;
                        continue;
                    }
                }
                hit = sphere_test(spheres, si, ray(), maxt, &t);
                if (hit && (flags & kPrimHitBox)) hit = table_box();
                if (hit && beside(boxes + (flags >> kPrimBoxShift), ix, iy, iz)) {
                    give_up();
                    break;
                }
            } else {
                hit = tri_test(r0, r1, r2, ray(), maxt, &t, &u, &v);
                if (hit && (flags & kPrimOwnBox)) {
                    float tr;
                    hit = slab(fminf(fminf(r0.x, r1.x), r2.x), fminf(fminf(r0.y, r1.y), r2.y),
                               fminf(fminf(r0.z, r1.z), r2.z), fmaxf(fmaxf(r0.x, r1.x), r2.x),
                               fmaxf(fmaxf(r0.y, r1.y), r2.y), fmaxf(fmaxf(r0.z, r1.z), r2.z), ray(), maxt, &tr);
                    // A hit whose box a direction of -0 rejects (the origin is
                    // on its boundary): the boxes above are likely rejected
                    // too, and without hits nothing here would be culled.
                    if (!hit && min3f(ix, iy, iz) == -kZeroInv) {
                        give_up();
                        break;
                    }
                }
            }
            if (hit) {
                accept(id, t, u, v);
                if (ANY) return stop();
            }
            if (flags & kPrimLastBit) break;
            ++off;
        }
        pop();
    }

    // The whole walk after start() returned kStartWalk.  Two visits per turn
    // before the leaves: the lanes of a warp that reach a leaf one visit apart
    // test it together (camera / shadow rays of a 1024 x 1024 x 16 terrain
    // frame: 2282 / 3911 us with node or leaf per turn, 2038 / 2676 with one
    // visit, 1952 / 2631 with two, 1985 / 2831 with three; waiting for 4 or
    // more lanes at leaves is slower, 2111 / 2757).
    __device__ __forceinline__ void run(const DevBVH4& bvh, Shared& sh, Ovf& ov) {
        for (;;) {
#pragma unroll
            for (int k = 0; k < 2; ++k)
                if ((int32_t)cur >= 0) node(bvh, ov);
            if ((int32_t)cur < 0 && cur != kWalkDone) leaf(bvh, sh, ov);
            if (cur == kWalkDone && !resume(ov)) return;
        }
    }
    // A hit at distance NaN, a flat box beside the ray, an instance ray that
    // was not clean or a full stack: the ray needs the exact walk.
    __device__ __forceinline__ bool gave_up() const { return !(maxt == maxt); }
    __device__ __forceinline__ bool found() const { return prim >= 0; }
    __device__ __forceinline__ float4 hit_record() const {
        return make_float4(__int_as_float(prim), prim >= 0 ? maxt : 0.0f, b1, b2);
    }
};

}  // namespace pbrt
