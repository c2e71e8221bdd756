// quads.cu - the 4-wide layout (layout.h: QuadNode) encoded from the binary
// one.  One thread per binary pair that starts a 4-wide node: the boxes of
// its grandchildren are all in it and its two children's pairs.  The grid
// arithmetic runs in 64 bits, so that a plane's rounding direction is decided
// on (nearly) exact values; what the 64-bit form rounds is far below the
// margin the walk gives every plane (trace4.cuh).
#include <cuda_runtime.h>

#include "host_scene.h"
#include "kernels.h"

namespace pbrt {

namespace {

constexpr uint32_t kNone = 0xffffffffu;  // HostBVH::quad_of: no 4-wide node starts here
constexpr uint32_t kAxisShift = 30u;     // kQuadAxisShift

__device__ __forceinline__ double code_value(int c) { return c < 128 ? 128.0 + c : 2.0 * c; }

// Largest float scale of the given kind at least `want`: 0 = any, 1 = a
// bfloat16, 2 = any with the low half `low`.
__device__ __forceinline__ float scale_of(int kind, float want, uint32_t low) {
    const uint32_t u = __float_as_uint(want);
    if (kind == 1) return __uint_as_float((u + 0xffffu) & 0xffff0000u);
    if (kind == 2) {
        uint32_t v = (u & 0xffff0000u) | low;
        if (v < u) v += 0x10000u;
        return __uint_as_float(v);
    }
    return want;
}

// Origin and scale of an axis' grid: org + v(0) * scale <= lo and
// org + v(255) * scale >= hi.
__device__ __forceinline__ void fit_axis(float lo, float hi, int kind, uint32_t low, float* org, float* scale) {
    float want = (float)(((double)hi - (double)lo) / 382.0 * (1.0 + 1e-6));
    if (!(want > 1e-30f)) want = 1e-30f;
    for (;;) {
        const float s = scale_of(kind, want, low);
        const float o = __double2float_rd((double)lo - 128.0 * (double)s);
        *org = o;
        *scale = s;
        if ((double)o + 510.0 * (double)s >= (double)hi) return;
        want = s * 1.5f;  // o was rounded down by more than the slack
    }
}

// Codes of the planes; inv = 1 / s.  Off by one towards the outside at most
// (this GPU divides doubles slowly: one division per axis, not per plane, took
// the kernel for 180000 triangles from 162 to 114 us).
__device__ __forceinline__ int code_down(double org, double s, double inv, float x) {
    const double v = ((double)x - org) * inv;
    int c = v < 256.0 ? (int)floor(v) - 128 : (int)floor(v * 0.5);
    c = min(max(c, 0), 255);
    while (c > 0 && org + code_value(c) * s > (double)x) --c;
    return c;
}
__device__ __forceinline__ int code_up(double org, double s, double inv, float x) {
    const double v = ((double)x - org) * inv;
    int c = v <= 255.0 ? (int)ceil(v) - 128 : (int)ceil(v * 0.5);
    c = min(max(c, 0), 255);
    while (c < 255 && org + code_value(c) * s < (double)x) ++c;
    return c;
}

__global__ void __launch_bounds__(128) k_make_quads(const NodePair* __restrict__ pairs,
                                                    const uint32_t* __restrict__ quad_of, uint32_t n_pairs,
                                                    uint32_t null_prim, QuadNode* __restrict__ quads) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_pairs || quad_of[p] == kNone) return;
    const uint32_t axis_n = quad_of[p] >> kAxisShift;
    constexpr uint32_t kIndex = (1u << kAxisShift) - 1u;
    QuadNode q;
    const ChildRec* kid[4] = {nullptr, nullptr, nullptr, nullptr};
    uint32_t axis[2] = {0, 0};
    for (int h = 0; h < 2; ++h) {
        const ChildRec& c = pairs[p].c[h];
        if (c.b & kLeafBit) {
            kid[2 * h] = &c;
        } else {
            kid[2 * h] = &pairs[c.a].c[0];
            kid[2 * h + 1] = &pairs[c.a].c[1];
            axis[h] = c.b;
        }
    }
    for (int k = 0; k < 4; ++k)
        q.ref[k] = !kid[k] ? (kNode4Leaf | null_prim)
                           : (kid[k]->b & kLeafBit ? (kNode4Leaf | kid[k]->a) : (quad_of[kid[k]->a] & kIndex));
    q.order = 0;
    for (uint32_t oct = 0; oct < 8; ++oct)
        q.order |= (((oct >> axis[0]) & 1u) | (((oct >> axis[1]) & 1u) << 1) | (((oct >> axis_n) & 1u) << 2))
                   << (3 * oct);
    uint32_t low = 0, lo_w[3], hi_w[3];
    float org[3], scale[3];
    for (int i = 0; i < 3; ++i) {
        const int ax = i == 0 ? 1 : (i == 1 ? 0 : 2);  // y first: its scale is the low half of x's
        float lo = 3.402823466e38f, hi = -3.402823466e38f;
        for (int k = 0; k < 4; ++k)
            if (kid[k]) {
                lo = fminf(lo, (&kid[k]->lo_x)[ax]);
                hi = fmaxf(hi, (&kid[k]->hi_x)[ax]);
            }
        fit_axis(lo, hi, ax == 1 ? 1 : (ax == 0 ? 2 : 0), low, &org[ax], &scale[ax]);
        if (ax == 1) low = __float_as_uint(scale[1]) >> 16;
        lo_w[ax] = hi_w[ax] = 0;
        const double inv = 1.0 / (double)scale[ax];
        for (int k = 0; k < 4; ++k) {
            // an empty slot: lower planes above the upper ones
            const int cl = kid[k] ? code_down(org[ax], scale[ax], inv, (&kid[k]->lo_x)[ax]) : 255;
            const int ch = kid[k] ? code_up(org[ax], scale[ax], inv, (&kid[k]->hi_x)[ax]) : 0;
            lo_w[ax] |= (uint32_t)cl << (8 * k);
            hi_w[ax] |= (uint32_t)ch << (8 * k);
        }
    }
    q.org_x = org[0];
    q.org_y = org[1];
    q.org_z = org[2];
    q.sxy = __float_as_uint(scale[0]);
    q.sz = scale[2];
    q.lo_x = lo_w[0];
    q.hi_x = hi_w[0];
    q.lo_y = lo_w[1];
    q.hi_y = hi_w[1];
    q.lo_z = lo_w[2];
    q.hi_z = hi_w[2];
    quads[quad_of[p] & kIndex] = q;
}

}  // namespace

cudaError_t launch_make_quads(const NodePair* d_pairs, const uint32_t* d_quad_of, uint32_t n_pairs, uint32_t null_prim,
                              QuadNode* d_quads, cudaStream_t s) {
    if (!n_pairs) return cudaSuccess;
    k_make_quads<<<(unsigned)((n_pairs + 127u) / 128u), 128, 0, s>>>(d_pairs, d_quad_of, n_pairs, null_prim, d_quads);
    return cudaGetLastError();
}

// ---------------------------------------------- layouts on the device ----
// What fill_host_layout computes, for a tree whose nodes are on the device:
// the host's passes over the nodes were 4.5 of the 11.9 ms that creating and
// first querying a terrain of 180000 triangles took, most of it page faults of
// 20 MB that the device then read once.  One thread per node; the numbers of
// pairs, boxed leaves and 4-wide nodes are their ranks in the nodes' order,
// from counts per block.
namespace {

constexpr uint32_t kLayoutBlock = 256;
constexpr uint32_t kSlotMask = 7u;       // node class: child slots of an inner node's 4-wide node's half (2..4)
constexpr uint32_t kClassBoxed = 0x10u;  // a leaf whose box goes to the table

struct LayoutTotals {
    uint32_t inner, boxed, starts, stack, bad;
    double area, length;  // of the boxes (tree_margins)
};

__device__ __forceinline__ bool usable(const V3& v) {  // false for NaN
    return fabsf(v.x) <= kWideReach && fabsf(v.y) <= kWideReach && fabsf(v.z) <= kWideReach;
}

// Blocks' numbers of inner nodes and boxed leaves (part[0..nb), part[nb..2 nb)),
// their boxes' half areas and edges (sums[0..nb)), every node's class and
// parent, and whether a coordinate is out of reach.
__global__ void __launch_bounds__(kLayoutBlock) k_layout_mark(const FlatNode* __restrict__ nodes, uint32_t m,
                                                              const HostPrim* __restrict__ prims,
                                                              const uint32_t* __restrict__ ordered,
                                                              uint32_t* __restrict__ parent, uint8_t* __restrict__ cls,
                                                              uint32_t* __restrict__ part, uint32_t nb,
                                                              float2* __restrict__ sums, LayoutTotals* totals) {
    __shared__ float2 warps[kLayoutBlock / 32];
    const uint32_t k = blockIdx.x * kLayoutBlock + threadIdx.x;
    bool inner = false, boxed = false, ok = true;
    float area = 0.0f, length = 0.0f;
    if (k < m) {
        const FlatNode& nd = nodes[k];
        const float ex = nd.box.hi.x - nd.box.lo.x, ey = nd.box.hi.y - nd.box.lo.y, ez = nd.box.hi.z - nd.box.lo.z;
        area = ex * ey + ey * ez + ez * ex;
        length = ex + ey + ez;
        if (k == 0) parent[0] = kNone;
        uint32_t c = 0;
        if (!nd.leaf) {
            inner = true;
            parent[k + 1] = k;
            parent[nd.offset] = k;
            c = (nodes[k + 1].leaf ? 1u : 2u) + (nodes[nd.offset].leaf ? 1u : 2u);
        } else {
            ok = usable(nd.box.lo) && usable(nd.box.hi);
            bool tri = false;
            for (uint32_t i = 0; i < nd.count; ++i) {
                const HostPrim& p = prims[ordered[nd.offset + i]];
                tri = p.kind == PBRT_SHAPE_TRIANGLE_MESH;
                if (tri) ok = ok && usable(p.p1) && usable(p.p2) && usable(p.p3);
            }
            boxed = nd.count > 1 || (nd.count == 1 && !tri);
            if (boxed) c = kClassBoxed;
        }
        cls[k] = (uint8_t)c;
    }
    for (uint32_t d = 16; d; d >>= 1) {
        area += __shfl_down_sync(0xffffffffu, area, d);
        length += __shfl_down_sync(0xffffffffu, length, d);
    }
    if ((threadIdx.x & 31u) == 0) warps[threadIdx.x >> 5] = make_float2(area, length);
    const int ni = __syncthreads_count(inner), nx = __syncthreads_count(boxed), nbad = __syncthreads_count(!ok);
    if (threadIdx.x == 0) {
        float2 s = warps[0];
        for (uint32_t w = 1; w < kLayoutBlock / 32; ++w) s = make_float2(s.x + warps[w].x, s.y + warps[w].y);
        sums[blockIdx.x] = s;
        part[blockIdx.x] = (uint32_t)ni;
        part[nb + blockIdx.x] = (uint32_t)nx;
        if (nbad) atomicOr(&totals->bad, 1u);
    }
}

// Which inner nodes start a 4-wide node (those at an even depth), blocks'
// numbers of them (part[2 nb..3 nb)), and the largest number of entries that a
// walk may hold above one: the sum over it and the starts above it of the
// slots but one.  Parents come before their children, so the climb ends.
__global__ void __launch_bounds__(kLayoutBlock) k_layout_starts(const uint32_t* __restrict__ parent, uint32_t m,
                                                                const uint8_t* __restrict__ cls,
                                                                uint8_t* __restrict__ start,
                                                                uint32_t* __restrict__ part, uint32_t nb,
                                                                LayoutTotals* totals) {
    const uint32_t k = blockIdx.x * kLayoutBlock + threadIdx.x;
    bool s = false;
    uint32_t held = 0;
    if (k < m && (cls[k] & kSlotMask)) {
        uint32_t same = 0, other = 0;  // sums over the levels of k's parity and the others
        for (uint32_t a = k; a != kNone; a = parent[a]) {
            same += (cls[a] & kSlotMask) - 1u;
            const uint32_t t = same;
            same = other;
            other = t;
            s = !s;
        }
        held = s ? other : 0u;  // s: k and the root have the same parity, swapped once more than not
    }
    if (k < m) start[k] = s ? 1u : 0u;
    held = __reduce_max_sync(0xffffffffu, held);
    if ((threadIdx.x & 31u) == 0 && held) atomicMax(&totals->stack, held);
    const int ns = __syncthreads_count(s);
    if (threadIdx.x == 0) part[2u * nb + blockIdx.x] = (uint32_t)ns;
}

// The exclusive sums of the three arrays of nb counts, their totals and those
// of the boxes (in a fixed order).
__global__ void __launch_bounds__(1024) k_layout_scan(uint32_t* __restrict__ part, uint32_t nb,
                                                      const float2* __restrict__ sums, LayoutTotals* totals) {
    __shared__ uint32_t warps[32];
    __shared__ double2 box_sums[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t a = 0; a < 3; ++a) {
        uint32_t carry = 0;
        for (uint32_t base = 0; base < nb; base += 1024u) {
            const uint32_t i = base + threadIdx.x;
            const uint32_t v = i < nb ? part[a * nb + i] : 0u;
            uint32_t sum = v;
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += o;
            }
            if (lane == 31) warps[warp] = sum;
            __syncthreads();
            uint32_t before = 0, all = 0;
            for (uint32_t w = 0; w < 32; ++w) {
                if (w < warp) before += warps[w];
                all += warps[w];
            }
            if (i < nb) part[a * nb + i] = carry + before + sum - v;
            carry += all;
            __syncthreads();
        }
        if (threadIdx.x == 0) (a == 0 ? totals->inner : a == 1 ? totals->boxed : totals->starts) = carry;
    }
    double area = 0.0, length = 0.0;
    for (uint32_t i = threadIdx.x; i < nb; i += 1024u) {
        area += (double)sums[i].x;
        length += (double)sums[i].y;
    }
    for (uint32_t d = 16; d; d >>= 1) {
        area += __shfl_down_sync(0xffffffffu, area, d);
        length += __shfl_down_sync(0xffffffffu, length, d);
    }
    if (lane == 0) box_sums[warp] = make_double2(area, length);
    __syncthreads();
    if (threadIdx.x == 0) {
        for (uint32_t w = 1; w < 32; ++w) {
            area += box_sums[w].x;
            length += box_sums[w].y;
        }
        totals->area = area;
        totals->length = length;
    }
}

// The calling thread's rank among the block's threads with `p`.
__device__ __forceinline__ uint32_t block_rank(bool p, uint32_t* warps) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t b = __ballot_sync(0xffffffffu, p);
    __syncthreads();
    if (lane == 0) warps[warp] = (uint32_t)__popc(b);
    __syncthreads();
    uint32_t r = (uint32_t)__popc(b & ((1u << lane) - 1u));
    for (uint32_t w = 0; w < warp; ++w) r += warps[w];
    return r;
}

// rank[k]: an inner node's pair, a boxed leaf's place in the table; quad_of of
// the pairs.
__global__ void __launch_bounds__(kLayoutBlock) k_layout_rank(const FlatNode* __restrict__ nodes, uint32_t m,
                                                              const uint8_t* __restrict__ cls,
                                                              const uint8_t* __restrict__ start,
                                                              const uint32_t* __restrict__ part, uint32_t nb,
                                                              uint32_t* __restrict__ rank,
                                                              uint32_t* __restrict__ quad_of) {
    __shared__ uint32_t warps[kLayoutBlock / 32];
    const uint32_t k = blockIdx.x * kLayoutBlock + threadIdx.x;
    const uint32_t c = k < m ? cls[k] : 0u;
    const bool inner = (c & kSlotMask) != 0, boxed = (c & kClassBoxed) != 0, s = k < m && start[k];
    const uint32_t ri = part[blockIdx.x] + block_rank(inner, warps);
    const uint32_t rb = part[nb + blockIdx.x] + block_rank(boxed, warps);
    const uint32_t rs = part[2u * nb + blockIdx.x] + block_rank(s, warps);
    if (inner) {
        rank[k] = ri;
        quad_of[ri] = s ? rs | (nodes[k].count << kAxisShift) : kNone;
    } else if (boxed) {
        rank[k] = rb;
    }
}

__global__ void __launch_bounds__(kLayoutBlock) k_layout_fill(const FlatNode* __restrict__ nodes, uint32_t m,
                                                              const HostPrim* __restrict__ prims,
                                                              const SphereRec* __restrict__ spheres,
                                                              const uint32_t* __restrict__ flat_id,
                                                              const uint32_t* __restrict__ ordered, uint32_t n,
                                                              const uint8_t* __restrict__ cls,
                                                              const uint32_t* __restrict__ rank,
                                                              NodePair* __restrict__ pairs, PrimRec* __restrict__ recs,
                                                              LeafBox* __restrict__ boxes) {
    const uint32_t k = blockIdx.x * kLayoutBlock + threadIdx.x;
    auto store = [&](uint32_t at, float4 r0, float4 r1, float4 r2) {
        float4* out = reinterpret_cast<float4*>(recs + at);
        out[0] = r0;
        out[1] = r1;
        out[2] = r2;
    };
    if (k == 0) store(n, make_float4(0, 0, 0, 0), make_float4(0, 0, 0, 0),
                      make_float4(0, 0, 0, __uint_as_float(kPrimLastBit)));  // the null record
    if (k >= m) return;
    const FlatNode nd = nodes[k];
    if (!nd.leaf) {
        float4* out = reinterpret_cast<float4*>(pairs + rank[k]);
        for (int h = 0; h < 2; ++h) {
            const uint32_t kid = h ? nd.offset : k + 1;
            const FlatNode c = nodes[kid];
            const uint32_t a = c.leaf ? c.offset : rank[kid], b = c.leaf ? kLeafBit | c.count : c.count;
            out[2 * h] = make_float4(c.box.lo.x, c.box.lo.y, c.box.lo.z, __uint_as_float(a));
            out[2 * h + 1] = make_float4(c.box.hi.x, c.box.hi.y, c.box.hi.z, __uint_as_float(b));
        }
        return;
    }
    for (uint32_t i = 0; i < nd.count; ++i) {
        const uint32_t ref = ordered[nd.offset + i];
        const HostPrim& p = prims[ref];
        uint32_t id = flat_id ? flat_id[ref] : ref, flags = i + 1 == nd.count ? kPrimLastBit : 0u;
        const bool tri = p.kind == PBRT_SHAPE_TRIANGLE_MESH;
        if (cls[k] & kClassBoxed) flags |= rank[k] << kPrimBoxShift;
        if (i == 0 && (cls[k] & kClassBoxed)) {
            const bool entry = nd.count > 1 || spheres[p.sphere].kind == kQuadInstance;
            flags |= entry ? kPrimBoxEntry : kPrimHitBox;
            float4* out = reinterpret_cast<float4*>(boxes + rank[k]);
            out[0] = make_float4(nd.box.lo.x, nd.box.lo.y, nd.box.lo.z, 0.0f);
            out[1] = make_float4(nd.box.hi.x, nd.box.hi.y, nd.box.hi.z, 0.0f);
        } else if (i == 0) {
            flags |= kPrimOwnBox;
        }
        if (tri)
            store(nd.offset + i, make_float4(p.p1.x, p.p1.y, p.p1.z, __uint_as_float(id)),
                  make_float4(p.p2.x, p.p2.y, p.p2.z, 0.0f),
                  make_float4(p.p3.x, p.p3.y, p.p3.z, __uint_as_float(flags)));
        else
            store(nd.offset + i, make_float4(0, 0, 0, __uint_as_float(id | kSphereBit)),
                  make_float4(0, 0, 0, __uint_as_float((uint32_t)p.sphere)),
                  make_float4(0, 0, 0, __uint_as_float(flags)));
    }
}

}  // namespace

DeviceLayout::~DeviceLayout() {
    for (void* p : {(void*)pairs, (void*)prims, (void*)boxes, (void*)quads})
        if (p) cudaFree(p);
}

void device_fill_layout(HostBVH& H, const FlatNode* d_nodes, uint32_t m, const uint32_t* d_ordered,
                        const HostPrim* d_prims) {
    const size_t n = H.ordered.size();
    const uint32_t nb = (m + kLayoutBlock - 1) / kLayoutBlock;
    const size_t n_pairs = (m - 1) / 2;
    auto L = std::make_shared<DeviceLayout>();
    // the workspace, one allocation
    size_t bytes = 0;
    auto take = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) & ~(size_t)255;
        return at;
    };
    const size_t o_tot = take(sizeof(LayoutTotals)), o_prims = take(d_prims ? 0 : n * sizeof(HostPrim)),
                 o_sph = take(H.spheres.size() * sizeof(SphereRec)), o_flat = take(H.flat_id.size() * 4),
                 o_parent = take((size_t)m * 4), o_rank = take((size_t)m * 4), o_cls = take(m), o_start = take(m),
                 o_part = take((size_t)nb * 12), o_quad = take(n_pairs * 4), o_sums = take((size_t)nb * sizeof(float2));
    char* ws = nullptr;
    struct Free {
        char*& p;
        ~Free() {
            if (p) cudaFree(p);
        }
    } free_ws{ws};
    auto fits = [](cudaError_t e) {  // false: the caller fills the layout on the host
        if (e == cudaSuccess) return true;
        (void)cudaGetLastError();
        return false;
    };
    if (!fits(cudaGetDevice(&L->device)) || !fits(cudaMalloc((void**)&ws, bytes)) ||
        !fits(cudaMalloc((void**)&L->prims, (n + 1) * sizeof(PrimRec))) ||
        (n_pairs && !fits(cudaMalloc((void**)&L->pairs, n_pairs * sizeof(NodePair)))))
        return;
    auto* totals = reinterpret_cast<LayoutTotals*>(ws + o_tot);
    const HostPrim* prims = d_prims ? d_prims : reinterpret_cast<HostPrim*>(ws + o_prims);
    auto* spheres = reinterpret_cast<SphereRec*>(ws + o_sph);
    auto* flat = H.flat_id.empty() ? nullptr : reinterpret_cast<uint32_t*>(ws + o_flat);
    auto* parent = reinterpret_cast<uint32_t*>(ws + o_parent);
    auto* rank = reinterpret_cast<uint32_t*>(ws + o_rank);
    auto* cls = reinterpret_cast<uint8_t*>(ws + o_cls);
    auto* start = reinterpret_cast<uint8_t*>(ws + o_start);
    auto* part = reinterpret_cast<uint32_t*>(ws + o_part);
    auto* quad_of = reinterpret_cast<uint32_t*>(ws + o_quad);
    auto* sums = reinterpret_cast<float2*>(ws + o_sums);
    if (!fits(cudaMemsetAsync(totals, 0, sizeof(LayoutTotals), 0)) ||
        (!d_prims && !fits(cudaMemcpy(ws + o_prims, H.prims.data(), n * sizeof(HostPrim), cudaMemcpyHostToDevice))) ||
        (!H.spheres.empty() && !fits(cudaMemcpy(spheres, H.spheres.data(), H.spheres.size() * sizeof(SphereRec),
                                                cudaMemcpyHostToDevice))) ||
        (flat && !fits(cudaMemcpy(flat, H.flat_id.data(), H.flat_id.size() * 4, cudaMemcpyHostToDevice))))
        return;
    k_layout_mark<<<nb, kLayoutBlock>>>(d_nodes, m, prims, d_ordered, parent, cls, part, nb, sums, totals);
    k_layout_starts<<<nb, kLayoutBlock>>>(parent, m, cls, start, part, nb, totals);
    k_layout_scan<<<1, 1024>>>(part, nb, sums, totals);
    k_layout_rank<<<nb, kLayoutBlock>>>(d_nodes, m, cls, start, part, nb, rank, quad_of);
    LayoutTotals T;
    if (!fits(cudaGetLastError()) || !fits(cudaMemcpy(&T, totals, sizeof(T), cudaMemcpyDeviceToHost))) return;
    if (T.inner != n_pairs || T.boxed >= (1u << (32u - kPrimBoxShift)) ||
        (T.boxed && !fits(cudaMalloc((void**)&L->boxes, T.boxed * sizeof(LeafBox)))))
        return;
    k_layout_fill<<<nb, kLayoutBlock>>>(d_nodes, m, prims, spheres, flat, d_ordered, (uint32_t)n, cls, rank, L->pairs,
                                        L->prims, L->boxes);
    const bool wide = !T.bad && n < 0x7ffffff0u && n_pairs < (1u << kQuadAxisShift);
    if (wide && T.starts &&
        (!fits(cudaMalloc((void**)&L->quads, T.starts * sizeof(QuadNode))) ||
         !fits(launch_make_quads(L->pairs, quad_of, (uint32_t)n_pairs, (uint32_t)n, L->quads, 0))))
        return;
    if (!fits(cudaGetLastError()) || !fits(cudaStreamSynchronize(0))) return;
    const FlatNode& root = H.nodes[0];
    H.root = ChildRec{root.box.lo.x, root.box.lo.y, root.box.lo.z, root.leaf ? root.offset : 0u,
                      root.box.hi.x, root.box.hi.y, root.box.hi.z, root.leaf ? kLeafBit | root.count : root.count};
    L->n_pairs = n_pairs;
    L->n_boxes = T.boxed;
    H.wide = wide;
    H.n_quads = T.starts;
    H.stack4_bound = T.stack;
    tree_margins(H, T.area, T.length);
    H.layout = std::move(L);
}

}  // namespace pbrt
