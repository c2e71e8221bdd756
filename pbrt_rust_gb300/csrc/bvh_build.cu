// bvh_build.cu - BVHAccelerator::new's tree built on the device.
//
// The same tree as the host restatement (host_scene.cpp build_tree, itself
// the reference's recursive_build, src/primitive/aggregates/bvh.rs:86-258):
// the same nodes, bounds, split axes and primitive order, bit for bit.  The
// recursion becomes two phases over one array of primitive indices, every
// node owning a contiguous range of it:
//
//   A. ranges above kSmall (32) primitives, one tree level per round: every range
//      of the level is cut into chunks; chunk kernels reduce its bounds and
//      centroid bounds, fill the twelve SAH buckets (or test the middle
//      split) and count the left side, one thread per range picks the split,
//      and a stable scatter writes the two sides in their original order
//      (Iterator::partition keeps order, bvh.rs:89, 174).  The host reads the
//      per-range decisions back, once per level, and lays out the next.
//   B. ranges of at most kSmall primitives: one warp runs the whole subtree,
//      one primitive per lane, with the host algorithm (including
//      partition_by for the equal-counts split of ranges of up to four,
//      utils/mod.rs:112-169), writing its nodes in pre-order.
//
// Bounds are combined with a min/max that ignores NaN and orders -0 below
// +0, in any order; f32 bucket indices and SAH costs repeat the host's
// operations (--fmad=false).  The nodes are then numbered in the reference's
// depth-first order (k_number), and the tree's layout is made from there
// (quads.cu: device_fill_layout).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/pbrt_gpu.h"
#include "host_scene.h"

namespace pbrt {

namespace {

constexpr uint32_t kSmall = 32;   // ranges of at most this many primitives go to phase B (a lane each)
constexpr uint32_t kChunk = 2048; // phase A chunk
constexpr int kNB = 12;           // SAH buckets (bvh.rs:188)

// ---- order-independent min / max ------------------------------------------
// Floats as ints whose signed order is the float order with -0 < +0.
__host__ __device__ inline int32_t ord(float f) {
    int32_t i;
    memcpy(&i, &f, 4);
    return i >= 0 ? i : (int32_t)(i ^ 0x7fffffff);
}
__host__ __device__ inline float unord(int32_t i) {
    int32_t b = i >= 0 ? i : (int32_t)(i ^ 0x7fffffff);
    float f;
    memcpy(&f, &b, 4);
    return f;
}
__device__ inline float dmin(float a, float b) {  // std::fmin, -0 below +0
    if (a != a) return b;
    if (b != b) return a;
    return ord(a) <= ord(b) ? a : b;
}
__device__ inline float dmax(float a, float b) {
    if (a != a) return b;
    if (b != b) return a;
    return ord(a) >= ord(b) ? a : b;
}

struct DBox {
    float lx, ly, lz, hx, hy, hz;
};
__device__ inline DBox dbox_empty() { return DBox{FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX}; }
__device__ inline DBox dunion(const DBox& a, const DBox& b) {
    return DBox{dmin(a.lx, b.lx), dmin(a.ly, b.ly), dmin(a.lz, b.lz),
                dmax(a.hx, b.hx), dmax(a.hy, b.hy), dmax(a.hz, b.hz)};
}
__device__ inline float darea(const DBox& b) {  // bbox.rs:73-78
    float dx = fmaxf(b.hx - b.lx, 0.0f), dy = fmaxf(b.hy - b.ly, 0.0f), dz = fmaxf(b.hz - b.lz, 0.0f);
    return 2.0f * (dx * dy + dx * dz + dy * dz);
}
__device__ inline int dmax_extent(const DBox& b) {  // bbox.rs:87-96
    float dx = b.hx - b.lx, dy = b.hy - b.ly, dz = b.hz - b.lz;
    if (dx > dy && dx > dz) return 0;
    if (dy > dz) return 1;
    return 2;
}
__device__ inline size_t to_usize(float f) {  // Rust `as usize`: saturating, NaN -> 0
    if (!(f > 0.0f)) return 0;
    if (f >= 18446744073709551615.0f) return (size_t)-1;
    return (size_t)f;
}
__device__ inline int bucket_of(float key, float cmin, float dist) {  // bvh.rs:118-131
    size_t b = to_usize((float)kNB * ((key - cmin) / dist));
    // key lies in [cmin, cmin + dist], so b <= kNB; the clamp only guards
    return b >= (size_t)kNB ? kNB - 1 : (int)b;
}

struct Prims {
    const float4* lo;   // bounds
    const float4* hi;
    const float* cen[3];  // centroids by axis
};
__device__ inline DBox pbox(const Prims& P, uint32_t p) {
    float4 a = __ldg(P.lo + p), b = __ldg(P.hi + p);
    return DBox{a.x, a.y, a.z, b.x, b.y, b.z};
}

// ---- phase A ---------------------------------------------------------------
struct Chunk {  // a range's piece; as a range's record: first chunk, lo, count, chunks
    uint32_t seg, lo, hi, pad;
};
// Per range: [0..5] bounds, [6..11] centroid bounds (ord ints, min fields
// stored as is, max fields too), then 12 buckets of count + 6 bounds.
constexpr int kAccWords = 12 + kNB * 7;

struct SegDecision {   // filled by k_decide / k_choose
    float cmin, dist, pmid;
    int32_t dim;
    int32_t action;    // 0 leaf, 1 split by bucket <= best, 2 split by key < pmid
    int32_t best;
    float lo[3], hi[3];  // range bounds
    uint32_t n_left;   // k_a_base: primitives that go left
};

__global__ void k_acc_init(int32_t* acc, uint32_t nseg) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nseg * kAccWords) return;
    const uint32_t w = i % kAccWords;
    int f;  // min fields start at +FLT_MAX, max fields at -FLT_MAX, counts at 0
    if (w < 12) {
        f = (w % 6) < 3 ? ord(FLT_MAX) : ord(-FLT_MAX);
    } else {
        const uint32_t k = (w - 12) % 7;
        f = k == 0 ? 0 : (k <= 3 ? ord(FLT_MAX) : ord(-FLT_MAX));
    }
    acc[i] = f;
}

__device__ inline void warp_min_to(int32_t v, int32_t* dst) {
    for (int o = 16; o; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) atomicMin(dst, v);
}
__device__ inline void warp_max_to(int32_t v, int32_t* dst) {
    for (int o = 16; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) atomicMax(dst, v);
}

// Bounds and centroid bounds of each range (NaN-free inputs: the int order
// then is the float order of dmin / dmax).
__global__ void __launch_bounds__(256) k_a_bounds(Prims P, const uint32_t* __restrict__ idx,
                                                  const Chunk* __restrict__ chunks, int32_t* acc) {
    const Chunk c = chunks[blockIdx.x];
    int32_t m[12];
    for (int k = 0; k < 12; ++k) m[k] = (k % 6) < 3 ? ord(FLT_MAX) : ord(-FLT_MAX);
    for (uint32_t i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) {
        const uint32_t p = __ldg(idx + i);
        const DBox b = pbox(P, p);
        const float cx = __ldg(P.cen[0] + p), cy = __ldg(P.cen[1] + p), cz = __ldg(P.cen[2] + p);
        m[0] = min(m[0], ord(b.lx)), m[1] = min(m[1], ord(b.ly)), m[2] = min(m[2], ord(b.lz));
        m[3] = max(m[3], ord(b.hx)), m[4] = max(m[4], ord(b.hy)), m[5] = max(m[5], ord(b.hz));
        m[6] = min(m[6], ord(cx)), m[7] = min(m[7], ord(cy)), m[8] = min(m[8], ord(cz));
        m[9] = max(m[9], ord(cx)), m[10] = max(m[10], ord(cy)), m[11] = max(m[11], ord(cz));
    }
    int32_t* a = acc + (size_t)c.seg * kAccWords;
    for (int k = 0; k < 12; ++k) {
        if ((k % 6) < 3)
            warp_min_to(m[k], a + k);
        else
            warp_max_to(m[k], a + k);
    }
}

// One thread per range: split axis and centroid extent (bvh.rs:208-217).
__global__ void k_a_decide(const int32_t* __restrict__ acc, SegDecision* dec, const Chunk* __restrict__ ranges,
                           uint32_t nseg, int split) {
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    const int32_t* a = acc + (size_t)s * kAccWords;
    DBox cb{unord(a[6]), unord(a[7]), unord(a[8]), unord(a[9]), unord(a[10]), unord(a[11])};
    SegDecision d;
    for (int k = 0; k < 3; ++k) {
        d.lo[k] = unord(a[k]);
        d.hi[k] = unord(a[3 + k]);
    }
    d.dim = dmax_extent(cb);
    const float cmin = d.dim == 0 ? cb.lx : (d.dim == 1 ? cb.ly : cb.lz);
    const float cmax = d.dim == 0 ? cb.hx : (d.dim == 1 ? cb.hy : cb.hz);
    d.cmin = cmin;
    d.dist = cmax - cmin;
    d.pmid = 0.5f * (cmin + cmax);
    d.best = 0;
    if (ranges[s].hi <= 1 || cmin == cmax)
        d.action = 0;
    else
        d.action = split == PBRT_SPLIT_MIDDLE ? 2 : 1;
    dec[s] = d;
}

// SAH buckets of each range.
__global__ void __launch_bounds__(256) k_a_buckets(Prims P, const uint32_t* __restrict__ idx,
                                                   const Chunk* __restrict__ chunks,
                                                   const SegDecision* __restrict__ dec, int32_t* acc) {
    __shared__ int32_t sb[kNB * 7];
    const Chunk c = chunks[blockIdx.x];
    const SegDecision d = dec[c.seg];
    if (d.action != 1) return;
    for (int i = threadIdx.x; i < kNB * 7; i += blockDim.x) {
        const int k = i % 7;
        sb[i] = k == 0 ? 0 : (k <= 3 ? ord(FLT_MAX) : ord(-FLT_MAX));
    }
    __syncthreads();
    const float* key = d.dim == 0 ? P.cen[0] : (d.dim == 1 ? P.cen[1] : P.cen[2]);
    for (uint32_t i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) {
        const uint32_t p = __ldg(idx + i);
        const int b = bucket_of(__ldg(key + p), d.cmin, d.dist);
        const DBox bx = pbox(P, p);
        int32_t* q = sb + b * 7;
        atomicAdd(q, 1);
        atomicMin(q + 1, ord(bx.lx)), atomicMin(q + 2, ord(bx.ly)), atomicMin(q + 3, ord(bx.lz));
        atomicMax(q + 4, ord(bx.hx)), atomicMax(q + 5, ord(bx.hy)), atomicMax(q + 6, ord(bx.hz));
    }
    __syncthreads();
    int32_t* a = acc + (size_t)c.seg * kAccWords + 12;
    for (int i = threadIdx.x; i < kNB * 7; i += blockDim.x) {
        const int k = i % 7;
        if (k == 0)
            atomicAdd(a + i, sb[i]);
        else if (k <= 3)
            atomicMin(a + i, sb[i]);
        else
            atomicMax(a + i, sb[i]);
    }
}

// The cheapest of the eleven splits and its cost (bvh.rs:133-160): the first
// whose cost is below every earlier one's and FLT_MAX.  The boxes of the left
// sides grow bucket by bucket and those of the right sides come from a
// backward pass; unions do not depend on their order (dmin / dmax), so the
// costs are those of the host's loop over all buckets per split.
__device__ inline int cheapest_split(const DBox* bb, const uint32_t* bc, float tsa, float* cost_out) {
    DBox right[kNB];  // union of buckets j ..
    uint32_t n_right[kNB];
    DBox u = dbox_empty();
    uint32_t n = 0;
#pragma unroll
    for (int j = kNB - 1; j > 0; --j) {
        u = dunion(u, bb[j]);
        n += bc[j];
        right[j] = u;
        n_right[j] = n;
    }
    int best = 0;
    float best_cost = FLT_MAX;
    u = dbox_empty();
    n = 0;
#pragma unroll
    for (int sp = 0; sp + 1 < kNB; ++sp) {
        u = dunion(u, bb[sp]);
        n += bc[sp];
        const float cost =
            0.125f * ((float)n * darea(u) + (float)n_right[sp + 1] * darea(right[sp + 1])) / tsa;
        if (cost < best_cost) {
            best_cost = cost;
            best = sp;
        }
    }
    *cost_out = best_cost;
    return best;
}

// One thread per range: the SAH costs in the host's order and the leaf test
// (bvh.rs:133-185).
__global__ void __launch_bounds__(32) k_a_choose(const int32_t* __restrict__ acc, SegDecision* dec,
                                                 const Chunk* __restrict__ ranges, uint32_t nseg, uint32_t mp) {
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    SegDecision d = dec[s];
    if (d.action != 1) return;
    const int32_t* a = acc + (size_t)s * kAccWords + 12;
    uint32_t bc[kNB];
    DBox bb[kNB];
#pragma unroll
    for (int i = 0; i < kNB; ++i) {
        const int32_t* q = a + i * 7;
        bc[i] = (uint32_t)q[0];
        bb[i] = DBox{unord(q[1]), unord(q[2]), unord(q[3]), unord(q[4]), unord(q[5]), unord(q[6])};
    }
    DBox total{d.lo[0], d.lo[1], d.lo[2], d.hi[0], d.hi[1], d.hi[2]};
    float best_cost;
    d.best = cheapest_split(bb, bc, darea(total), &best_cost);
    const size_t cnt = ranges[s].hi;
    if (!(mp < cnt || to_usize(best_cost) < cnt)) d.action = 0;  // a leaf of cnt primitives
    dec[s] = d;
}

__device__ inline bool goes_left(const Prims& P, const SegDecision& d, uint32_t p) {
    const float* key = d.dim == 0 ? P.cen[0] : (d.dim == 1 ? P.cen[1] : P.cen[2]);
    const float k = __ldg(key + p);
    if (d.action == 2) return k < d.pmid;
    return bucket_of(k, d.cmin, d.dist) <= d.best;
}

// Left-side count of every chunk.
__global__ void __launch_bounds__(256) k_a_count(Prims P, const uint32_t* __restrict__ idx,
                                                 const Chunk* __restrict__ chunks,
                                                 const SegDecision* __restrict__ dec, uint32_t* left) {
    const Chunk c = chunks[blockIdx.x];
    const SegDecision d = dec[c.seg];
    uint32_t n = 0;
    if (d.action != 0)
        for (uint32_t i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) n += goes_left(P, d, __ldg(idx + i));
    for (int o = 16; o; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    __shared__ uint32_t ws[8];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
        left[blockIdx.x] = t;
    }
}

// A range's left total and where each of its chunks' sides go (a leaf's
// chunks stay), one warp per range.  On the host this was a download, a pass
// and an upload in the middle of every level.
__global__ void __launch_bounds__(128) k_a_base(const Chunk* __restrict__ chunks, const Chunk* __restrict__ ranges,
                                                uint32_t nseg, const uint32_t* __restrict__ left, SegDecision* dec,
                                                uint2* __restrict__ base) {
    const uint32_t s = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (s >= nseg) return;  // the whole warp
    const Chunk r = ranges[s];
    const uint32_t first = r.seg, lo = r.lo, cnt = r.hi, nc = r.pad;
    const bool split = dec[s].action != 0;
    uint32_t total = 0;
    for (uint32_t c = lane; c < nc; c += 32u) total += left[first + c];
    total = __reduce_add_sync(0xffffffffu, total);
    const uint32_t mid = split ? lo + total : lo + cnt;
    uint32_t run = 0;  // left ones before these chunks
    for (uint32_t c0 = 0; c0 < nc; c0 += 32u) {
        const uint32_t c = c0 + lane;
        const Chunk k = c < nc ? chunks[first + c] : Chunk{0, 0, 0, 0};
        const uint32_t nl = c < nc ? (split ? left[first + c] : k.hi - k.lo) : 0u;
        uint32_t sum = nl;
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, sum, d);
            if (lane >= d) sum += o;
        }
        const uint32_t before = run + sum - nl;
        if (c < nc) base[first + c] = make_uint2(lo + before, mid + (k.lo - lo) - before);
        run += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) dec[s].n_left = total;
}

// Stable two-way scatter of every chunk: left side to base_left + rank,
// right side to base_right + rank, in index order.
__global__ void __launch_bounds__(256) k_a_scatter(Prims P, const uint32_t* __restrict__ idx, uint32_t* out,
                                                   const Chunk* __restrict__ chunks,
                                                   const SegDecision* __restrict__ dec,
                                                   const uint2* __restrict__ base) {
    __shared__ uint32_t ws[8];
    __shared__ uint32_t carry;  // left elements of the chunk before this round
    const Chunk c = chunks[blockIdx.x];
    const SegDecision d = dec[c.seg];
    const uint2 b = base[blockIdx.x];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t i0 = c.lo; i0 < c.hi; i0 += blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        const bool live = i < c.hi;
        const uint32_t p = live ? idx[i] : 0u;
        const bool left = live && (d.action == 0 || goes_left(P, d, p));  // leaves keep their order
        const unsigned m = __ballot_sync(0xffffffffu, left);
        if (lane == 0) ws[w] = __popc(m);
        __syncthreads();
        uint32_t before = 0, total = 0;
        for (unsigned k = 0; k < nw; ++k) {
            if (k < w) before += ws[k];
            total += ws[k];
        }
        // left elements before this one in the chunk, and right ones
        const uint32_t rank_l = carry + before + __popc(m & ((1u << lane) - 1u));
        const uint32_t rank_r = (i - c.lo) - rank_l;
        if (live) out[left ? b.x + rank_l : b.y + rank_r] = p;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
}

__global__ void k_copy_ranges(const uint32_t* __restrict__ src, uint32_t* dst, const Chunk* __restrict__ chunks) {
    const Chunk c = chunks[blockIdx.x];
    for (uint32_t i = c.lo + threadIdx.x; i < c.hi; i += blockDim.x) dst[i] = src[i];
}

// ---- phase B ---------------------------------------------------------------
struct Job {
    uint32_t lo, hi;   // primitive range
    uint32_t node0;    // first node slot in the pool
    uint32_t pad;
};
struct PoolNode {      // a = leaf ? first prim : second child (pool index); b = leaf ? kLeaf | count : axis
    float lo[3];
    uint32_t a;
    float hi[3];
    uint32_t b;
};
constexpr uint32_t kLeaf = 0x80000000u;
struct JobOut {
    uint32_t nodes, depth, err, pad;
};

// utils/mod.rs:112-169 (as host_scene.cpp partition_by_key)
__device__ void partition_by_key(uint8_t* v, uint32_t n, const float* key) {
    while (true) {
        if (n < 3) {
            if (n == 2 && key[v[1]] < key[v[0]]) {
                uint8_t t = v[0];
                v[0] = v[1];
                v[1] = t;
            }
            return;
        }
        float a = key[v[0]], b = key[v[n / 2]], c = key[v[n - 1]];
        float pivot = (a < b && b < c) ? b : ((b < a && a < c) ? a : c);
        uint32_t ls = 0, np = 0;
        for (uint32_t i = 0; i < n; ++i) {
            float k = key[v[i]];
            if (k < pivot) {
                uint8_t t = v[ls + np];
                v[ls + np] = v[i];
                v[i] = t;
                t = v[ls + np];
                v[ls + np] = v[ls];
                v[ls] = t;
                ++ls;
            } else if (k == pivot) {
                uint8_t t = v[ls + np];
                v[ls + np] = v[i];
                v[i] = t;
                ++np;
            }
        }
        uint32_t pi = ls > 1 ? ls : 1;
        if (pi + np <= n / 2) {
            v += pi;
            n -= pi;
        } else if (pi >= n / 2) {
            n = pi;
        } else {
            return;
        }
    }
}

// One warp per job: build_tree on [lo, hi) (host_scene.cpp), nodes in
// pre-order at pool[node0 ...], the range's primitive order in idx.  The
// range's boxes and centroids sit in shared memory, one slot per primitive;
// a lane holds the slot at its position of the range.  A node's bounds are
// warp reductions over the lanes of its sub-range (an inner node's box is the
// union of its children's, bvh.rs:247, which is the union of its primitives'
// boxes whatever the order), the twelve buckets are filled with shared-memory
// atomics and their eleven splits costed one per lane, and a split moves
// the slots by rank, which keeps their order.  As one thread per range, whose
// lanes diverge at every node, 180000 terrain triangles took 2.40 ms here.
constexpr int kBWarps = 4;
struct BScratch {
    float box[6][kSmall], cen[3][kSmall];  // by slot
    uint8_t order[kSmall];                 // slot at each position of the range
    int32_t bucket[kNB][7];                // count, bounds (ord)
    uint4 stack[kSmall];                   // (lo, hi, parent or ~0, depth)
};
__global__ void __launch_bounds__(32 * kBWarps) k_b_build(Prims P, uint32_t* idx, const Job* __restrict__ jobs,
                                                         uint32_t njobs, PoolNode* pool, JobOut* outs, uint32_t mp,
                                                         int split) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ BScratch scratch[kBWarps];
    BScratch& S = scratch[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t j = blockIdx.x * kBWarps + (threadIdx.x >> 5);
    if (j >= njobs) return;
    const Job J = jobs[j];
    const uint32_t n = J.hi - J.lo;
    uint32_t prim = 0;  // of slot `lane`
    if (lane < n) {
        prim = idx[J.lo + lane];
        const DBox b = pbox(P, prim);
        S.box[0][lane] = b.lx, S.box[1][lane] = b.ly, S.box[2][lane] = b.lz;
        S.box[3][lane] = b.hx, S.box[4][lane] = b.hy, S.box[5][lane] = b.hz;
        for (int k = 0; k < 3; ++k) S.cen[k][lane] = __ldg(P.cen[k] + prim);
    }
    uint32_t slot = lane;  // at this lane's position
    uint32_t sp = 1, nn = 0, maxd = 0, err = 0;  // warp-uniform
    if (lane == 0) S.stack[0] = make_uint4(0, n, kAll, 1);
    __syncwarp();
    const int32_t lowest = ord(FLT_MAX), highest = ord(-FLT_MAX);  // of an empty box
    // ord of a bound that takes part; NaNs and other lanes leave it alone
    auto part = [](bool in, float v, int32_t none) { return in && v == v ? ord(v) : none; };
    while (sp > 0) {
        const uint4 t = S.stack[--sp];
        const uint32_t k = nn++, cnt = t.y - t.x;
        const bool in = lane >= t.x && lane < t.y;
        __syncwarp();
        if (lane == 0 && t.z != kAll) pool[J.node0 + t.z].a = k;
        maxd = max(maxd, t.w);
        float box[6], cen[3];
        int32_t m[6], c[6];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            box[i] = S.box[i][slot];
            box[3 + i] = S.box[3 + i][slot];
            cen[i] = S.cen[i][slot];
            m[i] = min(lowest, __reduce_min_sync(kAll, part(in, box[i], lowest)));
            m[3 + i] = max(highest, __reduce_max_sync(kAll, part(in, box[3 + i], highest)));
            c[i] = min(lowest, __reduce_min_sync(kAll, part(in, cen[i], lowest)));
            c[3 + i] = max(highest, __reduce_max_sync(kAll, part(in, cen[i], highest)));
        }
        uint32_t mid = 0;
        bool split_it = false;
        int dim = 0;
        if (cnt > 1) {
            dim = dmax_extent(DBox{unord(c[0]), unord(c[1]), unord(c[2]), unord(c[3]), unord(c[4]), unord(c[5])});
            const float cmin = unord(dim == 0 ? c[0] : (dim == 1 ? c[1] : c[2]));
            const float cmax = unord(dim == 0 ? c[3] : (dim == 1 ? c[4] : c[5]));
            const float key = dim == 0 ? cen[0] : (dim == 1 ? cen[1] : cen[2]);
            bool left = false;  // a stable split sends this lane's primitive left
            bool stable = false;
            if (cmin != cmax) {
                if (split == PBRT_SPLIT_MIDDLE) {
                    left = key < 0.5f * (cmin + cmax);
                    stable = true;
                } else if (split == PBRT_SPLIT_EQUAL || cnt <= 4) {
                    S.order[lane] = (uint8_t)slot;
                    __syncwarp();
                    if (lane == 0) partition_by_key(S.order + t.x, cnt, S.cen[dim]);
                    __syncwarp();
                    slot = S.order[lane];
                    mid = t.x + cnt / 2;
                    split_it = true;
                } else {
                    for (uint32_t i = lane; i < kNB * 7; i += 32u)
                        (&S.bucket[0][0])[i] = i % 7u == 0u ? 0 : (i % 7u <= 3u ? lowest : highest);
                    __syncwarp();
                    const float dist = cmax - cmin;
                    int b = 0;
                    if (in) {
                        b = bucket_of(key, cmin, dist);
                        int32_t* q = S.bucket[b];
                        atomicAdd(q, 1);
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            atomicMin(q + 1 + i, part(true, box[i], lowest));
                            atomicMax(q + 4 + i, part(true, box[3 + i], highest));
                        }
                    }
                    __syncwarp();
                    // lane s < 11: the cost of the split after bucket s
                    float cost = FLT_MAX;
                    if (lane + 1u < (uint32_t)kNB) {
                        DBox u0 = dbox_empty(), u1 = dbox_empty();
                        uint32_t n0 = 0;
                        for (uint32_t q = 0; q < (uint32_t)kNB; ++q) {
                            const int32_t* e = S.bucket[q];
                            const DBox bq{unord(e[1]), unord(e[2]), unord(e[3]), unord(e[4]), unord(e[5]), unord(e[6])};
                            if (q <= lane) {
                                n0 += (uint32_t)e[0];
                                u0 = dunion(u0, bq);
                            } else {
                                u1 = dunion(u1, bq);
                            }
                        }
                        const float tsa = darea(DBox{unord(m[0]), unord(m[1]), unord(m[2]), unord(m[3]), unord(m[4]),
                                                     unord(m[5])});
                        cost = 0.125f * ((float)n0 * darea(u0) + (float)(cnt - n0) * darea(u1)) / tsa;
                        if (!(cost < FLT_MAX)) cost = FLT_MAX;  // also NaN: never below the best
                    }
                    const int32_t lo_cost = __reduce_min_sync(kAll, ord(cost));
                    const float best_cost = unord(lo_cost);
                    const int best = best_cost < FLT_MAX ? __ffs(__ballot_sync(kAll, ord(cost) == lo_cost)) - 1 : 0;
                    if (mp < cnt || to_usize(best_cost) < cnt) {
                        left = b <= best;
                        stable = true;
                    }
                }
            }
            if (stable) {
                const unsigned ml = __ballot_sync(kAll, in && left), below = (1u << lane) - 1u;
                const uint32_t nl = (uint32_t)__popc(ml);
                if (in) {
                    const uint32_t rank = (uint32_t)__popc(ml & below);
                    S.order[left ? t.x + rank : t.x + nl + (lane - t.x - rank)] = (uint8_t)slot;
                }
                __syncwarp();
                if (in) slot = S.order[lane];
                mid = t.x + nl;
                split_it = true;
            }
        }
        if (split_it && (mid == t.x || mid == t.y)) err = 1;
        __syncwarp();
        if (lane == 0) {
            PoolNode& N = pool[J.node0 + k];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                N.lo[i] = unord(m[i]);
                N.hi[i] = unord(m[3 + i]);
            }
            N.a = split_it ? 0u : J.lo + t.x;
            N.b = split_it ? (uint32_t)dim : (kLeaf | cnt);
            if (split_it) {
                S.stack[sp] = make_uint4(mid, t.y, k, t.w + 1);
                S.stack[sp + 1] = make_uint4(t.x, mid, kAll, t.w + 1);
            }
        }
        __syncwarp();
        if (err) break;
        if (split_it) sp += 2;
    }
    const uint32_t p = __shfl_sync(kAll, prim, (int)(slot & 31u));
    if (lane < n) idx[J.lo + lane] = p;
    if (lane == 0) outs[j] = JobOut{nn, maxd, err, 0};
}

// ---- host ------------------------------------------------------------------
struct Buf {  // a device allocation owned by the build
    void* p = nullptr;
    size_t cap = 0;
    Buf() = default;
    Buf(const Buf&) = delete;
    Buf& operator=(const Buf&) = delete;
    ~Buf() { reset(); }
    void reset() {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    }
    // At least `bytes`, contents not kept.  Grown ahead of the need: the
    // levels' buffers double from level to level, and an allocation and its
    // release synchronise the device.
    cudaError_t reserve(size_t bytes) {
        if (bytes <= cap) return cudaSuccess;
        reset();
        const size_t want = std::max<size_t>(4 * bytes, 1u << 16);
        cudaError_t e = cudaMalloc(&p, want);
        cap = want;
        if (e != cudaSuccess) {  // not that much room: what is needed
            (void)cudaGetLastError();
            p = nullptr;
            e = cudaMalloc(&p, bytes);
            cap = e == cudaSuccess ? bytes : 0;
        }
        return e;
    }
    template <class T>
    T* as() {
        return static_cast<T*>(p);
    }
};

#define CK(x)                                                          \
    do {                                                               \
        cudaError_t e_ = (x);                                          \
        if (e_ != cudaSuccess) {                                       \
            *err = std::string("device BVH build: ") + cudaGetErrorString(e_); \
            return PBRT_ERR_CUDA;                                      \
        }                                                              \
    } while (0)

// Host tree of phase A: nodes with children or a phase-B job.
struct ANode {
    bool leaf = false, small = false;  // small: the subtree is job `job`
    uint32_t lo = 0, cnt = 0, dim = 0, depth = 1;
    int32_t left = -1, right = -1, job = -1;
    Box box{};
};

// A phase-A node, at its place in the tree.
struct TopNode {
    uint32_t at;
    FlatNode node;
};

// The small ranges' roots.
__global__ void __launch_bounds__(128) k_b_roots(const PoolNode* __restrict__ pool, const Job* __restrict__ jobs,
                                                 uint32_t njobs, PoolNode* __restrict__ roots) {
    const uint32_t j = blockIdx.x * 128u + threadIdx.x;
    if (j < njobs) roots[j] = pool[jobs[j].node0];
}

// Every node in the reference's depth-first order: a small range's nodes
// start at at[job], one warp each (on the host, from the downloaded pool,
// this took 1.4 ms for 180000 triangles).
__global__ void __launch_bounds__(128) k_number(const PoolNode* __restrict__ pool, const Job* __restrict__ jobs,
                                                const JobOut* __restrict__ outs, const uint32_t* __restrict__ at,
                                                uint32_t njobs, const TopNode* __restrict__ top, uint32_t ntop,
                                                FlatNode* __restrict__ nodes) {
    const uint64_t t = (uint64_t)blockIdx.x * 128u + threadIdx.x;
    if (t < ntop) nodes[top[t].at] = top[t].node;
    const uint64_t j = t >> 5;
    if (j >= njobs) return;
    const uint32_t base = at[j], count = outs[j].nodes;
    const PoolNode* p = pool + jobs[j].node0;
    for (uint32_t k = threadIdx.x & 31u; k < count; k += 32u) {
        const PoolNode q = p[k];
        FlatNode f;
        f.box = Box{V3{q.lo[0], q.lo[1], q.lo[2]}, V3{q.hi[0], q.hi[1], q.hi[2]}};
        f.leaf = (q.b & kLeaf) != 0;
        f.offset = f.leaf ? q.a : base + q.a;
        f.count = f.leaf ? q.b & ~kLeaf : q.b;
        nodes[base + k] = f;
    }
}

// The bounds and centroids of triangles (as prim_bounds: mesh.rs:196-205,
// bvh.rs:77), and every primitive's index.  From the refined primitives, which
// the layout reads again, instead of arrays that the host computes first.
__global__ void __launch_bounds__(256) k_bounds(const HostPrim* __restrict__ prims, uint32_t n, float4* __restrict__ lo,
                                                float4* __restrict__ hi, float* __restrict__ cx,
                                                float* __restrict__ cy, float* __restrict__ cz,
                                                uint32_t* __restrict__ idx) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= n) return;
    idx[i] = i;
    const HostPrim& p = prims[i];
    if (p.kind != PBRT_SHAPE_TRIANGLE_MESH) return;  // k_set_bounds
    auto low = [](float a, float b, float c) { return dmin(dmin(dmin(FLT_MAX, a), b), c); };
    auto high = [](float a, float b, float c) { return dmax(dmax(dmax(-FLT_MAX, a), b), c); };
    const V3 a = p.p1, b = p.p2, c = p.p3;
    const float4 l = make_float4(low(a.x, b.x, c.x), low(a.y, b.y, c.y), low(a.z, b.z, c.z), 0.0f);
    const float4 h = make_float4(high(a.x, b.x, c.x), high(a.y, b.y, c.y), high(a.z, b.z, c.z), 0.0f);
    lo[i] = l;
    hi[i] = h;
    cx[i] = (l.x + h.x) * 0.5f;
    cy[i] = (l.y + h.y) * 0.5f;
    cz[i] = (l.z + h.z) * 0.5f;
}

// The same of the other primitives, from the host.
struct PrimBounds {
    uint32_t prim;
    Box box;
    V3 centroid;
};
__global__ void __launch_bounds__(256) k_set_bounds(const PrimBounds* __restrict__ b, uint32_t n,
                                                    float4* __restrict__ lo, float4* __restrict__ hi,
                                                    float* __restrict__ cx, float* __restrict__ cy,
                                                    float* __restrict__ cz) {
    const uint32_t k = blockIdx.x * 256u + threadIdx.x;
    if (k >= n) return;
    const PrimBounds q = b[k];
    lo[q.prim] = make_float4(q.box.lo.x, q.box.lo.y, q.box.lo.z, 0.0f);
    hi[q.prim] = make_float4(q.box.hi.x, q.box.hi.y, q.box.hi.z, 0.0f);
    cx[q.prim] = q.centroid.x;
    cy[q.prim] = q.centroid.y;
    cz[q.prim] = q.centroid.z;
}

// Up to this many the primitives stay on the device for the layout; beyond it
// (240 MB) they make room and are uploaded again.
constexpr size_t kKeepPrims = 1u << 22;

}  // namespace

int device_build_tree(HostBVH& H, uint32_t mp, int split, std::string* err) {
    const size_t n = H.prims.size();
    H.nodes.clear();
    H.ordered.resize(n);
    H.depth = 0;
    if (n == 0) return PBRT_OK;
    if (n >= (1u << 31)) {
        *err = "device BVH build: more than 2^31 primitives";
        return PBRT_ERR_UNSUPPORTED;
    }
    std::vector<PrimBounds> analytic;
    for (size_t i = 0; !H.spheres.empty() && i < n; ++i) {
        if (H.prims[i].kind == PBRT_SHAPE_TRIANGLE_MESH) continue;
        PrimBounds b;
        b.prim = (uint32_t)i;
        b.box = prim_bounds(H, i, &b.centroid);
        analytic.push_back(b);
    }
    Buf d_prims, d_analytic, d_lo, d_hi, d_c[3], d_idx, d_tmp, d_pool;
    CK(cudaMalloc(&d_prims.p, n * sizeof(HostPrim)));
    CK(cudaMalloc(&d_lo.p, n * sizeof(float4)));
    CK(cudaMalloc(&d_hi.p, n * sizeof(float4)));
    for (int k = 0; k < 3; ++k) CK(cudaMalloc(&d_c[k].p, n * sizeof(float)));
    CK(cudaMalloc(&d_idx.p, n * 4));
    CK(cudaMalloc(&d_tmp.p, n * 4));
    Prims P;
    P.lo = d_lo.as<float4>();
    P.hi = d_hi.as<float4>();
    for (int k = 0; k < 3; ++k) P.cen[k] = d_c[k].as<float>();
    CK(cudaMemcpy(d_prims.p, H.prims.data(), n * sizeof(HostPrim), cudaMemcpyHostToDevice));
    k_bounds<<<(unsigned)((n + 255) / 256), 256>>>(d_prims.as<HostPrim>(), (uint32_t)n, d_lo.as<float4>(),
                                                   d_hi.as<float4>(), d_c[0].as<float>(), d_c[1].as<float>(),
                                                   d_c[2].as<float>(), d_idx.as<uint32_t>());
    if (!analytic.empty()) {
        const uint32_t na = (uint32_t)analytic.size();
        CK(cudaMalloc(&d_analytic.p, na * sizeof(PrimBounds)));
        CK(cudaMemcpy(d_analytic.p, analytic.data(), na * sizeof(PrimBounds), cudaMemcpyHostToDevice));
        k_set_bounds<<<(na + 255) / 256, 256>>>(d_analytic.as<PrimBounds>(), na, d_lo.as<float4>(), d_hi.as<float4>(),
                                                d_c[0].as<float>(), d_c[1].as<float>(), d_c[2].as<float>());
    }
    CK(cudaGetLastError());
    if (n > kKeepPrims) d_prims.reset();

    // ---- phase A: one level per round
    std::vector<ANode> A;
    A.push_back(ANode{});
    A[0].lo = 0;
    A[0].cnt = (uint32_t)n;
    std::vector<uint32_t> level;  // phase-A nodes of this level
    std::vector<Job> jobs;
    auto to_small = [&](uint32_t a) {
        A[a].small = true;
        A[a].job = (int32_t)jobs.size();
        jobs.push_back(Job{A[a].lo, A[a].lo + A[a].cnt, 0, 0});
    };
    if (n <= kSmall)
        to_small(0);
    else
        level.push_back(0);
    std::vector<Chunk> chunks, ranges;
    std::vector<SegDecision> dec;
    Buf d_acc, d_dec, d_chunks, d_left, d_base;
    while (!level.empty()) {
        const uint32_t S = (uint32_t)level.size();
        // the level's chunks, then its ranges, in one upload
        chunks.clear();
        ranges.clear();
        for (uint32_t s = 0; s < S; ++s) {
            const ANode& a = A[level[s]];
            const uint32_t first = (uint32_t)chunks.size();
            for (uint32_t o = 0; o < a.cnt; o += kChunk)
                chunks.push_back(Chunk{s, a.lo + o, a.lo + std::min(a.cnt, o + kChunk), 0});
            ranges.push_back(Chunk{first, a.lo, a.cnt, (uint32_t)chunks.size() - first});
        }
        const uint32_t NC = (uint32_t)chunks.size();
        chunks.insert(chunks.end(), ranges.begin(), ranges.end());
        CK(d_acc.reserve((size_t)S * kAccWords * 4));
        CK(d_dec.reserve((size_t)S * sizeof(SegDecision)));
        CK(d_chunks.reserve(chunks.size() * sizeof(Chunk)));
        CK(d_left.reserve((size_t)NC * 4));
        CK(d_base.reserve((size_t)NC * sizeof(uint2)));
        CK(cudaMemcpy(d_chunks.p, chunks.data(), chunks.size() * sizeof(Chunk), cudaMemcpyHostToDevice));
        const Chunk* d_ranges = d_chunks.as<Chunk>() + NC;
        const uint32_t acc_words = S * kAccWords;
        k_acc_init<<<(acc_words + 255) / 256, 256>>>(d_acc.as<int32_t>(), S);
        k_a_bounds<<<NC, 256>>>(P, d_idx.as<uint32_t>(), d_chunks.as<Chunk>(), d_acc.as<int32_t>());
        k_a_decide<<<(S + 127) / 128, 128>>>(d_acc.as<int32_t>(), d_dec.as<SegDecision>(), d_ranges, S, split);
        if (split == PBRT_SPLIT_SAH) {
            k_a_buckets<<<NC, 256>>>(P, d_idx.as<uint32_t>(), d_chunks.as<Chunk>(), d_dec.as<SegDecision>(),
                                     d_acc.as<int32_t>());
            k_a_choose<<<(S + 31) / 32, 32>>>(d_acc.as<int32_t>(), d_dec.as<SegDecision>(), d_ranges, S, mp);
        }
        k_a_count<<<NC, 256>>>(P, d_idx.as<uint32_t>(), d_chunks.as<Chunk>(), d_dec.as<SegDecision>(),
                               d_left.as<uint32_t>());
        k_a_base<<<(S + 3) / 4, 128>>>(d_chunks.as<Chunk>(), d_ranges, S, d_left.as<uint32_t>(),
                                       d_dec.as<SegDecision>(), d_base.as<uint2>());
        CK(cudaGetLastError());
        dec.resize(S);
        CK(cudaMemcpy(dec.data(), d_dec.p, (size_t)S * sizeof(SegDecision), cudaMemcpyDeviceToHost));
        k_a_scatter<<<NC, 256>>>(P, d_idx.as<uint32_t>(), d_tmp.as<uint32_t>(), d_chunks.as<Chunk>(),
                                 d_dec.as<SegDecision>(), d_base.as<uint2>());
        k_copy_ranges<<<NC, 256>>>(d_tmp.as<uint32_t>(), d_idx.as<uint32_t>(), d_chunks.as<Chunk>());
        CK(cudaGetLastError());
        std::vector<uint32_t> next;
        for (uint32_t s = 0; s < S; ++s) {
            const uint32_t ai = level[s];
            const SegDecision& d = dec[s];
            A[ai].box = Box{v3(d.lo[0], d.lo[1], d.lo[2]), v3(d.hi[0], d.hi[1], d.hi[2])};
            if (d.action == 0) {
                A[ai].leaf = true;
                continue;
            }
            const uint32_t lo_ = A[ai].lo, cnt = A[ai].cnt, nl = d.n_left;
            if (nl == 0 || nl == cnt) {
                *err = "BVH build: empty partition (the reference asserts at bvh.rs:237-238)";
                return PBRT_ERR_BUILD;
            }
            A[ai].dim = (uint32_t)d.dim;
            const uint32_t depth = A[ai].depth + 1;
            for (int side = 0; side < 2; ++side) {
                ANode c;
                c.lo = side == 0 ? lo_ : lo_ + nl;
                c.cnt = side == 0 ? nl : cnt - nl;
                c.depth = depth;
                const uint32_t ci = (uint32_t)A.size();
                A.push_back(c);
                (side == 0 ? A[ai].left : A[ai].right) = (int32_t)ci;
                if (c.cnt <= kSmall)
                    to_small(ci);
                else
                    next.push_back(ci);
            }
        }
        level.swap(next);
    }

    // ---- phase B: every small range, one warp each
    const uint32_t NJ = (uint32_t)jobs.size();
    uint64_t pool_nodes = 0;
    for (Job& j : jobs) {
        j.node0 = (uint32_t)pool_nodes;
        pool_nodes += 2ull * (j.hi - j.lo) - 1;
    }
    Buf d_jobs, d_outs, d_roots;
    std::vector<JobOut> outs(NJ);
    std::vector<PoolNode> roots(NJ);
    if (NJ) {  // none if no range beyond kSmall primitives could be split
        CK(cudaMalloc(&d_pool.p, pool_nodes * sizeof(PoolNode)));
        CK(cudaMalloc(&d_jobs.p, (size_t)NJ * sizeof(Job)));
        CK(cudaMalloc(&d_outs.p, (size_t)NJ * sizeof(JobOut)));
        CK(cudaMalloc(&d_roots.p, (size_t)NJ * sizeof(PoolNode)));
        CK(cudaMemcpy(d_jobs.p, jobs.data(), (size_t)NJ * sizeof(Job), cudaMemcpyHostToDevice));
        k_b_build<<<(NJ + kBWarps - 1) / kBWarps, 32 * kBWarps>>>(P, d_idx.as<uint32_t>(), d_jobs.as<Job>(), NJ,
                                                                  d_pool.as<PoolNode>(), d_outs.as<JobOut>(), mp,
                                                                  split);
        k_b_roots<<<(NJ + 127) / 128, 128>>>(d_pool.as<PoolNode>(), d_jobs.as<Job>(), NJ, d_roots.as<PoolNode>());
        CK(cudaGetLastError());
        CK(cudaMemcpy(outs.data(), d_outs.p, (size_t)NJ * sizeof(JobOut), cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(roots.data(), d_roots.p, (size_t)NJ * sizeof(PoolNode), cudaMemcpyDeviceToHost));
    }
    CK(cudaMemcpy(H.ordered.data(), d_idx.p, n * 4, cudaMemcpyDeviceToHost));
    for (const JobOut& o : outs)
        if (o.err) {
            *err = "BVH build: empty partition (the reference asserts at bvh.rs:237-238)";
            return PBRT_ERR_BUILD;
        }

    // ---- number every node in the reference's depth-first order
    // subtree sizes of phase-A nodes, children first
    std::vector<uint64_t> size(A.size(), 0);
    std::vector<Box> abox(A.size());
    for (size_t i = A.size(); i-- > 0;) {
        const ANode& a = A[i];
        if (a.small) {
            size[i] = outs[a.job].nodes;
            const PoolNode& r = roots[a.job];
            abox[i] = Box{v3(r.lo[0], r.lo[1], r.lo[2]), v3(r.hi[0], r.hi[1], r.hi[2])};
        } else if (a.leaf) {
            size[i] = 1;
            abox[i] = a.box;
        } else {
            size[i] = 1 + size[a.left] + size[a.right];
            abox[i] = box_union(abox[a.left], abox[a.right]);  // bvh.rs:247
        }
    }
    struct Item {
        uint32_t a;
        uint64_t at;
    };
    std::vector<uint32_t> job_at(NJ);  // first node of each small range
    std::vector<TopNode> top;
    std::vector<Item> todo{{0, 0}};
    while (!todo.empty()) {
        const Item it = todo.back();
        todo.pop_back();
        const ANode& a = A[it.a];
        if (a.small) {
            job_at[a.job] = (uint32_t)it.at;
            H.depth = std::max(H.depth, a.depth + outs[a.job].depth - 1);
            continue;
        }
        top.push_back(TopNode{(uint32_t)it.at, FlatNode{}});
        FlatNode& f = top.back().node;
        f.box = abox[it.a];
        H.depth = std::max(H.depth, a.depth);
        if (a.leaf) {
            f.leaf = true;
            f.offset = a.lo;
            f.count = a.cnt;
            continue;
        }
        f.leaf = false;
        f.count = a.dim;
        const uint64_t right_at = it.at + 1 + size[a.left];
        f.offset = (uint32_t)right_at;
        todo.push_back(Item{(uint32_t)a.right, right_at});
        todo.push_back(Item{(uint32_t)a.left, it.at + 1});
    }
    const uint32_t m = (uint32_t)size[0];
    for (Buf* b : {&d_lo, &d_hi, &d_c[0], &d_c[1], &d_c[2], &d_tmp}) b->reset();  // room for the nodes
    Buf d_nodes, d_at, d_top;
    CK(cudaMalloc(&d_nodes.p, (size_t)m * sizeof(FlatNode)));
    if (NJ) {
        CK(cudaMalloc(&d_at.p, (size_t)NJ * 4));
        CK(cudaMemcpy(d_at.p, job_at.data(), (size_t)NJ * 4, cudaMemcpyHostToDevice));
    }
    if (!top.empty()) {
        CK(cudaMalloc(&d_top.p, top.size() * sizeof(TopNode)));
        CK(cudaMemcpy(d_top.p, top.data(), top.size() * sizeof(TopNode), cudaMemcpyHostToDevice));
    }
    const size_t threads = std::max<size_t>(32 * (size_t)NJ, top.size());
    k_number<<<(unsigned)((threads + 127) / 128), 128>>>(d_pool.as<PoolNode>(), d_jobs.as<Job>(), d_outs.as<JobOut>(),
                                                         d_at.as<uint32_t>(), NJ, d_top.as<TopNode>(),
                                                         (uint32_t)top.size(), d_nodes.as<FlatNode>());
    CK(cudaGetLastError());
    H.nodes.resize(m);
    CK(cudaMemcpy(H.nodes.data(), d_nodes.p, (size_t)m * sizeof(FlatNode), cudaMemcpyDeviceToHost));
    const bool big_leaf = std::any_of(top.begin(), top.end(), [](const TopNode& t) { return t.node.leaf; });
    d_pool.reset();
    // The layout is made here too, which is the faster at every size (creation and
    // a query of 50 / 500 / 4000 / 64000 terrain triangles, us: 692 / 954 / 1297 /
    // 3762, from the host's arrays 814 / 1109 / 1585 / 5644), unless a range beyond
    // kSmall primitives could not be split: one thread writes a leaf.
    if (!big_leaf)
        device_fill_layout(H, d_nodes.as<FlatNode>(), m, d_idx.as<uint32_t>(), d_prims.as<HostPrim>());
    return PBRT_OK;
}

}  // namespace pbrt
