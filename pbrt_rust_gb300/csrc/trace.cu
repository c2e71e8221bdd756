// trace.cu - batched closest-hit / any-hit kernels over PbrtRay arrays.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "../../include/pbrt_gpu.h"
#include "kernels.h"
#include "trace.cuh"
#include "trace4.cuh"

namespace pbrt {

// One thread per ray.  Rays are two float4 loads (32 B, coalesced); a
// closest hit is one 16-byte store, an any-hit answer one byte.
template <int STACK, bool ANY>
__global__ void __launch_bounds__(128) k_trace(const __grid_constant__ DevBVH bvh, const float4* __restrict__ rays,
                                               uint32_t n,
                                               const uint32_t* __restrict__ order, float4* __restrict__ hits,
                                               uint8_t* __restrict__ occ, int* __restrict__ status,
                                               uint32_t* __restrict__ replay) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (order) i = __ldg(order + i);
    float4 a = __ldg(rays + 2 * (size_t)i), b = __ldg(rays + 2 * (size_t)i + 1);
    DRay r = make_dray(a, b);
    TraceResult res;
    int st = 0;
    bool nan_hit = false;
    bool found = traverse<STACK, ANY>(bvh, r, &res, &st, &nan_hit);
    if (st) atomicMax(status, st);
    if (ANY) {
        occ[i] = found ? 1 : 0;
    } else if (nan_hit) {
        hits[i] = make_float4(__int_as_float(kReplayMark), 0.0f, 0.0f, 0.0f);
        *replay = 1u;
    } else {
        hits[i] = make_float4(__int_as_float(res.prim), res.t, res.b1, res.b2);
    }
}

// One thread per ray; a warp whose rays share their direction signs walks
// them together (traverse_packet), any other warp walks each lane's ray on
// its own (traverse).  Results equal k_trace's bit for bit.
template <int STACK, bool ANY>
__global__ void __launch_bounds__(128) k_trace_packet(const __grid_constant__ DevBVH bvh,
                                                      const float4* __restrict__ rays, uint32_t n,
                                                      const uint32_t* __restrict__ order, float4* __restrict__ hits,
                                                      uint8_t* __restrict__ occ, int* __restrict__ status,
                                                      uint32_t* __restrict__ replay) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = i < n;  // every lane stays for the warp's votes
    if (active && order) i = __ldg(order + i);
    DRay r = make_dray(active ? __ldg(rays + 2 * (size_t)i) : make_float4(0, 0, 0, 0),
                       active ? __ldg(rays + 2 * (size_t)i + 1) : make_float4(0, 0, 1, 0));
    TraceResult res;
    int st = 0;
    bool nan_hit = false, found = false;
    if (warp_signs_uniform(r, active))
        found = traverse_packet<STACK, ANY>(bvh, r, active, &res, &st, &nan_hit);
    else if (active)
        found = traverse<STACK, ANY>(bvh, r, &res, &st, &nan_hit);
    if (!active) return;
    if (st) atomicMax(status, st);
    if (ANY) {
        occ[i] = found ? 1 : 0;
    } else if (nan_hit) {
        hits[i] = make_float4(__int_as_float(kReplayMark), 0.0f, 0.0f, 0.0f);
        *replay = 1u;
    } else {
        hits[i] = make_float4(__int_as_float(res.prim), res.t, res.b1, res.b2);
    }
}

// Persistent warps: the grid holds exactly the resident warps; each warp
// owns a contiguous range of rays and, whenever at least REFILL of its
// lanes are idle, hands them the next rays of its range.  Rays of very
// different lengths then share warps without leaving lanes idle until the
// longest one finishes.  Each ray's own traversal is unchanged, so results
// are identical to k_trace.
template <int STACK, bool ANY, bool INST = false>
__global__ void __launch_bounds__(128) k_trace_persistent(const __grid_constant__ DevBVH bvh,
                                                          const float4* __restrict__ rays, uint32_t n,
                                                          const uint32_t* __restrict__ order, float4* __restrict__ hits,
                                                          uint8_t* __restrict__ occ, int* __restrict__ status,
                                                          uint32_t per_warp, uint32_t refill,
                                                          uint32_t* __restrict__ replay) {
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint64_t next = warp * per_warp;
    const uint64_t end = (next + per_warp < (uint64_t)n) ? next + per_warp : (uint64_t)n;
    const uint32_t kNone = 0xffffffffu;
    uint32_t ray = kNone;
    int st = 0;
    DRay r;
    Traversal<STACK, INST> T;
    T.found = false;
    auto finish = [&]() {
        if (ANY) {
            occ[ray] = T.found ? 1 : 0;
        } else {
            if (T.nan_hit) {
                hits[ray] = make_float4(__int_as_float(kReplayMark), 0.0f, 0.0f, 0.0f);
                *replay = 1u;
            } else {
                hits[ray] = make_float4(__int_as_float(T.res.prim), T.res.t, T.res.b1, T.res.b2);
            }
        }
        ray = kNone;
    };
    for (;;) {
        unsigned idle = __ballot_sync(0xffffffffu, ray == kNone);
        unsigned nidle = __popc(idle);
        if (next < end && nidle >= (next + nidle >= end ? 1u : refill)) {
            if (ray == kNone) {
                uint64_t my = next + __popc(idle & ((1u << lane) - 1u));
                if (my < end) {
                    ray = order ? __ldg(order + my) : (uint32_t)my;
                    r = make_dray(__ldg(rays + 2 * (size_t)ray), __ldg(rays + 2 * (size_t)ray + 1));
                    if (!T.start(bvh, r)) finish();
                }
            }
            next += nidle;
        }
        bool busy = ray != kNone;
        if (!__any_sync(0xffffffffu, busy)) {
            if (next >= end) break;
            continue;
        }
        if (busy && !T.template step<ANY>(bvh, r, &st)) finish();
    }
    if (st) atomicMax(status, st);
}

constexpr int kWalkBlock = 128;  // threads per block and stack rows of the 4-wide kernels
constexpr int kWalkRows = 16;

// 4-wide traversal, one thread per ray; the first per_warp lanes of each warp
// have one (rays_per_warp).  Blocks per SM: what the registers allow without
// spills (any hit, 8 / 9 / 10 blocks on a terrain frame's shadow rays: 2594 /
// 2553 / 2844 us; closest hit, 7 / 8 / 9 on its camera rays: 1916 / 1899 /
// 1935).
template <int OVF, bool ANY, bool INST>
__global__ void __launch_bounds__(kWalkBlock, INST ? 6 : (ANY ? 9 : 8)) k_trace4(const __grid_constant__ DevBVH4 bvh,
                                                       const float4* __restrict__ rays, uint32_t n,
                                                       const uint32_t* __restrict__ order, float4* __restrict__ hits,
                                                       uint8_t* __restrict__ occ, int* __restrict__ status,
                                                       uint32_t per_warp) {
    using Walk = Walk4<kWalkBlock, kWalkRows, OVF, ANY, INST>;
    __shared__ typename Walk::Shared sh;
    sh.init();
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t g = (uint64_t)(blockIdx.x * (kWalkBlock / 32) + (threadIdx.x >> 5)) * per_warp + lane;
    if (lane >= per_warp || g >= n) return;
    uint32_t i = (uint32_t)g;
    if (order) i = __ldg(order + i);
    const float4* ray = rays + 2 * (size_t)i;
    Walk T;
    typename Walk::Ovf ov;
    T.bind(sh);
    const int st = T.start(bvh, __ldg(ray), __ldg(ray + 1));
    if (st == kStartWalk) T.run(bvh, sh, ov);
    const bool exact = st == kStartExact || T.gave_up();
    if (ANY)
        occ[i] = (exact ? exact_any<OVF + 8, INST>(bvh.pair, ray, status) : T.found()) ? 1 : 0;
    else
        hits[i] = exact ? exact_hit<OVF + 8, INST>(bvh.pair, ray, status) : T.hit_record();
}

// A ray is read once: its lines go to L2 only, leaving L1 to the tree.
__device__ __forceinline__ float4 ld_stream(const float4* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p));
    return v;
}

// Streamed input: the rays arrive in pieces of 2^piece_shift rays while the
// traversal already runs, and ready[k] turns non-zero once piece k has
// landed (the copy stream writes it with a 4-byte copy queued behind the
// piece's own copy).  %globaltimer is the GPU's nanosecond clock.
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// A flag that has not come within `wait_ms` means the copies did not run
// beside the walk (or at all), and the warp gives up instead of hanging (at
// once when another warp already gave up: *status holds the timeout).
__device__ __noinline__ bool wait_piece(const uint32_t* ready, uint32_t k, uint32_t wait_ms, const int* status) {
    if (ld_acquire_u32(ready + k)) return true;
    const uint64_t t0 = global_ns(), limit = (uint64_t)wait_ms * 1000000ull;
    for (;;) {
        __nanosleep(256);
        if (ld_acquire_u32(ready + k)) return true;
        if (global_ns() - t0 > limit ||
            ld_acquire_u32(reinterpret_cast<const uint32_t*>(status)) == (uint32_t)PBRT_ERR_TIMEOUT)
            return false;
    }
}

// 4-wide traversal with persistent warps refilling idle lanes (see
// k_trace_persistent).  Without `work`, warp w owns rays
// [w * per_warp, (w + 1) * per_warp); with it, warps take chunks of
// per_warp rays from the shared counter *work (zero at launch) whenever
// their chunk is used up, so warps that drew short rays take more of them
// and no warp is left with a long tail.  With `ready` (streamed input; only
// with `work`, which hands out chunks in ray order) a warp that takes a
// chunk first waits for the piece holding its last ray, and reads rays
// through L2 (they are written while the kernel runs); a wait that runs out
// sets PBRT_ERR_TIMEOUT and the warp drops its chunk.
//
// A turn of the loop hands out rays, makes kNodeSteps visits of inner nodes
// and then tests the leaves that were reached: the votes and the leaf code,
// which a few of the warp's lanes need at a time, are paid once per
// kNodeSteps visits (one, two, three, four visits per turn: 586 / 501 / 480 /
// 494 us for 2^22 incoherent rays into a terrain of a million triangles).
//
// HOSTOUT (closest hits, with `work`): `hits` is a device staging array and
// `host_hits` the caller's pinned host memory mapped into the device's
// address space.  Scattered 16-byte stores across NVLink-C2C run at a fifth
// of its bandwidth (measured on GB300: 37 against 191 GB/s for 1 KiB runs),
// so each warp counts its chunks' finished rays in a ring of 4 slots in
// shared memory and copies a chunk's hits from the staging array to the
// host in coalesced rows once its last ray is done; a warp takes a new
// chunk only when a slot is free (always the case once all its lanes are
// idle).  The copies spread over the walk, sharing the link with the
// streamed input.
constexpr int kNodeSteps = 3;
constexpr uint32_t kRingWords = 10 + 32;  // HOSTOUT: per warp, see k_trace4_persistent
// HOSTOUT's copy of finished chunks (ring[9]: one bit per slot) from the
// staging array to the host, one row of the warp's lanes at a time; out of
// line, so that the walk keeps its registers.
static __device__ __noinline__ void write_out_chunks(uint32_t* ring, const float4* hits, float4* host_hits, uint32_t n,
                                                     uint32_t per_warp) {
    const unsigned lane = threadIdx.x & 31u;
    uint32_t dm = ring[9];
    __syncwarp();
    if (lane == 0) ring[9] = 0u;
    while (dm) {
        const uint32_t j = (uint32_t)(__ffs(dm) - 1);
        dm &= dm - 1u;
        const uint32_t base = ring[4 + j];
        const uint32_t cnt = min(per_warp, n - base);
        for (uint32_t k = lane; k < cnt; k += 32u) host_hits[base + k] = __ldcg(hits + base + k);
    }
}
template <int OVF, bool ANY, bool INST = false, bool HOSTOUT = false>
__global__ void __launch_bounds__(kWalkBlock, INST ? 6 : 8)
    k_trace4_persistent(const __grid_constant__ DevBVH4 bvh, const float4* __restrict__ rays, uint32_t n,
                        const uint32_t* __restrict__ order,
                        float4* __restrict__ hits, uint8_t* __restrict__ occ, int* __restrict__ status,
                        uint32_t per_warp, uint32_t refill, uint32_t* __restrict__ work,
                        uint32_t* __restrict__ replay, const StreamIn in, float4* __restrict__ host_hits) {
    static_assert(!(HOSTOUT && ANY), "host write-out is for closest hits");
    using Walk = Walk4<kWalkBlock, kWalkRows, OVF, ANY, INST>;
    __shared__ typename Walk::Shared sh;
    __shared__ uint32_t rings[HOSTOUT ? kWalkBlock / 32 : 1][HOSTOUT ? kRingWords : 1];
    sh.init();
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * kWalkBlock + threadIdx.x) >> 5;
    uint32_t next = 0, end = 0;
    if (!work) {
        const uint64_t lo = (uint64_t)warp * per_warp;
        next = lo < n ? (uint32_t)lo : n;
        end = lo + per_warp < n ? (uint32_t)lo + per_warp : n;
    }
    bool more = work != nullptr;  // the shared counter may still hold rays
    const uint32_t kNone = 0xffffffffu;
    uint32_t ray = kNone;
    Walk T;
    typename Walk::Ovf ov;
    T.bind(sh);
    // HOSTOUT: this warp's ring in shared memory: rays left in slot j at
    // ring[j], the slot's first ray at ring[4 + j], the slot of the chunk
    // being handed out at ring[8], the slots whose last ray finished (a bit
    // each) at ring[9], then each lane's slot at ring[10 + lane].  Nothing of
    // it lives in registers, which the walk needs.
    auto ring_of = [&]() -> uint32_t* {
        uint32_t tid;  // read afresh at each use: the address is not kept in a register across the walk
        asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
        return rings[tid >> 5];
    };
    if constexpr (HOSTOUT) {
        if (lane < 10) ring_of()[lane] = 0u;
        __syncwarp();
    }
    // HOSTOUT: the chunks whose last ray finished go out to the host.  Done
    // when the warp takes its next chunk (which needs a slot) and at the
    // end, not at every step of the walk.
    auto write_out = [&]() {
        if constexpr (HOSTOUT) {
            __syncwarp();  // the chunks' staged hits and the ring are visible to every lane
            uint32_t* ring = ring_of();
            if (ring[9]) write_out_chunks(ring, hits, host_hits, n, per_warp);
        }
    };
    // The lane's ray ends with what T found, or marked for the replay.
    auto finish = [&](bool exact) {
        if (exact) *replay = 1u;
        if (ANY) {
            occ[ray] = exact ? kReplayOcc : (T.found() ? 1 : 0);
        } else {
            const float4 h = exact ? make_float4(__int_as_float(kReplayMark), 0.0f, 0.0f, 0.0f) : T.hit_record();
            if constexpr (HOSTOUT) {
                hits[ray] = h;
                uint32_t* ring = ring_of();
                const uint32_t j = ring[10 + lane];
                if (atomicSub(ring + j, 1u) == 1u) atomicOr(ring + 9, 1u << j);
            } else {
                __stcs(hits + ray, h);  // written once and (but for marks) not read here
            }
        }
        ray = kNone;
        T.cur = kWalkDone;
    };
    for (;;) {
        unsigned idle = __ballot_sync(0xffffffffu, ray == kNone);
        unsigned nidle = __popc(idle);
        if (more && next >= end && nidle >= refill) {  // warp-uniform
            int fs = 0;  // HOSTOUT: a free slot for the next chunk, -1 when none is
            if constexpr (HOSTOUT) {
                write_out();  // frees the slots of finished chunks
                __syncwarp();
                const uint32_t* ring = ring_of();
                fs = -1;
                for (int j = 3; j >= 0; --j)
                    if (ring[j] == 0u) fs = j;
            }
            if (fs >= 0) {
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(work, per_warp);
                base = __shfl_sync(0xffffffffu, base, 0);
                if (base < n) {
                    next = base;
                    end = n - base > per_warp ? base + per_warp : n;
                    if (in.ready) {  // streamed input: the chunk's rays must have landed
                        int ok = 1;
                        if (lane == 0)
                            ok = wait_piece(in.ready, (uint32_t)((end - 1) >> in.shift), in.wait_ms, status) ? 1 : 0;
                        if (!__shfl_sync(0xffffffffu, ok, 0)) {
                            if (lane == 0) atomicMax(status, PBRT_ERR_TIMEOUT);
                            next = end;
                            more = false;
                        }
                    }
                    if constexpr (HOSTOUT) {
                        if (next < end) {
                            if (lane == 0) {
                                uint32_t* ring = ring_of();
                                ring[fs] = end - next;
                                ring[4 + fs] = base;
                                ring[8] = (uint32_t)fs;
                            }
                            __syncwarp();
                        }
                    }
                } else {
                    more = false;
                }
            }
        }
        const bool tail = !more && end - next <= nidle;
        if (next < end && nidle >= (tail ? 1u : refill)) {
            if (ray == kNone) {
                const uint32_t k = __popc(idle & ((1u << lane) - 1u));
                if (k < end - next) {
                    ray = order ? __ldg(order + next + k) : next + k;
                    if constexpr (HOSTOUT) {
                        uint32_t* ring = ring_of();
                        ring[10 + lane] = ring[8];
                    }
                    const float4* rp = rays + 2 * (size_t)ray;
                    float4 a, b;
                    if (in.ready) {
                        a = __ldcg(rp);
                        b = __ldcg(rp + 1);
                    } else {
                        a = ld_stream(rp);
                        b = ld_stream(rp + 1);
                    }
                    const int st = T.start(bvh, a, b);
                    if (st != kStartWalk) finish(st == kStartExact);
                }
            }
            next += min(nidle, end - next);
        }
        if (!__any_sync(0xffffffffu, ray != kNone)) {
            if (next >= end && !more) break;
            continue;
        }
        // an idle lane's `cur` is kWalkDone
#pragma unroll
        for (int k = 0; k < kNodeSteps; ++k)
            if ((int32_t)T.cur >= 0) T.node(bvh, ov);
        if ((int32_t)T.cur < 0 && T.cur != kWalkDone) T.leaf(bvh, sh, ov);
        if (T.cur == kWalkDone && ray != kNone && !T.resume(ov)) finish(T.gave_up());
    }
    write_out();
}

enum {
    kVariantPairPlain = 0,
    kVariantPairPersistent = 1,
    kVariantWidePlain = 2,
    kVariantWidePersistent = 3,
    kVariantWideSpeculative = 4,
    kVariantPairPacket = 5,
    kVariantAuto = PBRT_TRACE_AUTO  // renders: by the tree's size
};
static int g_kernel_variant = -1;
static unsigned g_refill = 4;
static unsigned g_min_blocks = 0;
static int g_render_kernel = kVariantAuto;
static unsigned g_reorder = 0;
static unsigned g_chunk = 64;

// Queries take the 4-wide persistent walk (under either of its names).
static bool wide_persistent() {
    return g_kernel_variant == kVariantWidePersistent || g_kernel_variant == kVariantWideSpeculative;
}

static int variant_from_name(const char* v, int dflt) {
    if (!strcmp(v, "plain")) return kVariantPairPlain;
    if (!strcmp(v, "pt")) return kVariantPairPersistent;
    if (!strcmp(v, "w4")) return kVariantWidePlain;
    if (!strcmp(v, "w4pt")) return kVariantWidePersistent;
    if (!strcmp(v, "w4spec")) return kVariantWideSpeculative;
    if (!strcmp(v, "packet")) return kVariantPairPacket;
    return dflt;
}

static void read_variant() {
    if (g_kernel_variant >= 0) return;
    g_kernel_variant = kVariantWidePersistent;
    if (const char* v = getenv("PBRT_TRACE_KERNEL")) g_kernel_variant = variant_from_name(v, g_kernel_variant);
    if (const char* r = getenv("PBRT_TRACE_REFILL")) {
        int x = atoi(r);
        if (x >= 1 && x <= 32) g_refill = (unsigned)x;
    }
    if (const char* m = getenv("PBRT_TRACE_MINB")) {
        int x = atoi(m);
        if (x == 0 || x == 7 || x == 8 || x == 9) g_min_blocks = (unsigned)x;
    }
    if (const char* v = getenv("PBRT_TRACE_CHUNK")) {
        int x = atoi(v);
        if (x == 0 || (x >= 32 && x <= 4096 && x % 32 == 0)) g_chunk = (unsigned)x;
    }
    if (const char* v = getenv("PBRT_TRACE_REORDER")) {
        if (!strcmp(v, "0") || !strcmp(v, "1")) g_reorder = (unsigned)(v[0] - '0');
    }
    if (const char* v = getenv("PBRT_RENDER_KERNEL")) {
        g_render_kernel = strcmp(v, "auto") ? variant_from_name(v, g_render_kernel) : (int)kVariantAuto;
    }
}

// Rewrites what a traversal marked kReplayMark (closest hits) or kReplayOcc
// (any hit) by the exact walk over the binary layout (see Traversal in
// trace.cuh, and trace4.cuh for the rays that 4-wide walks mark); returns at
// once when no ray of the launch was marked, so a launch without such rays
// pays one empty kernel.  `host_hits` (may be null): a second copy of the
// hits that the rewritten ones also go to (the host memory of a write-out
// walk).  Two blocks of 512 per SM: 2^20 rays, all marked, into 200000 random
// triangles / a terrain of 180000 / the forest 1901 / 577 / 1802 us, with four
// of 128 2822 / 775 / 2305; the empty launch takes 1 us more, with 16 or 32 of
// 128 3 to 5 us.
constexpr int kReplayBlock = 512;
template <int STACK, bool INST>
__global__ void __launch_bounds__(kReplayBlock)
    k_replay2(const __grid_constant__ DevBVH bvh, const float4* __restrict__ rays, uint32_t n,
              float4* __restrict__ hits, uint8_t* __restrict__ occ, const uint32_t* __restrict__ replay,
              int* __restrict__ status, float4* __restrict__ host_hits) {
    if (*(const volatile uint32_t*)replay == 0u) return;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (occ) {
            if (occ[i] == kReplayOcc) occ[i] = exact_any<STACK, INST>(bvh, rays + 2 * i, status) ? 1 : 0;
        } else if (__float_as_int(hits[i].x) == kReplayMark) {
            hits[i] = exact_hit<STACK, INST>(bvh, rays + 2 * i, status);
            if (host_hits) host_hits[i] = hits[i];
        }
    }
}

// `host_hits` (closest hits, with `work`): the HOSTOUT walk, `h4` its
// staging array.
template <int OVF, bool ANY, bool INST, bool HOSTOUT = false>
static cudaError_t launch_wide_persistent(const DevBVH4& bvh, const float4* r4, uint32_t n, const uint32_t* order,
                                          float4* h4, uint8_t* occ, int* d_status, cudaStream_t stream,
                                          uint32_t* work, uint32_t* replay, StreamIn in, float4* host_hits) {
    constexpr int warps_per_block = kWalkBlock / 32;
    auto kernel = k_trace4_persistent<OVF, ANY, INST, HOSTOUT>;
    static ShapeCache bps_cache;
    const int sms = device_sms();
    const int bps = resident_blocks(bps_cache, kernel, kWalkBlock, 0);
    uint64_t warps = (uint64_t)sms * bps * warps_per_block;
    uint32_t per_warp = (uint32_t)((n + warps - 1) / warps);
    if (per_warp < 32) per_warp = 32;
    if (work && g_chunk && n <= 0xF0000000u) {  // the counter cannot wrap past n
        // every resident warp, each taking g_chunk rays at a time; no more
        // warps than chunks
        uint64_t chunks = (n + g_chunk - 1) / g_chunk;
        uint64_t w = chunks < warps ? chunks : warps;
        unsigned grid = (unsigned)((w + warps_per_block - 1) / warps_per_block);
        kernel<<<grid, kWalkBlock, 0, stream>>>(bvh, r4, n, order, h4, occ, d_status, g_chunk, g_refill, work, replay,
                                                in, host_hits);
        return cudaGetLastError();
    }
    // fixed per-warp ranges would read rays out of order and have no chunks
    // to write out: no streamed input, no write-out
    if (in.ready || HOSTOUT) return cudaErrorInvalidValue;
    uint64_t need_warps = (n + (uint64_t)per_warp - 1) / per_warp;
    unsigned grid = (unsigned)((need_warps + warps_per_block - 1) / warps_per_block);
    kernel<<<grid, kWalkBlock, 0, stream>>>(bvh, r4, n, order, h4, occ, d_status, per_warp, g_refill, nullptr,
                                            replay, StreamIn{}, nullptr);
    return cudaGetLastError();
}

// A launch of few rays is as long as its longest walk.  A warp whose lanes
// walk different rays takes the sum of their detours, so few rays are spread
// over more warps than they would fill, up to 14 warps per SM (an SM keeps 32
// of them, but from there on they slow each other down more than sharing a
// warp does).  Closest hits of 64 / 1000 / 4000 / 16000 / 64000 rays into 4096
// random triangles, us: 33 / 33 / 42 / 58 / 72 with this rule (1 / 1 / 2 / 8 /
// 32 lanes), 59 / 58 / 58 / 62 / 72 with full warps, 121 with one lane at
// 16000; the persistent kernel 79 / 84 / 87 / 89 / 96.
uint32_t rays_per_warp(uint64_t n) {
    const uint64_t warps = 14ull * (uint64_t)device_sms();
    uint32_t r = 1;
    while (r < 32u && n > warps * r) r *= 2;
    return r;
}

// The most rays of a call that takes one thread per ray instead of the
// persistent kernel: what fits the chip at once (8 blocks of 128 per SM).
// 128000 / 256000 rays into 4096 and 200000 random triangles, us: 95 / 159 and
// 196 / 298 one thread per ray, 110 / 150 and 204 / 242 persistent; and such a
// call needs no work counter, no replay launch and no scratch.
static uint64_t small_call_rays() { return 8ull * kWalkBlock * (uint64_t)device_sms(); }
bool trace_is_small(const DevBVH4* wide, uint32_t wide_bound, uint32_t n) {
    read_variant();
    return wide && wide_stack_variant(wide_bound) && wide_persistent() && !g_reorder &&
           n <= small_call_rays();
}

// The 4-wide kernel for a call: closest hits into h4 (occ null) or answers
// into occ; persistent or one thread per ray.
template <int OVF>
static cudaError_t launch_wide(const DevBVH4& bvh, const float4* r4, uint32_t n, const uint32_t* order, float4* h4,
                               uint8_t* occ, int* d_status, cudaStream_t stream, bool persistent, uint32_t* work,
                               uint32_t* replay, StreamIn in = {}, float4* host_hits = nullptr) {
    auto pt = [&](auto launch) {
        return launch(bvh, r4, n, order, h4, occ, d_status, stream, work, replay, in, host_hits);
    };
    const bool inst = bvh.pair.insts != nullptr;
    if (inst && persistent)
        return host_hits ? pt(launch_wide_persistent<OVF, false, true, true>)
               : occ     ? pt(launch_wide_persistent<OVF, true, true>)
                         : pt(launch_wide_persistent<OVF, false, true>);
    if (host_hits) return pt(launch_wide_persistent<OVF, false, false, true>);
    if (persistent)
        return occ ? pt(launch_wide_persistent<OVF, true, false>) : pt(launch_wide_persistent<OVF, false, false>);
    const uint32_t per_warp = rays_per_warp(n);
    const uint64_t per_block = (uint64_t)per_warp * (kWalkBlock / 32);
    const unsigned grid = (unsigned)((n + per_block - 1) / per_block);
    auto plain = [&](auto kernel) {
        kernel<<<grid, kWalkBlock, 0, stream>>>(bvh, r4, n, order, h4, occ, d_status, per_warp);
        return cudaGetLastError();
    };
    if (inst) return occ ? plain(k_trace4<OVF, true, true>) : plain(k_trace4<OVF, false, true>);
    return occ ? plain(k_trace4<OVF, true, false>) : plain(k_trace4<OVF, false, false>);
}

int set_trace_config(const PbrtTraceConfig& c) {
    if (c.kernel < kVariantPairPlain || c.kernel > kVariantPairPacket || c.refill < 1 || c.refill > 32) return 1;
    if (!(c.min_blocks == 0 || c.min_blocks == 7 || c.min_blocks == 8 || c.min_blocks == 9)) return 1;
    if (c.render_kernel < kVariantPairPlain || c.render_kernel > kVariantAuto) return 1;
    if (c.reorder > 1) return 1;
    if (!(c.chunk == 0 || (c.chunk >= 32 && c.chunk <= 4096 && c.chunk % 32 == 0))) return 1;
    read_variant();
    g_kernel_variant = c.kernel;
    g_refill = c.refill;
    g_min_blocks = c.min_blocks;
    g_render_kernel = c.render_kernel;
    g_reorder = c.reorder;
    g_chunk = c.chunk;
    return 0;
}
void get_trace_config(PbrtTraceConfig* c) {
    read_variant();
    c->kernel = g_kernel_variant;
    c->refill = g_refill;
    c->min_blocks = g_min_blocks;
    c->render_kernel = g_render_kernel;
    c->reorder = g_reorder;
    c->chunk = g_chunk;
}
unsigned trace_chunk() {
    read_variant();
    return g_chunk;
}
bool trace_reorder() {
    read_variant();
    return g_reorder != 0;
}
// The choice of kVariantAuto.  Which walk a small tree's frame is faster with
// depends on the visits per ray, not on the tree's size alone.  Camera + shadow rays of
// 512 x 512 x 4 frames, binary against 4-wide, us: terrains of 300 / 2000 /
// 20000 triangles 84 / 134 / 251 against 95 / 144 / 221, 64 spheres 100 against
// 117, soups of 300 / 1000 / 4000 triangles 61 / 97 / 241 against 58 / 78 / 168.
// The line is where none of them is slower than with the binary walk; soups
// below it would be faster with PBRT_TRACE_WIDE.
constexpr uint32_t kWideRenderPrims = 4096;
int render_trace_kernel(uint32_t n_prims) {
    read_variant();
    if (g_render_kernel != kVariantAuto) return g_render_kernel;
    return n_prims < kWideRenderPrims ? kVariantPairPlain : kVariantWidePlain;
}

int wide_stack_variant(uint32_t bound) {
    if (bound <= 64) return 64;
    if (bound <= 256) return 256;
    return 0;
}

template <int STACK, bool ANY, bool INST = false>
static cudaError_t launch_persistent(const DevBVH& bvh, const float4* r4, uint32_t n, const uint32_t* order,
                                     float4* h4, uint8_t* occ, int* d_status, cudaStream_t stream,
                                     uint32_t* replay) {
    static ShapeCache bps_cache;  // one per instantiation
    const int block = 128;
    const int sms = device_sms();
    const int bps = resident_blocks(bps_cache, k_trace_persistent<STACK, ANY, INST>, block, 0);
    uint64_t warps = (uint64_t)sms * bps * (block / 32);
    uint32_t per_warp = (uint32_t)((n + warps - 1) / warps);
    if (per_warp < 32) per_warp = 32;
    uint64_t need_warps = (n + per_warp - 1) / per_warp;
    unsigned grid = (unsigned)((need_warps + (block / 32) - 1) / (block / 32));
    k_trace_persistent<STACK, ANY, INST><<<grid, block, 0, stream>>>(bvh, r4, n, order, h4, occ, d_status, per_warp,
                                                                     g_refill, replay);
    return cudaGetLastError();
}

int trace_stack_for_depth(uint32_t depth) {
    if (depth <= 64) return 64;
    if (depth <= 256) return 256;
    return 0;
}

// *replays: the launch marks rays for the replay kernel.
static cudaError_t launch_main(const DevBVH& bvh, uint32_t depth, const PbrtRay* rays, uint32_t n, PbrtHit* hits,
                               uint8_t* occluded, int* d_status, cudaStream_t stream, const DevBVH4* wide,
                               uint32_t wide_bound, int kernel, const uint32_t* order, uint32_t* work,
                               uint32_t* replay, bool* replays) {
    const int variant = kernel == kTraceSmall ? (int)kVariantWidePlain : (kernel >= 0 ? kernel : g_kernel_variant);
    // a scene with instances takes a walk with nested instance traversal
    // (4-wide when a variant covers the stack bound), whatever the configured
    // kernel
    const bool inst = bvh.insts != nullptr;
    const int v = wide ? wide_stack_variant(wide_bound) : 0;
    const float4* r4 = reinterpret_cast<const float4*>(rays);
    float4* h4 = reinterpret_cast<float4*>(hits);
    if (v && (inst || variant == kVariantWidePlain || variant == kVariantWidePersistent ||
              variant == kVariantWideSpeculative)) {
        // with instances: one thread per ray for a render's camera rays
        // (kernel >= 0; 390 -> 151 us for a 517 x 389 x 4 forest frame), the
        // persistent walk for batches
        const bool pt = kernel == kTraceSmall ? false : (inst ? kernel < 0 : variant != kVariantWidePlain);
        *replays = pt;
        return v == 64 ? launch_wide<64>(*wide, r4, n, order, h4, occluded, d_status, stream, pt, work, replay)
                       : launch_wide<256>(*wide, r4, n, order, h4, occluded, d_status, stream, pt, work, replay);
    }
    *replays = occluded == nullptr;
    if (inst) {
        const int stack = trace_stack_for_depth(depth);
        const bool any = occluded != nullptr;
        if (stack == 64)
            return any ? launch_persistent<64, true, true>(bvh, r4, n, order, nullptr, occluded, d_status, stream, replay)
                       : launch_persistent<64, false, true>(bvh, r4, n, order, h4, nullptr, d_status, stream, replay);
        if (stack == 256)
            return any ? launch_persistent<256, true, true>(bvh, r4, n, order, nullptr, occluded, d_status, stream, replay)
                       : launch_persistent<256, false, true>(bvh, r4, n, order, h4, nullptr, d_status, stream, replay);
        return cudaErrorInvalidValue;
    }
    const int block = 128;
    const unsigned grid = (unsigned)((n + block - 1) / block);
    int stack = trace_stack_for_depth(depth);
    bool any = occluded != nullptr;
    if (variant == kVariantPairPersistent) {
        if (stack == 64)
            return any ? launch_persistent<64, true>(bvh, r4, n, order, nullptr, occluded, d_status, stream, replay)
                       : launch_persistent<64, false>(bvh, r4, n, order, h4, nullptr, d_status, stream, replay);
        if (stack == 256)
            return any ? launch_persistent<256, true>(bvh, r4, n, order, nullptr, occluded, d_status, stream, replay)
                       : launch_persistent<256, false>(bvh, r4, n, order, h4, nullptr, d_status, stream, replay);
        return cudaErrorInvalidValue;
    }
    if (variant == kVariantPairPacket) {
        if (stack == 64) {
            if (any)
                k_trace_packet<64, true><<<grid, block, 0, stream>>>(bvh, r4, n, order, nullptr, occluded, d_status,
                                                                     replay);
            else
                k_trace_packet<64, false><<<grid, block, 0, stream>>>(bvh, r4, n, order, h4, nullptr, d_status, replay);
        } else if (stack == 256) {
            if (any)
                k_trace_packet<256, true><<<grid, block, 0, stream>>>(bvh, r4, n, order, nullptr, occluded, d_status,
                                                                      replay);
            else
                k_trace_packet<256, false><<<grid, block, 0, stream>>>(bvh, r4, n, order, h4, nullptr, d_status,
                                                                       replay);
        } else {
            return cudaErrorInvalidValue;
        }
        return cudaGetLastError();
    }
    if (stack == 64) {
        if (any)
            k_trace<64, true><<<grid, block, 0, stream>>>(bvh, r4, n, order, nullptr, occluded, d_status, replay);
        else
            k_trace<64, false><<<grid, block, 0, stream>>>(bvh, r4, n, order, h4, nullptr, d_status, replay);
    } else if (stack == 256) {
        if (any)
            k_trace<256, true><<<grid, block, 0, stream>>>(bvh, r4, n, order, nullptr, occluded, d_status, replay);
        else
            k_trace<256, false><<<grid, block, 0, stream>>>(bvh, r4, n, order, h4, nullptr, d_status, replay);
    } else {
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

bool trace_streams(const DevBVH& bvh, const DevBVH4* wide, uint32_t wide_bound, uint32_t n) {
    read_variant();
    if (!wide || !wide_stack_variant(wide_bound) || !g_chunk || g_reorder || n > 0xF0000000u) return false;
    // scenes with instances always take the 4-wide persistent walk
    return bvh.insts != nullptr || wide_persistent();
}

// The launch of a streamed-input or write-out call: the 4-wide persistent
// walk with its shared counter (the only kernel that takes rays in order).
static cudaError_t launch_streamed(const DevBVH& bvh, const PbrtRay* rays, uint32_t n, PbrtHit* hits,
                                   uint8_t* occ, int* d_status, cudaStream_t stream, const DevBVH4* wide,
                                   uint32_t wide_bound, uint32_t* work, uint32_t* replay, StreamIn in,
                                   PbrtHit* host_hits) {
    if (!work || !trace_streams(bvh, wide, wide_bound, n) || (host_hits && occ)) return cudaErrorInvalidValue;
    const float4* r4 = reinterpret_cast<const float4*>(rays);
    float4* h4 = reinterpret_cast<float4*>(hits);
    float4* hh = reinterpret_cast<float4*>(host_hits);
    return wide_stack_variant(wide_bound) == 64
               ? launch_wide<64>(*wide, r4, n, nullptr, h4, occ, d_status, stream, true, work, replay, in, hh)
               : launch_wide<256>(*wide, r4, n, nullptr, h4, occ, d_status, stream, true, work, replay, in, hh);
}

cudaError_t launch_trace(const DevBVH& bvh, uint32_t depth, const PbrtRay* rays, uint32_t n, PbrtHit* hits,
                         uint8_t* occluded, int* d_status, cudaStream_t stream, const DevBVH4* wide,
                         uint32_t wide_bound, int kernel, const uint32_t* order, uint32_t* work, uint32_t* replay,
                         StreamIn in, PbrtHit* host_hits) {
    if (n == 0) return cudaSuccess;
    if (!replay && kernel != kTraceSmall) return cudaErrorInvalidValue;
    read_variant();
    if ((in.ready || host_hits) && order) return cudaErrorInvalidValue;
    bool replays = true;
    cudaError_t e = in.ready || host_hits
                        ? launch_streamed(bvh, rays, n, hits, occluded, d_status, stream, wide, wide_bound, work,
                                          replay, in, host_hits)
                        : launch_main(bvh, depth, rays, n, hits, occluded, d_status, stream, wide, wide_bound, kernel,
                                      order, work, replay, &replays);
    if (e != cudaSuccess || !replays) return e;
    // the replay pass (one empty launch unless a ray was marked)
    const unsigned grid = (unsigned)(device_sms() * 2);
    const float4* r4 = reinterpret_cast<const float4*>(rays);
    float4* h4 = reinterpret_cast<float4*>(hits);
    const bool inst = bvh.insts != nullptr;
    float4* hh = reinterpret_cast<float4*>(host_hits);
    auto go = [&](auto kernel) {
        kernel<<<grid, kReplayBlock, 0, stream>>>(bvh, r4, n, h4, occluded, replay, d_status, hh);
    };
    if (trace_stack_for_depth(depth) == 64)
        inst ? go(k_replay2<64, true>) : go(k_replay2<64, false>);
    else
        inst ? go(k_replay2<256, true>) : go(k_replay2<256, false>);
    return cudaGetLastError();
}

}  // namespace pbrt
