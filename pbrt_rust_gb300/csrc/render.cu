// render.cu - the SamplerRenderer wavefront on the device.
//
//   generate : one thread per sampler pixel - stratified samples, light
//              sample arrays and camera rays (sampler/stratified.rs:60-127,
//              camera/mod.rs:168-271), reading the pixel's slice of its
//              task's ChaCha12 stream
//   extend   : closest hit of every camera ray (trace.cuh)
//   shade    : dg, emitted radiance, per-light sample_l, BSDF and the
//              unoccluded contribution; shadow rays go to a compacted queue
//              (integrator/whitted.rs:30-65, light/point.rs:28-35)
//   shadow   : any hit of every queued shadow ray
//   combine  : L = Le + sum over lights of the unoccluded contributions, in
//              light order
//   film     : every film pixel gathers the samples that land on it, from
//              its own task only, in the task's sample order
//              (camera/film.rs:192-249, 175-186, 316-354)
// The library is compiled with --fmad=false and IEEE div/sqrt, so each
// step repeats the reference's f32 operations.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "wavefront.cuh"

namespace pbrt {

constexpr uint32_t kCounterWords = 16;  // 64 bytes
constexpr uint32_t kCounterWork = 4, kCounterReplay = 5;  // k_shadow4_refill's
__global__ void __launch_bounds__(128) k_generate(RenderParams P) {
    __shared__ uint32_t words[16 * 128];  // the threads' ChaCha blocks
    uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix < kCounterWords) P.counters[pix] = 0u;  // the later kernels' (a memset of its own is 4 us of stream time)
    if (pix >= P.n_pixels) return;
    generate_pixel(P, pix, words + threadIdx.x, 128u);
}

// 9 blocks per SM: 363 us for 1024 x 1024 x 16 samples and one light, 386 with
// 8, 509 with 10 (spills).
__global__ void __launch_bounds__(128, 9) k_shade(RenderParams P) {
    const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const ShadowSink Q{P.shadow_rays, P.shadow_slot, nullptr, &P.counters[0]};
    shade_sample(P, s, s < P.n_samples, Q, 0u);
}

// ---------------------------------------------------------------- shadow ---
template <int STACK, bool INST = false>
__global__ void __launch_bounds__(128) k_shadow(RenderParams P) {
    uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= *(volatile uint32_t*)&P.counters[0]) return;
    const float4* r4 = reinterpret_cast<const float4*>(P.shadow_rays);
    DRay r = make_dray(r4[2 * (size_t)q], r4[2 * (size_t)q + 1]);
    TraceResult res;
    int st = 0;
    bool occ = traverse<STACK, true, INST>(P.bvh, r, &res, &st);
    if (st) atomicMax((int*)&P.counters[2], st);
    P.occluded[P.shadow_slot[q]] = occ ? 1 : 0;
}

// k_shadow with warps of shadow rays that share their direction signs
// walked together (traverse_packet); the same answers.
template <int STACK>
__global__ void __launch_bounds__(128) k_shadow_packet(RenderParams P) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = q < *(volatile uint32_t*)&P.counters[0];  // every lane stays for the warp's votes
    const float4* r4 = reinterpret_cast<const float4*>(P.shadow_rays);
    DRay r = make_dray(active ? r4[2 * (size_t)q] : make_float4(0, 0, 0, 0),
                       active ? r4[2 * (size_t)q + 1] : make_float4(0, 0, 1, 0));
    TraceResult res;
    int st = 0;
    bool occ = false;
    if (warp_signs_uniform(r, active))
        occ = traverse_packet<STACK, true>(P.bvh, r, active, &res, &st);
    else if (active)
        occ = traverse<STACK, true>(P.bvh, r, &res, &st);
    if (!active) return;
    if (st) atomicMax((int*)&P.counters[2], st);
    P.occluded[P.shadow_slot[q]] = occ ? 1 : 0;
}

// The first per_warp lanes of each warp have a ray (rays_per_warp).
template <int OVF, bool INST>
__global__ void __launch_bounds__(128, INST ? 6 : 9)
    k_shadow4(const __grid_constant__ RenderParams P, uint32_t per_warp) {
    using Walk = Walk4<128, 16, OVF, true, INST>;
    __shared__ typename Walk::Shared sh;
    sh.init();
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t q = (uint64_t)(blockIdx.x * 4u + (threadIdx.x >> 5)) * per_warp + lane;
    if (lane >= per_warp || q >= *(volatile uint32_t*)&P.counters[0]) return;
    const float4* ray = reinterpret_cast<const float4*>(P.shadow_rays) + 2 * (size_t)q;
    int* status = (int*)&P.counters[2];
    Walk T;
    typename Walk::Ovf ov;
    T.bind(sh);
    const int st = T.start(P.bvh4, ray[0], ray[1]);
    if (st == kStartWalk) T.run(P.bvh4, sh, ov);
    const bool exact = st == kStartExact || T.gave_up();
    P.occluded[P.shadow_slot[q]] = (exact ? exact_any<OVF + 8, INST>(P.bvh, ray, status) : T.found()) ? 1 : 0;
}

// k_shadow4 with persistent warps that take kShadowChunk rays of the queue at a
// time and refill their idle lanes once kShadowRefill are idle (see
// k_trace4_persistent): the rays of a warp go to points all over an area light
// and end where they hit, so 14 of 32 lanes were active.  1024 x 1024 x 16
// terrain frame 4816 -> 4553 us, 700 x 700 x 16 into 200000 random triangles
// 3098 -> 2828 (refill at 4 / 8 / 16 lanes: 4573 / 4553 / 4649).  A ray that
// needs the exact walk is marked for k_shadow_replay.
constexpr uint32_t kShadowChunk = 64, kShadowRefill = 8;
template <int OVF, bool INST>
__global__ void __launch_bounds__(128, INST ? 6 : 8) k_shadow4_refill(const __grid_constant__ RenderParams P) {
    using Walk = Walk4<128, 16, OVF, true, INST>;
    __shared__ typename Walk::Shared sh;
    sh.init();
    const uint32_t lane = threadIdx.x & 31u, n = *(volatile uint32_t*)&P.counters[0];
    constexpr uint32_t kNone = 0xffffffffu;
    uint32_t next = 0, end = 0, ray = kNone;
    bool more = true;
    Walk T;
    typename Walk::Ovf ov;
    T.bind(sh);
    auto finish = [&](bool exact) {
        if (exact) P.counters[kCounterReplay] = 1u;
        P.occluded[P.shadow_slot[ray]] = exact ? kReplayOcc : (T.found() ? 1 : 0);
        ray = kNone;
        T.cur = kWalkDone;
    };
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, ray == kNone), nidle = (uint32_t)__popc(idle);
        if (more && next >= end && nidle >= kShadowRefill) {  // warp-uniform
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&P.counters[kCounterWork], kShadowChunk);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base < n) {
                next = base;
                end = n - base > kShadowChunk ? base + kShadowChunk : n;
            } else {
                more = false;
            }
        }
        const bool tail = !more && end - next <= nidle;
        if (next < end && nidle >= (tail ? 1u : kShadowRefill)) {
            if (ray == kNone) {
                const uint32_t k = (uint32_t)__popc(idle & ((1u << lane) - 1u));
                if (k < end - next) {
                    ray = next + k;
                    const float4* r = reinterpret_cast<const float4*>(P.shadow_rays) + 2 * (size_t)ray;
                    const int st = T.start(P.bvh4, __ldg(r), __ldg(r + 1));
                    if (st != kStartWalk) finish(st == kStartExact);
                }
            }
            next += min(nidle, end - next);
        }
        if (!__any_sync(0xffffffffu, ray != kNone)) {
            if (next >= end && !more) break;
            continue;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if ((int32_t)T.cur >= 0) T.node(P.bvh4, ov);
        if ((int32_t)T.cur < 0 && T.cur != kWalkDone) T.leaf(P.bvh4, sh, ov);
        if (T.cur == kWalkDone && ray != kNone && !T.resume(ov)) finish(T.gave_up());
    }
}
template <int STACK, bool INST>
__global__ void __launch_bounds__(128) k_shadow_replay(const __grid_constant__ RenderParams P) {
    if (*(volatile uint32_t*)&P.counters[kCounterReplay] == 0u) return;
    const uint32_t n = *(volatile uint32_t*)&P.counters[0];
    for (uint32_t q = blockIdx.x * 128u + threadIdx.x; q < n; q += gridDim.x * 128u) {
        uint8_t* occ = P.occluded + P.shadow_slot[q];
        if (*occ == kReplayOcc)
            *occ = exact_any<STACK, INST>(P.bvh, reinterpret_cast<const float4*>(P.shadow_rays) + 2 * (size_t)q,
                                          (int*)&P.counters[2]) ? 1 : 0;
    }
}
// Where that pays: frames and trees so large that the walks, not their start
// and the tail of the last warps, take the time.  Frame time without / with it, us, at
// n = samples x lights: 17000 random triangles n = 4.3M 916 / 886, 5000 n = 6.5M
// 843 / 853, 20000 n = 2.2M 573 / 573, 200000 n = 1.6M 599 / 610; terrains of 10000
// n = 7.8M 1610 / 1667, 50000 n = 7.8M 1864 / 1866, 300000 n = 2.4M 853 / 864 and
// 3.9M 1395 / 1382.  With instances, by n alone (the definitions' sizes are not
// the scene's): n = 0.7M 421 / 435, 1.3M 569 / 560, 1.6M 678 / 633, 11.5M 3466 /
// 3158.
static bool shadow_refills(const RenderParams& P, uint64_t max_shadow) {
    const uint64_t from = P.bvh.insts ? 3ull << 19 : 1ull << 22;
    return max_shadow >= from && max_shadow < 0xF0000000ull && (P.bvh.insts || P.bvh.n_prims >= 16384u);
}
template <int OVF, bool INST>
static cudaError_t launch_shadow_refill(const RenderParams& P, uint64_t max_shadow, cudaStream_t s) {
    static ShapeCache bps_cache;
    const uint64_t resident = (uint64_t)device_sms() * resident_blocks(bps_cache, k_shadow4_refill<OVF, INST>, 128, 0);
    const uint64_t chunks = (max_shadow + 4 * kShadowChunk - 1) / (4 * kShadowChunk);
    k_shadow4_refill<OVF, INST><<<(unsigned)std::min(resident, chunks), 128, 0, s>>>(P);
    k_shadow_replay<OVF + 8, INST><<<(unsigned)device_sms(), 128, 0, s>>>(P);
    return cudaGetLastError();
}

// --------------------------------------------------------------- combine ---
__global__ void __launch_bounds__(256) k_combine(RenderParams P) {
    const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.n_samples) return;
    combine_sample(P, s);
}

// ------------------------------------------------------------------ film ---
__global__ void __launch_bounds__(128) k_film(RenderParams P) {
    const int32_t fw = P.fx1 - P.fx0, fh = P.fy1 - P.fy0;
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (uint32_t)(fw * fh)) return;
    film_pixel(P, idx);
}

// ------------------------------------------------------ sampler stream ---
// The sampler's ChaCha code, run on its own so that it can be compared with
// other implementations: thread i computes block ctr0 + i, 16 words a block.
struct Key8 {
    uint32_t k[8];
};
template <int DR>
__global__ void __launch_bounds__(128) k_chacha_blocks(Key8 key, uint64_t ctr0, uint64_t sid, uint32_t n_blocks,
                                                       uint32_t* out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_blocks) return;
    chacha12_block<DR>(key.k, ctr0 + i, out + 16ull * i, 1u, sid);
}

// Words [first, first + n) of one task's stream as generate_pixel reads
// them: thread t reads the seg words from first + t * seg (the last one
// fewer) through its window, block by block.
__global__ void __launch_bounds__(128) k_rng_words(Key8 key, uint64_t first, uint32_t n, uint32_t seg,
                                                   uint32_t* out) {
    __shared__ uint32_t words[16 * 128];
    const uint64_t lo = (uint64_t)(blockIdx.x * blockDim.x + threadIdx.x) * seg;
    if (lo >= n) return;
    const uint64_t hi = lo + seg < n ? lo + seg : n;
    WordWindow rng(key.k, words + threadIdx.x, 128u);
    for (uint64_t w = lo; w < hi;) {
        rng.load(first + w);
        do {
            out[w] = rng.word(first + w);
            ++w;
        } while (w < hi && ((first + w) & 15u));
    }
}

// ------------------------------------------------------------ launchers ---
static inline unsigned blocks_for(uint64_t n, int b) { return (unsigned)((n + b - 1) / b); }

cudaError_t launch_chacha_blocks(const uint32_t key[8], uint64_t ctr, uint64_t sid, uint32_t rounds, uint32_t n_blocks,
                                 uint32_t* d_out, cudaStream_t s) {
    Key8 k;
    for (int i = 0; i < 8; ++i) k.k[i] = key[i];
    const unsigned grid = blocks_for(n_blocks, 128);
    if (!grid) return cudaSuccess;
    if (rounds == 8)
        k_chacha_blocks<4><<<grid, 128, 0, s>>>(k, ctr, sid, n_blocks, d_out);
    else if (rounds == 12)
        k_chacha_blocks<6><<<grid, 128, 0, s>>>(k, ctr, sid, n_blocks, d_out);
    else if (rounds == 20)
        k_chacha_blocks<10><<<grid, 128, 0, s>>>(k, ctr, sid, n_blocks, d_out);
    else
        return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_rng_words(const uint32_t key[8], uint64_t first, uint32_t n, uint32_t seg, uint32_t* d_out,
                             cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    if (seg == 0) return cudaErrorInvalidValue;
    Key8 k;
    for (int i = 0; i < 8; ++i) k.k[i] = key[i];
    k_rng_words<<<blocks_for(((uint64_t)n + seg - 1) / seg, 128), 128, 0, s>>>(k, first, n, seg, d_out);
    return cudaGetLastError();
}

cudaError_t launch_render(const RenderParams& P, cudaStream_t s) {
    cudaError_t e;
    if (P.n_pixels) {
        k_generate<<<blocks_for(P.n_pixels, 128), 128, 0, s>>>(P);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    } else if ((e = cudaMemsetAsync(P.counters, 0, 4 * kCounterWords, s)) != cudaSuccess) {
        return e;
    }
    if (P.n_samples) {
        // camera rays of neighbouring pixels are coherent: one thread per
        // ray keeps them together in a warp
        const int rk = render_trace_kernel(P.bvh.n_prims);
        e = launch_trace(P.bvh, P.depth, P.rays, (uint32_t)P.n_samples, reinterpret_cast<PbrtHit*>(P.hits), nullptr,
                         (int*)&P.counters[2], s, P.has_wide ? &P.bvh4 : nullptr, P.wide_bound, rk, nullptr, nullptr,
                         &P.counters[3]);
        if (e != cudaSuccess) return e;
        k_shade<<<blocks_for(P.n_samples, 128), 128, 0, s>>>(P);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        uint64_t max_shadow = P.n_samples * P.n_lights;
        if (max_shadow) {
            const uint32_t pw = rays_per_warp(max_shadow);
            const unsigned grid4 = blocks_for(max_shadow, 4 * (int)pw);
            // scenes with instances: the 4-wide walk with instances when a
            // variant covers its stack bound, else the binary one
            const bool inst = P.bvh.insts != nullptr;
            const int iv = (inst && P.has_wide) ? wide_stack_variant(P.wide_bound) : 0;
            const bool wide_rk =
                rk == PBRT_TRACE_WIDE || rk == PBRT_TRACE_WIDE_PERSISTENT || rk == PBRT_TRACE_WIDE_SPECULATIVE;
            int wv = (P.has_wide && wide_rk && !inst) ? wide_stack_variant(P.wide_bound) : 0;
            const bool refill = shadow_refills(P, max_shadow);
            if (refill && (iv == 64 || wv == 64))
                e = iv ? launch_shadow_refill<64, true>(P, max_shadow, s)
                       : launch_shadow_refill<64, false>(P, max_shadow, s);
            else if (refill && (iv == 256 || wv == 256))
                e = iv ? launch_shadow_refill<256, true>(P, max_shadow, s)
                       : launch_shadow_refill<256, false>(P, max_shadow, s);
            else if (iv == 64)
                k_shadow4<64, true><<<grid4, 128, 0, s>>>(P, pw);
            else if (iv == 256)
                k_shadow4<256, true><<<grid4, 128, 0, s>>>(P, pw);
            else if (inst && trace_stack_for_depth(P.depth) == 64)
                k_shadow<64, true><<<blocks_for(max_shadow, 128), 128, 0, s>>>(P);
            else if (inst)
                k_shadow<256, true><<<blocks_for(max_shadow, 128), 128, 0, s>>>(P);
            else if (rk == PBRT_TRACE_PAIR_PACKET && trace_stack_for_depth(P.depth) == 64)
                k_shadow_packet<64><<<blocks_for(max_shadow, 128), 128, 0, s>>>(P);
            else if (rk == PBRT_TRACE_PAIR_PACKET)
                k_shadow_packet<256><<<blocks_for(max_shadow, 128), 128, 0, s>>>(P);
            else if (wv == 64)
                k_shadow4<64, false><<<grid4, 128, 0, s>>>(P, pw);
            else if (wv == 256)
                k_shadow4<256, false><<<grid4, 128, 0, s>>>(P, pw);
            else if (trace_stack_for_depth(P.depth) == 64)
                k_shadow<64><<<blocks_for(max_shadow, 128), 128, 0, s>>>(P);
            else
                k_shadow<256><<<blocks_for(max_shadow, 128), 128, 0, s>>>(P);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
        k_combine<<<blocks_for(P.n_samples, 256), 256, 0, s>>>(P);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    uint64_t npx = (uint64_t)(P.fx1 - P.fx0) * (uint64_t)(P.fy1 - P.fy0);
    if (npx) {
        k_film<<<blocks_for(npx, 128), 128, 0, s>>>(P);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace pbrt
