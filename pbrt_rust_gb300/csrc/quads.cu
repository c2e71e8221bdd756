// quads.cu - the 4-wide layout (layout.h: QuadNode) encoded from the binary
// one.  One thread per binary pair that starts a 4-wide node: the boxes of
// its grandchildren are all in it and its two children's pairs.  The grid
// arithmetic runs in 64 bits, so that a plane's rounding direction is decided
// on (nearly) exact values; what the 64-bit form rounds is far below the
// margin the walk gives every plane (trace4.cuh).
#include <cuda_runtime.h>

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

__device__ __forceinline__ int code_down(double org, double s, float x) {
    const double v = ((double)x - org) / s;
    int c = v < 256.0 ? (int)floor(v) - 128 : (int)floor(v * 0.5);
    c = min(max(c, 0), 255);
    while (c > 0 && org + code_value(c) * s > (double)x) --c;
    return c;
}
__device__ __forceinline__ int code_up(double org, double s, float x) {
    const double v = ((double)x - org) / s;
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
        q.order |= (((oct >> axis[0]) & 1u) | (((oct >> axis[1]) & 1u) << 1) | (((oct >> axis_n) & 1u) << 2)) << (3 * oct);
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
        for (int k = 0; k < 4; ++k) {
            // an empty slot: lower planes above the upper ones
            const int cl = kid[k] ? code_down(org[ax], scale[ax], (&kid[k]->lo_x)[ax]) : 255;
            const int ch = kid[k] ? code_up(org[ax], scale[ax], (&kid[k]->hi_x)[ax]) : 0;
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

}  // namespace pbrt
