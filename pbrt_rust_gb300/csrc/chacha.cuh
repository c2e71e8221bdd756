// chacha.cuh - the reference RNG stream on the device.
//
// src/rng.rs wraps rand 0.8.5's StdRng, which is ChaCha with 12 rounds
// (rand_chacha 0.3.1): 16-word state of the four constants, the 8-word key,
// a 64-bit block counter (words 12-13) and a zero 64-bit stream id (words
// 14-15); output words are the keystream words in order.  Because the
// keystream is a function of the block counter, a thread seeks directly to
// the first word of its pixel instead of replaying the task's stream.
// The key is expanded on the host from the task index (rand_core 0.6.4
// seed_from_u64, see host_scene.cpp).
#pragma once
#include <stdint.h>

namespace pbrt {

__device__ __forceinline__ uint32_t rotl32(uint32_t v, int c) { return __funnelshift_l(v, v, c); }

#define PBRT_QR(a, b, c, d) \
    a += b;                 \
    d ^= a;                 \
    d = rotl32(d, 16);      \
    c += d;                 \
    b ^= c;                 \
    b = rotl32(b, 12);      \
    a += b;                 \
    d ^= a;                 \
    d = rotl32(d, 8);       \
    c += d;                 \
    b ^= c;                 \
    b = rotl32(b, 7);

// out[k * stride] = keystream word k of block `ctr`.  DR double rounds (6:
// ChaCha12, StdRng's cipher) and stream id `sid` (0 for StdRng) are
// parameters only so that the same code can be checked against other
// ChaCha implementations (pbrtgpu_chacha_blocks); the sampler uses the
// defaults.
template <int DR = 6>
__device__ __forceinline__ void chacha12_block(const uint32_t* key, uint64_t ctr, uint32_t* out, uint32_t stride,
                                               uint64_t sid = 0) {
    const uint32_t s14 = (uint32_t)sid, s15 = (uint32_t)(sid >> 32);
    uint32_t x0 = 0x61707865u, x1 = 0x3320646eu, x2 = 0x79622d32u, x3 = 0x6b206574u;
    uint32_t x4 = key[0], x5 = key[1], x6 = key[2], x7 = key[3];
    uint32_t x8 = key[4], x9 = key[5], x10 = key[6], x11 = key[7];
    uint32_t x12 = (uint32_t)ctr, x13 = (uint32_t)(ctr >> 32), x14 = s14, x15 = s15;
#pragma unroll
    for (int r = 0; r < DR; ++r) {
        PBRT_QR(x0, x4, x8, x12);
        PBRT_QR(x1, x5, x9, x13);
        PBRT_QR(x2, x6, x10, x14);
        PBRT_QR(x3, x7, x11, x15);
        PBRT_QR(x0, x5, x10, x15);
        PBRT_QR(x1, x6, x11, x12);
        PBRT_QR(x2, x7, x8, x13);
        PBRT_QR(x3, x4, x9, x14);
    }
    out[0u * stride] = x0 + 0x61707865u;
    out[1u * stride] = x1 + 0x3320646eu;
    out[2u * stride] = x2 + 0x79622d32u;
    out[3u * stride] = x3 + 0x6b206574u;
    out[4u * stride] = x4 + key[0];
    out[5u * stride] = x5 + key[1];
    out[6u * stride] = x6 + key[2];
    out[7u * stride] = x7 + key[3];
    out[8u * stride] = x8 + key[4];
    out[9u * stride] = x9 + key[5];
    out[10u * stride] = x10 + key[6];
    out[11u * stride] = x11 + key[7];
    out[12u * stride] = x12 + (uint32_t)ctr;
    out[13u * stride] = x13 + (uint32_t)(ctr >> 32);
    out[14u * stride] = x14 + s14;
    out[15u * stride] = x15 + s15;
}
#undef PBRT_QR

// A thread's window on its task's word stream: one block at a time, in the
// caller's shared-memory column of 16 words (word k at buf[k * stride]; a
// per-thread array would go to local memory).  Readers load a block at one
// place in a loop and then use up the words of it that they need, so the
// lanes of a warp compute their blocks together although their positions
// inside a block differ: with a reader that computed a block whenever a word
// of it was asked for, lanes at different positions did so one after the
// other (1.77M blocks for 512 x 512 x 4 samples and two lights: the sampler
// 120 us, now 71).
struct WordWindow {
    uint32_t key[8];
    uint32_t* buf;
    uint32_t stride;

    __device__ __forceinline__ WordWindow(const uint32_t* k, uint32_t* column, uint32_t column_stride)
        : buf(column), stride(column_stride) {
#pragma unroll
        for (int i = 0; i < 8; ++i) key[i] = k[i];
    }
    // Loads the block that holds word w.
    __device__ __forceinline__ void load(uint64_t w) { chacha12_block(key, w >> 4, buf, stride); }
    // Word w of the block loaded last.
    __device__ __forceinline__ uint32_t word(uint64_t w) const { return buf[(uint32_t)(w & 15u) * stride]; }
    // rng.rs:15-17 - gen::<f32>(): (u32 >> 8) * 2^-24
    __device__ __forceinline__ float unit(uint64_t w) const { return (float)(word(w) >> 8) * (1.0f / 16777216.0f); }
};

// v % d for v = hi:lo and 1 <= d <= 64, where the RNG's random_uint is
// v % usize::MAX (rng.rs:19-21).
__device__ __forceinline__ uint32_t random_index(uint32_t lo, uint32_t hi, uint32_t d) {
    if ((lo & hi) == 0xffffffffu) return 0u;  // usize::MAX % usize::MAX
    uint32_t r = hi % d;
    r = ((r << 16) | (lo >> 16)) % d;
    return ((r << 16) | (lo & 0xffffu)) % d;
}

}  // namespace pbrt
