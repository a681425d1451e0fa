// A thread a row of 128 x 64 scores in tensor memory: what the two prompt attentions on tcgen05 share. Weights go back over
// the scores as two bf16 numbers each (16 bits), so that the values product takes them from tensor memory.
#pragma once

#include "typed.cuh"
#include "umma.cuh"

namespace leankv {

constexpr int kTile = 128;                       // rows of a CTA
constexpr int kKeys = 64;                        // keys of a tile
constexpr uint32_t kBlock = kTile * 128;         // 128 rows of 64 columns: 16 KB
constexpr uint32_t kKeyBlock = kKeys * 128;      // 64 keys of 64 columns: 8 KB
constexpr float kSlack = 8.f;                    // outputs are rescaled when a row's maximum grows by more than 2^kSlack

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two floats at a time.
struct Two { float x, y; };
__device__ __forceinline__ Two fma2(Two a, Two b, Two c) {
    Two d;
    asm("{\n\t.reg .b64 a, b, c, d;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ Two add2(Two a, Two b) {
    Two d;
    asm("{\n\t.reg .b64 a, b, d;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "add.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

__device__ __forceinline__ float largest(const uint32_t (&s)[2][32]) {
    float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int x = 0; x < 32; ++x) top[x & 3] = fmaxf(top[x & 3], __uint_as_float(s[c][x]));
    return fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
}

// Scores of this thread's row (lane row0 + lane id) become weights 2^(s c - m) at `tm`; their sum.
__device__ __forceinline__ float put_weights(const uint32_t (&s)[2][32], float c, float m, uint32_t tm, int row0) {
    Two sum[2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        uint32_t ph[16], pl[16];
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
            Two w = fma2({__uint_as_float(s[b][x]), __uint_as_float(s[b][x + 1])}, {c, c}, {-m, -m});
            w.x = ex2(w.x);
            w.y = ex2(w.y);
            sum[(x >> 1) & 1] = add2(sum[(x >> 1) & 1], w);
            const uint32_t hi = pack_bf16(w.x, w.y);
            const Two left = add2(w, {-__uint_as_float(hi << 16), -__uint_as_float(hi & 0xffff0000u)});
            ph[x / 2] = hi;
            pl[x / 2] = pack_bf16(left.x, left.y);
        }
        umma::st16_async(ph, tm, row0, b * 32);
        umma::st16_async(pl, tm, row0, b * 32 + 16);
    }
    return (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
}

__device__ __forceinline__ void scale_outputs(uint32_t tm_o, int row0, int cols, float f) {
#pragma unroll 1
    for (int c = 0; c < cols; c += 32) {
        uint32_t o[32];
        umma::ld32(o, tm_o, row0, c);
#pragma unroll
        for (int x = 0; x < 32; ++x) o[x] = __float_as_uint(__uint_as_float(o[x]) * f);
        umma::st32(o, tm_o, row0, c);
    }
}

}  // namespace leankv
