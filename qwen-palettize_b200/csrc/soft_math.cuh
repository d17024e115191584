// Per-weight arithmetic of the Gumbel-Softmax relaxation, shared by the pass that builds W_soft and by the gradient epilogue so that forward and
// backward see identical numbers (soft_tensors.cu has steps of its own, for tensors that a caller asks for: their last bits may differ).
//
// Semantics follow the reference's PyTorch/Triton path:
//   P = softmax((logits + g) / tau) in fp32, max-subtracted   (scripts/triton_soft_forward.py:119-141)
//   W_soft = sum_p P[p] * palette[p]                          (scripts/bench_triton_kernels.py:77-78)
//   hard index = argmax over the *plain* logits, ties -> lowest index (scripts/triton_soft_forward.py:160-168)
//   dLogits[p] = dW * P[p] * (palette[p] - W_soft), no 1/tau   (scripts/bench_triton_kernels.py:108-111)
//   dPalette[p] += dW * P[p]                                   (scripts/bench_triton_kernels.py:114-118)
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace plz {

enum NoiseMode { NOISE_NONE = 0, NOISE_TENSOR = 1, NOISE_HASH = 2 };

// Two fp32 numbers in a register pair: Blackwell adds, multiplies and fuses them by one instruction.
typedef uint64_t f32x2;
__device__ __forceinline__ f32x2 pair2(float a, float b) { f32x2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b)); return d; }
__device__ __forceinline__ void split2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ float exp2_approx(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// Counter-based Gumbel(0,1) samples of the four entries of a weight, added to s: the 32-bit hash-LCG of the reference sampler
// (scripts/fused_lut_kernel.cu:1245-1256), integer part bit-exact (its low 24 bits come out shifted up by eight, exact as a float either way);
// the float part, -log(-log(u)), is the device's log2 scaled, so values agree with the reference to a few ulp.
__device__ __forceinline__ void add_gumbel_hash(f32x2 (&s)[2], uint32_t seed, uint32_t first) {
    float u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t x = seed ^ ((first + q) * 0x9E3779B9u);
        x ^= x >> 13;
        x = x * 1103515245u + 12345u;
        x ^= x >> 17;
        x = x * (1103515245u << 8) + (12345u << 8);
        u[q] = __uint2float_rn(x);
    }
    constexpr float kLn2 = 0.69314718056f, kUnit = 1.0f / 4294967296.0f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        float a, b;
        split2(mul2(pair2(u[2 * i], u[2 * i + 1]), pair2(kUnit, kUnit)), a, b);
        split2(mul2(pair2(__log2f(fmaxf(a, 1e-7f)), __log2f(fmaxf(b, 1e-7f))), pair2(-kLn2, -kLn2)), a, b);
        s[i] = fma2(pair2(__log2f(a), __log2f(b)), pair2(-kLn2, -kLn2), s[i]);
    }
}

__device__ __forceinline__ int argmax4_first(float a, float b, float c, float d) {
    int i = 0;
    float m = a;
    if (b > m) { m = b; i = 1; }
    if (c > m) { m = c; i = 2; }
    if (d > m) { m = d; i = 3; }
    return i;
}

struct Soft4 {
    f32x2 P[2];
    float w_soft;
};

// s: logits plus noise; c: palette entries in fp32; scale: soft_scale(tau). exp(x / tau) is 2 to the scaled x. The largest is subtracted before anything is
// scaled: of logits of any size the largest then weighs exactly 1, where a product that is rounded, or overflows, by itself would leave its error as an
// exponent (one instruction less; a step of 1000 tokens through 9728 x 2560 353 against 354 us). Pairs in place of single numbers took the weight gradient's
// epilogue from 150 to 105 instructions per weight.
__device__ __forceinline__ Soft4 soft4(const f32x2 (&s)[2], const f32x2 (&c)[2], float scale) {
    float x[4], e[4];
    split2(s[0], x[0], x[1]);
    split2(s[1], x[2], x[3]);
    const float top = -fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        split2(mul2(add2(s[i], pair2(top, top)), pair2(scale, scale)), e[2 * i], e[2 * i + 1]);
        e[2 * i] = exp2_approx(e[2 * i]);
        e[2 * i + 1] = exp2_approx(e[2 * i + 1]);
    }
    const f32x2 e01 = pair2(e[0], e[1]), e23 = pair2(e[2], e[3]);
    float a, b;
    split2(add2(e01, e23), a, b);
    const float inv = __fdividef(1.0f, a + b);
    Soft4 r;
    r.P[0] = mul2(e01, pair2(inv, inv));
    r.P[1] = mul2(e23, pair2(inv, inv));
    split2(fma2(r.P[1], c[1], mul2(r.P[0], c[0])), a, b);
    r.w_soft = a + b;
    return r;
}
__host__ __device__ inline float soft_scale(float tau) { return (float)(1.4426950408889634 / (double)tau); }

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__half v) { return __half2float(v); }
__device__ __forceinline__ void from_f32(float& d, float v) { d = v; }
__device__ __forceinline__ void from_f32(__half& d, float v) { d = __float2half_rn(v); }

}  // namespace plz
