// Attention of one new token per sequence against a key / value cache (token decode), and the embedding-row gather that
// opens a forward pass. Both are single passes that should be bound by HBM: a decode step reads every cached key and value once
// (B * T * Hkv * 128 * 2 * 2 bytes per layer).
//
//   attn_decode_mma_kernel  bf16, head sizes above 64 and up to 128, long caches or many sequences. With scores and sums on FMAs (the kernel below) a step of 64 sequences over 1025
//     tokens of 8 key / value heads issued about 1000 instructions per 16 tokens and warp and took 68 us for 268 MB, bound by issue. Here the
//     scores are mma.sync m16n8k16 (A = the query heads of the group, 4 of 16 rows used; B = 8 keys straight from memory, the order of
//     the dimensions permuted alike on both sides so that a lane's operands are whole 16-byte loads): products of bf16 are exact and sums
//     are fp32 as before. The weights stay fp32: they pass through shared memory (16 tokens x 4 heads per warp and step) to the lanes that
//     hold the values, and weight x value runs on packed fp32 pairs.
//     Keys and values are requested one step ahead. 69 -> 51 us (5.3 TB/s); one sequence of 2049 tokens 6.2 -> 5.5 us.
//   attn_decode_partial_kernel  the other types and sizes, and few cached tokens: grid (splits, Hkv, B), 4 warps. The sequence is cut into `splits` contiguous chunks so that
//     the launch has a few CTAs per SM whatever B is. Inside a CTA a warp takes 8 tokens per step: 16 lanes per token, each
//     lane the 16 bytes (8 dims) of the key and of the value row that belong to it, so one load instruction of a warp covers
//     two whole 256-byte rows, and four such loads for K and four for V are in flight per lane before anything is used. The
//     up-to-4 query heads of the group share every key / value byte. The 16 partial scores of a step (4 heads x 4 token
//     slots) are summed over the 16 lanes by recursive halving (15 shuffles, after which lane i owns score i), so exp2 is
//     evaluated once per score; online softmax (running max and sum per head) across steps; the warps' partial results meet in
//     shared memory. With one split the CTA writes the bf16 output itself, else an unnormalised fp32 partial (o, max, sum).
//     Both kernels share the grid, the split and the merge.
//   attn_decode_combine_kernel  merges the splits.
//
// Template parameters widen it: element type (bf16, fp32), lanes per token (8, 16, 32: head sizes up to 64, 128, 256, key and value
// sizes independent), and EXT, which takes the length from device memory (a captured step replays at any position), adds a bias by
// distance to the scores and a sink (score 0, no value) to the denominator.
//
// The reference has no attention code (it calls the HuggingFace layer, scripts/qwen_model.py:454 selects SDPA); semantics are
// those of transformers' Qwen3Attention at q_len = 1 with a DynamicCache: softmax over all T cached positions, no mask.
#include "plz_launch.h"

namespace plz {
namespace {

constexpr float kLog2eDec = 1.4426950408889634f;
constexpr float kNegBig = -1.0e30f;
constexpr int kDecWarps = 4;
constexpr int kStepTokens = 8;                     // tokens of one warp step
constexpr int kCtaStep = kDecWarps * kStepTokens;  // tokens a CTA advances per step of its warps
constexpr int kMaxSplits = 128;

struct DecParams {
    const void* q; long long ldq;
    const void* k; const void* v; long long k_batch, v_batch, k_tok, v_tok;   // elements between sequences / positions
    void* out; long long ldo;
    float* ws_o; float* ws_ml;       // [B, Hq, splits, dv] and [B, Hq, splits, 2]
    int T, Hq, Hkv, chunk, splits;
    int group, passes;                       // Hq / Hkv; launches of up to four query heads of a group, side by side in the grid
    float scale_log2e;
    // EXT only: head sizes, device-side length, bias by distance, sink
    int dk, dv;
    const int* pos;                          // the new token's position; T = *pos + 1
    const float* bias; long long ldb; int n_bias;
    int sink;
};

__device__ __forceinline__ float ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// eight consecutive cached elements of a lane
template <typename T> struct Chunk;
template <> struct Chunk<__nv_bfloat16> {
    uint4 r;
    __device__ __forceinline__ void zero() { r = make_uint4(0u, 0u, 0u, 0u); }
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { r = __ldcs(reinterpret_cast<const uint4*>(p)); }
    __device__ __forceinline__ void unpack(float (&f)[8]) const {
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { f[2 * i] = __uint_as_float(w[i] << 16); f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u); }
    }
};
template <> struct Chunk<float> {
    float4 a, b;
    __device__ __forceinline__ void zero() { a = make_float4(0.f, 0.f, 0.f, 0.f); b = a; }
    __device__ __forceinline__ void load(const float* p) { a = __ldcs(reinterpret_cast<const float4*>(p)); b = __ldcs(reinterpret_cast<const float4*>(p + 4)); }
    __device__ __forceinline__ void unpack(float (&f)[8]) const {
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
};
__device__ __forceinline__ void store_elem(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
__device__ __forceinline__ void store_elem(float* p, float v) { *p = v; }

// the warps' partial results of a CTA, unnormalised (o, max, sum) per head: thread d takes dimension d (and d + 128) of every head
template <typename T, bool EXT, int D>
__device__ __forceinline__ void merge_warps(const DecParams& p, const float (&sm_o)[kDecWarps][4][D], const float (&sm_ml)[kDecWarps][4][2], int split, int b,
                                            int head0, int G, int dv) {
    for (int d = threadIdx.x; d < dv; d += kDecWarps * 32) {
        for (int g = 0; g < G; ++g) {
            float M = kNegBig;
#pragma unroll
            for (int w = 0; w < kDecWarps; ++w) M = fmaxf(M, sm_ml[w][g][0]);
            const bool sink = EXT && p.sink && p.splits == 1;
            if (sink) M = fmaxf(M, 0.f);
            float acc = 0.f, l = sink ? ex2(-M) : 0.f;
#pragma unroll
            for (int w = 0; w < kDecWarps; ++w) {
                const float c = ex2(sm_ml[w][g][0] - M);
                acc = fmaf(c, sm_o[w][g][d], acc);
                l = fmaf(c, sm_ml[w][g][1], l);
            }
            const int head = head0 + g;
            if (p.splits == 1) {
                store_elem((T*)p.out + (long long)b * p.ldo + (long long)head * dv + d, l > 0.f ? acc / l : 0.f);
            } else {
                const long long slot = ((long long)b * p.Hq + head) * p.splits + split;
                p.ws_o[slot * dv + d] = acc;
                if (d == 0) { p.ws_ml[slot * 2] = M; p.ws_ml[slot * 2 + 1] = l; }
            }
        }
    }
}

// T: element type; LPT: lanes per token (head sizes up to 8 * LPT); EXT: the head sizes, bias, sink and length of the params
template <typename T, int LPT, bool EXT>
__global__ void __launch_bounds__(kDecWarps * 32)
attn_decode_partial_kernel(const DecParams p) {
    constexpr int U = LPT / 4;                      // token groups of a step: U * (32 / LPT) = 8 tokens
    constexpr int D = 8 * LPT;
    __shared__ float sm_o[kDecWarps][4][D];
    __shared__ float sm_ml[kDecWarps][4][2];
    const int split = blockIdx.x, hk = blockIdx.y / p.passes, g0 = (blockIdx.y % p.passes) * 4, b = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tl = lane / LPT, dl = lane % LPT;
    const int G = min(4, p.group - g0);
    const int head0 = hk * p.group + g0;            // first q head of this CTA's part of the group
    const int dk = EXT ? p.dk : 128, dv = EXT ? p.dv : 128;
    const bool in_k = !EXT || dl * 8 < dk, in_v = !EXT || dl * 8 < dv;
    pdl_launch_dependents();
    pdl_wait();
    const int T_all = EXT ? *p.pos + 1 : p.T;
    int chunk = p.chunk;
    if (EXT) chunk = ((T_all + p.splits - 1) / p.splits + kCtaStep - 1) / kCtaStep * kCtaStep;
    const int t0 = split * chunk, t1 = min(T_all, t0 + chunk);

    float q[4][8];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        Chunk<T> r;
        r.zero();
        if (g < G && in_k) r.load((const T*)p.q + (long long)b * p.ldq + (long long)(head0 + g) * dk + dl * 8);
        r.unpack(q[g]);
#pragma unroll
        for (int d = 0; d < 8; ++d) q[g][d] *= p.scale_log2e;
    }
    float o[4][8];
#pragma unroll
    for (int g = 0; g < 4; ++g)
#pragma unroll
        for (int d = 0; d < 8; ++d) o[g][d] = 0.f;
    float m_own = kNegBig, l_own = 0.f;             // of head dl / U, this lane's share of the sum
    const T* kb = (const T*)p.k + (long long)b * p.k_batch + (long long)hk * dk + dl * 8;
    const T* vb = (const T*)p.v + (long long)b * p.v_batch + (long long)hk * dv + dl * 8;
    const int u_own = dl % U, g_own = dl / U;
    const float* brow = nullptr;
    if (EXT && p.bias && g_own < G) brow = p.bias + (long long)(head0 + g_own) * p.ldb;

    for (int base = t0 + warp * kStepTokens; base < t1; base += kCtaStep) {
        Chunk<T> kr[U], vr[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = base + (32 / LPT) * u + tl;
            kr[u].zero(); vr[u].zero();
            if (t < t1) {
                if (in_k) kr[u].load(kb + (long long)t * p.k_tok);
                if (in_v) vr[u].load(vb + (long long)t * p.v_tok);
            }
        }
        float val[LPT];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float kf[8];
            kr[u].unpack(kf);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                float s = 0.f;
#pragma unroll
                for (int d = 0; d < 8; ++d) s = fmaf(q[g][d], kf[d], s);
                val[g * U + u] = s;
            }
        }
        // sum over the LPT lanes of a token by recursive halving: afterwards lane dl holds the total of val[dl]
#pragma unroll
        for (int half = LPT / 2; half >= 1; half >>= 1) {
            const bool up = (dl & half) != 0;
#pragma unroll
            for (int i = 0; i < half; ++i) {
                const float send = up ? val[i] : val[i + half];
                const float keep = up ? val[i + half] : val[i];
                val[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, half);
            }
        }
        const int t_own = base + (32 / LPT) * u_own + tl;
        const bool ok = t_own < t1;
        float s = ok ? val[0] : kNegBig;
        if (EXT && ok && brow) s = fmaf(__ldg(brow + min(T_all - 1 - t_own, p.n_bias - 1)), kLog2eDec, s);
        float mx = s;
#pragma unroll
        for (int i = 1; i < U; i <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, i));
#pragma unroll
        for (int i = LPT; i < 32; i <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, i));
        const float m_new = fmaxf(m_own, mx);
        const float corr = ex2(m_own - m_new);
        const float pr = ok ? ex2(s - m_new) : 0.f;
        l_own = l_own * corr + pr;
        m_own = m_new;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const float cg = __shfl_sync(0xFFFFFFFFu, corr, g * U);
#pragma unroll
            for (int d = 0; d < 8; ++d) o[g][d] *= cg;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float vf[8];
            vr[u].unpack(vf);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const float pgu = __shfl_sync(0xFFFFFFFFu, pr, tl * LPT + g * U + u);
#pragma unroll
                for (int d = 0; d < 8; ++d) o[g][d] = fmaf(pgu, vf[d], o[g][d]);
            }
        }
    }
    // the token slots of a warp, then the sum of a head over its lanes
#pragma unroll
    for (int i = LPT; i < 32; i <<= 1) {
#pragma unroll
        for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int d = 0; d < 8; ++d) o[g][d] += __shfl_xor_sync(0xFFFFFFFFu, o[g][d], i);
        l_own += __shfl_xor_sync(0xFFFFFFFFu, l_own, i);
    }
#pragma unroll
    for (int i = 1; i < U; i <<= 1) l_own += __shfl_xor_sync(0xFFFFFFFFu, l_own, i);
    if (tl == 0) {
#pragma unroll
        for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int d = 0; d < 8; ++d) sm_o[warp][g][dl * 8 + d] = o[g][d];
        if (u_own == 0) { sm_ml[warp][g_own][0] = m_own; sm_ml[warp][g_own][1] = l_own; }
    }
    __syncthreads();
    merge_warps<T, EXT, D>(p, sm_o, sm_ml, split, b, head0, G, dv);
}

__device__ __forceinline__ uint64_t pack2(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ uint32_t word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// A warp takes 16 tokens per step. Scores: lane (g, t) = (lane / 4, lane % 4) loads chunks t, t + 4, t + 8, t + 12 (of 8 dimensions) of the keys of tokens
// g and g + 8, and of query head g; words 2 h, 2 h + 1 of a chunk are the operand registers of one MMA. It ends up with the scores of head g for tokens
// 2 t, 2 t + 1, 2 t + 8, 2 t + 9. Values: lane (tl, dl) = (lane / 16, lane % 16) holds dimensions 8 dl .. of tokens 2 u + tl, as in the kernel above.
template <bool EXT>
__global__ void __launch_bounds__(kDecWarps * 32, 4)
attn_decode_mma_kernel(const DecParams p) {
    constexpr int D = 128, kStep = 16;
    __shared__ float sm_o[kDecWarps][4][D];
    __shared__ float sm_ml[kDecWarps][4][2];
    __shared__ float4 sm_p[kDecWarps][kStep];       // weights of a step: token -> four heads
    __shared__ uint4 sm_q[8][17];                   // query heads (rows of absent heads zero)
    const int split = blockIdx.x, hk = blockIdx.y / p.passes, g0 = (blockIdx.y % p.passes) * 4, b = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, tl = lane >> 4, dl = lane & 15;
    const int G = min(4, p.group - g0);
    const int head0 = hk * p.group + g0;
    const int dk = EXT ? p.dk : 128, dv = EXT ? p.dv : 128;
    const bool in_v = !EXT || dl * 8 < dv;
    pdl_launch_dependents();
    pdl_wait();
    const int T_all = EXT ? *p.pos + 1 : p.T;
    int chunk = p.chunk;
    if (EXT) chunk = ((T_all + p.splits - 1) / p.splits + kCtaStep - 1) / kCtaStep * kCtaStep;
    const int t0 = split * chunk, t1 = min(T_all, t0 + chunk);

    for (int i = threadIdx.x; i < 8 * 16; i += kDecWarps * 32) {
        const int h = i >> 4, c = i & 15;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (h < G && (!EXT || c * 8 < dk)) v = __ldcs(reinterpret_cast<const uint4*>((const __nv_bfloat16*)p.q + (long long)b * p.ldq + (long long)(head0 + h) * dk + c * 8));
        sm_q[h][c] = v;
    }
    __syncthreads();
    uint64_t o[4][4];
#pragma unroll
    for (int h = 0; h < 4; ++h)
#pragma unroll
        for (int d = 0; d < 4; ++d) o[h][d] = 0ull;
    float m_own = kNegBig, l_own = 0.f;             // of head g, this lane's share of the sum
    const __nv_bfloat16* kb = (const __nv_bfloat16*)p.k + (long long)b * p.k_batch + (long long)hk * dk + t * 8;
    const __nv_bfloat16* vb = (const __nv_bfloat16*)p.v + (long long)b * p.v_batch + (long long)hk * dv + dl * 8;
    const float* brow = nullptr;
    if (EXT && p.bias && g < G) brow = p.bias + (long long)(head0 + g) * p.ldb;

    uint4 kr[2][4], vr[8];
    float bias[4];
    auto load_k = [&](int base) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int tok = base + 8 * r + g;
            const __nv_bfloat16* row = kb + (long long)tok * p.k_tok;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                kr[r][j] = make_uint4(0u, 0u, 0u, 0u);
                if (tok < t1 && (!EXT || (t + 4 * j) * 8 < dk)) kr[r][j] = __ldcs(reinterpret_cast<const uint4*>(row + 32 * j));
            }
        }
        if (EXT && p.bias) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int tok = base + (i >> 1) * 8 + 2 * t + (i & 1);
                bias[i] = brow && tok < t1 ? __ldg(brow + min(T_all - 1 - tok, p.n_bias - 1)) : 0.f;
            }
        }
    };
    auto load_v = [&](int base) {
        const __nv_bfloat16* row = vb + (long long)(base + tl) * p.v_tok;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            vr[u] = make_uint4(0u, 0u, 0u, 0u);
            if (base + 2 * u + tl < t1 && in_v) vr[u] = __ldcs(reinterpret_cast<const uint4*>(row));
            row += 2 * p.v_tok;
        }
    };
    // keys and values of a step are requested one step ahead, each as soon as the registers of the step before are used up
    load_k(t0 + warp * kStep);
    load_v(t0 + warp * kStep);
    for (int base = t0 + warp * kStep; base < t1; base += kDecWarps * kStep) {
        float s[4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint4 q = sm_q[g][t + 4 * j];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                                 : "r"(word(q, 2 * h)), "r"(0u), "r"(word(q, 2 * h + 1)), "r"(0u), "r"(word(kr[r][j], 2 * h)), "r"(word(kr[r][j], 2 * h + 1)));
            }
            s[2 * r] = c[0]; s[2 * r + 1] = c[1];
        }
        float mx = m_own;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int tok = base + (i >> 1) * 8 + 2 * t + (i & 1);
            s[i] *= p.scale_log2e;
            if (EXT && p.bias) s[i] = fmaf(bias[i], kLog2eDec, s[i]);
            if (tok >= t1) s[i] = kNegBig;
            mx = fmaxf(mx, s[i]);
        }
        load_k(base + kDecWarps * kStep);
        mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 2));
        const float corr = ex2(m_own - mx);
        const bool grew = mx > m_own;
        m_own = mx;
        l_own *= corr;
        __syncwarp();                               // the previous step's weights have been read
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int at = (i >> 1) * 8 + 2 * t + (i & 1);
            const float w = base + at < t1 ? ex2(s[i] - mx) : 0.f;
            l_own += w;
            if (g < 4) reinterpret_cast<float*>(&sm_p[warp][at])[g] = w;
        }
        if (__any_sync(0xFFFFFFFFu, grew)) {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const float ch = __shfl_sync(0xFFFFFFFFu, corr, 4 * h);
                const uint64_t c2 = pack2(ch, ch);
#pragma unroll
                for (int d = 0; d < 4; ++d) o[h][d] = mul2(o[h][d], c2);
            }
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const float4 w = sm_p[warp][2 * u + tl];
            const uint64_t w2[4] = {pack2(w.x, w.x), pack2(w.y, w.y), pack2(w.z, w.z), pack2(w.w, w.w)};
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                const uint32_t v = word(vr[u], d);
                const uint64_t v2 = pack2(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u));
#pragma unroll
                for (int h = 0; h < 4; ++h) o[h][d] = fma2(w2[h], v2, o[h][d]);
            }
        }
        load_v(base + kDecWarps * kStep);
    }
    l_own += __shfl_xor_sync(0xFFFFFFFFu, l_own, 1);
    l_own += __shfl_xor_sync(0xFFFFFFFFu, l_own, 2);
    if (t == 0 && g < 4) { sm_ml[warp][g][0] = m_own; sm_ml[warp][g][1] = l_own; }
#pragma unroll
    for (int h = 0; h < 4; ++h)
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            float lo, hi;
            unpack2(o[h][d], lo, hi);
            lo += __shfl_xor_sync(0xFFFFFFFFu, lo, 16);      // the two token slots
            hi += __shfl_xor_sync(0xFFFFFFFFu, hi, 16);
            if (tl == 0) { sm_o[warp][h][dl * 8 + 2 * d] = lo; sm_o[warp][h][dl * 8 + 2 * d + 1] = hi; }
        }
    __syncthreads();
    merge_warps<__nv_bfloat16, EXT, D>(p, sm_o, sm_ml, split, b, head0, G, dv);
}

// Merge of the splits: one block per (head, sequence), thread d = dimension d (and d + 128). The weights exp2(m_s - M) of the
// splits are computed once (thread s for split s, at most kMaxSplits of them) and shared; the sum over splits then has
// independent loads.
template <typename T>
__global__ void __launch_bounds__(128)
attn_decode_combine_kernel(const float* ws_o, const float* ws_ml, int splits, int Hq, int dv, int sink,
                           T* out, long long ldo) {
    __shared__ float wgt[kMaxSplits];
    __shared__ float red[8];
    const int head = blockIdx.x, b = blockIdx.y, t = threadIdx.x, lane = t & 31, wib = t >> 5;
    const long long slot0 = ((long long)b * Hq + head) * splits;
    pdl_launch_dependents();
    pdl_wait();
    const float m = t < splits ? ws_ml[(slot0 + t) * 2] : kNegBig;
    const float l = t < splits ? ws_ml[(slot0 + t) * 2 + 1] : 0.f;
    float M = m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xFFFFFFFFu, M, o));
    if (lane == 0) red[wib] = M;
    __syncthreads();
    M = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    if (sink) M = fmaxf(M, 0.f);
    const float c = ex2(m - M);
    wgt[t] = c;
    float ls = c * l;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ls += __shfl_xor_sync(0xFFFFFFFFu, ls, o);
    if (lane == 0) red[4 + wib] = ls;
    __syncthreads();
    const float L = red[4] + red[5] + red[6] + red[7] + (sink ? ex2(-M) : 0.f);
    for (int d = t; d < dv; d += 128) {
        float acc = 0.f;
        const float* src = ws_o + slot0 * dv + d;
#pragma unroll 8
        for (int s = 0; s < splits; ++s) acc = fmaf(wgt[s], __ldcs(src + (long long)s * dv), acc);
        store_elem(out + (long long)b * ldo + (long long)head * dv + d, L > 0.f ? acc / L : 0.f);
    }
}

// The same with a chain of one trip to memory instead of two: a warp takes every `parts`-th split and four dimensions per lane, requests its partial sums together with the
// maxima of all splits, of which every warp works out the weights for itself. dv a multiple of 4 up to 128. 2048 keys, 32 heads: 4.5 -> 2.05 us, of a step of one sequence 242 -> 232 us.
template <typename T>
__global__ void __launch_bounds__(512)
attn_decode_combine4_kernel(const float* ws_o, const float* ws_ml, int splits, int Hq, int dv, int sink, T* out, long long ldo) {
    __shared__ float4 red[16][32];
    const int head = blockIdx.x, b = blockIdx.y, lane = threadIdx.x & 31, part = threadIdx.x >> 5, parts = blockDim.x >> 5;
    const long long slot0 = ((long long)b * Hq + head) * splits;
    const bool live = lane * 4 < dv;
    pdl_launch_dependents();
    pdl_wait();
    constexpr int kEach = kMaxSplits / 16, kMl = kMaxSplits / 32;
    float4 o[kEach];
#pragma unroll
    for (int j = 0; j < kEach; ++j) {
        const int s = part + j * parts;
        o[j] = live && s < splits ? __ldcs(reinterpret_cast<const float4*>(ws_o + (slot0 + s) * dv) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float m[kMl], l[kMl], M = sink ? 0.f : kNegBig;
#pragma unroll
    for (int i = 0; i < kMl; ++i) {
        const int s = lane + 32 * i;
        const float2 ml = s < splits ? *reinterpret_cast<const float2*>(ws_ml + (slot0 + s) * 2) : make_float2(kNegBig, 0.f);
        m[i] = ml.x;
        l[i] = ml.y;
        M = fmaxf(M, ml.x);
    }
#pragma unroll
    for (int i = 16; i > 0; i >>= 1) M = fmaxf(M, __shfl_xor_sync(0xFFFFFFFFu, M, i));
    float L = 0.f;
#pragma unroll
    for (int i = 0; i < kMl; ++i) {
        m[i] = ex2(m[i] - M);
        L = fmaf(m[i], l[i], L);
    }
#pragma unroll
    for (int i = 16; i > 0; i >>= 1) L += __shfl_xor_sync(0xFFFFFFFFu, L, i);
    if (sink) L += ex2(-M);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < kEach; ++j) {
        const int s = part + j * parts;             // the same in all lanes
        if (s >= splits) break;
        const float w = s < 32 ? m[0] : s < 64 ? m[1] : s < 96 ? m[2] : m[3];
        const float c = __shfl_sync(0xFFFFFFFFu, w, s & 31);
        acc.x = fmaf(c, o[j].x, acc.x); acc.y = fmaf(c, o[j].y, acc.y); acc.z = fmaf(c, o[j].z, acc.z); acc.w = fmaf(c, o[j].w, acc.w);
    }
    red[part][lane] = acc;
    __syncthreads();
    if (part == 0 && live) {
        for (int i = 1; i < parts; ++i) {
            const float4 v = red[i][lane];
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        T* to = out + (long long)b * ldo + (long long)head * dv + lane * 4;
        const float v[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) store_elem(to + e, L > 0.f ? v[e] / L : 0.f);
    }
}

template <typename T>
int launch_combine(const DecParams& p, int B, int dv, int sink, cudaStream_t stream) {
    if (dv % 4 == 0 && dv <= 128 && !((uintptr_t)p.ws_o & 15) && !((uintptr_t)p.ws_ml & 7)) {
        int parts = 1;
        while (parts < p.splits && parts < 16) parts *= 2;
        PLZ_LAUNCH_CHAIN(attn_decode_combine4_kernel<T>, dim3(p.Hq, B), dim3(32 * parts), 0, stream, (const float*)p.ws_o, (const float*)p.ws_ml, p.splits, p.Hq, dv, sink,
                         (T*)p.out, p.ldo);
    } else {
        PLZ_LAUNCH_CHAIN(attn_decode_combine_kernel<T>, dim3(p.Hq, B), dim3(128), 0, stream, (const float*)p.ws_o, (const float*)p.ws_ml, p.splits, p.Hq, dv, sink, (T*)p.out,
                         p.ldo);
    }
    return PLZ_OK;
}

// out[i, :] = table[ids[i], :] (bf16 rows of `width`, width % 8 == 0); an id outside [0, vocab) gives a zero row and sets *bad
__global__ void __launch_bounds__(256)
embed_gather_kernel(const __nv_bfloat16* __restrict__ table, long long ldt, const long long* __restrict__ ids, long long n, int width,
                    long long vocab, __nv_bfloat16* __restrict__ out, long long ldo, int* __restrict__ bad) {
    pdl_launch_dependents();
    const int vec = width >> 3;
    const long long total = n * vec;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / vec;
        const int c = (int)(i - r * vec) << 3;
        const long long id = ids[r];
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (id >= 0 && id < vocab) v = __ldg(reinterpret_cast<const uint4*>(table + id * ldt + c));
        else if (bad && c == 0) *bad = 1;
        *reinterpret_cast<uint4*>(out + r * ldo + c) = v;
    }
}

int sm_count_now() {
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// tokens per split (a multiple of the CTA step) and the number of splits for a launch of B * Hkv groups over T tokens
void decode_split(int B, int Hkv, int T, int* chunk, int* splits) {
    const int want_ctas = 2 * sm_count_now();
    int s = (want_ctas + B * Hkv - 1) / (B * Hkv);
    const int max_s = (T + kCtaStep - 1) / kCtaStep;
    if (s > max_s) s = max_s;
    if (s > kMaxSplits) s = kMaxSplits;
    if (s < 1) s = 1;
    int c = (T + s - 1) / s;
    c = ((c + kCtaStep - 1) / kCtaStep) * kCtaStep;
    *chunk = c;
    *splits = (T + c - 1) / c;
}

}  // namespace

long long attn_decode_ws_bytes(int B, int T, int Hq, int Hkv) {
    int chunk = 0, splits = 1;
    decode_split(B, Hkv, T, &chunk, &splits);
    return splits == 1 ? 0 : (long long)B * Hq * splits * 130 * (long long)sizeof(float);
}

int launch_attn_decode(const AttnDecodeArgs& a, cudaStream_t stream) {
    if (a.B <= 0) return PLZ_OK;
    DecParams p = {};
    decode_split(a.B, a.Hkv, a.T, &p.chunk, &p.splits);
    const long long need = p.splits == 1 ? 0 : (long long)a.B * a.Hq * p.splits * 130 * (long long)sizeof(float);
    if (need > a.ws_bytes) { set_last_error("attn_decode: workspace of %lld bytes needed, %lld given", need, a.ws_bytes); return PLZ_ERR_TOO_LARGE; }
    p.q = a.q; p.ldq = a.ldq;
    p.k = a.k; p.v = a.v; p.k_batch = p.v_batch = a.batch_stride; p.k_tok = p.v_tok = a.tok_stride;
    p.out = a.out; p.ldo = a.ldo;
    p.ws_o = (float*)a.ws;
    p.ws_ml = p.ws_o ? p.ws_o + (long long)a.B * a.Hq * p.splits * 128 : nullptr;
    p.T = a.T; p.Hq = a.Hq; p.Hkv = a.Hkv; p.group = a.Hq / a.Hkv; p.passes = (p.group + 3) / 4;
    p.scale_log2e = a.scale * kLog2eDec;
    // Few cached tokens in all: a step of half the size. us there / here: 1 x 16 tokens of 8 heads 3.0 / 3.2, 1 x 300 6.1 / 6.4, 64 x 16 4.0 / 4.6, 16 x 100 of one 6.3 / 6.6,
    // 4 x 300 7.6 either way, 1 x 2049 9.3 / 8.8, 2 x 1000 7.8 / 7.5, 64 x 1025 67 / 46.
    const dim3 grid(p.splits, a.Hkv * p.passes, a.B), block(kDecWarps * 32);
    if ((long long)a.B * a.Hkv * a.T <= 8192) PLZ_LAUNCH_CHAIN((attn_decode_partial_kernel<__nv_bfloat16, 16, false>), grid, block, 0, stream, p);
    else PLZ_LAUNCH_CHAIN(attn_decode_mma_kernel<false>, grid, block, 0, stream, p);
    return p.splits > 1 ? launch_combine<__nv_bfloat16>(p, a.B, 128, 0, stream) : PLZ_OK;
}

// splits for a cache of `cap` positions whose length is known on the device only
static int ext_splits(int B, int groups, int cap) {
    int chunk = 0, splits = 1;
    decode_split(B, groups, cap, &chunk, &splits);
    return splits;
}
long long attn_bias_decode_ws_bytes(int B, int H, int G, int dv, int cap) {
    const int passes = (H / G + 3) / 4, splits = ext_splits(B, G * passes, cap);
    return splits == 1 ? 0 : (long long)B * H * splits * (dv + 2) * (long long)sizeof(float);
}
template <typename T>
static int launch_attn_bias_decode_t(const AttnBiasArgs& a, int cap, float* ws, cudaStream_t stream) {
    DecParams p = {};
    p.group = a.H / a.G; p.passes = (p.group + 3) / 4;
    p.splits = ext_splits(a.B, a.G * p.passes, cap);
    p.q = a.q; p.ldq = a.ldq; p.k = a.k; p.v = a.v; p.k_batch = a.k_batch; p.v_batch = a.v_batch;
    p.k_tok = (long long)a.G * a.dk; p.v_tok = (long long)a.G * a.dv;
    p.out = a.o; p.ldo = a.ldo; p.ws_o = ws; p.ws_ml = ws ? ws + (long long)a.B * a.H * p.splits * a.dv : nullptr;
    p.Hq = a.H; p.Hkv = a.G; p.scale_log2e = a.scale * kLog2eDec;
    p.dk = a.dk; p.dv = a.dv; p.pos = a.pos; p.bias = a.bias; p.ldb = a.ldb; p.n_bias = a.n_bias; p.sink = a.sink;
    const dim3 grid(p.splits, a.G * p.passes, a.B), block(kDecWarps * 32);
    const int d = a.dk > a.dv ? a.dk : a.dv;
    if (d <= 64) PLZ_LAUNCH_CHAIN((attn_decode_partial_kernel<T, 8, true>), grid, block, 0, stream, p);
    else if (d <= 128 && sizeof(T) == 2) PLZ_LAUNCH_CHAIN(attn_decode_mma_kernel<true>, grid, block, 0, stream, p);
    else if (d <= 128) PLZ_LAUNCH_CHAIN((attn_decode_partial_kernel<float, 16, true>), grid, block, 0, stream, p);
    else PLZ_LAUNCH_CHAIN((attn_decode_partial_kernel<T, 32, true>), grid, block, 0, stream, p);
    return p.splits > 1 ? launch_combine<T>(p, a.B, a.dv, a.sink, stream) : PLZ_OK;
}
int launch_attn_bias_decode(int dtype, const AttnBiasArgs& a, int cap, void* ws, long long ws_bytes, cudaStream_t stream) {
    if (a.B <= 0) return PLZ_OK;
    if (a.n != 1) { set_last_error("attention decode: one token per sequence (%d given)", a.n); return PLZ_ERR_BAD_SHAPE; }
    const long long need = attn_bias_decode_ws_bytes(a.B, a.H, a.G, a.dv, cap);
    if (need > ws_bytes) { set_last_error("attention decode: workspace of %lld bytes needed, %lld given", need, ws_bytes); return PLZ_ERR_TOO_LARGE; }
    return dtype == 1 ? launch_attn_bias_decode_t<float>(a, cap, (float*)ws, stream) : launch_attn_bias_decode_t<__nv_bfloat16>(a, cap, (float*)ws, stream);
}

int launch_embed_gather(const void* table, long long ldt, const long long* ids, long long n, int width, long long vocab, void* out,
                        long long ldo, int* bad, cudaStream_t stream) {
    if (n <= 0) return PLZ_OK;
    long long blocks = (n * (width >> 3) + 255) / 256;
    const long long cap = (long long)sm_count_now() * 16;
    if (blocks > cap) blocks = cap;
    embed_gather_kernel<<<(unsigned)blocks, 256, 0, stream>>>((const __nv_bfloat16*)table, ldt, ids, n, width, vocab, (__nv_bfloat16*)out, ldo, bad);
    PLZ_LAUNCH_CHECK();
    return PLZ_OK;
}

}  // namespace plz
