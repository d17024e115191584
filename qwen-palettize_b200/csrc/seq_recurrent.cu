// Token-by-token form of the two linear recurrences, state fp32 [B, H, dk, dv] in HBM, read and written once per call:
//
//   decayed linear attention   S <- lambda_h S + k v^T ;                                   o = S^T q   (q, k, v = silu of the projections)
//   gated delta rule           S <- g S (rows) ; u = beta (v - S^T k) ; S <- S + k u^T ;   o = S^T q
//
// This form serves token decode (bound by streaming the state), short portions and the 32-bit mode. A warp holds 8 value columns
// x dk key rows in registers: lane = 8 * (key row group) + column, row group g owning rows g, g + 4, g + 8, ..., so a warp's access
// to the state is whole 32-byte sectors, a token's key and query are conflict-free broadcasts from shared memory, and the sums
// over the key dimension take two shuffles. A single token moves the state through 16-byte accesses instead (recurrent_step_kernel).
#include "seq_math.cuh"

namespace plz {
namespace {

constexpr int kTok = 8;      // tokens staged in shared memory at a time

struct RecParams {
    // DELTA: q, k [rows, G * dk], v [rows, H * dv], logg [rows, H * dk], beta [rows, H], all fp32.  else: T slices of the projections
    const void* q; const void* k; const void* v; long long ldq, ldk, ldv;
    const float* logg; const float* beta; const float* decay;
    float* S;
    float* o;                // [rows, H * dv]
    int n, H, G, dk, dv;
};

// RK: key rows of a thread (dk <= 4 * RK). T: type of q, k, v.
template <typename T, bool DELTA, int RK>
__global__ void __launch_bounds__(128)
recurrent_kernel(const RecParams p) {
    extern __shared__ float sm[];
    constexpr int DK = 4 * RK;
    float* sq = sm;                      // [kTok][DK], zero past dk
    float* sk = sq + kTok * DK;
    float* sg = sk + kTok * DK;          // DELTA only
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kg = lane >> 3;
    const int col = (int)blockIdx.x * 32 + warp * 8 + (lane & 7);
    const int h = blockIdx.y;
    const long long b = blockIdx.z;
    const int hk = DELTA ? h / (p.H / p.G) : h;
    const bool live = col < p.dv;
    float* Sp = p.S + ((b * p.H + h) * p.dk) * (long long)p.dv + col;
    pdl_launch_dependents();
    pdl_wait();
    float s[RK];
#pragma unroll
    for (int i = 0; i < RK; ++i) {
        const int r = i * 4 + kg;
        s[i] = (live && r < p.dk) ? Sp[(long long)r * p.dv] : 0.f;
    }
    const float lam = DELTA ? 0.f : p.decay[h];
    for (int t0 = 0; t0 < p.n; t0 += kTok) {
        const int nt = min(kTok, p.n - t0);
        __syncthreads();
        for (int e = threadIdx.x; e < nt * DK; e += 128) {
            const int t = e / DK, c = e - t * DK;
            const long long row = b * p.n + t0 + t;
            float q = 0.f, k = 0.f, g = 0.f;
            if (c < p.dk) {
                q = to_f(((const T*)p.q)[row * p.ldq + (long long)hk * p.dk + c]);
                k = to_f(((const T*)p.k)[row * p.ldk + (long long)hk * p.dk + c]);
                if (DELTA) g = expf(p.logg[(row * p.H + h) * p.dk + c]);
                else { q = silu_f(q); k = silu_f(k); }
            }
            sq[t * DK + c] = q;
            sk[t * DK + c] = k;
            if (DELTA) sg[t * DK + c] = g;
        }
        __syncthreads();
        for (int t = 0; t < nt; ++t) {
            const long long row = b * p.n + t0 + t;
            float v = live ? to_f(((const T*)p.v)[row * p.ldv + (long long)h * p.dv + col]) : 0.f;
            float acc = 0.f;
            if (DELTA) {
                float pred = 0.f;
#pragma unroll
                for (int i = 0; i < RK; ++i) {
                    s[i] *= sg[t * DK + i * 4 + kg];
                    pred = fmaf(s[i], sk[t * DK + i * 4 + kg], pred);
                }
                pred += __shfl_xor_sync(0xFFFFFFFFu, pred, 8);
                pred += __shfl_xor_sync(0xFFFFFFFFu, pred, 16);
                const float u = p.beta[row * p.H + h] * (v - pred);
#pragma unroll
                for (int i = 0; i < RK; ++i) {
                    s[i] = fmaf(sk[t * DK + i * 4 + kg], u, s[i]);
                    acc = fmaf(s[i], sq[t * DK + i * 4 + kg], acc);
                }
            } else {
                v = silu_f(v);
#pragma unroll
                for (int i = 0; i < RK; ++i) {
                    s[i] = fmaf(sk[t * DK + i * 4 + kg], v, lam * s[i]);
                    acc = fmaf(s[i], sq[t * DK + i * 4 + kg], acc);
                }
            }
            acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 8);
            acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 16);
            if (live && kg == 0) p.o[(row * p.H + h) * (long long)p.dv + col] = acc;
        }
    }
#pragma unroll
    for (int i = 0; i < RK; ++i) {
        const int r = i * 4 + kg;
        if (live && r < p.dk) Sp[(long long)r * p.dv] = s[i];
    }
}

// One token, dk a multiple of 16 up to 128: bound by reading and writing the state once. A warp of the kernel above moves it 4 bytes per lane, 32 bytes of a row at a
// time; here a lane holds four columns of eight rows, a warp access is 128 bytes of four rows, and the four warps of a block share the key rows of 32 columns, so the
// sums over keys meet in shared memory. 64 sequences, 20 heads of 128 x 128 (168 MB), in a decode chain: decayed 41 -> 30 us, delta 42 -> 25.
constexpr int kStepRows = 8;       // key rows of a lane
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xFFFF0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xFFFF0000u));
}
__device__ __forceinline__ void fma4(float4& d, float a, const float4& b) { d.x = fmaf(a, b.x, d.x); d.y = fmaf(a, b.y, d.y); d.z = fmaf(a, b.z, d.z); d.w = fmaf(a, b.w, d.w); }
// over the four row groups of a warp
__device__ __forceinline__ float4 sum_groups(float4 v) {
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1) {
        v.x += __shfl_xor_sync(0xFFFFFFFFu, v.x, o); v.y += __shfl_xor_sync(0xFFFFFFFFu, v.y, o);
        v.z += __shfl_xor_sync(0xFFFFFFFFu, v.z, o); v.w += __shfl_xor_sync(0xFFFFFFFFu, v.w, o);
    }
    return v;
}
__device__ __forceinline__ float4 sum_warps(const float4 (&part)[4][8], int c) {
    float4 v = part[0][c];
#pragma unroll
    for (int w = 1; w < 4; ++w) { v.x += part[w][c].x; v.y += part[w][c].y; v.z += part[w][c].z; v.w += part[w][c].w; }
    return v;
}

template <typename T, bool DELTA>
__global__ void __launch_bounds__(128)
recurrent_step_kernel(const RecParams p) {
    __shared__ float sq[128], sk[128], sg[128];
    __shared__ float4 part[2][4][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kg = lane >> 3, c = lane & 7;
    const int col = (int)blockIdx.x * 32 + c * 4, h = blockIdx.y;
    const long long b = blockIdx.z;
    const int hk = DELTA ? h / (p.H / p.G) : h;
    const bool live = col < p.dv;
    const int row0 = warp * (p.dk >> 2) + kg, rows = p.dk >> 4;      // key rows of this lane: row0 + 4 i, i < rows
    float* Sp = p.S + ((b * p.H + h) * p.dk + row0) * (long long)p.dv + col;
    const long long step = 4ll * p.dv;
    pdl_launch_dependents();
    pdl_wait();
    float4 s[kStepRows];
#pragma unroll
    for (int i = 0; i < kStepRows; ++i) s[i] = live && i < rows ? __ldcs(reinterpret_cast<const float4*>(Sp + i * step)) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v = live ? load4((const T*)p.v + b * p.ldv + (long long)h * p.dv + col) : make_float4(0.f, 0.f, 0.f, 0.f);
    if ((int)threadIdx.x < p.dk) {
        float q = to_f(((const T*)p.q)[b * p.ldq + (long long)hk * p.dk + threadIdx.x]), k = to_f(((const T*)p.k)[b * p.ldk + (long long)hk * p.dk + threadIdx.x]);
        if (DELTA) sg[threadIdx.x] = expf(p.logg[(b * p.H + h) * p.dk + threadIdx.x]);
        else { q = silu_f(q); k = silu_f(k); }
        sq[threadIdx.x] = q;
        sk[threadIdx.x] = k;
    }
    const float lam = DELTA ? p.beta[b * p.H + h] : p.decay[h];
    __syncthreads();
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f), u = v;
    if (DELTA) {
        float4 pred = acc;
#pragma unroll
        for (int i = 0; i < kStepRows; ++i) {
            if (i >= rows) break;
            const float g = sg[row0 + 4 * i];
            s[i] = make_float4(s[i].x * g, s[i].y * g, s[i].z * g, s[i].w * g);
            fma4(pred, sk[row0 + 4 * i], s[i]);
        }
        pred = sum_groups(pred);
        if (kg == 0) part[0][warp][c] = pred;
        __syncthreads();
        pred = sum_warps(part[0], c);
        u = make_float4(lam * (v.x - pred.x), lam * (v.y - pred.y), lam * (v.z - pred.z), lam * (v.w - pred.w));
    } else {
        u = make_float4(silu_f(v.x), silu_f(v.y), silu_f(v.z), silu_f(v.w));
    }
#pragma unroll
    for (int i = 0; i < kStepRows; ++i) {
        if (i >= rows) break;
        if (!DELTA) s[i] = make_float4(lam * s[i].x, lam * s[i].y, lam * s[i].z, lam * s[i].w);
        fma4(s[i], sk[row0 + 4 * i], u);
        fma4(acc, sq[row0 + 4 * i], s[i]);
        if (live) __stcs(reinterpret_cast<float4*>(Sp + i * step), s[i]);
    }
    acc = sum_groups(acc);
    if (kg == 0) part[1][warp][c] = acc;
    __syncthreads();
    if (threadIdx.x < 8 && live) *reinterpret_cast<float4*>(p.o + (b * p.H + h) * (long long)p.dv + col) = sum_warps(part[1], c);
}

template <typename T, bool DELTA>
bool step_form(const RecParams& p) {
    return p.n == 1 && p.dk <= 128 && p.dk % 16 == 0 && p.dv % 4 == 0 && !(((uintptr_t)p.S | (uintptr_t)p.o) & 15) && !((uintptr_t)p.v & (4 * sizeof(T) - 1)) && p.ldv % 4 == 0;
}

template <typename T, bool DELTA, int RK>
int launch_rk(const RecParams& p, int B, cudaStream_t stream) {
    const size_t smem = (size_t)(DELTA ? 3 : 2) * kTok * 4 * RK * sizeof(float);
    PLZ_LAUNCH_CHAIN((recurrent_kernel<T, DELTA, RK>), dim3((p.dv + 31) / 32, p.H, B), dim3(128), smem, stream, p);
    return PLZ_OK;
}
template <typename T, bool DELTA>
int launch_any(const RecParams& p, int B, cudaStream_t stream) {
    if (step_form<T, DELTA>(p)) {
        PLZ_LAUNCH_CHAIN((recurrent_step_kernel<T, DELTA>), dim3((p.dv + 31) / 32, p.H, B), dim3(128), 0, stream, p);
        return PLZ_OK;
    }
    if (p.dk <= 32) return launch_rk<T, DELTA, 8>(p, B, stream);
    if (p.dk <= 64) return launch_rk<T, DELTA, 16>(p, B, stream);
    if (p.dk <= 128) return launch_rk<T, DELTA, 32>(p, B, stream);
    if (p.dk <= 256) return launch_rk<T, DELTA, 64>(p, B, stream);
    set_last_error("recurrence: key size %d (at most 256)", p.dk);
    return PLZ_ERR_UNSUPPORTED;
}

}  // namespace

int launch_recurrent_decay(int dtype, const DecayAttnArgs& a, cudaStream_t stream) {
    if (a.B <= 0 || a.n <= 0) return PLZ_OK;
    RecParams p = {};
    p.q = a.q; p.k = a.k; p.v = a.v; p.ldq = p.ldk = p.ldv = a.ld; p.decay = a.decay; p.S = a.state; p.o = a.o;
    p.n = a.n; p.H = a.H; p.G = a.H; p.dk = a.dk; p.dv = a.dv;
    return dtype == 1 ? launch_any<float, false>(p, a.B, stream) : launch_any<__nv_bfloat16, false>(p, a.B, stream);
}

int launch_recurrent_delta(const DeltaRuleArgs& a, cudaStream_t stream) {
    if (a.B <= 0 || a.n <= 0) return PLZ_OK;
    RecParams p = {};
    p.q = a.q; p.k = a.k; p.v = a.v; p.ldq = p.ldk = (long long)a.G * a.dk; p.ldv = (long long)a.H * a.dv;
    p.logg = a.logg; p.beta = a.beta; p.S = a.state; p.o = a.o;
    p.n = a.n; p.H = a.H; p.G = a.G; p.dk = a.dk; p.dv = a.dv;
    return launch_any<float, true>(p, a.B, stream);
}

}  // namespace plz
