// Causal attention with a per-head bias by distance and a sink on the tensor cores (tcgen05.mma, accumulators in TMEM), for a portion of
// n new tokens against the key / value cache that already holds them. bf16, key head sizes up to 192 in 64-column blocks, value head
// sizes up to 128 (multiples of 8), any n and any cache length.
//
// The structure is that of the plain causal kernel (attention.cu): one CTA takes two neighbouring 128-query tiles of a head and walks
// the key / value tiles they share once; warps 0-3 / 4-7 are the softmax groups of the two tiles (thread = query row = TMEM lane), warp 8
// issues TMA copies and MMAs, so that one group's exponentials run under the other group's products. What differs:
//   - tiles come through 4-D tensor maps (head column, head, token, sequence), so head sizes that are no multiple of 64, ragged token
//     counts and the end of the cache read as zeros and are clipped on the store;
//   - the first query sits at position pos of the sequence: a key tile may straddle the diagonal of two query rows' tiles, and every
//     element is masked by position where a tile touches the diagonal;
//   - the bias depends on i - j only: a tile row r, column c reads table[d0 + r - c], i.e. consecutive lanes read consecutive words.
//     A tile that lies wholly beyond the last table entry adds one constant per head, folded into the exponent;
//   - the running maximum uses the head's largest bias as a bound (any bound serves the softmax), so the bias is added once, in the
//     exponent of the second pass;
//   - with a sink the running maximum starts at its score (0 if it is not learned) and the denominator at 1;
//   - the last key columns may come from a second tensor that all heads share (a rotated part beside the heads' own), as blocks of their
//     own of the key tile;
//   - the weights P go back to TMEM over the scores they came from and are the A operand of P V from there; shared memory holds queries,
//     keys and values only, and the output leaves through the space of the queries;
//   - the output may be multiplied by the sigmoid of a gate on its way out.
#include "attention_tiles.cuh"

namespace plz {
namespace {

constexpr int kThreads = 288;   // warps 0..3 / 4..7: softmax of tile A / B, warp 8: TMA + MMA

struct TcParams {
    int n, H, G, pos;            // pos: position of the first query
    int k1_blocks;               // 64-column blocks of the heads' own keys; the others come from the shared tensor
    int k_steps[3];              // 16-wide reduction steps of Q K^T in each block
    int dv_blocks;               // 64-column boxes of the output
    float scale_log2e;
    const float* bias; long long ldb; int n_bias; const float* bias_top;
    int sink; const float* sinks;
    int heads_first;
    const __nv_bfloat16* gate; long long ldg; int dv;
    StatusWord* status;
};

template <int DKB, int DVB>
struct TcCfg {
    static constexpr uint32_t QK = DKB * kBlk, V = DVB * kBlk, QS = (DKB > DVB ? DKB : DVB) * kBlk;   // QS: a query tile, later the output
    static constexpr uint32_t OFF_K = 2 * QS, OFF_V = OFF_K + 2 * QK, OFF_BAR = OFF_V + V;
    static constexpr uint32_t SMEM = OFF_BAR + 1024 + 256;
};

template <int BLOCKS>
__device__ __forceinline__ void load_boxes(uint32_t dst, const CUtensorMap* map, uint32_t bar, int head, int tok, int b) {
#pragma unroll
    for (int i = 0; i < BLOCKS; ++i) tma_load_4d(dst + i * kBlk, map, bar, i * 64, head, tok, b);
}
// the first k1 blocks from one tensor, the others from a second one
template <int BLOCKS>
__device__ __forceinline__ void load_boxes2(uint32_t dst, const CUtensorMap* map, const CUtensorMap* map2, int k1, uint32_t bar, int head, int head2, int tok, int b) {
#pragma unroll
    for (int i = 0; i < BLOCKS; ++i) {
        if (i < k1) tma_load_4d(dst + i * kBlk, map, bar, i * 64, head, tok, b);
        else tma_load_4d(dst + i * kBlk, map2, bar, (i - k1) * 64, head2, tok, b);
    }
}

// S = Q K^T: both K-major
template <int DKB>
__device__ __forceinline__ void mma_qk(uint32_t d, uint32_t sQ, uint32_t sK, const int (&steps)[3]) {
    const uint32_t idesc = make_idesc(128, 128, 0, 0);
    const uint64_t ad = make_sdesc(sQ, 16u, 1024u), bd = make_sdesc(sK, 16u, 1024u);
#pragma unroll
    for (int i = 0; i < DKB; ++i) {
        for (int ks = 0; ks < steps[i]; ++ks) {
            const uint32_t off = (uint32_t)(i * (kBlk >> 4) + ks * 2);
            umma_bf16_words<1>(d, (uint32_t)ad + off, (uint32_t)(ad >> 32), (uint32_t)bd + off, (uint32_t)(bd >> 32), idesc, (i > 0 || ks > 0) ? 1u : 0u);
        }
    }
}
// O (+)= P V: P in TMEM, V MN-major (rows = keys)
template <int DVB>
__device__ __forceinline__ void mma_pv(uint32_t d, uint32_t tP, uint32_t sV, bool accumulate) {
    const uint32_t idesc = make_idesc(128, 64 * DVB, 0, 1);
    const uint64_t bd = make_sdesc(sV, kBlk, 1024u);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks)
        umma_ts(d, tP + ks * 8u, (uint32_t)bd + (uint32_t)(ks * 128), (uint32_t)(bd >> 32), idesc, (ks > 0 || accumulate) ? 1u : 0u);
}

struct Group {
    uint32_t tS, tO, s_full, p_full, o_full, out_ready;
    uint8_t* pOut; uint32_t sOut;   // space of the query tile, free once the last scores are in
    int qt, n_kv;              // query tile; key tiles it walks
};

// The weights of a row from its scores v, over the scores in TMEM; their sum.
// NEAR: the bias varies over the tile.
template <bool NEAR>
__device__ __forceinline__ float exp_pass(uint32_t tP, const uint32_t (&v)[128], float c, float add, const float* brow) {
    const uint64_t c2 = pair_f32(c, c);
    uint64_t l_tile = 0ull;         // even and odd columns
#pragma unroll
    for (int cb = 0; cb < 8; ++cb) {
        float bb[16];
        if (NEAR) {
#pragma unroll
            for (int i = 0; i < 16; ++i) bb[i] = __ldg(brow - (cb * 16 + i));
        }
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int c0 = cb * 16 + 2 * i;
            const uint64_t a2 = NEAR ? pair_f32(fmaf(bb[2 * i], kLog2e, add), fmaf(bb[2 * i + 1], kLog2e, add)) : pair_f32(add, add);
            float p0, p1;
            split_f32(fma_f32x2(pair_f32(__uint_as_float(v[c0]), __uint_as_float(v[c0 + 1])), c2, a2), p0, p1);
            p0 = ex2(p0);
            p1 = ex2(p1);
            l_tile = add_f32x2(l_tile, pair_f32(p0, p1));
            o[i] = pack_bf16x2(p0, p1);
        }
        tmem_st_32x8(tP + cb * 8, o);
    }
    tmem_wait_st();
    float even, odd;
    split_f32(l_tile, even, odd);
    return even + odd;
}

// The same where biases vary and columns beyond lim are masked, from the scores in TMEM once more, 16 at a time: masked columns read nothing. Only where what
// stands in front of a head's biases would spoil them (odd_front): a choice per column in the pass above costs every tile (20 heads over 4 of 128, 2048 tokens, 48.3 us
// without any, 54 with one, 49.1 so).
__device__ __forceinline__ float exp_pass_masked(uint32_t tP, float c, float add, const float* brow, int lim) {
    float l_tile = 0.f;
#pragma unroll 1
    for (int cb = 0; cb < 8; ++cb) {
        uint32_t v[16], o[8];
        tmem_ld_32x16(tP + cb * 16, v);
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            const int c0 = cb * 16 + i;
            const float p0 = c0 <= lim ? ex2(fmaf(__uint_as_float(v[i]), c, fmaf(__ldg(brow - c0), kLog2e, add))) : 0.f;
            const float p1 = c0 < lim ? ex2(fmaf(__uint_as_float(v[i + 1]), c, fmaf(__ldg(brow - c0 - 1), kLog2e, add))) : 0.f;
            l_tile += p0 + p1;
            o[i / 2] = pack_bf16x2(p0, p1);
        }
        tmem_st_32x8(tP + cb * 8, o);
    }
    tmem_wait_st();
    return l_tile;
}

template <int DVB>
__device__ __forceinline__ void softmax_group(const Group& G, const TcParams& p, const CUtensorMap* tmO, int h, int b, int warp_in_group, int lane,
                                              volatile uint32_t* abort_flag) {
    const int r = warp_in_group * 32 + lane;
    const uint32_t lane_off = (uint32_t)(warp_in_group * 32) << 16;
    const float c = fmaxf(p.scale_log2e, 1.17549435e-38f);   // positive: masked scores, -inf, get the weight 0
    const int i0 = p.pos + G.qt * kT;                       // position of the tile's first query
    // As in attention.cu: a row's scores stay in registers between the maximum and the exponentials, the maximum runs in four chains, and O is rescaled where
    // those registers are free again. 2048 tokens of one sequence: 20 heads over 4 of 128 with a bias 74 -> 58 us, 16 heads of 128 without one 51 -> 40,
    // 16 of 192 + 128 55 -> 43, 16 over 2 of 64 with a bias 64 -> 50.
    float m_run = p.sink ? (p.sinks ? p.sinks[h] * kLog2e : 0.f) : -INFINITY, l_run = p.sink ? 1.f : 0.f;
    // what stands in front of the head's biases, which masked columns read, may be anything; their exponents stay -inf where it is no NaN and nothing large
    bool odd_front = false;
    if (p.bias)
        for (int i = lane; i < 2 * kT; i += 32) odd_front |= !(__ldg(p.bias + (long long)h * p.ldb - 1 - i) < 1e30f);
    odd_front = __any_sync(0xFFFFFFFFu, odd_front);
    bool ok = true;
    for (int j = 0; j < G.n_kv && ok; ++j) {
        ok = mbar_wait(G.s_full, j & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 20);
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t v[128];
        tmem_ld_32x128(G.tS + lane_off, v);
        const int d0 = i0 - j * kT;                         // distance of (row 0, column 0)
        const bool mask = d0 < kT - 1;
        const bool near = p.bias != nullptr && d0 - (kT - 1) < p.n_bias - 1;
        const float shift = (!p.bias ? 0.f : __ldg(near ? p.bias_top + h : p.bias + (long long)h * p.ldb + p.n_bias - 1)) * kLog2e;   // near: a bound of the biases
        const int lim = d0 + r;                             // last visible column of this row
        if (mask) {
#pragma unroll
            for (int i = 0; i < 128; ++i)
                if (i > lim) v[i] = 0xFF800000u;            // -inf
        }
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 128; i += 8)
#pragma unroll
            for (int k = 0; k < 4; ++k) m4[k] = fmaxf(fmaxf(m4[k], __uint_as_float(v[i + k])), __uint_as_float(v[i + 4 + k]));
        const float bound = fmaf(fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])), c, shift);
        const float m_new = fmaxf(m_run, bound), alpha = m_run == -INFINITY ? 0.f : exp2f(m_run - m_new);
        const bool moved = m_new > m_run;
        m_run = m_new;
        if (j > 0) {
            ok = mbar_wait(G.o_full, (j - 1) & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 21);
            if (!ok) break;
            tc_fence_after_sync();
        }
        // a row that has seen no key yet (all of the tile masked, no sink) keeps m = -inf: its exponents are all masked
        const float add = (m_run == -INFINITY ? 0.f : -m_run) + (near ? 0.f : shift);
        const float* brow = p.bias ? p.bias + (long long)h * p.ldb + lim : nullptr;   // read where near
        const uint32_t tP = G.tS + lane_off;
        const float l_tile = !near ? exp_pass<false>(tP, v, c, add, brow) : mask && odd_front ? exp_pass_masked(tP, c, add, brow, lim) : exp_pass<true>(tP, v, c, add, brow);
        l_run = fmaf(l_run, alpha, l_tile);
        if (j > 0 && __any_sync(0xFFFFFFFFu, moved)) rescale<DVB>(G.tO + lane_off, alpha);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(G.p_full);
    }
    if (ok) ok = mbar_wait(G.o_full, (G.n_kv - 1) & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 22);
    if (ok) {
        tc_fence_after_sync();
        const float inv_l = l_run > 0.f ? 1.0f / l_run : 0.f;
        const __nv_bfloat16* gate = p.gate && G.qt * kT + r < p.n ? p.gate + ((long long)b * p.n + G.qt * kT + r) * p.ldg + (long long)h * p.dv : nullptr;
#pragma unroll 1
        for (int cb = 0; cb < 2 * DVB; ++cb) {
            uint32_t v[32];
            tmem_ld_32x32(G.tO + lane_off + cb * 32, v);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint32_t o[4];
                float f[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(v[g * 8 + i]) * inv_l;
                if (gate && cb * 32 + g * 8 < p.dv) {
                    const uint4 q = *reinterpret_cast<const uint4*>(gate + cb * 32 + g * 8);
                    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        f[2 * i] *= __fdividef(1.0f, 1.0f + __expf(-__uint_as_float(w[i] << 16)));
                        f[2 * i + 1] *= __fdividef(1.0f, 1.0f + __expf(-__uint_as_float(w[i] & 0xFFFF0000u)));
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) o[i] = pack_bf16x2(f[2 * i], f[2 * i + 1]);
                *reinterpret_cast<uint4*>(tile_chunk(G.pOut, r, cb * 4 + g)) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(G.out_ready);
        if (r == 0 && mbar_wait(G.out_ready, 0, abort_flag, p.status, ST_TIMEOUT_ACCUM, 23)) {
            for (int i = 0; i < p.dv_blocks; ++i) tma_store_4d(tmO, G.sOut + i * kBlk, i * 64, h, G.qt * kT, b);
            tma_store_commit();
            tma_store_wait_all();
        }
    }
}

template <int DKB, int DVB>
__global__ void __launch_bounds__(kThreads, 1)
attn_bias_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                    const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmQ2, const __grid_constant__ CUtensorMap tmK2, const TcParams p) {
    using C = TcCfg<DKB, DVB>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    const uint32_t sQ0 = base, sK0 = base + C::OFF_K, sV = base + C::OFF_V;
    const uint32_t bar = base + C::OFF_BAR;
    const uint32_t q_full = bar, k_full0 = bar + 8, k_empty0 = bar + 24, v_full = bar + 40, v_empty = bar + 48;
    auto s_full = [&](int g) { return bar + 56u + 8u * g; };
    auto p_full = [&](int g) { return bar + 72u + 8u * g; };
    auto o_full = [&](int g) { return bar + 88u + 8u * g; };
    auto out_ready = [&](int g) { return bar + 104u + 8u * g; };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + C::OFF_BAR + 128);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // uniform to the compiler too
    const int n_qt = (p.n + kT - 1) / kT;
    const int n_pairs = (n_qt + 1) / 2;
    // heavy pairs first: over all heads where the CTAs make more than a wave, else within a head, whose pairs then share keys and values in L2
    const int heads = gridDim.x / n_pairs, order = (int)blockIdx.x;
    const int pi = n_pairs - 1 - (p.heads_first ? order / heads : order % n_pairs), hb = p.heads_first ? order % heads : order / n_pairs;
    const int qtA = 2 * pi, qtB = 2 * pi + 1;
    const bool hasB = qtB < n_qt;
    const int h = hb % p.H, b = hb / p.H;
    const int hk = h / (p.H / p.G);
    auto kv_tiles = [&](int qt) { return (p.pos + min(p.n, (qt + 1) * kT) + kT - 1) / kT; };
    const int n_kvA = kv_tiles(qtA);
    const int n_kv = hasB ? kv_tiles(qtB) : n_kvA;

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1); mbar_init(v_full, 1); mbar_init(v_empty, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(k_full0 + 8 * i, 1); mbar_init(k_empty0 + 8 * i, 1);
            mbar_init(s_full(i), 1); mbar_init(p_full(i), 4); mbar_init(o_full(i), 1); mbar_init(out_ready(i), 4);
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 8) { tmem_alloc(smem_u32((const void*)tmem_slot), 512); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    pdl_launch_dependents();
    auto tS = [&](int g) { return tmem + 128u * g; };
    auto tO = [&](int g) { return tmem + 256u + 128u * g; };

    if (warp == 8) {
        // the whole warp walks the tiles and one elected lane issues (narrow_gemm.cu: operands stay in uniform registers)
        {
            if (elect_one()) { tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); }
            if (elect_one()) { mbar_arrive_expect_tx(q_full, hasB ? 2 * C::QK : C::QK); }
            if (elect_one()) { load_boxes2<DKB>(sQ0, &tmQ, &tmQ2, p.k1_blocks, q_full, h, h, qtA * kT, b); }
            if (hasB && elect_one()) load_boxes2<DKB>(sQ0 + C::QS, &tmQ, &tmQ2, p.k1_blocks, q_full, h, h, qtB * kT, b);
            bool ok = true;
            for (int j = 0; j < 2 && j < n_kv; ++j) {
                if (elect_one()) { mbar_arrive_expect_tx(k_full0 + 8 * j, C::QK); }
                if (elect_one()) { load_boxes2<DKB>(sK0 + j * C::QK, &tmK, &tmK2, p.k1_blocks, k_full0 + 8 * j, hk, 0, j * kT, b); }
            }
            if (elect_one()) { mbar_arrive_expect_tx(v_full, C::V); }
            if (elect_one()) { load_boxes<DVB>(sV, &tmV, v_full, hk, 0, b); }
            ok = mbar_wait_warp(q_full, 0, abort_flag, p.status, ST_TIMEOUT_FULL, 10);
            if (ok) ok = mbar_wait_warp(k_full0, 0, abort_flag, p.status, ST_TIMEOUT_FULL, 11);
            if (ok) {
                tc_fence_after_sync();
                if (elect_one()) { mma_qk<DKB>(tS(0), sQ0, sK0, p.k_steps); }
                if (elect_one()) { umma_commit(s_full(0)); }
                if (hasB && elect_one()) { mma_qk<DKB>(tS(1), sQ0 + C::QS, sK0, p.k_steps); umma_commit(s_full(1)); }
            }
            for (int j = 0; j < n_kv && ok; ++j) {
                const int s = j & 1, s1 = (j + 1) & 1;
                ok = mbar_wait_warp(v_full, j & 1, abort_flag, p.status, ST_TIMEOUT_FULL, 15);
                if (!ok) break;
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const int n_g = g == 0 ? n_kvA : n_kv;
                    if ((g == 1 && !hasB) || j >= n_g) continue;
                    ok = mbar_wait_warp(p_full(g), j & 1, abort_flag, p.status, ST_TIMEOUT_FULL, 12);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (elect_one()) { mma_pv<DVB>(tO(g), tS(g), sV, j > 0); }
                    if (elect_one()) { umma_commit(o_full(g)); }
                    if (j + 1 < n_g) {
                        ok = mbar_wait_warp(k_full0 + 8 * s1, ((j + 1) >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_FULL, 13);
                        if (!ok) break;
                        tc_fence_after_sync();
                        if (elect_one()) { mma_qk<DKB>(tS(g), sQ0 + g * C::QS, sK0 + s1 * C::QK, p.k_steps); }
                        if (elect_one()) { umma_commit(s_full(g)); }
                    }
                }
                if (!ok) break;
                if (elect_one()) { umma_commit(v_empty); }
                if (elect_one()) { umma_commit(k_empty0 + 8 * s); }
                if (j + 1 < n_kv) {
                    ok = mbar_wait_warp(v_empty, j & 1, abort_flag, p.status, ST_TIMEOUT_EMPTY, 16);
                    if (!ok) break;
                    if (elect_one()) { mbar_arrive_expect_tx(v_full, C::V); }
                    if (elect_one()) { load_boxes<DVB>(sV, &tmV, v_full, hk, (j + 1) * kT, b); }
                }
                if (j + 2 < n_kv) {
                    ok = mbar_wait_warp(k_empty0 + 8 * s, (j >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_EMPTY, 14);
                    if (!ok) break;
                    if (elect_one()) { mbar_arrive_expect_tx(k_full0 + 8 * s, C::QK); }
                    if (elect_one()) { load_boxes2<DKB>(sK0 + s * C::QK, &tmK, &tmK2, p.k1_blocks, k_full0 + 8 * s, hk, 0, (j + 2) * kT, b); }
                }
            }
        }
    } else {
        const int g = warp >> 2;
        if (g == 0 || hasB) {
            Group G;
            G.tS = tS(g); G.tO = tO(g); G.s_full = s_full(g); G.p_full = p_full(g); G.o_full = o_full(g); G.out_ready = out_ready(g);
            G.pOut = smem + g * C::QS; G.sOut = sQ0 + g * C::QS; G.qt = g == 0 ? qtA : qtB; G.n_kv = g == 0 ? n_kvA : n_kv;
            softmax_group<DVB>(G, p, &tmO, h, b, warp & 3, lane, abort_flag);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 8) { tc_fence_after_sync(); tmem_dealloc(tmem, 512); }
}

template <int DKB, int DVB>
int launch_t(const AttnBiasArgs& a, cudaStream_t stream) {
    using C = TcCfg<DKB, DVB>;
    CUtensorMap tmQ, tmK, tmV, tmO;
    int rc;
    const uint64_t keys = (uint64_t)a.host_pos + a.n;
    const int dk1 = a.dk - a.dk2;
    const uint64_t qb = (uint64_t)a.n * a.ldq;
    if ((rc = make_tmap_bf16_heads(&tmQ, a.q, dk1, a.H, a.n, a.B, a.ldq, qb, kT, a.dk))) return rc;
    if ((rc = make_tmap_bf16_heads(&tmK, a.k, dk1, a.G, keys, a.B, a.k_tok, a.k_batch, kT))) return rc;
    if ((rc = make_tmap_bf16_heads(&tmV, a.v, a.dv, a.G, keys, a.B, a.v_tok, a.v_batch, kT))) return rc;
    if ((rc = make_tmap_bf16_heads(&tmO, a.o, a.dv, a.H, a.n, a.B, a.ldo, (uint64_t)a.n * a.ldo, kT))) return rc;
    CUtensorMap tmQ2 = tmQ, tmK2 = tmK;
    if (a.k2) {
        if ((rc = make_tmap_bf16_heads(&tmQ2, (const __nv_bfloat16*)a.q + dk1, a.dk2, a.H, a.n, a.B, a.ldq, qb, kT, a.dk))) return rc;
        if ((rc = make_tmap_bf16_heads(&tmK2, a.k2, a.dk2, 1, keys, a.B, a.dk2, a.k2_batch, kT))) return rc;
    }
    TcParams p = {};
    p.n = a.n; p.H = a.H; p.G = a.G; p.pos = a.host_pos; p.dv_blocks = (a.dv + 63) / 64;
    p.k1_blocks = (dk1 + 63) / 64;
    for (int i = 0; i < DKB; ++i) {
        const int left = i < p.k1_blocks ? dk1 - 64 * i : a.dk2 - 64 * (i - p.k1_blocks);
        p.k_steps[i] = ((left < 64 ? left : 64) + 15) / 16;
    }
    p.scale_log2e = a.scale * kLog2e; p.bias = a.bias; p.ldb = a.ldb; p.n_bias = a.n_bias; p.bias_top = a.bias_top; p.sink = a.sink || a.sinks; p.sinks = a.sinks;
    p.gate = (const __nv_bfloat16*)a.gate; p.ldg = a.ldg; p.dv = a.dv;
    p.status = device_status_ptr();
    auto kern = attn_bias_tc_kernel<DKB, DVB>;
    static bool once[64] = {};
    int dev = 0;
    PLZ_CUDA_CHECK(cudaGetDevice(&dev));
    if (!once[dev & 63]) { PLZ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM)); once[dev & 63] = true; }
    const int n_qt = (a.n + kT - 1) / kT;
    const long long ctas = (long long)(n_qt + 1) / 2 * a.H * a.B;
    if (ctas > 0x7FFFFFFF) { set_last_error("attention: too many query tiles"); return PLZ_ERR_TOO_LARGE; }
    // us by pairs of a head / by heads: 4 x 1024 tokens, 32 heads over 8, 82 / 71; 2048, 20 heads (160 CTAs) 56 / 49; one wave: 2048, 16 heads over 2 of 64 48.5 / 51.7
    p.heads_first = ctas > seq_sm_count();
    PLZ_LAUNCH_BEHIND(kern, dim3((unsigned)ctas), dim3(kThreads), C::SMEM, stream, tmQ, tmK, tmV, tmO, tmQ2, tmK2, p);
    return PLZ_OK;
}

}  // namespace

// n >= 2 tokens, bf16, key parts and dv multiples of 8, at most three 64-column blocks of keys and dv <= 128, 16-byte aligned rows,
// positive scale, host_pos known
int launch_attn_bias_tc(const AttnBiasArgs& a, cudaStream_t stream) {
    const int blocks = (a.dk - a.dk2 + 63) / 64 + (a.dk2 + 63) / 64;
    if (blocks == 1) return a.dv <= 64 ? launch_t<1, 1>(a, stream) : launch_t<1, 2>(a, stream);
    if (blocks == 2) return a.dv <= 64 ? launch_t<2, 1>(a, stream) : launch_t<2, 2>(a, stream);
    return a.dv <= 64 ? launch_t<3, 1>(a, stream) : launch_t<3, 2>(a, stream);
}

}  // namespace plz
