// Causal grouped-query attention, forward and backward, for the decoder layers around the palettized Linears
// (head_dim 128, tokens-major activations: q [B*S, Hq*128], k / v [B*S, Hkv*128], exactly what the q/k/v projections
// write and what o_proj reads, so nothing is transposed).
//
// The reference has no attention code of its own: it trains through the HuggingFace decoder layer
// (scripts/train_qwen.py:1259-1266) with SDPA selected at scripts/qwen_model.py:454. Semantics follow
// transformers' Qwen3Attention: softmax(q k^T / sqrt(d) + causal mask) v, fp32 softmax, bf16 operands.
//
// All products run on the 5th-generation tensor cores (tcgen05.mma, 128 x 128 x 16, accumulators in TMEM), operands
// staged by TMA in 128-byte-swizzled tiles. One CTA handles one (batch, head) and one or two 128-token tiles:
//   forward        two neighbouring query tiles per CTA: S = Q K^T -> online softmax by 128 threads per tile (one row each,
//                  TMEM -> registers) -> P (bf16) to shared memory -> O += P V, O rescaled in TMEM when a row maximum grows;
//                  the softmax of one tile runs under the MMAs of the other; also writes the row log-sum-exp.
//   backward dQ    per q tile: S, dP = dO V^T -> dS = P (dP - D) / sqrt(d) -> dQ += dS K
//   backward dKdV  per kv tile and kv head, over the q heads of the group and the q tiles at or after it:
//                  S^T = K Q^T, dP^T = V dO^T -> P^T, dS^T in TMEM -> dV += P^T dO, dK += dS^T Q
// D[row] = sum_d dO O is a small pre-pass. Every barrier wait is bounded (status word, as in the GEMM kernels).
#include <type_traits>

#include "attention_tiles.cuh"

namespace plz {
namespace {

constexpr int kD = 128;                         // head dimension
constexpr uint32_t kTile = 2 * kBlk;            // a 128 x 128 bf16 tile: 32 KB

struct AttnParams {
    int B, S, Hq, Hkv;
    float scale;          // 1 / sqrt(head_dim)
    float* lse;           // [B, Hq, S] natural-log sum-exp of the scaled scores
    const float* dsum;    // [B, Hq, S] sum_d dO * O (backward)
    StatusWord* status;
};

// eight MMAs of one 128 x 128 x 128 product. A / B tiles are 128-row bf16 tiles of two 64-column blocks.
//   K-major operand (A, and B unless b_mn; rows = M or N index, reduction along the 128-byte row):  step ks -> block ks / 4, 32 bytes * (ks % 4)
//   MN-major B (rows = reduction index, N along the row): step ks -> 16 rows = 2048 bytes, blocks 16 KB apart
__device__ __forceinline__ void mma_128(uint32_t d_tmem, uint32_t sA, uint32_t sB, bool b_mn, bool accumulate) {
    const uint32_t idesc = make_idesc(128, 128, 0, b_mn ? 1 : 0);
    const uint64_t ad0 = make_sdesc(sA, 16u, 1024u);
    const uint64_t bd0 = b_mn ? make_sdesc(sB, kBlk, 1024u) : make_sdesc(sB, 16u, 1024u);
    const uint32_t a_hi = (uint32_t)(ad0 >> 32), b_hi = (uint32_t)(bd0 >> 32), a_lo = (uint32_t)ad0, b_lo = (uint32_t)bd0;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
        const uint32_t off_k = (uint32_t)((ks >> 2) * (kBlk >> 4) + (ks & 3) * 2);
        const uint32_t off_mn = (uint32_t)(ks * 128);
        umma_bf16_words<1>(d_tmem, a_lo + off_k, a_hi, b_lo + (b_mn ? off_mn : off_k), b_hi, idesc,
                           (ks > 0 || accumulate) ? 1u : 0u);
    }
}

__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int col0, int row0) {
    tma_load_2d(dst, map, bar, col0, row0);
    tma_load_2d(dst + kBlk, map, bar, col0 + 64, row0);
}

// ---------------------------------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------------------------------
// One CTA takes TWO neighbouring 128-query tiles (A = tile 2i, B = tile 2i + 1) of one head and walks the key / value tiles
// they share once. Warps 0-3 are the softmax group of A, warps 4-7 of B (thread = query row = TMEM lane), warp 8 issues the
// MMAs, warp 9 the TMA copies. S_A, S_B, O_A, O_B fill the 512 TMEM columns; Q_A, Q_B, a ring of three key or value tiles and one P tile
// per group (7 x 32 KB) fill the shared memory. A group takes its scores S(j) into registers at once, and S(j + 1) is computed
// while it works on them, so that it waits for neither product: the exponentials (MUFU, 16 per clock) and the MMAs cost about the same per tile
// and each hides the other. The ring takes the tiles in the order of their use, K_0 K_1 V_0 K_2 V_1 .., each requested a whole step ahead.
constexpr int kFwdThreads = 320;   // warps 0..3 / 4..7: softmax of tile A / B, warp 8: MMA, warp 9: TMA
constexpr uint32_t kFwdSmem = 7 * kTile + 1024 + 256;   // Q x 2, K / V x 3, P x 2

struct FwdGroup {          // what one softmax group works on
    uint32_t tS, tO;       // TMEM columns of its score and output accumulators
    uint32_t s_full, s_free, p_full, o_full;
    uint8_t* pP; uint32_t sP;
    int qt;                // its query tile; it attends key tiles 0 .. qt
};

__device__ __forceinline__ void fwd_softmax_group(const FwdGroup& G, const AttnParams& p, const CUtensorMap* tmO, int h, int b, int row0,
                                                  int warp_in_group, int lane, int bar_id, volatile uint32_t* abort_flag) {
    const int r = warp_in_group * 32 + lane;                       // query row of the tile = TMEM lane
    const uint32_t lane_off = (uint32_t)(warp_in_group * 32) << 16;
    const float c = p.scale * kLog2e;
    const int n_kv = G.qt + 1;
    // The scores of a row stay in registers between the maximum and the exponentials (128 of them, one read of TMEM instead of two), the maximum runs in
    // four chains, only the tile on the diagonal is compared with the row, and O is rescaled where those registers are free again. 32 heads over 8,
    // 8 x 512 tokens: 53 -> 44 us, 4 x 1024 84 -> 55, 1 x 4096 255 -> 130, 8 x 2048 461 -> 297.
    // The exponentials alone are 17 us. Rescaling O only when a maximum has grown by 2^8 gives 53, 120, 285, but the largest weight is then
    // no longer 1 and its rounding shows: error of O against 64 bits at 1024 keys 1.74e-3 -> 2.04e-3 with scores of spread 4.
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < n_kv && ok; ++j) {
        ok = mbar_wait(G.s_full, j & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 20);
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t v[128];
        tmem_ld_32x128(G.tS + lane_off, v);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(G.s_free);
        const bool diag = (j == G.qt);
        if (diag) {
#pragma unroll
            for (int i = 0; i < 128; ++i)
                if (i > r) v[i] = 0xFF800000u;                 // -inf
        }
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 128; i += 8)
#pragma unroll
            for (int k = 0; k < 4; ++k) m4[k] = fmaxf(fmaxf(m4[k], __uint_as_float(v[i + k])), __uint_as_float(v[i + 4 + k]));
        const float m_tile = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
        const bool moved = m_tile > m_run;
        const float alpha = !moved ? 1.f : m_run == -INFINITY ? 0.f : exp2f((m_run - m_tile) * c);
        if (moved) m_run = m_tile;
        // the previous P V product must have landed before P is overwritten and before O is rescaled
        if (j > 0) {
            ok = mbar_wait(G.o_full, (j - 1) & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 21);
            if (!ok) break;
            tc_fence_after_sync();
        }
        // P = exp2(s c - m c), row sum, bf16 row into the swizzled P tile; of the diagonal tile only the 32-column blocks that some row of this warp attends
        const uint64_t c2 = pair_f32(c, c), mc2 = pair_f32(-m_run * c, -m_run * c);
        uint64_t l_tile = 0ull;                        // even and odd columns
        auto weights = [&](auto on_diagonal) {
            constexpr bool kDiag = decltype(on_diagonal)::value;
#pragma unroll
            for (int cb = 0; cb < 4; ++cb) {
                if (!kDiag || cb <= warp_in_group) {
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        uint32_t o[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int c0 = cb * 32 + g * 8 + 2 * i;
                            float p0, p1;
                            split_f32(fma_f32x2(pair_f32(__uint_as_float(v[c0]), __uint_as_float(v[c0 + 1])), c2, mc2), p0, p1);
                            p0 = ex2(p0);
                            p1 = ex2(p1);
                            if (kDiag) { if (c0 > r) p0 = 0.f; if (c0 + 1 > r) p1 = 0.f; }
                            l_tile = add_f32x2(l_tile, pair_f32(p0, p1));
                            o[i] = pack_bf16x2(p0, p1);
                        }
                        *reinterpret_cast<uint4*>(tile_chunk(G.pP, r, cb * 4 + g)) = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                } else {
#pragma unroll
                    for (int g = 0; g < 4; ++g) *reinterpret_cast<uint4*>(tile_chunk(G.pP, r, cb * 4 + g)) = make_uint4(0u, 0u, 0u, 0u);
                }
            }
        };
        if (diag) weights(std::true_type());
        else weights(std::false_type());
        float even, odd;
        split_f32(l_tile, even, odd);
        l_run = fmaf(l_run, alpha, even + odd);
        if (j > 0 && __any_sync(0xFFFFFFFFu, moved)) rescale<2>(G.tO + lane_off, alpha);
        tc_fence_before_sync();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(G.p_full);
    }
    // epilogue: O / l -> bf16 -> the P tile as staging -> TMA store; log-sum-exp for the backward
    if (ok) ok = mbar_wait(G.o_full, (n_kv - 1) & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 22);
    if (ok) {
        tc_fence_after_sync();
        const float inv_l = 1.0f / l_run;
#pragma unroll 1
        for (int cb = 0; cb < 4; ++cb) {
            uint32_t v[32];
            tmem_ld_32x32(G.tO + lane_off + cb * 32, v);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint32_t o[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    o[i] = pack_bf16x2(__uint_as_float(v[g * 8 + 2 * i]) * inv_l, __uint_as_float(v[g * 8 + 2 * i + 1]) * inv_l);
                *reinterpret_cast<uint4*>(tile_chunk(G.pP, r, cb * 4 + g)) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
        if (p.lse) p.lse[((long long)b * p.Hq + h) * p.S + G.qt * kT + r] = m_run * p.scale + logf(l_run);
        fence_proxy_async_smem();
    }
    asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");
    if (ok && r == 0) {
        tma_store_2d(tmO, G.sP, h * kD, row0 + G.qt * kT);
        tma_store_2d(tmO, G.sP + kBlk, h * kD + 64, row0 + G.qt * kT);
        tma_store_commit();
        tma_store_wait_all();
    }
}

__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                const __grid_constant__ CUtensorMap tmO, const AttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    const uint32_t sQ0 = base, sKV = base + 2 * kTile, sP0 = base + 5 * kTile;
    const uint32_t bar = base + 7 * kTile;
    const uint32_t q_full = bar;
    auto full = [&](int i) { return bar + 8u + 8u * i; };
    auto empty = [&](int i) { return bar + 32u + 8u * i; };
    auto s_full = [&](int g) { return bar + 56u + 8u * g; };
    auto p_full = [&](int g) { return bar + 72u + 8u * g; };
    auto o_full = [&](int g) { return bar + 88u + 8u * g; };
    auto s_free = [&](int g) { return bar + 104u + 8u * g; };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + 7 * kTile + 120);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // uniform to the compiler too
    const int n_qt = p.S / kT;
    const int n_pairs = (n_qt + 1) / 2;
    const int pi = n_pairs - 1 - (int)blockIdx.y;   // heavy pairs first, over all heads
    const int qtA = 2 * pi, qtB = 2 * pi + 1;
    const bool hasB = qtB < n_qt;
    const int h = blockIdx.x % p.Hq, b = blockIdx.x / p.Hq;
    const int hk = h / (p.Hq / p.Hkv);
    const int n_kvA = qtA + 1;
    const int n_kv = hasB ? qtB + 1 : n_kvA;
    const int row0 = b * p.S;

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int i = 0; i < 3; ++i) { mbar_init(full(i), 1); mbar_init(empty(i), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(s_full(i), 1); mbar_init(s_free(i), 4); mbar_init(p_full(i), 4); mbar_init(o_full(i), 1); }
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

    // the ring's items: K_0, then K_{j + 1} and V_j in turns (the last V_j without a K_{j + 1})
    const int last = 2 * n_kv;
    auto k_item = [](int j) { return j == 0 ? 0 : 2 * j - 1; };
    auto v_item = [](int j) { return 2 * j + 2; };
    if (warp == 9) {
        if (elect_one()) { tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); }
        if (elect_one()) { mbar_arrive_expect_tx(q_full, hasB ? 2 * kTile : kTile); }
        if (elect_one()) { load_tile(sQ0, &tmQ, q_full, h * kD, row0 + qtA * kT); }
        bool ok = true;
        for (int i = 0, s = 0; i <= last && ok; ++i, s = s == 2 ? 0 : s + 1) {
            if (i == 1 && hasB && elect_one()) load_tile(sQ0 + kTile, &tmQ, q_full, h * kD, row0 + qtB * kT);
            if (i == last - 1) continue;
            if (i >= 3) ok = mbar_wait_warp(empty(s), (i / 3 - 1) & 1, abort_flag, p.status, ST_TIMEOUT_EMPTY, 14);
            if (!ok) break;
            const bool is_k = i == 0 || (i & 1);
            const int row = row0 + (i == 0 ? 0 : is_k ? (i + 1) / 2 : i / 2 - 1) * kT;
            if (elect_one()) { mbar_arrive_expect_tx(full(s), kTile); }
            if (elect_one()) { load_tile(sKV + s * kTile, is_k ? &tmK : &tmV, full(s), hk * kD, row); }
        }
    } else if (warp == 8) {
        // the whole warp walks the tiles and one elected lane issues (narrow_gemm.cu: operands stay in uniform registers)
        auto ready = [&](int item) { return mbar_wait_warp(full(item % 3), (item / 3) & 1, abort_flag, p.status, ST_TIMEOUT_FULL, 11); };
        auto done = [&](int item) { if (item + 3 <= last && elect_one()) umma_commit(empty(item % 3)); };
        bool ok = mbar_wait_warp(q_full, 0, abort_flag, p.status, ST_TIMEOUT_FULL, 10);
        for (int j = -1; j < n_kv && ok; ++j) {
            if (j + 1 < n_kv) {                     // S_g(j + 1) = Q_g K_{j + 1}^T once S_g(j) is in registers
                const int item = k_item(j + 1);
                ok = ready(item);
#pragma unroll
                for (int g = 0; g < 2 && ok; ++g) {
                    if ((g == 1 && !hasB) || j + 1 >= (g == 0 ? n_kvA : n_kv)) continue;
                    if (j >= 0) ok = mbar_wait_warp(s_free(g), j & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 12);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (elect_one()) { mma_128(tS(g), sQ0 + g * kTile, sKV + item % 3 * kTile, false, false); }
                    if (elect_one()) { umma_commit(s_full(g)); }
                }
                if (!ok) break;
                done(item);
            }
            if (j >= 0) {                           // O_g += P_g V_j
                const int item = v_item(j);
                ok = ready(item);
#pragma unroll
                for (int g = 0; g < 2 && ok; ++g) {
                    if ((g == 1 && !hasB) || j >= (g == 0 ? n_kvA : n_kv)) continue;
                    ok = mbar_wait_warp(p_full(g), j & 1, abort_flag, p.status, ST_TIMEOUT_FULL, 13);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (elect_one()) { mma_128(tO(g), sP0 + g * kTile, sKV + item % 3 * kTile, true, j > 0); } // V: rows = kv = reduction index
                    if (elect_one()) { umma_commit(o_full(g)); }
                }
                if (!ok) break;
                done(item);
            }
        }
    } else {
        const int g = warp >> 2;
        if (g == 0 || hasB) {
            FwdGroup G;
            G.tS = tS(g); G.tO = tO(g); G.s_full = s_full(g); G.s_free = s_free(g); G.p_full = p_full(g); G.o_full = o_full(g);
            G.pP = smem + 5 * kTile + g * kTile; G.sP = sP0 + g * kTile; G.qt = g == 0 ? qtA : qtB;
            fwd_softmax_group(G, p, &tmO, h, b, row0, warp & 3, lane, 1 + g, abort_flag);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 8) { tc_fence_after_sync(); tmem_dealloc(tmem, 512); }
}

// ---------------------------------------------------------------------------------------------------------------------
// backward pre-pass: dsum[b, h, s] = sum_d dO * O   (one warp per (token, head) row)
// ---------------------------------------------------------------------------------------------------------------------
template <bool O16>      // o aligned to 16 bytes; else to 8
__global__ void __launch_bounds__(256)
attn_dsum_kernel(const __nv_bfloat16* o, const __nv_bfloat16* d_o, long long ld, int B, int S, int Hq, float* dsum) {
    // sixteen lanes per (token, head) row, eight rows of a warp at once: four 16-byte loads of each operand in flight per lane (4096 tokens x 32
    // heads 23 -> 18 us against one row per warp)
    const int lane = threadIdx.x & 31, l = lane & 15;
    const long long rows = (long long)B * S * Hq, row0 = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * 8 + (lane >> 4);
    uint4 a[4], g[4];
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long row = row0 + 2 * i;
        a[i] = g[i] = make_uint4(0u, 0u, 0u, 0u);
        if (row < rows) {
            const long long at = row / Hq * ld + row % Hq * kD + l * 8;
            if (O16) a[i] = __ldcs(reinterpret_cast<const uint4*>(o + at));
            else {
                const uint2 lo = __ldcs(reinterpret_cast<const uint2*>(o + at)), hi = __ldcs(reinterpret_cast<const uint2*>(o + at + 4));
                a[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
            }
            g[i] = *reinterpret_cast<const uint4*>(d_o + at);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t aw[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, gw[4] = {g[i].x, g[i].y, g[i].z, g[i].w};
        float s = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e)
            s += __uint_as_float(aw[e] << 16) * __uint_as_float(gw[e] << 16) + __uint_as_float(aw[e] & 0xFFFF0000u) * __uint_as_float(gw[e] & 0xFFFF0000u);
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, off);
        const long long row = row0 + 2 * i;
        if (l == 0 && row < rows) {
            const long long tok = row / Hq;
            dsum[(tok / S * Hq + row % Hq) * S + tok % S] = s;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// backward: dK and dV (KV: one CTA per kv tile and kv head, walking the q heads of the group and the q tiles), or dQ (one CTA per
// q tile and q head, walking the kv tiles)
// ---------------------------------------------------------------------------------------------------------------------
// Either way two tiles X1, X2 stay (K, V or Q, dO) and pairs Y1, Y2 walk by (Q, dO or K, V) in halves of 64 tokens, one half to each of two groups of four warps:
//   S = X1 Y1^T, dP = X2 Y2^T        X's tokens are the accumulators' rows, so with KV both come out transposed
//   P, dS = P (dP - D) scale         in registers, written over S and dP in TMEM as bf16
//   dV += P Y2 (KV), dX1 += dS Y1    P and dS as operands in TMEM
// P and dS never go through shared memory, which leaves room for a second pair Y; while one group works on its half, the tensor core runs the products of the
// other's. Before, four warps and the tensor core took turns and every pair was loaded when the last one was done with. 32 heads over 8, all three
// backward launches: 8 x 512 tokens 191 -> 126 us, 4 x 1024 298 -> 167, 1 x 4096 902 -> 444.
constexpr int kBwdThreads = 320;   // warps 0..3 / 4..7: halves 0 / 1, warp 8: MMA, warp 9: TMA
constexpr uint32_t kBwdSmem = 6 * kTile + 1024 + 256 + 8 * 2 * 128 * 4;   // X1, X2, (Y1, Y2) x 2, [warp][parity][lse, dsum of its 64 queries]

// eight MMAs S_half = X Y_half^T: 128 rows, 64 tokens, 128 head columns
__device__ __forceinline__ void mma_half(uint32_t d_tmem, uint32_t sX, uint32_t sY, int half) {
    const uint32_t idesc = make_idesc(128, 64, 0, 0);
    const uint64_t ad = make_sdesc(sX, 16u, 1024u), bd = make_sdesc(sY + (uint32_t)half * 8192u, 16u, 1024u);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
        const uint32_t off = (uint32_t)((ks >> 2) * (kBlk >> 4) + (ks & 3) * 2);
        umma_bf16_words<1>(d_tmem, (uint32_t)ad + off, (uint32_t)(ad >> 32), (uint32_t)bd + off, (uint32_t)(bd >> 32), idesc, ks > 0 ? 1u : 0u);
    }
}
// four MMAs acc += A Y_half with A (128 rows, 64 tokens) in TMEM: 128 rows, 128 head columns
__device__ __forceinline__ void mma_grad(uint32_t acc, uint32_t tA, uint32_t sY, int half, bool accumulate) {
    const uint32_t idesc = make_idesc(128, 128, 0, 1);
    const uint64_t bd = make_sdesc(sY + (uint32_t)half * 8192u, kBlk, 1024u);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
        umma_ts(acc, tA + ks * 8u, (uint32_t)bd + (uint32_t)(ks * 128), (uint32_t)(bd >> 32), idesc, (ks > 0 || accumulate) ? 1u : 0u);
}

// One half's rows, 32 columns at a time: thread r (row r) turns its scores and dP into bf16 P (KV) and dS over them. nl, nd: -lse (log2 units) and -dsum of the
// row, or with KV of the 64 columns in shared memory. masked: of the tile on the diagonal.
template <bool KV>
__device__ __forceinline__ void bwd_rows(uint32_t tS, uint32_t tdP, int half, int r, bool diag, float c, float scale, float nl, float nd, const float* col_stats) {
    const uint64_t c2 = pair_f32(c, c), scale2 = pair_f32(scale, scale);
#pragma unroll
    for (int cb = 0; cb < 2; ++cb) {
        uint32_t vs[32], vd[32], op[16], od[16];
        tmem_ld_32x32_two(tS + cb * 32, tdP + cb * 32, vs, vd);
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            float4 l4 = make_float4(nl, nl, nl, nl), d4 = make_float4(nd, nd, nd, nd);
            if (KV) {
                l4 = *reinterpret_cast<const float4*>(col_stats + cb * 32 + i);
                d4 = *reinterpret_cast<const float4*>(col_stats + 64 + cb * 32 + i);
            }
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                const uint64_t l2 = e == 0 ? pair_f32(l4.x, l4.y) : pair_f32(l4.z, l4.w), n2 = e == 0 ? pair_f32(d4.x, d4.y) : pair_f32(d4.z, d4.w);
                float p0, p1, d0, d1;
                split_f32(fma_f32x2(pair_f32(__uint_as_float(vs[i + e]), __uint_as_float(vs[i + e + 1])), c2, l2), p0, p1);
                p0 = ex2(p0);
                p1 = ex2(p1);
                if (diag) {
                    const int t = half * 64 + cb * 32 + i + e;      // a key comes no later than its query
                    if (KV ? t < r : t > r) p0 = 0.f;
                    if (KV ? t + 1 < r : t + 1 > r) p1 = 0.f;
                }
                split_f32(mul_f32x2(mul_f32x2(pair_f32(p0, p1), add_f32x2(pair_f32(__uint_as_float(vd[i + e]), __uint_as_float(vd[i + e + 1])), n2)), scale2), d0, d1);
                op[(i + e) / 2] = pack_bf16x2(p0, p1);
                od[(i + e) / 2] = pack_bf16x2(d0, d1);
            }
        }
        if (KV) tmem_st_32x16(tS + cb * 16, op);
        tmem_st_32x16(tdP + cb * 16, od);
    }
    tmem_wait_st();
}

// 64 columns of a finished fp32 accumulator as one swizzled bf16 block
__device__ __forceinline__ void stage_block(uint32_t tacc, int r, uint8_t* block) {
#pragma unroll 1
    for (int cb = 0; cb < 2; ++cb) {
        uint32_t v[32];
        tmem_ld_32x32(tacc + cb * 32, v);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            uint32_t o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = pack_bf16x2(__uint_as_float(v[g * 8 + 2 * i]), __uint_as_float(v[g * 8 + 2 * i + 1]));
            *reinterpret_cast<uint4*>(tile_chunk(block, r, cb * 4 + g)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
}

// the maps of X1, X2, Y1, Y2 and of the gradients of X1 and (KV) X2
template <bool KV>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmX1, const __grid_constant__ CUtensorMap tmX2, const __grid_constant__ CUtensorMap tmY1,
                const __grid_constant__ CUtensorMap tmY2, const __grid_constant__ CUtensorMap tmG1, const __grid_constant__ CUtensorMap tmG2, const AttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    const uint32_t sX1 = base, sX2 = base + kTile, bar = base + 6 * kTile;
    auto sY1 = [&](int s) { return base + (2 + 2 * s) * kTile; };
    auto sY2 = [&](int s) { return base + (3 + 2 * s) * kTile; };
    const uint32_t x_full = bar, acc_full = bar + 8;
    auto full = [&](int s) { return bar + 16u + 8u * s; };
    auto empty = [&](int s) { return bar + 32u + 8u * s; };
    auto sd_full = [&](int g) { return bar + 48u + 8u * g; };
    auto ds_full = [&](int g) { return bar + 64u + 8u * g; };
    auto done = [&](int g) { return bar + 80u + 8u * g; };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + 6 * kTile + 96);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    float* stats = reinterpret_cast<float*>(smem + 6 * kTile + 256);

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // uniform to the compiler too
    const int heads = KV ? p.Hkv : p.Hq, group = p.Hq / p.Hkv;
    const int head = blockIdx.x % heads, b = blockIdx.x / heads;
    const int n_qt = p.S / kT;
    const int xt = KV ? (int)blockIdx.y : n_qt - 1 - (int)blockIdx.y;      // the tile that stays; those with the most work first
    const int n_i = KV ? n_qt - xt : xt + 1;                                // pairs per walk
    const int n_it = KV ? group * n_i : n_i;
    const int row0 = b * p.S;

    if (threadIdx.x == 0) {
        mbar_init(x_full, 1); mbar_init(acc_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(full(i), 1); mbar_init(empty(i), 1);
            mbar_init(sd_full(i), 1); mbar_init(ds_full(i), 4); mbar_init(done(i), 1);
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
    auto tdP = [&](int g) { return tmem + 128u * g + 64u; };
    const uint32_t tG1 = tmem + 256, tG2 = tmem + 384;

    if (warp == 9) {
        if (elect_one()) { mbar_arrive_expect_tx(x_full, 2 * kTile); }
        if (elect_one()) { load_tile(sX1, &tmX1, x_full, head * kD, row0 + xt * kT); }
        if (elect_one()) { load_tile(sX2, &tmX2, x_full, head * kD, row0 + xt * kT); }
        bool ok = true;
        int yh = KV ? head * group : head / group, yt = KV ? xt : 0;
        for (int it = 0; it < n_it; ++it) {
            const int s = it & 1;
            if (it >= 2) ok = mbar_wait_warp(empty(s), ((it >> 1) - 1) & 1, abort_flag, p.status, ST_TIMEOUT_EMPTY, 30);
            if (!ok) break;
            if (elect_one()) { mbar_arrive_expect_tx(full(s), 2 * kTile); }
            if (elect_one()) { load_tile(sY1(s), &tmY1, full(s), yh * kD, row0 + yt * kT); }
            if (elect_one()) { load_tile(sY2(s), &tmY2, full(s), yh * kD, row0 + yt * kT); }
            if (++yt == (KV ? n_qt : n_it)) { yt = KV ? xt : 0; ++yh; }
        }
    } else if (warp == 8) {
        // the whole warp walks the tiles and one elected lane issues (narrow_gemm.cu: operands stay in uniform registers)
        bool ok = mbar_wait_warp(x_full, 0, abort_flag, p.status, ST_TIMEOUT_FULL, 31);
        auto scores = [&](int it, int g) {          // over P and dS of the half before, whose products must be done
            if (g == 0) ok = mbar_wait_warp(full(it & 1), (it >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_FULL, 32);
            if (ok && it > 0) ok = mbar_wait_warp(done(g), (it - 1) & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 33);
            if (!ok) return;
            tc_fence_after_sync();
            if (elect_one()) { mma_half(tS(g), sX1, sY1(it & 1), g); }
            if (elect_one()) { mma_half(tdP(g), sX2, sY2(it & 1), g); }
            if (elect_one()) { umma_commit(sd_full(g)); }
        };
        if (ok) scores(0, 0);
        if (ok) scores(0, 1);
        for (int it = 0; it < n_it && ok; ++it) {
#pragma unroll
            for (int g = 0; g < 2 && ok; ++g) {
                ok = mbar_wait_warp(ds_full(g), it & 1, abort_flag, p.status, ST_TIMEOUT_FULL, 34);
                if (!ok) break;
                tc_fence_after_sync();
                if (KV && elect_one()) mma_grad(tG2, tS(g), sY2(it & 1), g, it > 0 || g > 0);
                if (elect_one()) { mma_grad(tG1, tdP(g), sY1(it & 1), g, it > 0 || g > 0); }
                if (elect_one()) { umma_commit(done(g)); }
                if (g == 1 && it + 2 < n_it && elect_one()) umma_commit(empty(it & 1));
                if (it + 1 < n_it) scores(it + 1, g);
                else if (g == 1 && elect_one()) umma_commit(acc_full);
            }
        }
    } else {
        const int g = warp >> 2, t = threadIdx.x & 127;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const float c = p.scale * kLog2e;
        float nl = 0.f, nd = 0.f;
        int yh = head * group, yt = xt;             // KV: the queries whose statistics are requested next
        float st[4] = {};
        auto request = [&]() {
            const long long at = ((long long)b * p.Hq + yh) * p.S + yt * kT + g * 64 + lane;
            st[0] = p.lse[at]; st[1] = p.lse[at + 32]; st[2] = p.dsum[at]; st[3] = p.dsum[at + 32];
            if (++yt == n_qt) { yt = xt; ++yh; }
        };
        if (KV) {
            request();
        } else {
            const long long at = ((long long)b * p.Hq + head) * p.S + xt * kT + t;
            nl = -p.lse[at] * kLog2e;
            nd = -p.dsum[at];
        }
        bool ok = true;
        for (int it = 0, i = 0; it < n_it; ++it) {
            float* mine = stats + (warp * 2 + (it & 1)) * 128;
            if (KV) {
                mine[lane] = -st[0] * kLog2e; mine[lane + 32] = -st[1] * kLog2e; mine[lane + 64] = -st[2]; mine[lane + 96] = -st[3];
                __syncwarp();
                if (it + 1 < n_it) request();
            }
            ok = mbar_wait_warp(sd_full(g), it & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 40);
            if (!ok) break;
            tc_fence_after_sync();
            bwd_rows<KV>(tS(g) + lane_off, tdP(g) + lane_off, g, t, KV ? i == 0 : it == n_it - 1, c, p.scale, nl, nd, mine);
            if (++i == n_i) i = 0;
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(ds_full(g));
        }
        if (ok) ok = mbar_wait_warp(acc_full, 0, abort_flag, p.status, ST_TIMEOUT_ACCUM, 41);
        // KV: the first group stores dK, the second dV; else each half the columns of dQ. The walk is over: its tiles serve as staging.
        const uint32_t stage = (KV ? 2 + g : 2) * kTile + (KV ? 0 : g * kBlk), acc = (KV && g ? tG2 : tG1) + lane_off + (KV ? 0 : 64 * g);
        if (ok) {
            tc_fence_after_sync();
            stage_block(acc, t, smem + stage);
            if (KV) stage_block(acc + 64, t, smem + stage + kBlk);
            fence_proxy_async_smem();
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");
        if (ok && t == 0) {
            const CUtensorMap* map = KV && g ? &tmG2 : &tmG1;
            tma_store_2d(map, base + stage, head * kD + (KV ? 0 : 64 * g), row0 + xt * kT);
            if (KV) tma_store_2d(map, base + stage + kBlk, head * kD + 64, row0 + xt * kT);
            tma_store_commit();
            tma_store_wait_all();
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 8) { tc_fence_after_sync(); tmem_dealloc(tmem, 512); }
}

int check_attn(const AttnArgs& a) {
    if (a.B <= 0 || a.S <= 0 || a.Hq <= 0 || a.Hkv <= 0 || a.Hq % a.Hkv) { set_last_error("attention: bad shape B=%d S=%d Hq=%d Hkv=%d", a.B, a.S, a.Hq, a.Hkv); return PLZ_ERR_BAD_SHAPE; }
    if (a.S % kT) { set_last_error("attention: the sequence length %d must be a multiple of 128", a.S); return PLZ_ERR_BAD_SHAPE; }
    if (a.head_dim != kD) { set_last_error("attention: head_dim %d (only 128 is built)", a.head_dim); return PLZ_ERR_UNSUPPORTED; }
    return PLZ_OK;
}

template <typename K>
int set_smem(K kern, uint32_t bytes) {
    PLZ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    return PLZ_OK;
}

}  // namespace

int launch_attn_fwd(const AttnArgs& a, cudaStream_t stream) {
    int rc = check_attn(a);
    if (rc) return rc;
    if (!a.q || !a.k || !a.v || !a.o) { set_last_error("attention: null pointer"); return PLZ_ERR_NULL; }
    const uint64_t rows = (uint64_t)a.B * a.S;
    CUtensorMap tmQ, tmK, tmV, tmO;
    if ((rc = make_tmap_bf16(&tmQ, a.q, rows, (uint64_t)a.Hq * kD, a.ldq, 64, kT))) return rc;
    if ((rc = make_tmap_bf16(&tmK, a.k, rows, (uint64_t)a.Hkv * kD, a.ldk, 64, kT))) return rc;
    if ((rc = make_tmap_bf16(&tmV, a.v, rows, (uint64_t)a.Hkv * kD, a.ldv, 64, kT))) return rc;
    if ((rc = make_tmap_bf16(&tmO, a.o, rows, (uint64_t)a.Hq * kD, a.ldo, 64, kT))) return rc;
    AttnParams p = {};
    p.B = a.B; p.S = a.S; p.Hq = a.Hq; p.Hkv = a.Hkv; p.scale = a.scale; p.lse = a.lse; p.status = device_status_ptr();
    static bool once = false;
    if (!once) { if ((rc = set_smem(attn_fwd_kernel, kFwdSmem))) return rc; once = true; }
    PLZ_LAUNCH_BEHIND(attn_fwd_kernel, dim3(a.Hq * a.B, (a.S / kT + 1) / 2), dim3(kFwdThreads), kFwdSmem, stream, tmQ, tmK, tmV, tmO, p);
    return PLZ_OK;
}

int launch_attn_bwd(const AttnArgs& a, cudaStream_t stream) {
    int rc = check_attn(a);
    if (rc) return rc;
    if (!a.q || !a.k || !a.v || !a.o || !a.d_o || !a.dq || !a.dk || !a.dv || !a.lse || !a.dsum) { set_last_error("attention backward: null pointer"); return PLZ_ERR_NULL; }
    if ((uintptr_t)a.o & 7) { set_last_error("attention backward: o must be 8-byte aligned"); return PLZ_ERR_BAD_ALIGN; }
    const uint64_t rows = (uint64_t)a.B * a.S;
    CUtensorMap tmQ, tmK, tmV, tmdO, tmdQ, tmdK, tmdV;
    if ((rc = make_tmap_bf16(&tmQ, a.q, rows, (uint64_t)a.Hq * kD, a.ldq, 64, kT))) return rc;
    if ((rc = make_tmap_bf16(&tmK, a.k, rows, (uint64_t)a.Hkv * kD, a.ldk, 64, kT))) return rc;
    if ((rc = make_tmap_bf16(&tmV, a.v, rows, (uint64_t)a.Hkv * kD, a.ldv, 64, kT))) return rc;
    if ((rc = make_tmap_bf16(&tmdO, a.d_o, rows, (uint64_t)a.Hq * kD, a.ldo, 64, kT))) return rc;
    if ((rc = make_tmap_bf16(&tmdQ, a.dq, rows, (uint64_t)a.Hq * kD, a.ldq, 64, kT))) return rc;
    if ((rc = make_tmap_bf16(&tmdK, a.dk, rows, (uint64_t)a.Hkv * kD, a.ldk, 64, kT))) return rc;
    if ((rc = make_tmap_bf16(&tmdV, a.dv, rows, (uint64_t)a.Hkv * kD, a.ldv, 64, kT))) return rc;
    AttnParams p = {};
    p.B = a.B; p.S = a.S; p.Hq = a.Hq; p.Hkv = a.Hkv; p.scale = a.scale; p.lse = a.lse; p.dsum = a.dsum; p.status = device_status_ptr();
    static bool once = false;
    if (!once) {
        if ((rc = set_smem(attn_bwd_kernel<false>, kBwdSmem))) return rc;
        if ((rc = set_smem(attn_bwd_kernel<true>, kBwdSmem))) return rc;
        once = true;
    }
    const long long n_rows = (long long)a.B * a.S * a.Hq;
    const auto dsum = ((uintptr_t)a.o & 15) ? attn_dsum_kernel<false> : attn_dsum_kernel<true>;   // o passes no tensor map that would refuse it
    PLZ_LAUNCH_BEHIND(dsum, dim3((unsigned)((n_rows + 63) / 64)), dim3(256), 0, stream, (const __nv_bfloat16*)a.o, (const __nv_bfloat16*)a.d_o, a.ldo, a.B, a.S, a.Hq, a.dsum);
    PLZ_LAUNCH_BEHIND(attn_bwd_kernel<false>, dim3(a.Hq * a.B, a.S / kT), dim3(kBwdThreads), kBwdSmem, stream, tmQ, tmdO, tmK, tmV, tmdQ, tmdQ, p);
    PLZ_LAUNCH_BEHIND(attn_bwd_kernel<true>, dim3(a.Hkv * a.B, a.S / kT), dim3(kBwdThreads), kBwdSmem, stream, tmK, tmV, tmQ, tmdO, tmdK, tmdV, p);
    return PLZ_OK;
}

}  // namespace plz
