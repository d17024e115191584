// Large products with a dense bf16 matrix on CTA PAIRS (tcgen05.mma.cta_group::2, M = 256): the Linears of the hybrid decoders over prompts
// (optional bias, squared relu or gated gelu) and the soft-weight products with their LoRA block. The counterpart of lut_gemm_pair.cu, whose
// split, barriers and tile plan it shares; here both operands come by TMA, so a CTA is a producer warp, an MMA warp and four epilogue warps.
//
// Bound by the tensor cores where the tiles fill the waves. Against a CTA per 256 x 256 tile (lut_gemm.cu) an SM reads 8 instead of 12 KB of
// operands per 128 x 256 x 16 of work and holds two accumulators, so that a tile's epilogue runs under the next one's main loop; a last wave
// of few tiles is cut, and few tiles are made narrow enough to fill the chip once.
// us there / here: 1000 rows, 2560 x 9728 97 / 49, 19456 x 2560 gated 90 / 72; 2048 rows, 2560 x 9728 103 / 90, 9728 x 2560 88 / 73.
#include "plz_launch.h"

namespace plz {
namespace {

constexpr int kDpEpiWarps = 4;
constexpr int kDpThreads = (2 + kDpEpiWarps) * 32;
constexpr int kDpStages = 3;
constexpr int kDpBK = 128;                       // reduction elements per stage: two 64-wide swizzle blocks
// Tiles are dealt out row tile fastest inside bands of eight row tiles: the 74 tiles in flight are then about 8 x 9, whose operands are a few MB
// per pass; column tile fastest would stream the whole matrix once per row tile (100 MB of gate / up weights do not stay in L2).
constexpr int kDpBand = 8;
constexpr uint32_t kDpBlkBytes = 128 * 64 * 2;
constexpr uint32_t kDpABytes = 2 * kDpBlkBytes;
constexpr uint32_t kDpStageBytes = 2 * kDpABytes;
constexpr uint32_t kDpEpiOff = kDpStages * kDpStageBytes;
constexpr uint32_t kDpEpiBytes = 32 * 64 * 2;
constexpr uint32_t kDpBarOff = kDpEpiOff + kDpEpiWarps * kDpEpiBytes;
constexpr uint32_t kDpSmemBytes = kDpBarOff + 1024 + 256;

struct DpParams {
    int lets_next;           // let the next kernel start behind this one's wait
    int M, J, R, out_cols;
    int n_extra;             // 0 or 1 extra 64-wide reduction block from (A2, B2)
    int tiles_m, tiles_j, tile_w, n_whole, n_items;   // plan_pair_tiles
    float alpha;
    const __nv_bfloat16* bias;               // optional [J]
    int relu2;
    StatusWord* status;
};

// tanh form of gelu, z * sigmoid(2 sqrt(2 / pi) (z + 0.044715 z^3))
__device__ __forceinline__ float gelu_gate(float z) {
    return __fdividef(z, 1.0f + exp2f(fminf(-2.302208198f * fmaf(0.044715f * z * z, z, z), 80.0f)));
}

// BMN: B is [R, J] (else [J, R]); GLU: columns 2 i, 2 i + 1 are a gate / up pair of output i
template <bool BMN, bool GLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kDpThreads, 1)
dense_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmBh,
                       const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmD,
                       const __grid_constant__ CUtensorMap tmD16, const DpParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    const uint32_t bar_base = base + kDpBarOff;
    auto full = [&](int s) { return bar_base + 8u * s; };                         // leader's copy: the bytes of both CTAs
    auto empty = [&](int s) { return bar_base + 8u * (kDpStages + s); };          // own copy: multicast commit of the leader
    auto acc_full = [&](int b) { return bar_base + 8u * (2 * kDpStages + b); };   // own copy
    auto acc_empty = [&](int b) { return bar_base + 8u * (2 * kDpStages + 2 + b); };   // leader's copy: epilogue warps of both CTAs
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + kDpBarOff + 8 * (2 * kDpStages + 4));
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0);   // uniform to the compiler too
    const int lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    const uint32_t lead_bar_base = leader_addr(bar_base);
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int nkb = (p.R + kDpBK - 1) / kDpBK, nkb_total = nkb + p.n_extra;   // columns past R read as zero on both sides

    if (threadIdx.x == 0) {
        for (int s = 0; s < kDpStages; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 2 * kDpEpiWarps); }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        tma_prefetch_desc(&tmD);
        if (p.n_extra) { tma_prefetch_desc(&tmA2); tma_prefetch_desc(&tmB2); }
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32((const void*)tmem_slot), 512);
        tmem_relinquish_pair();
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();   // both CTAs' barriers are initialised before anyone arrives on the other's
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    if (p.lets_next) pdl_launch_dependents();

    auto item_width = [&](int t) { return t < p.n_whole ? p.tile_w : 128; };
    auto item_origin = [&](int t, int& m0, int& j0) {
        const int cut = t - p.n_whole;                       // >= 0: a half tile
        const int tile = cut < 0 ? t : p.n_whole + (cut >> 1);
        const int band = tile / (kDpBand * p.tiles_j), in = tile - band * kDpBand * p.tiles_j, rows = min(kDpBand, p.tiles_m - band * kDpBand);
        j0 = (in / rows) * p.tile_w + (cut < 0 ? 0 : (cut & 1) * 128);
        m0 = (band * kDpBand + in % rows) * 256;
    };

    int issued = 0;        // stages the producing thread has filled
    if (warp == 0) {
        // ------------------------------------------------------------- TMA producer (one per CTA)
        if (lane == 0) {
            bool ok = true;
            int s = 0;
            uint32_t ph = 0;
            for (int t = pair; t < p.n_items && ok; t += n_pairs) {
                int m0, j0;
                item_origin(t, m0, j0);
                const int half = item_width(t) >> 1, boxes = (half + 63) >> 6;     // BMN: boxes of 64 columns
                const int mrow = m0 + 128 * rank, jr = j0 + half * rank;
                const CUtensorMap* mb = t < p.n_whole ? &tmB : &tmBh;
                const uint32_t b_bytes = BMN ? (uint32_t)boxes * kDpBlkBytes : (uint32_t)half * 256u;
                for (int it = 0; it < nkb_total; ++it) {
                    ok = mbar_wait(empty(s), ph ^ 1u, abort_flag, p.status, ST_TIMEOUT_EMPTY, 0);
                    if (!ok) break;
                    const uint32_t sA = base + s * kDpStageBytes, sB = sA + kDpABytes, bar = lead_bar_base + 8u * s;
                    if (it < nkb) {
                        // the leader announces the bytes of BOTH CTAs for this stage
                        if (rank == 0) mbar_arrive_expect_tx(full(s), 2u * (kDpABytes + b_bytes));
                        tma_load_2d_pair(sA, &tmA, bar, it * kDpBK, mrow);
                        tma_load_2d_pair(sA + kDpBlkBytes, &tmA, bar, it * kDpBK + 64, mrow);
                        if (BMN) {
                            for (int b = 0; b < boxes; ++b) tma_load_2d_pair(sB + b * kDpBlkBytes, &tmB, bar, jr + 64 * b, it * kDpBK);
                        } else {
                            tma_load_2d_pair(sB, mb, bar, it * kDpBK, jr);
                            tma_load_2d_pair(sB + kDpBlkBytes, mb, bar, it * kDpBK + 64, jr);
                        }
                    } else {
                        // the LoRA block is one 64-wide block (BMN: two boxes of 64 columns by 64 rows)
                        if (rank == 0) mbar_arrive_expect_tx(full(s), 4u * kDpBlkBytes);
                        tma_load_2d_pair(sA, &tmA2, bar, 0, mrow);
                        if (BMN) {
                            tma_load_2d_pair(sB, &tmB2, bar, jr, 0);
                            tma_load_2d_pair(sB + kDpBlkBytes, &tmB2, bar, jr + 64, 0);
                        } else {
                            tma_load_2d_pair(sB, &tmB2, bar, 0, jr);
                        }
                    }
                    ++issued;
                    if (++s == kDpStages) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------- MMA issuer (leader only)
        // the whole warp walks the stages and one elected lane issues (narrow_gemm.cu: operands stay in uniform registers)
        if (rank == 0) {
            const uint32_t idesc_whole = make_idesc(256, p.tile_w, 0, BMN ? 1 : 0), idesc_half = make_idesc(256, 128, 0, BMN ? 1 : 0);
            const uint64_t ad0 = make_sdesc(base, 16u, 1024u);
            const uint64_t bd0 = BMN ? make_sdesc(base + kDpABytes, kDpBlkBytes, 1024u) : make_sdesc(base + kDpABytes, 16u, 1024u);
            const uint32_t a_hi = (uint32_t)(ad0 >> 32), b_hi = (uint32_t)(bd0 >> 32), a_lo0 = (uint32_t)ad0, b_lo0 = (uint32_t)bd0;
            uint32_t a_lo = a_lo0, b_lo = b_lo0;
            bool ok = true;
            int s = 0, lt = 0;
            uint32_t ph = 0;
            for (int t = pair; t < p.n_items && ok; t += n_pairs, ++lt) {
                const uint32_t d_tmem = tmem_base + (uint32_t)(lt & 1) * 256u;
                const uint32_t idesc = t < p.n_whole ? idesc_whole : idesc_half;
                ok = __all_sync(0xFFFFFFFFu, mbar_wait_lean(acc_empty(lt & 1), ((lt >> 1) & 1) ^ 1u, abort_flag, p.status, ST_TIMEOUT_ACCUM, 1));
                if (!ok) break;
                tc_fence_after_sync();
                for (int it = 0; it < nkb_total; ++it) {
                    ok = __all_sync(0xFFFFFFFFu, mbar_wait_lean(full(s), ph, abort_flag, p.status, ST_TIMEOUT_FULL, 1));
                    if (!ok) break;
                    tc_fence_after_sync();
                    // k step ks: A and K-major B advance 32 bytes inside a 64-wide block and one block after four steps;
                    // MN-major B advances 16 rows of 128 bytes. The LoRA block is 64 wide: four steps
                    const uint32_t more = it > 0 ? 1u : 0u;
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks)
                            umma_bf16_words<2>(d_tmem, a_lo + ks * 2, a_hi, b_lo + (BMN ? ks * (2048 >> 4) : ks * 2), b_hi, idesc, ks > 0 ? 1u : more);
                        if (it < nkb) {
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks)
                                umma_bf16_words<2>(d_tmem, a_lo + (kDpBlkBytes >> 4) + ks * 2, a_hi, b_lo + (BMN ? (ks + 4) * (2048 >> 4) : (int)(kDpBlkBytes >> 4) + ks * 2), b_hi, idesc, 1u);
                        }
                        umma_commit_pair(empty(s));
                    }
                    __syncwarp();
                    if (++s == kDpStages) { s = 0; ph ^= 1u; a_lo = a_lo0; b_lo = b_lo0; }
                    else { a_lo += kDpStageBytes >> 4; b_lo += kDpStageBytes >> 4; }
                }
                if (ok && elect_one()) umma_commit_pair(acc_full(lt & 1));
                __syncwarp();
            }
        }
    } else {
        // ------------------------------------------------------------- epilogue warps: TMEM lanes 32 * (warp % 4), boxes of 64 outputs (of 16 where the tile ends sooner)
        const int lane_group = warp & 3;
        uint8_t* stage = smem + kDpEpiOff + (warp - 2) * kDpEpiBytes;
        const uint32_t stage_u32 = base + kDpEpiOff + (warp - 2) * kDpEpiBytes;
        const uint32_t lane_base = tmem_base + ((uint32_t)(lane_group * 32) << 16);
        bool ok = true;
        int lt = 0;
        for (int t = pair; t < p.n_items && ok; t += n_pairs, ++lt) {
            int m0, j0;
            item_origin(t, m0, j0);
            const int buf = lt & 1, w = item_width(t), w_out = GLU ? w >> 1 : w, o0 = GLU ? j0 >> 1 : j0;
            const int mrow = m0 + 128 * rank + lane_group * 32;
            ok = mbar_wait(acc_full(buf), (lt >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 4);
            if (!ok) break;
            tc_fence_after_sync();
#pragma unroll 1
            for (int col = 0; col < w_out; col += 64) {
                const int left = w_out - col;
                const bool wide = left >= 64;
                if (lane == 0) tma_store_wait_read();       // the previous box must have been read out of the staging buffer
                __syncwarp();
                // 32 accumulator columns: 32 outputs, or 16 gated ones
                constexpr int kChunks = GLU ? 4 : 2, kOut = GLU ? 16 : 32;
#pragma unroll
                for (int c = 0; c < kChunks; ++c) {
                    if (c * kOut >= left) break;
                    uint32_t v[32];
                    const int at = (GLU ? 2 * col : col) + c * 32;
                    tmem_ld_32x32(lane_base + buf * 256u + at, v);
                    if (at + 32 >= w) {
                        // last read of this accumulator: hand it back to the MMA thread of the leader
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(lead_bar_base + 8u * (2 * kDpStages + 2 + buf));
                    }
#pragma unroll
                    for (int g = 0; g < kOut / 8; ++g) {
                        float f[8];
                        if (GLU) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) f[i] = gelu_gate(__uint_as_float(v[g * 16 + 2 * i])) * __uint_as_float(v[g * 16 + 2 * i + 1]);
                        } else {
                            uint4 bb = make_uint4(0u, 0u, 0u, 0u);
                            const int jc = j0 + col + c * 32 + g * 8;        // J is a multiple of 8
                            if (p.bias != nullptr && jc < p.J) bb = __ldg(reinterpret_cast<const uint4*>(p.bias + jc));
                            const uint32_t bw[4] = {bb.x, bb.y, bb.z, bb.w};
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const float b = __uint_as_float((i & 1) ? (bw[i >> 1] & 0xFFFF0000u) : (bw[i >> 1] << 16));
                                f[i] = __uint_as_float(v[g * 8 + i]) * p.alpha + b;
                                if (p.relu2) { const float r = fmaxf(f[i], 0.f); f[i] = r * r; }
                            }
                        }
                        const int chunk = c * (kOut / 8) + g;
                        const uint32_t to = wide ? swz128(lane, chunk) : (uint32_t)((chunk >> 1) * 1024 + lane * 32 + ((chunk & 1) << 4));
                        *reinterpret_cast<uint4*>(stage + to) = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
                    }
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0 && o0 + col < p.out_cols && mrow < p.M) {
                    if (wide) tma_store_2d(&tmD, stage_u32, o0 + col, mrow);
                    else
                        for (int b = 0; b * 16 < left && o0 + col + b * 16 < p.out_cols; ++b) tma_store_2d(&tmD16, stage_u32 + b * 1024u, o0 + col + b * 16, mrow);
                    tma_store_commit();
                }
            }
        }
        if (lane == 0) tma_store_wait_all();
    }
    // neither CTA may leave while its partner can still touch its shared or tensor memory
    tc_fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0 && rank == 0 && *abort_flag) {
        // somebody gave up: the copies of both CTAs, which arrive on this CTA's barriers, get a bounded chance to land
        const uint64_t t0 = globaltimer_ns();
        for (int it = issued > kDpStages ? issued - kDpStages : 0; it < issued; ++it)
            while (!mbar_try_wait(full(it % kDpStages), (it / kDpStages) & 1))
                if (globaltimer_ns() - t0 > 100000000ull) { report(p.status, ST_TIMEOUT_DRAIN, 0); break; }
    }
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

template <bool BMN, bool GLU>
int launch_dp(const LutGemmArgs& a, int sms, cudaStream_t stream) {
    DpParams p = {};
    p.M = a.M; p.J = a.J; p.R = a.R; p.out_cols = GLU ? a.J / 2 : a.J; p.n_extra = a.r2 > 0 ? 1 : 0;
    p.alpha = a.alpha; p.bias = (const __nv_bfloat16*)a.bias; p.relu2 = a.fuse == 3 && a.act == 1;
    p.status = device_status_ptr();
    p.lets_next = !g_smallm_overlap;
    int pairs = sms / 2;
    // columns of a row-major B come in boxes of 64, so there other widths would read what they do not use
    const PairTiles pt = GLU ? plan_pair_tiles(a.M, a.J, pairs, 64) : BMN ? plan_pair_tiles(a.M, a.J, pairs, 32) : plan_pair_waves(a.M, a.J, pairs, 16);
    p.tiles_m = (a.M + 255) / 256; p.tiles_j = pt.tiles_j; p.tile_w = pt.tile_w; p.n_whole = pt.n_whole; p.n_items = pt.n_items;
    if (pairs > p.n_items) pairs = p.n_items;
    CUtensorMap tmA, tmB, tmBh, tmA2, tmB2, tmD, tmD16;
    int rc;
    if ((rc = make_tmap_bf16(&tmA, a.A, a.M, a.R, a.lda, 64, 128))) return rc;
    if (BMN) {
        if ((rc = make_tmap_bf16(&tmB, a.Bdense, a.R, a.J, a.ldb, 64, 128))) return rc;
        tmBh = tmB;
    } else {
        if ((rc = make_tmap_bf16(&tmB, a.Bdense, a.J, a.R, a.ldb, 64, (uint32_t)p.tile_w / 2))) return rc;
        if ((rc = make_tmap_bf16(&tmBh, a.Bdense, a.J, a.R, a.ldb, 64, 64))) return rc;
    }
    tmA2 = tmA; tmB2 = tmA;
    if (a.r2 > 0) {
        if ((rc = make_tmap_bf16(&tmA2, a.A2, a.M, a.r2, a.lda2, 64, 128))) return rc;
        if (BMN) {
            if ((rc = make_tmap_bf16(&tmB2, a.B2, a.r2, a.J, a.ldb2, 64, 64))) return rc;
        } else {
            if ((rc = make_tmap_bf16(&tmB2, a.B2, a.J, a.r2, a.ldb2, 64, 128))) return rc;
        }
    }
    if ((rc = make_tmap_bf16(&tmD, a.out, a.M, p.out_cols, a.ld_out, 64, 32))) return rc;
    if ((rc = make_tmap_bf16(&tmD16, a.out, a.M, p.out_cols, a.ld_out, 16, 32))) return rc;
    auto kern = dense_gemm_pair_kernel<BMN, GLU>;
    static bool attr_set[64] = {};
    int dev = 0;
    PLZ_CUDA_CHECK(cudaGetDevice(&dev));
    if (!attr_set[dev & 63]) {
        PLZ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kDpSmemBytes));
        attr_set[dev & 63] = true;
    }
    PLZ_LAUNCH_BEHIND(kern, dim3(2 * pairs), dim3(kDpThreads), kDpSmemBytes, stream, tmA, tmB, tmBh, tmA2, tmB2, tmD, tmD16, p);
    return PLZ_OK;
}

}  // namespace

// PLZ_ERR_UNSUPPORTED: not a shape for this kernel, the caller falls back to the single-CTA kernel.
int launch_dense_gemm_pair(const LutGemmArgs& a, cudaStream_t stream) {
    const bool mn = a.bmode == B_TMA_MN;
    if (!g_pair_gemm || (!mn && a.bmode != B_TMA_K) || a.M < 256 || a.J < 256) return PLZ_ERR_UNSUPPORTED;
    if ((a.fuse != 0 && a.fuse != 3 && a.fuse != 4) || (a.fuse && (mn || a.r2)) || (a.fuse == 4 && (a.J % 16 || a.alpha != 1.0f))) return PLZ_ERR_UNSUPPORTED;
    if (((uintptr_t)a.bias & 15) || (a.bias && a.fuse != 3)) return PLZ_ERR_UNSUPPORTED;
    int dev = 0, sms = 0;
    PLZ_CUDA_CHECK(cudaGetDevice(&dev));
    PLZ_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (a.sm_limit > 0 && a.sm_limit < sms) sms = a.sm_limit;
    if (g_cta_limit > 0 && g_cta_limit < sms) sms = g_cta_limit;
    if (sms < 2) return PLZ_ERR_UNSUPPORTED;
    if (mn) return launch_dp<true, false>(a, sms, stream);
    return a.fuse == 4 ? launch_dp<false, true>(a, sms, stream) : launch_dp<false, false>(a, sms, stream);
}

}  // namespace plz
