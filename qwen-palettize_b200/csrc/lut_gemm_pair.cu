// lut_gemm_pair: the two large palettized products, y = x W^T and dX = dY W (+ the LoRA block), on CTA PAIRS
// (tcgen05.mma.cta_group::2, M = 256): two CTAs of a cluster share one 256 x 256 output tile.
//
//   CTA r of the pair (r = rank in the cluster, 0 = leader)
//     - loads by TMA the 128 rows [m0 + 128 r, +128) of A into ITS shared memory,
//     - decodes the 128 B columns [j0 + 128 r, +128) of the tile (half of the packed weights) into ITS shared memory,
//     - owns the accumulator rows [128 r, +128) x 256 columns in ITS tensor memory and writes them out.
//   The leader's one MMA thread issues a single 256 x 256 x 16 instruction per 16 reduction elements; the hardware reads A
//   from each CTA's own shared memory and each half of B from the CTA that holds it.
//
// Against one CTA per tile (lut_gemm.cu: two 128 x 256 x 16 instructions that both re-read the 8 KB of B) this
//   * cuts shared-memory operand reads per SM from 12 KB to 8 KB per 128 x 256 x 16 of work (the single-CTA kernel ran at
//     about 140 B/cycle of demand against 128 B/cycle of shared-memory bandwidth),
//   * halves each CTA's accumulator to 256 of the 512 tensor-memory columns, so TWO accumulators fit and the epilogue of
//     tile i overlaps the main loop of tile i + 1,
//   * lets a stage span 128 reduction elements (32 KB A + 32 KB B per CTA): eight MMAs per barrier round trip.
// The thread that issues the MMAs is kept lean (precomputed descriptor words, one wait and one commit per stage): a lone
// thread retires a dependent instruction every five or six cycles, an MMA lasts 128, so two dozen instructions per MMA
// are enough to starve the tensor pipe.
//
// Synchronisation (every barrier named here lives at the same shared-memory offset in both CTAs):
//   full[s]     leader's copy: the leader's producer announces both CTAs' TMA bytes (each CTA's copies complete on the
//               LEADER's barrier) and the decode warps of one group of BOTH CTAs arrive once (remote arrive from the peer)
//   empty[s]    own copy in each CTA: tcgen05.commit of the leader, multicast to both CTAs
//   acc_full[b] own copy in each CTA: tcgen05.commit multicast after the last reduction block of a tile
//   acc_empty[b] leader's copy: one arrival per epilogue warp of BOTH CTAs
// No load uses cluster multicast: every CTA issues its own plain TMA copies.
//
// Tiles narrower than 256 columns (plan_pair_tiles). A launch ends when its last wave does, and a wave of a few tiles costs as much as a full one:
// 4096 x 2560 outputs are 160 tiles on 74 pairs, two full waves and one with twelve tiles. So where the tiles of the last wave, cut in halves of
// 128 columns, still fit one wave, they are; and a launch with fewer tiles than pairs takes the narrowest tile (32-column steps) that still
// fits one wave. Below 128 columns the rows of A, 32 KB per stage and CTA, arrive no faster than the tensor cores would use them up.
// The order of every sum is that of a 256-column tile.
//
// Replaces, in the reference: fused_lut_linear_fwd_tc_kernel (scripts/fused_lut_kernel.cu:309),
// fused_lut_linear_bwd_grad_x_tc_kernel (:551) and the cuBLAS calls of the soft path
// (scripts/fused_lut_linear_cuda.py:912, :944), as lut_gemm.cu does for the shapes this kernel does not take.
#include "plz_launch.h"

namespace plz {

int g_pair_gemm = 1;  // 0: never use the CTA-pair kernel (comparisons, tests of the single-CTA kernel)

namespace {

struct PairParams {
    int lets_next;           // let the next kernel start behind this one's wait
    int M, J, R;
    int n_extra;             // 0 or 1 extra 64-wide reduction block from (A2, B2)
    int tiles_j, tile_w;     // column tiles of tile_w columns
    int n_whole, n_items;    // items [0, n_whole) are whole tiles, the others halves of 128 columns of the tiles behind (tile_w = 256 then)
    const uint8_t* packed; long long packed_pitch;
    const __nv_bfloat16* palette;
    const uint8_t* packed2; const __nv_bfloat16* palette2;   // GLU: the up projection
    int gs_n, gs_k, n_kgroups, gs_n_shift;
    int gs_k_shift;          // log2(gs_k / 64) or -1
    int Wn, Wk;
    float alpha;
    const __nv_bfloat16* bias;   // optional [J], added in fp32 before the rounding
    StatusWord* status;
    unsigned long long* prof;  // diagnostics build: [gridDim][8] cycle counters (MMA thread 0..4, one decode thread 5..6)
};

constexpr int kDecodeWarps = 16;
constexpr int kEpiWarps = 4;   // one per TMEM lane group; the epilogue of a tile overlaps the main loop of the next
constexpr int kFirstEpiWarp = 2 + kDecodeWarps;
constexpr int kThreads = (2 + kDecodeWarps + kEpiWarps) * 32;  // 704
constexpr int kStages = 3;
constexpr int kBK = 128;                      // reduction elements per stage: two 64-wide (128-byte) swizzle blocks
constexpr uint32_t kBlkBytes = 128 * 64 * 2;  // one 64-wide block of 128 rows
constexpr uint32_t kABytes = 2 * kBlkBytes;   // this CTA's 128 rows of A
constexpr uint32_t kBBytes = 2 * kBlkBytes;   // this CTA's 128 columns of B
constexpr uint32_t kStageBytes = kABytes + kBBytes;
constexpr uint32_t kEpiStageBytes = 32 * 64 * 2;
constexpr uint32_t kEpiOff = kStages * kStageBytes;
constexpr uint32_t kBarOff = kEpiOff + kEpiWarps * kEpiStageBytes;
constexpr uint32_t kSmemBytes = kBarOff + 1024 + 256;

// GLU (forward): the tile's columns are the same outputs of a gate and of an up projection, half and half, one decoded by either CTA, and the
// epilogue writes silu(gate) * up: of a feed-forward's 4096 x 9728 outputs 80 MB reach memory, where the products apart and an element-wise pass move 400.
template <int BMODE, bool GLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
lut_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmA2,
                     const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmD32,
                     const PairParams p) {
    constexpr bool kBMn = (BMODE == B_DECODE_MN);
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    const uint32_t bar_base = base + kBarOff;
    auto full = [&](int s) { return bar_base + 8u * s; };
    auto empty = [&](int s) { return bar_base + 8u * (kStages + s); };
    auto acc_full = [&](int b) { return bar_base + 8u * (2 * kStages + b); };
    auto acc_empty = [&](int b) { return bar_base + 8u * (2 * kStages + 2 + b); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + kBarOff + 8 * (2 * kStages + 4));
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0);   // uniform to the compiler too
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();   // 0 = leader
    const uint32_t lead_bar_base = leader_addr(bar_base);   // the leader's barrier block as a shared::cluster address
    auto lead_full = [&](int s) { return lead_bar_base + 8u * s; };
    auto lead_acc_empty = [&](int b) { return lead_bar_base + 8u * (2 * kStages + 2 + b); };
    const int pair = blockIdx.x >> 1;
    const int n_pairs = gridDim.x >> 1;
    const int nkb = (p.R + kBK - 1) / kBK;   // a last stage that is only half covered reads zeros (TMA fill, decode bounds)
    const int nkb_total = nkb + p.n_extra;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full(s), 1 + kDecodeWarps);   // half of the decode warps of both CTAs
            mbar_init(empty(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full(b), 1);
            mbar_init(acc_empty(b), 2 * kEpiWarps);
        }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmD);
        if (p.tile_w & 32) tma_prefetch_desc(&tmD32);
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
        j0 = ((tile % p.tiles_j) * p.tile_w + (cut < 0 ? 0 : (cut & 1) * 128)) >> (GLU ? 1 : 0);
        m0 = (tile / p.tiles_j) * 256;
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
                const int mrow = m0 + 128 * (int)rank;
                const int jr = j0 + (item_width(t) >> 1) * (int)rank;
                for (int it = 0; it < nkb_total; ++it) {
                    ok = mbar_wait(empty(s), ph ^ 1u, abort_flag, p.status, ST_TIMEOUT_EMPTY, 0);
                    if (!ok) break;
                    const uint32_t sA = base + s * kStageBytes;
                    const uint32_t sB = sA + kABytes;
                    const bool extra = it >= nkb;
                    // the leader announces the bytes of BOTH CTAs for this stage
                    if (rank == 0) mbar_arrive_expect_tx(full(s), extra ? 4u * kBlkBytes : 2u * kABytes);
                    if (!extra) {
                        tma_load_2d_pair(sA, &tmA, lead_full(s), it * kBK, mrow);
                        tma_load_2d_pair(sA + kBlkBytes, &tmA, lead_full(s), it * kBK + 64, mrow);
                    } else {
                        // the LoRA block is one 64-wide block: A2 into block 0 of A, B2 by TMA into block 0 of B
                        tma_load_2d_pair(sA, &tmA2, lead_full(s), 0, mrow);
                        if (kBMn) {
                            tma_load_2d_pair(sB, &tmB2, lead_full(s), jr, 0);
                            tma_load_2d_pair(sB + kBlkBytes, &tmB2, lead_full(s), jr + 64, 0);
                        } else {
                            tma_load_2d_pair(sB, &tmB2, lead_full(s), 0, jr);
                        }
                    }
                    ++issued;
                    if (++s == kStages) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------- MMA issuer (leader only)
        // the whole warp walks the stages and one elected lane issues (narrow_gemm.cu: operands stay in uniform registers): 1000 rows,
        // 2560 x 9728 52 -> 46 us, input gradient at 512 rows 51 -> 40, 4096 rows, 9728 x 2560 165 -> 149
        if (rank == 0) {
            const uint32_t idesc_whole = make_idesc(256, p.tile_w, 0, kBMn ? 1 : 0), idesc_half = make_idesc(256, 128, 0, kBMn ? 1 : 0);
            // descriptor words of stage 0; a stage is kStageBytes >> 4 = 4096 further in the low word
            const uint64_t ad0 = make_sdesc(base, 16u, 1024u);
            const uint64_t bd0 = kBMn ? make_sdesc(base + kABytes, kBlkBytes, 1024u) : make_sdesc(base + kABytes, 16u, 1024u);
            const uint32_t a_hi = (uint32_t)(ad0 >> 32), b_hi = (uint32_t)(bd0 >> 32);
            uint32_t a_lo = (uint32_t)ad0, b_lo = (uint32_t)bd0;
            const uint32_t a_lo0 = a_lo, b_lo0 = b_lo;
            bool ok = true;
            int s = 0, lt = 0;
            uint32_t ph = 0;
            long long wait_f = 0, wait_t = 0;
            const long long t_begin = PLZ_PROF_ON(p.prof) ? clock64() : 0;
            for (int t = pair; t < p.n_items && ok; t += n_pairs, ++lt) {
                const uint32_t d_tmem = tmem_base + (uint32_t)(lt & 1) * 256u;
                const uint32_t idesc = t < p.n_whole ? idesc_whole : idesc_half;
                const long long c_t = PLZ_PROF_ON(p.prof) ? clock64() : 0;
                ok = __all_sync(0xFFFFFFFFu, mbar_wait_lean(acc_empty(lt & 1), ((lt >> 1) & 1) ^ 1u, abort_flag, p.status, ST_TIMEOUT_ACCUM, 1));
                if (PLZ_PROF_ON(p.prof)) wait_t += clock64() - c_t;
                if (!ok) break;
                tc_fence_after_sync();
                for (int it = 0; it < nkb_total; ++it) {
                    const long long c0 = PLZ_PROF_ON(p.prof) ? clock64() : 0;
                    ok = __all_sync(0xFFFFFFFFu, mbar_wait_lean(full(s), ph, abort_flag, p.status, ST_TIMEOUT_FULL, 1));
                    if (PLZ_PROF_ON(p.prof)) wait_f += clock64() - c0;
                    if (!ok) break;
                    tc_fence_after_sync();
                    // k step ks: A and K-major B advance 32 bytes inside a 64-wide block and one block (16 KB) after four
                    // steps; MN-major B advances 16 rows of 128 bytes. The LoRA block is 64 wide: four steps
                    const uint32_t more = it > 0 ? 1u : 0u;
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks)
                            umma_bf16_words<2>(d_tmem, a_lo + ks * 2, a_hi, b_lo + (kBMn ? ks * (2048 >> 4) : ks * 2), b_hi, idesc, ks > 0 ? 1u : more);
                        if (it < nkb) {
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks)
                                umma_bf16_words<2>(d_tmem, a_lo + (kBlkBytes >> 4) + ks * 2, a_hi, b_lo + (kBMn ? (ks + 4) * (2048 >> 4) : (int)(kBlkBytes >> 4) + ks * 2), b_hi, idesc, 1u);
                        }
                        umma_commit_pair(empty(s));
                    }
                    __syncwarp();
                    if (++s == kStages) { s = 0; ph ^= 1u; a_lo = a_lo0; b_lo = b_lo0; }
                    else { a_lo += kStageBytes >> 4; b_lo += kStageBytes >> 4; }
                }
                if (ok && elect_one()) umma_commit_pair(acc_full(lt & 1));
                __syncwarp();
            }
            if (PLZ_PROF_ON(p.prof) && lane == 0) {
                unsigned long long* o = p.prof + 8ull * blockIdx.x;
                o[0] = wait_f; o[1] = 0; o[2] = wait_t; o[3] = clock64() - t_begin; o[4] = lt;
            }
        }
    } else if (warp < kFirstEpiWarp) {
        // ------------------------------------------------------------- decode warps
        // Two groups of eight warps take the stages in turn: what a warp does per stage is a chain (wait, decode, store, proxy fence, arrive) of
        // about 0.7 us, as long as the MMAs of a whole stage, so with all warps on every stage it set the pace of narrow tiles.
        // 1000 rows, 2560 x 9728: 65 us with 256-column tiles and all warps on a stage, 58 with 160 columns, 52 with two groups; input gradient at
        // 512 rows 58 / 53 / 51 us; 4096 rows, 9728 x 2560 177 / 176 / 165 us.
        // The 256 threads of a group produce this CTA's half of the B stage, 128 columns x 128 reduction elements: 64 weights (twice eight bytes
        // of packed indices, eight 16-byte chunks of 128-byte operand rows) per thread, in the two 64-wide blocks b = 0, 1
        //   forward  (rows of the operand = n, blocks along k):                  row n = t / 2, half h = t % 2
        //   backward (rows of the operand = n of the stage, blocks of k columns): row = t / 2, h
        // Eight consecutive lanes cover four rows x two halves of one block, whose swizzled chunk positions are all different.
        // The index / palette loads run two of the group's stages ahead of the one being written, ACROSS tile boundaries: the sequence
        // of (tile, stage) positions of this pair is one stream, so a new tile does not start with an exposed load latency.
        const int grp = (threadIdx.x - 64) >> 8, t = (threadIdx.x - 64) & 255;
        const int h = t & 1, rr = t >> 1;
        const int blocks_per_kgroup = p.gs_k / 64;
        struct Pos {
            int tile, it;
            const uint8_t* ip;            // packed indices of this thread at stage 0 of the tile, block 0
            const __nv_bfloat16* pp;      // forward: palettes of this thread's row; backward: palette base
            int kg0, kg1;                 // backward: k groups of the two blocks
            bool ok0, ok1;                // the fixed coordinate (forward: n, backward: k of the block) lies inside the matrix and the tile
        };
        auto set_tile = [&](Pos& q) {
            int m0, j0;
            item_origin(q.tile, m0, j0);
            const int half = item_width(q.tile) >> 1;       // columns of this CTA; threads beyond them have nothing to fetch
            const int jr = j0 + half * (int)rank;
            if (kBMn) {
                const int k = jr + h * 32;
                q.ok0 = k < p.Wk && h * 32 < half;
                q.ok1 = k + 64 < p.Wk && h * 32 + 64 < half;
                q.kg0 = q.ok0 ? k / p.gs_k : 0;
                q.kg1 = q.ok1 ? (k + 64) / p.gs_k : 0;
                q.ip = p.packed + (long long)rr * p.packed_pitch + (k >> 2);
                q.pp = p.palette;
            } else {
                const int n = (GLU ? j0 : jr) + rr;
                q.ok0 = q.ok1 = n < p.Wn && rr < half;
                q.ip = (GLU && rank ? p.packed2 : p.packed) + (long long)n * p.packed_pitch + h * 8;
                const int ng = q.ok0 ? ((p.gs_n_shift >= 0) ? (n >> p.gs_n_shift) : (n / p.gs_n)) : 0;
                q.pp = (GLU && rank ? p.palette2 : p.palette) + (long long)ng * p.n_kgroups * 4;
            }
        };
        auto normalise = [&](int& tile, int& it) {          // true: another tile
            bool moved = false;
            while (it >= nkb_total) { it -= nkb_total; tile += n_pairs; moved = true; }
            return moved;
        };
        auto load_pos = [&](const Pos& q, uint2 (&idx)[2], uint2 (&pal)[2]) {
            idx[0] = idx[1] = pal[0] = pal[1] = make_uint2(0u, 0u);
            if (q.it >= nkb || q.tile >= p.n_items) return;
            if (kBMn) {
                const int n = q.it * kBK + rr;
                if (n >= p.Wn) return;
                const uint8_t* ip = q.ip + (long long)(q.it * kBK) * p.packed_pitch;
                const int ng = (p.gs_n_shift >= 0) ? (n >> p.gs_n_shift) : (n / p.gs_n);
                const __nv_bfloat16* pp = q.pp + (long long)ng * p.n_kgroups * 4;
                if (q.ok0) { idx[0] = __ldg(reinterpret_cast<const uint2*>(ip)); pal[0] = __ldg(reinterpret_cast<const uint2*>(pp + q.kg0 * 4)); }
                if (q.ok1) { idx[1] = __ldg(reinterpret_cast<const uint2*>(ip + 16)); pal[1] = __ldg(reinterpret_cast<const uint2*>(pp + q.kg1 * 4)); }
            } else if (q.ok0) {
                const int kb = q.it * 2;                    // blocks of 64 along k
                const uint8_t* ip = q.ip + q.it * (kBK / 4);
                int g0, g1;
                if (p.gs_k_shift >= 0) { g0 = kb >> p.gs_k_shift; g1 = (kb + 1) >> p.gs_k_shift; }
                else { g0 = kb / blocks_per_kgroup; g1 = (kb + 1) / blocks_per_kgroup; }
                if (kb * 64 + h * 32 < p.Wk) { idx[0] = __ldg(reinterpret_cast<const uint2*>(ip)); pal[0] = __ldg(reinterpret_cast<const uint2*>(q.pp + g0 * 4)); }
                if (kb * 64 + 64 + h * 32 < p.Wk) { idx[1] = __ldg(reinterpret_cast<const uint2*>(ip + 16)); pal[1] = __ldg(reinterpret_cast<const uint2*>(q.pp + g1 * 4)); }
            }
        };
        // Two stages per trip, so that the queue slot of every step is a compile-time constant: no slot is ever copied, which would make
        // the copy wait for a load that has just been issued.
        uint2 idx_q[2][2], pal_q[2][2];
        Pos pf; pf.tile = pair; pf.it = grp;
        normalise(pf.tile, pf.it);
        set_tile(pf);
        int c_tile = pf.tile, c_it = pf.it;   // the position being written
        auto pos_next = [&](Pos& q) {
            q.it += 2;
            if (normalise(q.tile, q.it) && q.tile < p.n_items) set_tile(q);
        };
#pragma unroll
        for (int u = 0; u < 2; ++u) { load_pos(pf, idx_q[u], pal_q[u]); pos_next(pf); }
        int s = grp;                          // ring slot and phase of the stage being written
        uint32_t ph = 0;
        bool ok = true;
        while (ok && c_tile < p.n_items) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (!ok || c_tile >= p.n_items) break;
                const bool is_extra = c_it >= nkb;
                const int half = item_width(c_tile) >> 1;
                uint2 idx[2] = {idx_q[u][0], idx_q[u][1]}, pl[2] = {pal_q[u][0], pal_q[u][1]};
                load_pos(pf, idx_q[u], pal_q[u]);
                pos_next(pf);
                ok = mbar_wait(empty(s), ph ^ 1u, abort_flag, p.status, ST_TIMEOUT_EMPTY, 3);
                if (!ok) break;
                if (!is_extra) {              // the LoRA block comes by TMA; arrive all the same, after the stage is free, to keep the phases in step
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        if ((kBMn ? b * 64 + h * 32 : rr) >= half) continue;
                        uint8_t* row = smem + s * kStageBytes + kABytes + b * kBlkBytes + rr * 128;
                        const PalRegs pal = pal_split(pl[b].x, pl[b].y);
                        const uint32_t w[2] = {idx[b].x, idx[b].y};
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            uint32_t o[8];
                            decode16(w[i], pal, o);
                            *reinterpret_cast<uint4*>(row + (((4 * h + 2 * i) ^ (rr & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
                            *reinterpret_cast<uint4*>(row + (((4 * h + 2 * i + 1) ^ (rr & 7)) << 4)) = make_uint4(o[4], o[5], o[6], o[7]);
                        }
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                }
                if (lane == 0) mbar_arrive_cluster(lead_full(s));
                s += 2;
                if (s >= kStages) { s -= kStages; ph ^= 1u; }
                c_it += 2;
                normalise(c_tile, c_it);
            }
        }
    } else {
        // ------------------------------------------------------------- epilogue warps
        // warp e reads TMEM lanes 32 * (warp % 4) (its 32 output rows of this CTA's 128) and walks the 256 columns 64 at a
        // time: fp32 -> bf16 -> 128-byte-swizzled box in shared memory -> TMA store (clipped at M and J).
        const int e = warp - kFirstEpiWarp;
        const int lane_group = warp & 3;
        uint8_t* stage = smem + kEpiOff + e * kEpiStageBytes;
        const uint32_t stage_u32 = base + kEpiOff + e * kEpiStageBytes;
        bool ok = true;
        int lt = 0;
        for (int t = pair; t < p.n_items && ok; t += n_pairs, ++lt) {
            int m0, j0;
            item_origin(t, m0, j0);
            const int w = GLU ? item_width(t) >> 1 : item_width(t);     // outputs
            const int buf = lt & 1;
            const int mrow = m0 + 128 * (int)rank + lane_group * 32;
            ok = mbar_wait(acc_full(buf), (lt >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 4);
            if (!ok) break;
            tc_fence_after_sync();
#pragma unroll 1
            for (int col = 0; col < w; col += 64) {
                const bool wide = col + 32 < w;            // a box of 64 columns, or the last 32 of a tile
                if (lane == 0) tma_store_wait_read();
                __syncwarp();
                if (GLU) {
                    const uint32_t at = tmem_base + ((uint32_t)(lane_group * 32) << 16) + buf * 256u + col;
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        if (c == 4 && !wide) break;
                        uint32_t vg[8], vu[8], o[4];
                        tmem_ld_32x8(at + c * 8, vg);
                        tmem_ld_32x8(at + w + c * 8, vu);
                        if (col + 8 * (c + 1) >= w) {
                            tc_fence_before_sync();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_cluster(lead_acc_empty(buf));
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float a0 = __uint_as_float(vg[2 * i]), a1 = __uint_as_float(vg[2 * i + 1]);
                            o[i] = pack_bf16x2(__fdividef(a0, 1.0f + __expf(-a0)) * __uint_as_float(vu[2 * i]), __fdividef(a1, 1.0f + __expf(-a1)) * __uint_as_float(vu[2 * i + 1]));
                        }
                        const uint32_t to = wide ? swz128(lane, c) : (uint32_t)(lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4));
                        *reinterpret_cast<uint4*>(stage + to) = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                }
#pragma unroll
                for (int c = 0; c < (GLU ? 0 : 2); ++c) {
                    if (c == 1 && !wide) break;
                    uint32_t v[32];
                    tmem_ld_32x32(tmem_base + ((uint32_t)(lane_group * 32) << 16) + buf * 256u + col + c * 32, v);
                    if (col + 32 * (c + 1) >= w) {
                        // last read of this accumulator: hand it back to the MMA thread of the leader
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(lead_acc_empty(buf));
                    }
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        float f[8];
                        uint4 bb = make_uint4(0u, 0u, 0u, 0u);
                        const int jc = j0 + col + c * 32 + g * 8;      // J is a multiple of 8
                        if (p.bias != nullptr && jc < p.J) bb = __ldg(reinterpret_cast<const uint4*>(p.bias + jc));
                        const uint32_t bw[4] = {bb.x, bb.y, bb.z, bb.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            f[2 * i] = __uint_as_float(v[g * 8 + 2 * i]) * p.alpha + __uint_as_float(bw[i] << 16);
                            f[2 * i + 1] = __uint_as_float(v[g * 8 + 2 * i + 1]) * p.alpha + __uint_as_float(bw[i] & 0xFFFF0000u);
                        }
                        const uint32_t at = wide ? swz128(lane, c * 4 + g) : (uint32_t)(lane * 64 + ((g ^ ((lane >> 1) & 3)) << 4));
                        *reinterpret_cast<uint4*>(stage + at) = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
                    }
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0 && j0 + col < p.J && mrow < p.M) {
                    tma_store_2d(wide ? &tmD : &tmD32, stage_u32, j0 + col, mrow);
                    tma_store_commit();
                }
            }
        }
        if (lane == 0) tma_store_wait_all();
    }
    // Neither CTA may leave while its partner can still touch its shared memory (operand reads of the pair MMA, remote
    // barrier arrivals) or its tensor memory.
    tc_fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0 && rank == 0 && *abort_flag) {
        // somebody gave up: the copies of both CTAs, which arrive on this CTA's barriers, get a bounded chance to land
        const uint64_t t0 = globaltimer_ns();
        for (int it = issued > kStages ? issued - kStages : 0; it < issued; ++it)
            while (!mbar_try_wait(full(it % kStages), (it / kStages) & 1))
                if (globaltimer_ns() - t0 > 100000000ull) { report(p.status, ST_TIMEOUT_DRAIN, 0); break; }
    }
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

template <int BMODE, bool GLU = false>
int launch_pair_t(const LutGemmArgs& a, cudaStream_t stream) {
    const int J = GLU ? a.J / 2 : a.J;     // columns of the result
    CUtensorMap tmA, tmA2, tmB2, tmD, tmD32;
    int rc;
    if ((rc = make_tmap_bf16(&tmA, a.A, a.M, a.R, a.lda, 64, 128))) return rc;
    tmA2 = tmA; tmB2 = tmA;
    if (a.r2 > 0) {
        if ((rc = make_tmap_bf16(&tmA2, a.A2, a.M, a.r2, a.lda2, 64, 128))) return rc;
        if (BMODE == B_DECODE_MN) {
            if ((rc = make_tmap_bf16(&tmB2, a.B2, a.r2, a.J, a.ldb2, 64, 64))) return rc;
        } else {
            if ((rc = make_tmap_bf16(&tmB2, a.B2, a.J, a.r2, a.ldb2, 64, 128))) return rc;
        }
    }
    if ((rc = make_tmap_bf16(&tmD, a.out, a.M, J, a.ld_out, 64, 32))) return rc;
    if ((rc = make_tmap_bf16(&tmD32, a.out, a.M, J, a.ld_out, 32, 32))) return rc;
    PairParams p = {};
    p.M = a.M; p.J = J; p.R = a.R; p.n_extra = a.r2 > 0 ? 1 : 0;
    p.packed = (const uint8_t*)a.packed; p.packed_pitch = a.packed_pitch;
    p.palette = (const __nv_bfloat16*)a.palette;
    p.packed2 = (const uint8_t*)a.packed2; p.palette2 = (const __nv_bfloat16*)a.palette2;
    p.gs_n = a.gs_n > 0 ? a.gs_n : 1; p.gs_k = a.gs_k > 0 ? a.gs_k : kBK;
    p.n_kgroups = a.gs_k > 0 ? (a.Wk / a.gs_k) : 1;
    p.gs_n_shift = -1;
    for (int sh = 0; sh < 31; ++sh) if ((1 << sh) == p.gs_n) p.gs_n_shift = sh;
    p.gs_k_shift = -1;
    for (int sh = 0; sh < 26; ++sh) if ((64ll << sh) == p.gs_k) p.gs_k_shift = sh;
    p.Wn = a.Wn; p.Wk = a.Wk;
    p.alpha = a.alpha; p.bias = (const __nv_bfloat16*)a.bias;
    p.status = device_status_ptr();
    p.lets_next = !g_smallm_overlap;
    p.prof = (unsigned long long*)a.prof;
    auto kern = lut_gemm_pair_kernel<BMODE, GLU>;
    static bool attr_set[64] = {};
    int dev = 0, sms = 0;
    PLZ_CUDA_CHECK(cudaGetDevice(&dev));
    if (!attr_set[dev & 63]) {
        PLZ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        attr_set[dev & 63] = true;
    }
    PLZ_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (a.sm_limit > 0 && a.sm_limit < sms) sms = a.sm_limit;
    if (g_cta_limit > 0 && g_cta_limit < sms) sms = g_cta_limit;
    int pairs = sms / 2;
    if (pairs < 1) return PLZ_ERR_UNSUPPORTED;
    // backward product: a decode thread's 32 columns start at a multiple of 32 (8-byte loads of indices, one palette group)
    // gated: half of a tile's columns is a multiple of 32 outputs
    const PairTiles pt = plan_pair_tiles(a.M, a.J, pairs, BMODE == B_DECODE_MN || GLU ? 64 : 32);
    p.tiles_j = pt.tiles_j; p.tile_w = pt.tile_w; p.n_whole = pt.n_whole; p.n_items = pt.n_items;
    if (pairs > p.n_items) pairs = p.n_items;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr; cfg.numAttrs = behind_attr(stream, attr);
    PLZ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tmA, tmA2, tmB2, tmD, tmD32, p));
    ++g_launch_count;
    return PLZ_OK;
}

}  // namespace

// Waves of a launch in units of a 256-column tile, the shortest of
//   whole tiles, the last wave cut in halves where the halves fit one wave;
//   fewer tiles than pairs: the narrowest tile that fits one wave.
PairTiles plan_pair_tiles(int M, int J, int pairs, int step) {
    const int tiles_m = (M + 255) / 256;
    PairTiles t;
    t.tile_w = 256; t.tiles_j = (J + 255) / 256;
    const int tiles = tiles_m * t.tiles_j;
    t.n_whole = t.n_items = tiles;
    if (tiles <= pairs) {
        for (int w = 128; w < 256; w += step) {
            const int tj = (J + w - 1) / w;
            if (tiles_m * tj <= pairs) { t.tile_w = w; t.tiles_j = tj; t.n_whole = t.n_items = tiles_m * tj; break; }
        }
        return t;
    }
    const int rem = tiles % pairs;
    if (rem > 0 && 2 * rem <= pairs) { t.n_whole = tiles - rem; t.n_items = t.n_whole + 2 * rem; }
    return t;
}

// One or two waves of narrower tiles where they are fewer columns in all: 2048 x 2560 outputs are 80 tiles of 256 on 74 pairs, a wave and one of halves, 384
// columns; or 144 tiles of 144, two nearly full waves, 288. For the dense kernel (packed weights are decoded in chains that cost 160 columns at least).
// us plan_pair_tiles / here, one after the other: 2048 rows, 2560 x 2560 27.1 / 25.6, 2560 x 4096 39.3 / 37.5, 2560 x 9728 87.4 / 84.8; 1000 rows, 7680 x 2560 33.6 / 31.6; 512 rows,
// 9728 x 2560 28.7 / 27.6. More waves or more rows do not pay, as narrow tiles read more of both operands: 1536 rows, 9728 x 2560 in four waves of 208 columns 57.6 / 62.5, 4096 rows,
// 2560 x 9728 in four of 144 151 / 178; nor do gated outputs (512 rows, 19456 x 2560 44.2 / 45.4).
PairTiles plan_pair_waves(int M, int J, int pairs, int step) {
    PairTiles best = plan_pair_tiles(M, J, pairs, 32);
    const int tiles_m = (M + 255) / 256;
    if (tiles_m > 8) return best;
    auto waves = [&](int tiles) { return (tiles + pairs - 1) / pairs; };
    int cost = best.n_items > best.n_whole ? waves(best.n_whole) * 256 + 128 : waves(best.n_whole) * best.tile_w;
    for (int w = 256 - step; w >= 128; w -= step) {
        const int tj = (J + w - 1) / w, n = waves(tiles_m * tj);
        if (n <= 2 && n * w * 100 < cost * 97) {
            cost = n * w;
            best.tile_w = w; best.tiles_j = tj; best.n_whole = best.n_items = tiles_m * tj;
        }
    }
    return best;
}

// PLZ_ERR_UNSUPPORTED: not a shape for this kernel, the caller falls back to the single-CTA kernel.
int launch_lut_gemm_pair(const LutGemmArgs& a, cudaStream_t stream) {
    if (!g_pair_gemm) return PLZ_ERR_UNSUPPORTED;
    if (a.bmode != B_DECODE_K && a.bmode != B_DECODE_MN) return PLZ_ERR_UNSUPPORTED;
    const bool factors = a.col_scale || a.row_scale;
    if (a.fuse == 1 && !factors && !a.gate_out && !a.up_out && a.r2 == 0 && a.alpha == 1.0f && a.M >= 256 && a.J >= 512 && a.Wk % 16 == 0 && a.bmode == B_DECODE_K &&
        !((uintptr_t)a.packed2 & 15) && !((uintptr_t)a.palette2 & 7))
        return launch_pair_t<B_DECODE_K, true>(a, stream);
    const bool plain = a.fuse == 0 || (a.fuse == 2 && !factors);   // fuse 2 without norm factors: at most a bias
    if (!plain || a.M < 256 || a.J < 256) return PLZ_ERR_UNSUPPORTED;
    if ((uintptr_t)a.bias & 15) return PLZ_ERR_UNSUPPORTED;
    if (a.bmode == B_DECODE_MN && (a.J % 16)) return PLZ_ERR_UNSUPPORTED;
    if (a.bmode == B_DECODE_K && (a.Wk % 16)) return PLZ_ERR_UNSUPPORTED;
    return a.bmode == B_DECODE_K ? launch_pair_t<B_DECODE_K>(a, stream) : launch_pair_t<B_DECODE_MN>(a, stream);
}

}  // namespace plz
