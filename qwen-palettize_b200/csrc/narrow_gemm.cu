// Linear products with few rows, y[m, n] = sum_k x[m, k] W[n, k] for M <= 128: token decode and short portions. What such a launch cannot do
// without is one pass over W, so everything here serves that stream.
//
//   shape     The operands change sides: 128 rows of W are the 128 TMEM lanes, the tokens are the N side (16 .. 128 columns). A tile of 128
//             weight rows and all tokens is shared by a cluster of up to eight CTAs that split the reduction, because N / 128 tiles alone
//             leave most SMs idle (2560 rows are 20 tiles). Each CTA leaves its partial tile in its own shared memory and every CTA of the
//             cluster adds up its share of the outputs over distributed shared memory, in rank order: no workspace, no atomics, the same
//             bits on every run.
//   operands  dense bf16 W by TMA (requested before the wait on the previous kernel of the stream, for callers whose weights are constant), or packed 2-bit indices: a decode
//             thread is one weight row, fetches the 16 bytes of a block of 64 columns several blocks ahead and writes the decoded row to
//             TMEM, from where it is the A operand (lane = row: no shared memory, no swizzle, no proxy fence in between). x by TMA into a
//             ring of its own, since TMEM has room for a few blocks of W only. A single issuing lane took 0.6 us a block (see there).
//             Shared memory and TMEM are kept to half of an SM's, so that two CTAs share one and hide each other's start and end.
//   turned    (transposed) W is an activation matrix of any number of rows and x the few rows of a LoRA factor, t = s x A^T and dt = s dY B: the
//             same launch with y stored [row of W][row of x], x from [M, K] or (x_mn) from [K, M]. Where the rows alone fill the chip a kernel of its
//             own takes a row tile per CTA (turned_gemm_kernel).
//   extra     an optional block of up to 64 more reduction elements (the LoRA up-projection: t [M, r] against B [N, r]).
//
// Accumulating into the tile the previous MMA still writes costs a TMEM round trip, so the four MMAs of a block go to several accumulators,
// as many as fit, which the epilogue adds.
#include <type_traits>

#include "attention_tiles.cuh"
#include "seq_math.cuh"

namespace plz {
namespace {

constexpr int kNgMaxMats = 4;
constexpr int kNgDecodeWarps = 8;                 // two groups of 128 threads, pairs of blocks alternate between them
constexpr uint32_t kNgWBytes = 128 * 64 * 2;
// shared memory of the stages; two CTAs per SM. LUT: four x tiles of 128 tokens and the W tile of the extra block
template <bool LUT>
constexpr uint32_t kNgRingBytes = LUT ? 80 * 1024 : 96 * 1024;
constexpr int kNgMaxStages = 16;                  // slots for copies
constexpr int kNgMaxW = 3;                        // pairs of blocks of decoded W in TMEM
constexpr uint32_t kNgBarBytes = 512;
constexpr int kNgAhead = 4;                       // blocks of packed indices a decode thread has in flight

struct NarrowMat {
    int N, first_tile;
    const uint8_t* packed; long long pitch; const __nv_bfloat16* palette;
    void* y; long long ldy;
};
struct NarrowParams {
    int M, npad, n_acc, stages, w_stages;   // slots for copies (dense: W and x of a block; LUT: x of two blocks, a power of two of them), LUT: pairs of blocks of W in TMEM
    int x_mn, transposed;
    uint32_t x_bytes;              // of a tile of x
    uint32_t tmem_cols;
    int group_blocks, group_shift; // blocks of 64 columns per palette group, its logarithm or -1
    int nkb, n_blocks;             // blocks of 64 columns of W; the same plus the extra block
    int count; NarrowMat mat[kNgMaxMats];
    int gs_n, gs_k, n_kgroups;
    int glu;                       // a tile is 64 rows of mat[0] and the same rows of mat[1]
    int early;                     // W is read ahead of the wait for the kernel before
    int lets_next;                 // let the next kernel start behind this one's wait
    const __nv_bfloat16* bias; int act, y_f32; float alpha;
    StatusWord* status;
};

__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// dense: four warps read the accumulators, two more help with the cluster's sums
template <bool LUT>
constexpr int kNgThreads = 64 + 32 * (LUT ? kNgDecodeWarps : 6);

template <bool LUT>
__global__ void __launch_bounds__(kNgThreads<LUT>, 2)
narrow_gemm_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX2,
                   const __grid_constant__ CUtensorMap tmW2, const NarrowParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    // dense: a stage is a W tile and an x tile; LUT: the x tiles of two blocks, behind the stages one W tile for the extra block (W is decoded to TMEM)
    const uint32_t x_bytes = p.x_bytes, stage_bytes = LUT ? 2u * x_bytes : kNgWBytes + x_bytes;
    const uint32_t w2_off = LUT ? (uint32_t)p.stages * stage_bytes : 0u;
    const uint32_t bar_off = kNgRingBytes<LUT>;
    auto full = [&](int s) { return base + bar_off + 8u * s; };
    auto empty = [&](int s) { return base + bar_off + 8u * (kNgMaxStages + s); };
    auto empty_w = [&](int s) { return base + bar_off + 8u * (2 * kNgMaxStages + s); };            // LUT only
    constexpr int kBars = 2 * kNgMaxStages + kNgMaxW + 1;
    static_assert(8 * kBars + 8 <= kNgBarBytes, "barriers");
    const uint32_t acc_full = base + bar_off + 8u * (kBars - 1);
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + bar_off + 8 * kBars);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    // the warp's number as a value the compiler knows to be uniform: what the issuing warp computes then stays in uniform registers
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int n_ranks = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
    const int tile = (int)blockIdx.x / n_ranks;
    int mi = 0;
#pragma unroll
    for (int i = 1; i < kNgMaxMats; ++i)
        if (i < p.count && tile >= p.mat[i].first_tile) mi = i;
    const NarrowMat& mat = p.mat[mi];
    const bool glu = LUT && p.glu;
    const int n0 = (tile - mat.first_tile) * (glu ? 64 : 128);
    const int b_begin = (int)((long long)rank * p.n_blocks / n_ranks), b_end = (int)((long long)(rank + 1) * p.n_blocks / n_ranks);
    const int nb = b_end - b_begin;        // at least one: the cluster is no larger than the number of blocks

    // Steps: a block (dense), or a pair of blocks (LUT). What the issuing warp does once per step (a wait, the election, the commits: 470 clocks beside the 90 that four
    // MMAs take) and what a decoding group does once (waits, the store's completion, an arrival: 450 beside 430 of decoding) made 650 clocks a block. By blocks / by pairs, 64 rows in a row of
    // launches, us: 19456 x 2560 23.6 / 20.4, 12288 x 4096 19.4 / 17.4, 9728 x 2560 12.6 / 11.0, 2560 x 9728 14.6 / 12.7.
    const int steps = LUT ? (nb + 1) >> 1 : nb;
    // the bytes of all copies of a stage are announced with the first one
    auto load_w = [&](int st, int s) {
        const int b = b_begin + (LUT ? 2 * st : st), n = LUT && 2 * st + 1 < nb ? 2 : 1;
        const bool extra = b + n > p.nkb, by_tma = !LUT || extra;
        mbar_arrive_expect_tx(full(s), n * x_bytes + (by_tma ? kNgWBytes : 0u));
        if (by_tma) tma_load_2d(base + (LUT ? w2_off : s * stage_bytes), extra ? &tmW2 : &tmW, full(s), extra ? 0 : b * 64, n0);
    };
    auto load_x = [&](int st, int s) {
        const int b = b_begin + (LUT ? 2 * st : st);
        const bool extra = b >= p.nkb;
        const bool mn = !LUT && p.x_mn;
        const uint32_t to = base + s * stage_bytes + (LUT ? 0u : kNgWBytes);
        tma_load_2d(to, extra ? &tmX2 : &tmX, full(s), extra || mn ? 0 : b * 64, mn ? b * 64 : 0);
        if (LUT && 2 * st + 1 < nb) tma_load_2d(to + x_bytes, b + 1 >= p.nkb ? &tmX2 : &tmX, full(s), b + 1 >= p.nkb ? 0 : (b + 1) * 64, 0);
    };
    const int pre = steps < p.stages ? steps : p.stages;

    // weights do not depend on the previous kernel and do not wait for this block's own set-up either
    constexpr int kAhead = LUT ? kNgAhead : 1;
    const int row = (warp & 3) * 32 + lane;                         // decode: thread = one weight row = its TMEM lane
    const int grp = LUT && warp >= 6 ? 1 : 0;
    const int nw = b_end < p.nkb ? nb : p.nkb - b_begin;            // blocks of W in this CTA's range
    const NarrowMat& own = glu && row >= 64 ? p.mat[1] : mat;
    const int wrow = n0 + (glu ? row & 63 : row);
    const bool row_ok = wrow < mat.N;
    const uint8_t* prow = LUT ? own.packed + (row_ok ? (long long)wrow * own.pitch : 0ll) + (long long)b_begin * 16 : nullptr;
    const __nv_bfloat16* pal = LUT ? own.palette + (row_ok ? (long long)(wrow / p.gs_n) * p.n_kgroups * 4 : 0ll) : nullptr;
    uint4 w[kAhead];
    uint2 pr[kAhead];
    auto fetch = [&](int it, int j) {
        w[j] = make_uint4(0u, 0u, 0u, 0u);
        pr[j] = make_uint2(0u, 0u);
        if (row_ok && it < nw) {
            const int kg = p.group_shift >= 0 ? (b_begin + it) >> p.group_shift : (b_begin + it) / p.group_blocks;
            w[j] = __ldg(reinterpret_cast<const uint4*>(prow + it * 16));
            pr[j] = __ldg(reinterpret_cast<const uint2*>(pal + kg * 4));
        }
    };
    if (LUT && warp >= 2) {
        if (!p.early) pdl_wait();
#pragma unroll
        for (int j = 0; j < kAhead; ++j) fetch(4 * (j >> 1) + 2 * grp + (j & 1), j);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kNgMaxStages; ++s) {
            mbar_init(full(s), LUT ? 1 + kNgDecodeWarps / 2 : 1);    // LUT: the copies and the decoded weights
            mbar_init(empty(s), 1);
        }
        for (int s = 0; LUT && s < kNgMaxW; ++s) mbar_init(empty_w(s), 1);
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmX);
        if (p.n_blocks > p.nkb) { tma_prefetch_desc(&tmX2); tma_prefetch_desc(&tmW2); }
        if (!p.early) pdl_wait();
        for (int it = 0; it < pre; ++it) load_w(it, it);
    }
    if (warp == 1) { tmem_alloc(smem_u32((const void*)tmem_slot), p.tmem_cols); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_w = tmem_base + (uint32_t)(p.n_acc * p.npad);      // LUT: 32 columns per stage
    if (!p.early) pdl_wait();
    if (p.lets_next) pdl_launch_dependents();

    // every wait below that x holds up starts after the previous kernel of the stream has finished: its time is not the wait's
    int issued = pre;                      // stages the producing thread has filled
    if (warp == 0) {
        if (lane == 0) {
            pdl_wait();
            for (int it = 0; it < pre; ++it) load_x(it, it);
            for (int it = pre; it < steps; ++it) {
                const int s = it % p.stages;
                if (!mbar_wait(empty(s), ((it / p.stages) & 1) ^ 1u, abort_flag, p.status, ST_TIMEOUT_EMPTY, 0)) break;
                load_w(it, s);
                load_x(it, s);
                issued = it + 1;
            }
        }
    } else if (warp == 1) {
        // The whole warp walks the blocks and one elected lane issues. In a branch of one lane the operands of every MMA live in vector registers
        // and are moved to uniform ones first: 630 clocks for the four MMAs and two commits of a block, longer than all else. Packed, 64 rows: 19456 x 2560 33 -> 24 us,
        // 2560 x 9728 18.8 -> 14.1, 1024 x 2560 7.7 -> 6.3.
        const bool mn = !LUT && p.x_mn;
        const uint32_t idesc = make_idesc(128, p.npad, 0, mn ? 1 : 0), x_step = mn ? 2048u >> 4 : 2u;   // 16 reduction elements of x
        const uint64_t desc = make_sdesc(base, 16u, 1024u);
        const uint32_t hi = (uint32_t)(desc >> 32), lo0 = (uint32_t)desc, slot = stage_bytes >> 4, x_off = LUT ? 0u : kNgWBytes >> 4;
        const uint32_t d1 = tmem_base + (p.n_acc > 1 ? (uint32_t)p.npad : 0u), d2 = tmem_base + (p.n_acc > 2 ? 2u * (uint32_t)p.npad : 0u),
                       d3 = p.n_acc > 2 ? tmem_base + 3u * (uint32_t)p.npad : d1;
        bool ok = true;
        int s = 0, iw = 0;
        uint32_t ph = 0, lo = lo0;
        // a block: accumulators start with their first MMA
        auto block = [&](bool from_tmem, uint32_t wt, uint32_t wd, uint32_t xd, uint32_t first) {
            const uint32_t m1 = p.n_acc > 1 ? first : 1u, m2 = p.n_acc > 2 ? first : 1u;
            if (from_tmem) {
                umma_ts(tmem_base, wt, xd, hi, idesc, first);
                umma_ts(d1, wt + 8u, xd + 2u, hi, idesc, m1);
                umma_ts(d2, wt + 16u, xd + 4u, hi, idesc, m2);
                umma_ts(d3, wt + 24u, xd + 6u, hi, idesc, m2);
            } else {
                umma_bf16_words<1>(tmem_base, wd, hi, xd, hi, idesc, first);
                umma_bf16_words<1>(d1, wd + 2u, hi, xd + x_step, hi, idesc, m1);
                umma_bf16_words<1>(d2, wd + 4u, hi, xd + 2u * x_step, hi, idesc, m2);
                umma_bf16_words<1>(d3, wd + 6u, hi, xd + 3u * x_step, hi, idesc, m2);
            }
        };
        pdl_wait();
        for (int st = 0; st < steps; ++st) {
            ok = mbar_wait_warp(full(s), ph, abort_flag, p.status, ST_TIMEOUT_FULL, 1);
            if (!ok) break;
            tc_fence_after_sync();
            if (LUT) {
                const int b = b_begin + 2 * st;
                const uint32_t wt = tmem_w + iw * 64u, w2 = lo0 + (w2_off >> 4);
                if (b + 1 < p.nkb && 2 * st + 1 < nb) {
                    if (elect_one()) {
                        block(true, wt, 0u, lo, st > 0 ? 1u : 0u);
                        block(true, wt + 32u, 0u, lo + (x_bytes >> 4), 1u);
                        umma_commit(empty(s));
                        umma_commit(empty_w(iw));
                    }
                } else if (elect_one()) {           // the last step: one block, or the extra one
                    block(b < p.nkb, wt, w2, lo, st > 0 ? 1u : 0u);
                    if (2 * st + 1 < nb) block(b + 1 < p.nkb, wt + 32u, w2, lo + (x_bytes >> 4), 1u);
                    umma_commit(empty(s));
                    umma_commit(empty_w(iw));
                }
                if (++iw == p.w_stages) iw = 0;
            } else if (elect_one()) {
                block(false, 0u, lo, lo + x_off, st > 0 ? 1u : 0u);
                umma_commit(empty(s));
            }
            __syncwarp();
            lo += slot;
            if (++s == p.stages) { s = 0; ph ^= 1u; lo = lo0; }
        }
        if (ok && elect_one()) umma_commit(acc_full);
        __syncwarp();
    } else {
        bool ok = true;
        if (LUT) {
            // ------------------------------------------------------ decode: the two groups of four warps take pairs of blocks in turn
            // The groups share three slots (two beyond 64 rows, then one each): a group that comes to a slot has, one of its steps before, waited for a product issued behind the
            // slot's last but one use, so the barrier's parity tells the rounds apart. Three groups gain nothing (64 rows of 19456 x 2560 20.4 / 19.8 us, 6144 x 2560 8.8 / 9.0), and on two
            // slots one of them could be a whole round ahead.
            const uint32_t lanes = tmem_w + ((uint32_t)((warp & 3) * 32) << 16);
            int iw = grp;
            uint32_t phw = 1;                       // the slots are free at first
            for (int st0 = grp; st0 < steps && ok; st0 += kAhead) {
#pragma unroll
                for (int j = 0; j < kAhead; j += 2) {
                    const int st = st0 + j, it = 2 * st;
                    if (st >= steps || !ok) continue;
                    if (st >= 2 && st < 4) pdl_wait();
                    uint32_t o[32];
                    auto decode = [&](int i) {
                        const PalRegs pl = pal_split(pr[i].x, pr[i].y);
                        decode16(w[i].x, pl, o);
                        decode16(w[i].y, pl, o + 8);
                        decode16(w[i].z, pl, o + 16);
                        decode16(w[i].w, pl, o + 24);
                    };
                    if (it < nw) decode(j);
                    fetch(it + 2 * kAhead, j);
                    ok = mbar_wait_warp(empty_w(iw), phw, abort_flag, p.status, ST_TIMEOUT_EMPTY, 3);
                    if (!ok) continue;
                    const uint32_t to = lanes + iw * 64u;
                    tc_fence_after_sync();
                    if (it < nw) tmem_st_32x32_begin(to, o);
                    if (it + 1 < nw) {
                        decode(j + 1);
                        tmem_st_32x32_begin(to + 32u, o);
                    }
                    fetch(it + 1 + 2 * kAhead, j + 1);
                    tmem_wait_st();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full(st & (p.stages - 1)));
                    iw += 2;
                    if (iw >= p.w_stages) { iw -= p.w_stages; phw ^= 1u; }
                }
            }
        }
        // ---------------------------------------------------------- this CTA's partial tile in the ring's space: [token][weight row], transposed
        // [weight row][npad tokens]
        // The accumulators of 16 columns are read behind one wait, packed by both groups of decode warps in turn. Read one after the other, they and the
        // sums below were half of what a launch costs beside its blocks. 64 rows, microseconds in a row of launches: dense 2560 x 2560 8.1 -> 7.6,
        // 9728 x 2560 13.7 -> 13.0; packed 2560 x 2560 8.6 -> 8.1, 19456 x 2560 24.7 -> 23.7. Pushing the shares to their owner with bulk copies
        // instead of fetching them behind the cluster's barrier is slower by 0.8 - 1.4 (dense 2560 x 2560 8.7, packed 9.4).
        if (LUT || warp < 6) {
            pdl_wait();
            if (ok) ok = mbar_wait(acc_full, 0, abort_flag, p.status, ST_TIMEOUT_ACCUM, 4);
            if (ok) {
                tc_fence_after_sync();
                const int lg = warp & 3;
                float* part = reinterpret_cast<float*>(smem) + lg * 32 + lane;
                constexpr int kGroups = LUT ? 2 : 1;
                for (int c0 = LUT && warp >= 6 ? 16 : 0; c0 < p.npad && c0 < p.M; c0 += 16 * kGroups) {
                    const uint32_t at = tmem_base + ((uint32_t)(lg * 32) << 16) + c0;
                    float sum[16];
                    if (p.n_acc == 4) {
                        uint32_t v[4][16];
                        tmem_ld_sets(at, (uint32_t)p.npad, v);
#pragma unroll
                        for (int c = 0; c < 16; ++c) sum[c] = __uint_as_float(v[0][c]) + __uint_as_float(v[1][c]) + __uint_as_float(v[2][c]) + __uint_as_float(v[3][c]);
                    } else if (p.n_acc == 2) {
                        uint32_t v[2][16];
                        tmem_ld_sets(at, (uint32_t)p.npad, v);
#pragma unroll
                        for (int c = 0; c < 16; ++c) sum[c] = __uint_as_float(v[0][c]) + __uint_as_float(v[1][c]);
                    } else {
                        uint32_t v[16];
                        tmem_ld_32x16(at, v);
#pragma unroll
                        for (int c = 0; c < 16; ++c) sum[c] = __uint_as_float(v[c]);
                    }
                    if (!LUT && p.transposed) {
                        float4* to = reinterpret_cast<float4*>(smem) + ((lg * 32 + lane) * p.npad + c0) / 4;
#pragma unroll
                        for (int c = 0; c < 16; c += 4) to[c / 4] = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
                        continue;
                    }
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        if (c0 + c < p.M) part[(c0 + c) * 128] = sum[c];
                }
            }
        }
    }
    tc_fence_before_sync();
    __syncwarp();
    cluster_sync_all();        // every CTA's partial tile is complete and visible
    if (threadIdx.x == 0 && *abort_flag) {
        // somebody gave up: copies in flight get a bounded chance to land before the CTA exits
        const uint64_t t0 = globaltimer_ns();
        for (int it = issued > p.stages ? issued - p.stages : 0; it < issued; ++it)
            while (!mbar_try_wait(full(it % p.stages), (it / p.stages) & 1))
                if (globaltimer_ns() - t0 > 100000000ull) { report(p.status, ST_TIMEOUT_DRAIN, 0); break; }
    }
    pdl_wait();                // outputs may be what the previous kernel still reads
    {
        uint32_t from[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) from[i] = map_rank(base, i < n_ranks ? i : 0);
        const bool turned = !LUT && p.transposed;
        const int quads = p.npad / 4;
        // one unit of the results with its sums: (token, 4 weight rows), turned: (weight row, 4 tokens), glu: (token, 4 outputs), gate sums behind up sums
        auto finish = [&](int u, float (&v)[4]) {
            const int m = turned ? u % quads * 4 : u >> 5, r = turned ? u / quads : (u & 31) * 4, n = n0 + r;
            if (n >= mat.N) return;
            if (turned) {
                __nv_bfloat16* y = (__nv_bfloat16*)mat.y + (long long)n * mat.ldy + m;
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] *= p.alpha;
                if (m + 3 < p.M && !((uintptr_t)y & 7)) *reinterpret_cast<uint2*>(y) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
                else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (m + e < p.M) y[e] = __float2bfloat16_rn(v[e]);
                }
                return;
            }
            if (p.act == ACT_GLU_GELU) {      // N is even
                const long long o = (long long)m * mat.ldy + (n >> 1);
                const float a = gelu_tanh_f(v[0]) * v[1], b = gelu_tanh_f(v[2]) * v[3];
                if (p.y_f32) {
                    float* y = (float*)mat.y + o;
                    y[0] = a;
                    if (n + 2 < mat.N) y[1] = b;
                } else {
                    __nv_bfloat16* y = (__nv_bfloat16*)mat.y + o;
                    y[0] = __float2bfloat16_rn(a);
                    if (n + 2 < mat.N) y[1] = __float2bfloat16_rn(b);
                }
                return;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                v[e] *= p.alpha;
                if (p.bias && n + e < mat.N) v[e] += __bfloat162float(p.bias[n + e]);
                v[e] = activate(v[e], p.act);
            }
            const long long o = (long long)m * mat.ldy + n;
            if (p.y_f32) {
                float* y = (float*)mat.y + o;
                if (n + 3 < mat.N && !((uintptr_t)y & 15)) { *reinterpret_cast<float4*>(y) = make_float4(v[0], v[1], v[2], v[3]); return; }
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < mat.N) y[e] = v[e];
            } else {
                __nv_bfloat16* y = (__nv_bfloat16*)mat.y + o;
                if (n + 3 < mat.N && !((uintptr_t)y & 7)) { *reinterpret_cast<uint2*>(y) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3])); return; }
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < mat.N) y[e] = __float2bfloat16_rn(v[e]);
            }
        };
        auto finish_glu = [&](int u, const float (&g)[4], const float (&h)[4]) {
            const int m = u >> 4, n = n0 + (u & 15) * 4;
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = swiglu_of_sums(g[e], h[e]);
            __nv_bfloat16* y = (__nv_bfloat16*)mat.y + (long long)m * mat.ldy + n;
            if (n + 3 < mat.N && !((uintptr_t)y & 7)) { *reinterpret_cast<uint2*>(y) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3])); return; }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n + e < mat.N) y[e] = __float2bfloat16_rn(v[e]);
        };
        const int units = glu ? p.M * 16 : turned ? 128 * quads : p.M * 32;
        const int u0 = (int)((long long)rank * units / n_ranks), u1 = (int)((long long)(rank + 1) * units / n_ranks);
        // packed: two units at a time in a cluster of two, whose trips to the partner's shared memory would come one after the other; no gain where W is dense
        auto gather = [&](auto ranks_at_most) {
            constexpr int kRanks = decltype(ranks_at_most)::value, kUnits = LUT && kRanks < 4 ? 4 / kRanks : 1;
            for (int at = u0 + (int)threadIdx.x; at < u1; at += kNgThreads<LUT> * kUnits) {
                float v[kUnits][4] = {};
                auto sums = [&](int half, float (&to)[kUnits][4]) {
                    float4 f[kUnits][kRanks];
#pragma unroll
                    for (int b = 0; b < kUnits; ++b) {
                        const int u = at + b * kNgThreads<LUT>;
                        const uint32_t off = (uint32_t)(glu ? (u >> 4) * 32 + half * 16 + (u & 15) : u) * 16u;
#pragma unroll
                        for (int i = 0; i < kRanks; ++i)
                            if (u < u1 && i < n_ranks) f[b][i] = ld_cluster_f4(from[i] + off);
                    }
#pragma unroll
                    for (int b = 0; b < kUnits; ++b)
#pragma unroll
                        for (int i = 0; i < kRanks; ++i)
                            if (i < n_ranks) { to[b][0] += f[b][i].x; to[b][1] += f[b][i].y; to[b][2] += f[b][i].z; to[b][3] += f[b][i].w; }
                };
                sums(0, v);
                if (glu) {
                    float h[kUnits][4] = {};
                    sums(1, h);
#pragma unroll
                    for (int b = 0; b < kUnits; ++b)
                        if (at + b * kNgThreads<LUT> < u1) finish_glu(at + b * kNgThreads<LUT>, v[b], h[b]);
                } else {
#pragma unroll
                    for (int b = 0; b < kUnits; ++b)
                        if (at + b * kNgThreads<LUT> < u1) finish(at + b * kNgThreads<LUT>, v[b]);
                }
            }
        };
        if (n_ranks <= 2) gather(std::integral_constant<int, 2>());
        else if (n_ranks <= 4) gather(std::integral_constant<int, 4>());
        else gather(std::integral_constant<int, 8>());
    }
    cluster_sync_all();        // nobody leaves while its partial tile may still be read
    if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, p.tmem_cols); }
}

// CTAs per tile: the shortest schedule when tiles * c CTAs of ceil(blocks / c) blocks each, plus about `fixed` for start, sum and end, are dealt to
// two places per SM, of which clusters can fill about nine tenths. Two CTAs of an SM slow each other down a little. Measured over 8 to 152
// tiles, 40 to 152 blocks, 20 to 128 rows: within 5 % of the best of 1 .. 8. A rule that counted one place per SM gave 2560 x 9728 packed 22 us at 64 rows
// for 19, 6144 x 2560 14.7 for 12.7, 19456 x 2560 36 for 33.
int cluster_size(int tiles, int blocks, int sms, int fixed) {
    int best = 1;
    double best_cost = 0;
    for (int c = 1; c <= 8; ++c) {
        if (c > 1 && blocks / c < 2) break;
        if (c == 5 || c == 7) continue;           // leave SMs of a processing cluster without a partner
        const long long ctas = (long long)tiles * c, places = c > 1 ? 2 * sms * 9 / 10 : 2 * sms;
        const double shared = ctas <= sms ? 0.0 : ctas >= 2 * sms ? 1.0 : (double)(ctas - sms) / sms;
        const double cost = (double)((ctas + places - 1) / places) * ((blocks + c - 1) / c + fixed) * (1.0 + 0.3 * shared);
        if (c == 1 || cost < best_cost) { best = c; best_cost = cost; }
    }
    return best;
}

// The same for packed W, whose blocks come out of a CTA at 0.25 us: start, sum and end are 14 of them, 18 in clusters of more than four, which moreover share SMs
// from about three fifths of one CTA per SM on; pairs fill every place; and without clusters one SM with two CTAs sets the time. us at 64 rows in a row of launches, by clusters
// of 1 / 2 / 3 / 4 / 6 / 8: 2560 x 2560 13.4 / 8.5 / 7.8 / 6.6 / 7.3 / 7.7, x 9728 39 / 21 / 18 / 15.6 / 13.4 / 12.7, 4096 x 4096 19 / 11.8 / 10.5 / 9.4 / 10.3 / 10.8, 6144 x 2560 13.9 / 9.3 /
// 9.4 / 8.8 / 15 / 16, 9728 x 2560 14.3 / 11.5 / 10.9 / 15 / 18 / 23, 18944 x 2560 (148 tiles) 15.4 / 14.4 / 21 / 24 / 34 / 41, 19456 x 2560 (152) 20.4 / 20.7 / 21 / 25 / 35 / 42.
int cluster_size_packed(int tiles, int blocks, int sms) {
    int best = 1;
    double best_cost = 0;
    for (int c = 1; c <= 8; ++c) {
        if (c > 1 && blocks / c < 2) break;
        if (c == 5 || c == 7) continue;
        const long long ctas = (long long)tiles * c, places = c <= 2 ? 2 * sms : 2 * sms * 9 / 10;
        const double alone = c > 4 ? 0.6 * sms : sms;
        double shared = ctas <= alone ? 0.0 : ctas >= alone + sms ? 1.0 : (ctas - alone) / sms;
        if (c == 1 && shared > 0.0) shared = 1.0;
        const double cost = (double)((ctas + places - 1) / places) * ((blocks + c - 1) / c + (c > 4 ? 18 : 14)) * (1.0 + 0.3 * shared);
        if (c == 1 || cost < best_cost) { best = c; best_cost = cost; }
    }
    return best;
}

// Parts of the reduction of a turned product: by the reduction alone, so that a row's result does not depend on how many rows there are (a step over
// all tokens and the sum of steps over parts of them then agree); eight to twenty blocks per part.
int turned_parts(int n_blocks) { return n_blocks >= 64 ? 8 : n_blocks >= 32 ? 4 : n_blocks >= 16 ? 2 : 1; }

template <bool LUT>
int launch_ng(const NarrowParams& p, int tiles, int ranks, const CUtensorMap (&tm)[4], cudaStream_t stream) {
    auto kern = narrow_gemm_kernel<LUT>;
    constexpr uint32_t smem = kNgRingBytes<LUT> + kNgBarBytes + 1024;
    static bool attr_set[64] = {};
    int dev = 0;
    PLZ_CUDA_CHECK(cudaGetDevice(&dev));
    if (!attr_set[dev & 63]) {
        PLZ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attr_set[dev & 63] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * ranks)); cfg.blockDim = dim3(kNgThreads<LUT>); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    const unsigned behind = behind_attr(stream, &attr[1]);
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ranks; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1 + (p.early ? 1u : behind);
    PLZ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tm[0], tm[1], tm[2], tm[3], p));
    ++g_launch_count;
    return PLZ_OK;
}

}  // namespace

// PLZ_ERR_UNSUPPORTED: not a call for this kernel.
int launch_narrow_gemm(const NarrowArgs& a, cudaStream_t stream) {
    const bool lut = a.mat[0].packed != nullptr;
    if (a.M < 1 || a.M > 128 || a.count < 1 || a.count > kNgMaxMats || (!lut && a.count != 1) || a.K < 8 || a.K % (lut ? 64 : 8)) return PLZ_ERR_UNSUPPORTED;
    if ((a.transposed || a.x_mn) && (lut || a.count != 1 || a.r2 || a.bias || a.act || a.y_f32 || !a.transposed || (a.x_mn && a.M > 64))) return PLZ_ERR_UNSUPPORTED;
    if (a.r2 < 0 || a.r2 > 64 || a.r2 % 8 || (a.r2 && a.count != 1)) return PLZ_ERR_UNSUPPORTED;
    if (((uintptr_t)a.x & 15) || a.ldx % 8) return PLZ_ERR_UNSUPPORTED;
    if (lut && (a.gs_n <= 0 || a.gs_k <= 0 || a.gs_k % 64 || a.K % a.gs_k)) return PLZ_ERR_UNSUPPORTED;
    if (!lut && (((uintptr_t)a.mat[0].w & 15) || a.mat[0].ldw % 8)) return PLZ_ERR_UNSUPPORTED;
    NarrowParams p = {};
    p.M = a.M; p.npad = a.M <= 16 ? 16 : a.M <= 32 ? 32 : a.M <= 64 ? 64 : 128;
    p.x_mn = a.x_mn; p.transposed = a.transposed;
    p.x_bytes = a.x_mn ? 64u * 128u : (uint32_t)p.npad * 128u;       // x_mn: 64 reduction rows of 64 columns
    if (lut) {      // 256 TMEM columns: accumulators, then 32 columns per stage
        p.n_acc = p.npad == 16 ? 4 : p.npad == 32 ? 2 : 1;
        p.w_stages = (256 - p.n_acc * p.npad) / 64;                              // 3, or 2 beyond 64 rows: never more than the slots for copies
        p.stages = (int)((kNgRingBytes<true> - kNgWBytes) / (2u * p.x_bytes));   // 2 to 16, behind them the W tile of the extra block
        p.tmem_cols = 256;
        p.group_blocks = a.gs_k / 64; p.group_shift = -1;
        for (int i = 0; i < 16; ++i) if (p.group_blocks == 1 << i) p.group_shift = i;
    } else {
        p.n_acc = p.npad <= 64 ? 4 : 2;
        p.stages = (int)(kNgRingBytes<false> / (kNgWBytes + p.x_bytes));
        p.tmem_cols = (uint32_t)(p.n_acc * p.npad);     // 64, 128 or 256
    }
    if (p.stages > kNgMaxStages) p.stages = kNgMaxStages;
    p.nkb = (a.K + 63) / 64; p.n_blocks = p.nkb + (a.r2 > 0 ? 1 : 0);
    p.count = a.count;
    p.gs_n = a.gs_n; p.gs_k = a.gs_k; p.n_kgroups = lut ? a.K / a.gs_k : 0;
    if (a.glu && (!lut || a.count != 2 || a.mat[0].N != a.mat[1].N || a.r2 || a.bias || a.act || a.y_f32 || a.alpha != 1.0f)) return PLZ_ERR_UNSUPPORTED;
    p.glu = a.glu;
    p.bias = (const __nv_bfloat16*)a.bias; p.act = a.act; p.y_f32 = a.y_f32; p.alpha = a.alpha;
    p.status = device_status_ptr();
    int tiles = 0, rc;
    for (int i = 0; i < a.count; ++i) {
        const NarrowArgs::Mat& s = a.mat[i];
        if (s.N < 1 || (a.act == ACT_GLU_GELU && s.N % 2) || (lut && (((uintptr_t)s.packed & 15) || s.pitch % 16 || ((uintptr_t)s.palette & 7)))) return PLZ_ERR_UNSUPPORTED;
        p.mat[i] = NarrowMat{s.N, tiles, (const uint8_t*)s.packed, s.pitch, (const __nv_bfloat16*)s.palette, s.y, s.ldy};
        tiles += (s.N + 127) / 128;
    }
    if (a.glu) {
        tiles = (a.mat[0].N + 63) / 64;
        p.mat[1].first_tile = 0x7FFFFFFF;        // every tile belongs to the first
    }
    CUtensorMap tm[4];
    if ((rc = a.x_mn ? make_tmap_bf16(&tm[0], a.x, a.K, a.M, a.ldx, 64, 64) : make_tmap_bf16(&tm[0], a.x, a.M, a.K, a.ldx, 64, (uint32_t)p.npad))) return rc;
    tm[1] = tm[2] = tm[3] = tm[0];
    if (!lut && (rc = make_tmap_bf16(&tm[1], a.mat[0].w, a.mat[0].N, a.K, a.mat[0].ldw, 64, 128))) return rc;
    if (a.r2) {
        if ((rc = make_tmap_bf16(&tm[2], a.x2, a.M, a.r2, a.ldx2, 64, (uint32_t)p.npad))) return rc;
        if ((rc = make_tmap_bf16(&tm[3], a.w2, a.mat[0].N, a.r2, a.ldw2, 64, 128))) return rc;
    }
    const int ranks = a.transposed ? turned_parts(p.n_blocks) : lut ? cluster_size_packed(tiles, p.n_blocks, seq_sm_count()) : cluster_size(tiles, p.n_blocks, seq_sm_count(), 12);
    const bool chain = a.early && !a.transposed;                  // else W may be what the previous kernel writes, and the result what the next one reads as W
    p.early = chain && g_smallm_overlap;
    p.lets_next = chain || !g_smallm_overlap;
    return lut ? launch_ng<true>(p, tiles, ranks, tm, stream) : launch_ng<false>(p, tiles, ranks, tm, stream);
}

namespace {
// ---- turned round, a whole row tile per CTA ----------------------------------------------------------------------------------------------
// Many row tiles, or a reduction of one part: no cluster. A CTA walks its tiles (grid: at most one CTA per SM, or the limit on CTAs) and of each the
// parts of the reduction that the CTAs of a cluster would take; four output warps (thread = row) add up a part's accumulators and then the parts in
// the same order, so that a row has the same bits either way. Two sets of accumulators, the next part's MMAs run under the sums of this one; the
// ring takes the whole SM, with 16 KB of rows and the factor's tile (out of L2) per stage. Bound by streaming the rows: 16384 rows of 9728, rank 16, 62 -> 52 us
// (6.1 TB/s) against clusters, rank 64 76 -> 53; of 2560 18 -> 14.5 and 23 -> 12.6; 1000 rows of 512, rank 64, 10.5 -> 5.1.
constexpr int kTgThreads = 6 * 32;
constexpr int kTgMaxStages = 11;
constexpr uint32_t kTgRingBytes = 200 * 1024;
struct TurnedParams {
    int M, N, tiles, parts, n_blocks, x_mn, stages;
    int lets_next;           // let the next kernel start behind this one's wait
    uint32_t x_bytes;
    __nv_bfloat16* y; long long ldy;
    float alpha;
    StatusWord* status;
};

template <int NPAD>
__global__ void __launch_bounds__(kTgThreads, 1)
turned_gemm_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const TurnedParams p) {
    constexpr int kAcc = 4;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    const uint32_t stage_bytes = kNgWBytes + p.x_bytes, bar = base + kTgRingBytes;
    auto full = [&](int s) { return bar + 8u * s; };
    auto empty = [&](int s) { return bar + 8u * (kTgMaxStages + s); };
    auto acc_full = [&](int b) { return bar + 8u * (2 * kTgMaxStages + b); };
    auto acc_empty = [&](int b) { return bar + 8u * (2 * kTgMaxStages + 2 + b); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + kTgRingBytes + 8 * (2 * kTgMaxStages + 4));
    volatile uint32_t* abort_flag = tmem_slot + 1;
    static_assert(8 * (2 * kTgMaxStages + 4) + 8 <= kNgBarBytes, "barriers");

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kTgMaxStages; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 4); }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmX);
        tma_prefetch_desc(&tmW);
    }
    if (warp == 1) { tmem_alloc(smem_u32((const void*)tmem_slot), 2 * kAcc * NPAD); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    if (p.lets_next) pdl_launch_dependents();

    int issued = 0;                        // stages the producing thread has filled
    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int s = 0;
            uint32_t ph = 0;
            for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
                for (int b = 0; b < p.n_blocks; ++b) {
                    ok = mbar_wait(empty(s), ph ^ 1u, abort_flag, p.status, ST_TIMEOUT_EMPTY, 0);
                    if (!ok) break;
                    const uint32_t at = base + s * stage_bytes;
                    mbar_arrive_expect_tx(full(s), kNgWBytes + p.x_bytes);
                    tma_load_2d(at, &tmW, full(s), b * 64, t * 128);
                    tma_load_2d(at + kNgWBytes, &tmX, full(s), p.x_mn ? 0 : b * 64, p.x_mn ? b * 64 : 0);
                    ++issued;
                    if (++s == p.stages) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = make_idesc(128, NPAD, 0, p.x_mn ? 1 : 0), x_step = p.x_mn ? 2048u >> 4 : 2u;
        const uint64_t desc = make_sdesc(base, 16u, 1024u);
        const uint32_t hi = (uint32_t)(desc >> 32), lo0 = (uint32_t)desc, slot = stage_bytes >> 4;
        bool ok = true;
        int s = 0, q = 0;
        uint32_t ph = 0, lo = lo0;
        for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
            for (int part = 0; part < p.parts && ok; ++part, ++q) {
                const int b0 = (int)((long long)part * p.n_blocks / p.parts), b1 = (int)((long long)(part + 1) * p.n_blocks / p.parts);
                const uint32_t d = tmem_base + (uint32_t)(q & 1) * (kAcc * NPAD);
                ok = mbar_wait_warp(acc_empty(q & 1), ((q >> 1) & 1) ^ 1u, abort_flag, p.status, ST_TIMEOUT_ACCUM, 1);
                for (int b = b0; b < b1 && ok; ++b) {
                    ok = mbar_wait_warp(full(s), ph, abort_flag, p.status, ST_TIMEOUT_FULL, 1);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const uint32_t xd = lo + (kNgWBytes >> 4), more = b > b0 ? 1u : 0u;
                    if (elect_one()) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) umma_bf16_words<1>(d + i * NPAD, lo + 2u * i, hi, xd + x_step * i, hi, idesc, more);
                        umma_commit(empty(s));
                    }
                    __syncwarp();
                    lo += slot;
                    if (++s == p.stages) { s = 0; ph ^= 1u; lo = lo0; }
                }
                if (ok && elect_one()) umma_commit(acc_full(q & 1));
                __syncwarp();
            }
        }
    } else {
        const int lg = warp & 3;
        const uint32_t lane_base = tmem_base + ((uint32_t)(lg * 32) << 16);
        bool ok = true;
        int q = 0;
        for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
            float tot[NPAD];
#pragma unroll
            for (int c = 0; c < NPAD; ++c) tot[c] = 0.f;
            for (int part = 0; part < p.parts && ok; ++part, ++q) {
                ok = mbar_wait(acc_full(q & 1), (q >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_ACCUM, 4);
                if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
                tc_fence_after_sync();
#pragma unroll
                for (int c0 = 0; c0 < NPAD; c0 += 16) {
                    float sum[16];
#pragma unroll
                    for (int a = 0; a < kAcc; ++a) {
                        uint32_t v[16];
                        tmem_ld_32x16(lane_base + (uint32_t)(((q & 1) * kAcc + a) * NPAD + c0), v);
#pragma unroll
                        for (int c = 0; c < 16; ++c) sum[c] = a == 0 ? __uint_as_float(v[c]) : sum[c] + __uint_as_float(v[c]);
                    }
#pragma unroll
                    for (int c = 0; c < 16; ++c) tot[c0 + c] += sum[c];
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty(q & 1));
            }
            const int n = t * 128 + lg * 32 + lane;
            if (ok && n < p.N) {
                __nv_bfloat16* y = p.y + (long long)n * p.ldy;
#pragma unroll
                for (int c = 0; c < NPAD; c += 8)      // M is a multiple of 8, rows of y are aligned to 16 bytes
                    if (c < p.M)
                        *reinterpret_cast<uint4*>(y + c) = make_uint4(pack_bf16x2(tot[c] * p.alpha, tot[c + 1] * p.alpha), pack_bf16x2(tot[c + 2] * p.alpha, tot[c + 3] * p.alpha),
                                                                      pack_bf16x2(tot[c + 4] * p.alpha, tot[c + 5] * p.alpha), pack_bf16x2(tot[c + 6] * p.alpha, tot[c + 7] * p.alpha));
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) {
        const uint64_t t0 = globaltimer_ns();
        for (int it = issued > p.stages ? issued - p.stages : 0; it < issued; ++it)
            while (!mbar_try_wait(full(it % p.stages), (it / p.stages) & 1))
                if (globaltimer_ns() - t0 > 100000000ull) { report(p.status, ST_TIMEOUT_DRAIN, 0); break; }
    }
    __syncthreads();
    if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, 2 * kAcc * NPAD); }
}

template <int NPAD>
int launch_tg(const NarrowArgs& a, const CUtensorMap& tmX, const CUtensorMap& tmW, int ctas, cudaStream_t stream) {
    TurnedParams p = {};
    p.M = a.M; p.N = a.mat[0].N; p.tiles = (p.N + 127) / 128; p.n_blocks = (a.K + 63) / 64; p.parts = turned_parts(p.n_blocks); p.x_mn = a.x_mn;
    p.x_bytes = a.x_mn ? 64u * 128u : NPAD * 128u;
    p.stages = (int)(kTgRingBytes / (kNgWBytes + p.x_bytes));
    if (p.stages > kTgMaxStages) p.stages = kTgMaxStages;
    p.y = (__nv_bfloat16*)a.mat[0].y; p.ldy = a.mat[0].ldy; p.alpha = a.alpha; p.status = device_status_ptr();
    p.lets_next = !g_smallm_overlap;
    auto kern = turned_gemm_kernel<NPAD>;
    constexpr uint32_t smem = kTgRingBytes + kNgBarBytes + 1024;
    static bool attr_set[64] = {};
    int dev = 0;
    PLZ_CUDA_CHECK(cudaGetDevice(&dev));
    if (!attr_set[dev & 63]) {
        PLZ_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attr_set[dev & 63] = true;
    }
    PLZ_LAUNCH_BEHIND(kern, dim3(p.tiles < ctas ? p.tiles : ctas), dim3(kTgThreads), smem, stream, tmX, tmW, p);
    return PLZ_OK;
}

}  // namespace

// y [N, M] = alpha W x^T, M <= 64: x A^T and dY B of a LoRA branch. ctas > 0: a limit on the CTAs.
int launch_turned_gemm(const NarrowArgs& a, int ctas, cudaStream_t stream) {
    if (a.M < 8 || a.M > 64 || a.M % 8 || a.mat[0].N < 1 || a.K % 8) return PLZ_ERR_UNSUPPORTED;
    const int sms = seq_sm_count(), tiles = (a.mat[0].N + 127) / 128, npad = a.M <= 16 ? 16 : a.M <= 32 ? 32 : 64, parts = turned_parts((a.K + 63) / 64);
    CUtensorMap tmX, tmW;
    int rc;
    // A cluster per row tile while the rows leave SMs idle. us cluster / whole: 9728 columns, rank 16, 4096 rows 13.8 / 30, 6144 28 / 32, 8192 33 / 34, rank 64 35 / 34, 40 / 35 at the
    // last two; 2560 columns, 6144 rows 9.0 / 11.2, 8192 9.9 / 11.7, 12288 16 / 13; 1024 columns, whatever the rows and the rank 6.3 to 9.3 / 5.9 to 6.8.
    const bool few = (parts == 8 && tiles <= sms / 3) || (parts == 4 && tiles <= 9 * sms / 20);
    if (ctas <= 0 && few && (rc = launch_narrow_gemm(a, stream)) != PLZ_ERR_UNSUPPORTED) return rc;   // which the maps below refuse
    if ((rc = a.x_mn ? make_tmap_bf16(&tmX, a.x, a.K, a.M, a.ldx, 64, 64) : make_tmap_bf16(&tmX, a.x, a.M, a.K, a.ldx, 64, (uint32_t)npad))) return rc;
    if ((rc = make_tmap_bf16(&tmW, a.mat[0].w, a.mat[0].N, a.K, a.mat[0].ldw, 64, 128))) return rc;
    if (ctas <= 0 || ctas > sms) ctas = sms;
    return npad == 16 ? launch_tg<16>(a, tmX, tmW, ctas, stream) : npad == 32 ? launch_tg<32>(a, tmX, tmW, ctas, stream) : launch_tg<64>(a, tmX, tmW, ctas, stream);
}

}  // namespace plz
