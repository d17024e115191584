"""Linear products with 1 to 128 rows on the swapped tcgen05 kernel (csrc/narrow_gemm.cu): edges of its tiles, clusters and epilogues, against
the same product in 64 bits. One bf16 rounding of the result bounds every element by 2^-8 of it; sums over K in fp32 add at most K 2^-24 of the sum
of magnitudes."""
import pytest
import torch

import plz_ops as ops
import seq_ops as S

pytestmark = pytest.mark.gpu


def check(y, ref, mag, K, half_ulp=2.0 ** -8):
    bound = half_ulp * ref.abs() + K * 2.0 ** -24 * mag + 1e-30
    assert bool(((y.double() - ref).abs() <= bound).all())


# rows around the MMA widths 16 / 32 / 64 / 128, outputs around a 128-row tile, reductions of one block, of ragged last blocks, and long enough
# for clusters of several CTAs (2560 x 1000: split; 20000 columns: no split)
@pytest.mark.parametrize("M,N,K", [(17, 8, 8), (17, 136, 72), (32, 128, 64), (33, 120, 200), (64, 1032, 2560), (65, 264, 2056), (128, 2560, 1000), (127, 1000, 4096), (24, 20000, 320), (16, 1024, 2560), (9, 1000, 2104)])
def test_dense(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(N, generator=g, device="cuda").bfloat16()
    ref, mag = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    check(S.linear(x, w), ref, mag, K)
    check(S.linear(x, w, b), ref + b.double(), mag + b.double().abs(), K)
    y = S.linear(x, w, act=S.ACT_RELU2)
    r = ref.clamp(min=0)
    assert bool(((y.double() - r * r).abs() <= 2.0 ** -8 * r * r + (2 * r + 1) * (K * 2.0 ** -24 * mag) + 1e-30).all())
    if M <= 16:
        check(S.linear(x, w, out_f32=True), ref, mag, K, 2.0 ** -24)
    out = torch.full((M, N + 24), 7.0, device="cuda", dtype=torch.bfloat16)      # a pitched destination: nothing beside it is written
    S.linear(x, w, out=out[:, 8:8 + N])
    check(out[:, 8:8 + N], ref, mag, K)
    assert bool((out[:, :8] == 7).all()) and bool((out[:, 8 + N:] == 7).all())


@pytest.mark.parametrize("M,N,K", [(20, 6, 64), (64, 1032, 2560), (100, 130, 2304)])
def test_gated_pairs(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(2 * N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    z = x.double() @ w.double().T
    ref = torch.nn.functional.gelu(z[:, 0::2], approximate="tanh") * z[:, 1::2]
    y = S.linear(x, w, act=S.ACT_GLU_GELU)
    # |d gelu| <= 1.13; each of the two factors carries K 2^-24 times the row's magnitude
    mag = x.double().abs() @ w.double().abs().T
    slack = K * 2.0 ** -24 * (1.13 * mag[:, 0::2] * z[:, 1::2].abs() + mag[:, 1::2] * z[:, 0::2].abs()) + 1e-6 * ref.abs() + 1e-7
    assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + slack).all())


# palette groups of 64, 192 (no power of two), 256 columns and of the whole reduction with 256 shared rows; LoRA ranks that fill part of a block
@pytest.mark.parametrize("M,N,K,gs_n,gs_k,rank", [(17, 8, 64, 1, 64, 0), (33, 136, 384, 1, 192, 8), (64, 2560, 2560, 1, 256, 16), (128, 1000, 1024, 1, 256, 64), (1, 512, 2560, 256, 2560, 32),
                                                  (65, 768, 2624, 256, 2624, 0), (16, 520, 9728, 1, 256, 0), (40, 9728, 320, 1, 64, 16)])
def test_packed(M, N, K, gs_n, gs_k, rank):
    g = torch.Generator(device="cuda").manual_seed(K)
    idx = torch.randint(0, 4, (N, K), generator=g, device="cuda", dtype=torch.int8)
    pal = torch.randn((N // gs_n) * (K // gs_k), 4, generator=g, device="cuda").bfloat16()
    w = ops.PackedWeight(ops.pack_indices(idx, n_major=True), pal, N, K, gs_n, gs_k)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    W = torch.gather(pal.view(N // gs_n, 1, K // gs_k, 1, 4).expand(-1, gs_n, -1, gs_k, -1).reshape(N, K, 4), 2, idx.long()[:, :, None])[:, :, 0].double()
    ref, mag = x.double() @ W.T, x.double().abs() @ W.abs().T
    if rank:
        a, b = torch.randn(rank, K, generator=g, device="cuda").bfloat16(), torch.randn(N, rank, generator=g, device="cuda").bfloat16()
        y, t = ops.hard_forward(w, x, (a, b, 0.5))
        check(t, 0.5 * x.double() @ a.double().T, 0.5 * x.double().abs() @ a.double().abs().T, K)
        ref, mag = ref + t.double() @ b.double().T, mag + t.double().abs() @ b.double().abs().T
    else:
        y = ops.hard_forward(w, x)[0]
        if 16 < M <= 64:
            check(ops.hard_forward_smallm(w, x), ref, mag, K)
    check(y, ref, mag, K + rank)
    assert torch.equal(y, ops.hard_forward(w, x, (a, b, 0.5) if rank else None)[0])


# x A^T and dY B of a LoRA branch: rows around a 128-row tile, ranks around the MMA widths, reductions of one block, of a few, and split over a cluster
@pytest.mark.parametrize("M,K,rank", [(1, 64, 8), (127, 128, 16), (129, 192, 24), (1000, 9728, 32), (300, 2560, 64), (4097, 1024, 40), (20000, 256, 16)])
def test_lora_factors(M, K, rank):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, a, b = rnd(M, K + 8)[:, :K], rnd(rank, K), rnd(K, rank)
    ref, mag = 0.5 * x.double() @ b.double(), 0.5 * x.double().abs() @ b.double().abs()
    check(ops.lora_dt((a, b, 0.5), x), ref, mag, K)
    w = ops.PackedWeight(ops.pack_indices(torch.zeros(64, K, dtype=torch.int8, device="cuda"), n_major=True), torch.zeros(64, 4, device="cuda", dtype=torch.bfloat16), 64, K, 1, K)
    t = ops.hard_forward(w, x, (a, rnd(64, rank), 0.5))[1]
    check(t, 0.5 * x.double() @ a.double().T, 0.5 * x.double().abs() @ a.double().abs().T, K)


@pytest.mark.parametrize("K,rank", [(64, 8), (1088, 16), (2560, 32), (9728, 64)])
def test_lora_rows_do_not_depend_on_their_number(K, rank):
    g = torch.Generator(device="cuda").manual_seed(K)
    x, b = torch.randn(20000, K, generator=g, device="cuda").bfloat16(), torch.randn(K, rank, generator=g, device="cuda").bfloat16()
    a = torch.zeros(rank, K, device="cuda", dtype=torch.bfloat16)
    t = ops.lora_dt((a, b, 1.0), x)
    for lo, hi in ((0, 1), (100, 1100), (1100, 9000)):
        assert torch.equal(ops.lora_dt((a, b, 1.0), x[lo:hi]), t[lo:hi])


# the same for x A^T, at the row counts where other products change their kernel, at ones with more row tiles than SMs, and with a limit on the CTAs
@pytest.mark.parametrize("K,rank", [(64, 64), (1088, 16), (2560, 24), (9728, 32), (4160, 64)])
def test_lora_rows_and_cta_limit(K, rank):
    import plz_native as P
    g = torch.Generator(device="cuda").manual_seed(K + 1)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, a, b = rnd(20011, K), rnd(rank, K), rnd(K, rank)
    w = ops.PackedWeight(ops.pack_indices(torch.zeros(64, K, dtype=torch.int8, device="cuda"), n_major=True), torch.zeros(64, 4, device="cuda", dtype=torch.bfloat16), 64, K, 1, K)
    t = ops.hard_forward(w, x, (a, rnd(64, rank), 0.5))[1]
    dt = ops.lora_dt((a, b, 0.5), x)
    check(t, 0.5 * x.double() @ a.double().T, 0.5 * x.double().abs() @ a.double().abs().T, K)
    check(dt, 0.5 * x.double() @ b.double(), 0.5 * x.double().abs() @ b.double().abs(), K)
    for limit in (0, 5, 140):
        P.lib().plz_set_cta_limit(limit)
        try:
            for rows in (1, 16, 17, 64, 65, 128, 129, 1000, 9000, 20011):
                lo = 20011 - rows
                assert torch.equal(ops.hard_forward(w, x[lo:], (a, b[:64], 0.5))[1], t[lo:]), (limit, rows)
                assert torch.equal(ops.lora_dt((a, b, 0.5), x[lo:]), dt[lo:]), (limit, rows)
        finally:
            P.lib().plz_set_cta_limit(0)
    P.device_status()


# reductions around the lines between this kernel and one CTA per 128 x 256 tile, at every padding of the rows and tiles that fill a part of the chip, most of it, and more
@pytest.mark.parametrize("N,K", [(72, 128), (72, 192), (520, 256), (520, 320), (9728, 512), (9728, 576), (24576, 384), (24576, 640), (40, 960), (40, 1024)])
def test_short_reductions(N, K):
    g = torch.Generator(device="cuda").manual_seed(N + K)
    idx = torch.randint(0, 4, (N, K), generator=g, device="cuda", dtype=torch.int8)
    pal = torch.randn(N * (K // 64), 4, generator=g, device="cuda").bfloat16()
    w = ops.PackedWeight(ops.pack_indices(idx, n_major=True), pal, N, K, 1, 64)
    W = torch.gather(pal.view(N, K // 64, 1, 4).expand(-1, -1, 64, -1).reshape(N, K, 4), 2, idx.long()[:, :, None])[:, :, 0]
    for M in (1, 16, 17, 33, 64, 65, 128):
        x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
        ref, mag = x.double() @ W.double().T, x.double().abs() @ W.double().abs().T
        check(ops.hard_forward(w, x)[0], ref, mag, K)
        check(ops.dense_forward(W, x)[0], ref, mag, K)
        if 16 < M <= 64:
            check(ops.hard_forward_smallm(w, x), ref, mag, K)
            out = torch.full((M, N + 8), 3.0, device="cuda", dtype=torch.bfloat16)
            ops.hard_forward_smallm(w, x, out[:, 4:4 + N])           # not aligned to 16 bytes
            check(out[:, 4:4 + N], ref, mag, K)
            assert bool((out[:, :4] == 3).all()) and bool((out[:, 4 + N:] == 3).all())
