"""Weight gradient with the soft epilogue where its requests run ahead: edges of tiles and of the tensors, several tiles per CTA, each noise, both
layouts; packed indices written by the same launch; indices of planar fp16 logits."""
import contextlib

import pytest
import torch

import plz_oracle as O
from helpers import assert_close, check_status

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _ctas(n):
    import plz_native as P
    P.lib().plz_set_cta_limit(n)
    try:
        yield
    finally:
        P.lib().plz_set_cta_limit(0)


def _noise(kind, seed, N, K, g):
    if kind == "hash":
        return "hash", O.gumbel_hash(seed, N, K)
    t = None if kind == "none" else torch.randn(N, K, 4, generator=g)
    return t, t


# a last round of quarters (five tiles on four pairs) and of halves (on two), a column tile of 8, CTAs without rows (K = 384: 256 + 128), less than a pair's tile either way, one pair (limit 2) walking eight tiles,
# and the form with eight epilogue warps (from 10241 rows on). Logits in steps of a half: every other argmax is a tie.
@pytest.mark.parametrize("M,N,K,limit", [(65, 264, 384, 0), (64, 200, 256, 0), (40, 520, 128, 0), (96, 776, 512, 2), (70, 1256, 256, 8), (70, 1256, 256, 4), (10304, 264, 384, 2), (7200, 776, 512, 2)])
@pytest.mark.parametrize("noise", ["none", "hash", "tensor"])
@pytest.mark.parametrize("rank", [0, 16])
def test_weight_gradient_writes_the_indices(M, N, K, limit, noise, rank):
    import plz_ops as ops
    g = torch.Generator().manual_seed(M + N + K)
    x, dy = torch.randn(M, K, generator=g).bfloat16(), torch.randn(M, N, generator=g).bfloat16()
    pal = (torch.randn(N * (K // 128), 4, generator=g) * 0.02).bfloat16()
    logits = (torch.randn(N, K, 4, generator=g) * 2).round() / 2
    given, want_noise = _noise(noise, 5, N, K, g)
    t, dt = (torch.randn(M, rank, generator=g).bfloat16() for _ in range(2)) if rank else (None, None)
    w = ops.PackedWeight(ops.empty_packed(N, K, "cuda").fill_(0xAB), pal.cuda(), N, K, 1, 128)
    nz = given.cuda() if isinstance(given, torch.Tensor) else given
    with _ctas(limit):
        dlog, dpal, da, db = ops.backward_dw_soft_select(w, x.cuda(), dy.cuda(), logits.cuda(), "nk4", noise=nz, tau=0.7, seed=5,
                                                         lora_ws=(t.cuda(), dt.cuda()) if rank else None)
    check_status()
    p, _, hard, w_hard = O.soft_weights(logits, want_noise, pal, 0.7, 1, 128)
    assert torch.equal(ops.unpack_indices(w.packed, K).cpu().long(), hard)
    _, want_log, want_pal, _ = O.soft_backward(x, dy, w_hard, p, pal, 1, 128)
    assert_close(dlog, want_log, "dLogits")
    assert_close(dpal, want_pal, "dPalette")
    if rank:
        assert_close(da, dt.float().t() @ x.float(), "dA")
        assert_close(db, dy.float().t() @ t.float(), "dB")


# Without a palette gradient nothing holds the epilogue's warps at the same tile: whole tiles followed by quarters and by halves (as above), by quarters of all 74 pairs, and
# one pair that walks whole tiles alone. The logits' gradients have the bits that they have with one, every time.
@pytest.mark.parametrize("M,N,K,limit", [(70, 1256, 256, 8), (70, 1256, 256, 4), (64, 9728, 2560, 0), (10304, 1256, 256, 8), (96, 776, 512, 2)])
@pytest.mark.parametrize("noise", ["none", "tensor"])
def test_logit_gradient_alone(M, N, K, limit, noise):
    import plz_ops as ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, dy = (torch.randn(M, n, generator=g, device="cuda").bfloat16() for n in (K, N))
    w = ops.PackedWeight(ops.empty_packed(N, K, "cuda"), torch.randn(N * (K // 128), 4, generator=g, device="cuda").bfloat16(), N, K, 1, 128)
    logits = torch.randn(N, K, 4, generator=g, device="cuda") * 2
    nz = None if noise == "none" else torch.randn(N, K, 4, generator=g, device="cuda")
    with _ctas(limit):
        want = ops.backward_dw_soft(w, x, dy, logits, "nk4", noise=nz, tau=0.7)[0]
        got = [ops.backward_dw_soft(w, x, dy, logits, "nk4", noise=nz, tau=0.7, want_dpalette=False) for _ in range(5)]
    check_status()
    assert all(p is None and torch.equal(d, want) for d, p in got)


# logits far beyond any temperature: large ones, the type's lowest in one and in all four entries, the same large value four times
@pytest.mark.parametrize("tau", [1.0, 0.01])
@pytest.mark.parametrize("layout,dtype", [("nk4", torch.float32), ("4kn", torch.float32), ("4kn", torch.float16)])
def test_extreme_logits(layout, dtype, tau):
    import plz_ops as ops
    M, N, K = 65, 264, 384
    g = torch.Generator().manual_seed(7)
    x, dy = torch.randn(M, K, generator=g).bfloat16(), torch.randn(M, N, generator=g).bfloat16()
    pal = (torch.randn(N, 4, generator=g) * 0.02).bfloat16()
    big, lowest = (6e4 if dtype == torch.float16 else 1e10), torch.finfo(dtype).min
    logits = (torch.randn(N, K, 4, generator=g) * 2).round() / 2
    logits[0::6] = torch.tensor([big, 0.0, 0.0, 0.0])
    logits[1::6] = lowest
    logits[2::6, :, 1] = lowest
    logits[3::6] = -big
    logits[4::6] = (logits[4::6] * 1e9).clamp(-big, big)
    logits = logits.to(dtype)
    p = torch.softmax(logits.double() / tau, -1).float()
    _, want_log, want_pal, _ = O.soft_backward(x, dy, torch.zeros(N, K).bfloat16(), p, pal, 1, K)
    lg = (logits if layout == "nk4" else O.from_nk_logits(logits)).cuda()
    w = ops.PackedWeight(ops.empty_packed(N, K, "cuda"), pal.cuda(), N, K, 1, K)
    w_soft = ops.soft_select(w, lg, layout, tau=tau, want_soft=True)
    dlog, dpal = ops.backward_dw_soft(w, x.cuda(), dy.cuda(), lg, layout, tau=tau)
    check_status()
    assert_close(w_soft, (p * O.group_palette(pal, N, K, 1, K)).sum(-1), "W_soft")
    assert_close(dlog, want_log if layout == "nk4" else O.from_nk_logits(want_log), "dLogits")
    assert_close(dpal, want_pal, "dPalette")


# five tiles on four pairs, cut along k, a palette per row (or 128 of them) and 256 columns: what meets at an address adds up the same every time
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("gs_n", [1, 128])
def test_palette_gradient_repeats(dtype, gs_n):
    import plz_ops as ops
    M, N, K = 70, 256, 1280
    g = torch.Generator(device="cuda").manual_seed(3)
    x, dy = (torch.randn(M, n, generator=g, device="cuda").bfloat16() for n in (K, N))
    w = ops.PackedWeight(ops.empty_packed(N, K, "cuda"), torch.randn(N // gs_n * (K // 256), 4, generator=g, device="cuda").bfloat16(), N, K, gs_n, 256)
    lg = torch.randn(4, K, N, generator=g, device="cuda").to(dtype)
    with _ctas(8):
        first = ops.backward_dw_soft(w, x, dy, lg, "4kn", tau=0.7)[1]
        assert all(torch.equal(ops.backward_dw_soft(w, x, dy, lg, "4kn", tau=0.7)[1], first) for _ in range(100))
    check_status()


def test_no_rows_still_select():
    import plz_ops as ops
    N, K = 264, 384
    logits = torch.randn(N, K, 4, generator=torch.Generator().manual_seed(1))
    w = ops.PackedWeight(ops.empty_packed(N, K, "cuda"), torch.zeros(N * 3, 4).bfloat16().cuda(), N, K, 1, 128)
    _, dpal, _, _ = ops.backward_dw_soft_select(w, torch.empty(0, K, device="cuda").bfloat16(), torch.empty(0, N, device="cuda").bfloat16(), logits.cuda(), "nk4")
    check_status()
    assert torch.equal(ops.unpack_indices(w.packed, K).cpu().long(), logits.argmax(-1)) and not dpal.any()


# lead = 0: 16-byte requests; otherwise the planes begin at an odd multiple of 2 bytes and take the loads of one logit
@pytest.mark.parametrize("M,N,K,limit,lead", [(65, 768, 320, 0, 0), (96, 768, 512, 2, 0), (96, 768, 512, 2, 3)])
@pytest.mark.parametrize("noise", ["none", "hash", "tensor"])
def test_planar_fp16_logits(M, N, K, limit, lead, noise):
    import plz_ops as ops
    g = torch.Generator().manual_seed(M + N + K)
    x, dy = torch.randn(M, K, generator=g).bfloat16(), torch.randn(M, N, generator=g).bfloat16()
    pal = (torch.randn(N // 256, 4, generator=g) * 0.02).bfloat16()
    logits = ((torch.randn(4, K, N, generator=g) * 2).round() / 2).half()
    given, want_noise = _noise(noise, 5, N, K, g)
    nz = O.from_nk_logits(given).cuda() if isinstance(given, torch.Tensor) else given
    room = torch.empty(4 * K * N + lead, dtype=torch.float16, device="cuda")
    lg = room[lead:].view(4, K, N).copy_(logits.cuda())
    w = ops.PackedWeight(ops.empty_packed(N, K, "cuda").fill_(0xAB), pal.cuda(), N, K, 256, K)
    ops.soft_select(w, lg, "4kn")
    with _ctas(limit):
        dlog, dpal = ops.backward_dw_soft(w, x.cuda(), dy.cuda(), lg, "4kn", noise=nz, tau=0.7, seed=5)
    check_status()
    p, _, hard, w_hard = O.soft_weights(O.to_nk_logits(logits), want_noise, pal, 0.7, 256, K)
    assert torch.equal(ops.unpack_indices(w.packed, K).cpu().long(), hard)
    _, want_log, want_pal, _ = O.soft_backward(x, dy, w_hard, p, pal, 256, K)
    assert_close(dlog, O.from_nk_logits(want_log), "dLogits")
    assert_close(dpal, want_pal, "dPalette")
