"""Attention where its sums are put together: the merge of a decode step's splits over head sizes, split counts and empty splits, and the
prompt kernel's running maximum when scores grow along the sequence.  Checked against softmax in 64 bits (32 bits for the prompt)."""
import pytest
import torch

from helpers import assert_close, check_status

pytestmark = pytest.mark.gpu


# positions: fewer keys than a split takes, splits without keys (few keys in a long cache), all of them at work
@pytest.mark.parametrize("B,H,G,dk,dv,cap,pos", [(1, 2, 1, 16, 8, 4096, 0), (1, 4, 2, 64, 40, 4096, 70), (2, 3, 3, 128, 120, 900, 899), (1, 1, 1, 128, 128, 20000, 17777),
                                                 (1, 4, 1, 64, 128, 300, 299), (1, 2, 2, 128, 136, 2048, 1500)])
@pytest.mark.parametrize("dtype,sink", [(torch.float32, True), (torch.bfloat16, False)])
def test_splits_of_a_decode_step(B, H, G, dk, dv, cap, pos, dtype, sink):
    import seq_ops as S
    g = torch.Generator().manual_seed(cap + pos)
    q = torch.randn(B, H * dk, generator=g).to(dtype).cuda()
    kc = torch.randn(B, cap, G * dk, generator=g).to(dtype).cuda()
    vc = torch.randn(B, cap, G * dv, generator=g).to(dtype).cuda()
    got = S.attention_bias(q, kc, vc, None, torch.tensor([pos], dtype=torch.int32, device="cuda"), -1, B, 1, H, G, dk, dv, dk ** -0.5, sink)
    check_status()
    qf = q.double().view(B, G, H // G, dk)
    kf, vf = (t[:, :pos + 1].double().view(B, pos + 1, G, -1).transpose(1, 2) for t in (kc, vc))
    s = qf @ kf.transpose(-1, -2) * dk ** -0.5
    if sink: s = torch.cat([s, torch.zeros_like(s[..., :1])], -1)
    want = (torch.softmax(s, -1)[..., :pos + 1] @ vf).reshape(B, H * dv)
    if dtype == torch.float32:
        # scores of size < 8 with a relative error of about dk 2^-24: weights within 1e-4, values below 6
        assert (got.double() - want).abs().max() < 6e-4
    else:
        assert_close(got, want.float(), "decode", rel=1e-2, cos=0.9999)


@pytest.mark.parametrize("S", [128, 384, 1024])
@pytest.mark.parametrize("growth", [0.0, 0.5, 3.0, -3.0])       # by tile of 128 keys, in units of the score's spread
def test_scores_that_grow_along_the_sequence(S, growth):
    import plz_ops as ops
    B, Hq, Hkv, D = 1, 2, 1, 128
    g = torch.Generator().manual_seed(S)
    q, do = (torch.randn(B * S, Hq * D, generator=g) for _ in range(2))
    k, v = (torch.randn(B * S, Hkv * D, generator=g) for _ in range(2))
    q[:, ::D] = 4.0
    k[:, 0] = growth * (torch.arange(S) // 128 + torch.arange(S) / 512) * D ** 0.5 / 4
    q, k, v, do = (t.to(torch.bfloat16).cuda() for t in (q, k, v, do))
    o, lse = ops.attention_forward(q, k, v, B, S, Hq, Hkv)
    check_status()
    s = (q.double().view(S, Hq, D).transpose(0, 1) @ k.double().t()) * D ** -0.5
    s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    assert_close(o, (torch.softmax(s, -1) @ v.double()).transpose(0, 1).reshape(S, Hq * D).float(), "o")
    assert_close(lse, torch.logsumexp(s, -1).float().view(B, Hq, S), "log-sum-exp", rel=1e-3)


@pytest.mark.parametrize("B,n,pos", [(1, 300, 0), (3, 300, 0), (3, 520, 70)])      # 64, 192 and 288 CTAs: within a wave and beyond
def test_order_of_the_query_tiles(B, n, pos):
    import seq_ops as S
    H, G, d, T, g = 32, 8, 64, pos + n, torch.Generator(device="cuda").manual_seed(n + B)
    q, k, v = (torch.randn(B, t, h * d, generator=g, device="cuda").bfloat16() for t, h in ((n, H), (T, G), (T, G)))
    tab = torch.randn(H, 100, generator=g, device="cuda")
    o = S.attention_bias(q.view(B * n, H * d), k, v, S.DistanceBias.from_distances(tab), torch.tensor([pos], dtype=torch.int32, device="cuda"), pos, B, n, H, G, d, d, d ** -0.5, True)
    check_status()
    kf, vf = (t.double().view(B, T, G, d).repeat_interleave(H // G, 2) for t in (k, v))
    at = torch.arange(pos, T, device="cuda")[:, None] - torch.arange(T, device="cuda")
    s = torch.einsum("bihd,bjhd->bhij", q.double().view(B, n, H, d), kf) * d ** -0.5 + tab.double()[:, at.clamp(0, 99)]
    s = torch.cat([s.masked_fill(at < 0, float("-inf")), torch.zeros_like(s[..., :1])], -1)
    assert_close(o, torch.einsum("bhij,bjhd->bihd", torch.softmax(s, -1)[..., :-1], vf).reshape(B * n, H * d).float(), "o")


# the entries in front of distance 0 are there to be read with a tile and may hold anything: a prompt, a portion behind cached tokens, more distances than the table has;
# heads of either kind beside each other
@pytest.mark.parametrize("n,pos,D", [(130, 0, 40), (300, 70, 100), (300, 70, 1000)])
def test_what_stands_in_front_of_the_biases(n, pos, D):
    import seq_ops as S
    B, H, G, d, T, g = 1, 4, 2, 64, pos + n, torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn(B, t, h * d, generator=g, device="cuda").bfloat16() for t, h in ((n, H), (T, G), (T, G)))
    b = S.DistanceBias.from_distances(torch.randn(H, D, generator=g, device="cuda"))
    out = []
    for fill in (0.0, 1e29, float("nan"), float("inf"), torch.finfo(torch.float32).max):
        b.rows[::2, :S.BIAS_FRONT] = fill
        out.append(S.attention_bias(q.view(B * n, H * d), k, v, b, torch.tensor([pos], dtype=torch.int32, device="cuda"), pos, B, n, H, G, d, d, d ** -0.5, True))
    check_status()
    # the other pass over a masked tile adds its weights in another order: 128 fp32 sums, then bf16
    assert torch.isfinite(out[0]).all() and torch.equal(out[0], out[1]) and all((o.float() - out[0].float()).abs().max() <= 2.0 ** -7 * out[0].float().abs().max() for o in out)
