"""Linears of one bf16 row whose matrix streams through shared memory, against the same product in 64 bits: ragged row pairs, reductions that end inside a piece, fewer pairs than
CTAs, pitched rows, each activation and type of result, and a chain with early starts. Sums of K products in fp32 add at most K 2^-24 of the sum of magnitudes;
a bf16 result is rounded once (2^-8)."""
import pytest
import torch

import plz_native as P
import seq_ops as S
from helpers import check_status

pytestmark = pytest.mark.gpu


def _rnd(g, *s):
    return torch.randn(*s, generator=g, device="cuda").bfloat16()


@pytest.mark.parametrize("N,K", [(19456, 2560), (2560, 9728), (1601, 2560), (4097, 264), (130, 16384), (2051, 520), (32768, 128), (8193, 1032)])
@pytest.mark.parametrize("pad", [0, 24])
def test_one_row(N, K, pad):
    g = torch.Generator(device="cuda").manual_seed(N + K)
    x, w, bias = _rnd(g, 1, K), _rnd(g, N, K + pad)[:, :K], _rnd(g, N)
    z = x.double() @ w.double().T
    slack = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 1e-30
    assert bool(((S.linear(x, w).double() - z).abs() <= 2.0 ** -8 * z.abs() + slack).all())
    assert bool(((S.linear(x, w, out_f32=True).double() - z).abs() <= slack).all())
    zb = z + bias.double()
    assert bool(((S.linear(x, w, bias, out_f32=True).double() - zb).abs() <= slack + 2.0 ** -23 * zb.abs()).all())
    r = z.clamp(min=0)
    assert bool(((S.linear(x, w, act=S.ACT_RELU2, out_f32=True).double() - r * r).abs() <= (2 * r + slack) * slack + 2.0 ** -22 * r * r).all())
    if N % 2 == 0:
        w2 = (w * K ** -0.5).bfloat16()
        z, mag = x.double() @ w2.double().T, x.double().abs() @ w2.double().abs().T
        ref = torch.nn.functional.gelu(z[:, 0::2], approximate="tanh") * z[:, 1::2]
        # |d gelu| <= 1.13, tanh of fp32 to 2^-20
        slack = K * 2.0 ** -24 * (1.13 * mag[:, 0::2] * z[:, 1::2].abs() + mag[:, 1::2] * z[:, 0::2].abs()) + 2.0 ** -20 * (z[:, 0::2] * z[:, 1::2]).abs() + 1e-7
        assert bool(((S.linear(x, w2, act=S.ACT_GLU_GELU, out_f32=True).double() - ref).abs() <= slack).all())
    check_status()


def test_chain_with_early_starts_repeats():
    g = torch.Generator(device="cuda").manual_seed(3)
    up, down, x = (_rnd(g, 9728, 2560) * 2560 ** -0.5).bfloat16(), (_rnd(g, 2560, 9728) * 9728 ** -0.5).bfloat16(), _rnd(g, 1, 2560)

    def chain():
        h = x
        for _ in range(4):
            h = S.linear(S.linear(h, up, act=S.ACT_RELU2), down)
        return h
    want = chain()
    P.lib().plz_set_smallm_overlap(1)
    try:
        for _ in range(20):
            assert torch.equal(chain(), want)
    finally:
        P.lib().plz_set_smallm_overlap(0)
    check_status()
