"""Gate and up projection with silu(gate) * up in the same launch: on CTA pairs (prompts), and in the two kernels of a decode step against the same step with the products and the
activation apart, which it follows in every rounding to bf16."""
import contextlib

import pytest
import torch

import plz_native as P
import plz_ops as ops
from helpers import check_status

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _ctas(n):
    P.lib().plz_set_cta_limit(n)
    try:
        yield
    finally:
        P.lib().plz_set_cta_limit(0)


def _weight(g, N, K, gs_n=1, gs_k=64):
    idx = torch.randint(0, 4, (N, K), generator=g, device="cuda", dtype=torch.int8)
    pal = torch.randn((N // gs_n) * (K // gs_k), 4, generator=g, device="cuda").bfloat16()
    W = torch.gather(pal.view(N // gs_n, 1, K // gs_k, 1, 4).expand(-1, gs_n, -1, gs_k, -1).reshape(N, K, 4), 2, idx.long()[:, :, None])[:, :, 0].double()
    return ops.PackedWeight(ops.pack_indices(idx, n_major=True), pal, N, K, gs_n, gs_k), W


# outputs of narrow tiles (64, 96 and 128 of a tile), two waves with halves behind (8 x 20 tiles of 128 outputs on 74 pairs), several tiles of one pair, reductions that end inside a
# stage, palettes shared by rows
@pytest.mark.parametrize("M,N,K,gs_n,limit", [(256, 256, 128, 1, 0), (300, 384, 192, 1, 0), (1000, 2688, 64, 1, 0), (2048, 2560, 128, 1, 0), (700, 1280, 320, 128, 0), (600, 896, 192, 1, 2)])
def test_on_pairs(M, N, K, gs_n, limit):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    (wg, Wg), (wu, Wu) = _weight(g, N, K, gs_n), _weight(g, N, K, gs_n)
    x = torch.randn(M, K, generator=g, device="cuda").mul(K ** -0.5).bfloat16()
    with _ctas(limit):
        act = ops.mlp_gate_up_forward(wg, wu, x)
    check_status()
    gate, up, mag_g, mag_u = x.double() @ Wg.T, x.double() @ Wu.T, x.double().abs() @ Wg.abs().T, x.double().abs() @ Wu.abs().T
    ref = torch.nn.functional.silu(gate) * up
    # |d silu| <= 1.1; K products summed in fp32, fast exponential and division 2^-20 of the gate, one rounding to bf16
    slack = K * 2.0 ** -24 * (1.1 * mag_g * up.abs() + mag_u * gate.abs()) + 2.0 ** -20 * (gate * up).abs() + 1e-7
    assert bool(((act.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + slack).all())


# a CTA's share of 132 rows and of 4, 16 rows of x (two accumulator tiles), and the few-row kernel
@pytest.mark.parametrize("B", [1, 8, 16, 17, 64])
@pytest.mark.parametrize("inter", [512, 9728])
def test_in_a_decode_step(B, inter):
    import decode_model as DM
    cfg = DM.ModelConfig(hidden=256, n_heads=2, n_kv_heads=1, head_dim=128, intermediate=inter, n_layers=1, vocab=512)
    dev = torch.device("cuda", 0)
    model = DM.PalettizedQwen.random(cfg, dev, seed=5, max_positions=64)
    model.embed = (torch.randn(cfg.vocab, cfg.hidden, device=dev) * 0.5).to(torch.bfloat16)
    ids = torch.randint(0, cfg.vocab, (B,), device=dev)
    got = model.decode_hidden(ids, model.new_cache(B, 8), 0)[0]
    check_status()
    L, lin = model.layers[0], ops.hard_forward_smallm
    h = model.embed[ids]
    v = lin(L["v"], ops.rmsnorm_forward(h, L["input_ln"], cfg.eps)[0])          # one cached position: attention returns its value
    x2, n2 = ops.add_rmsnorm_forward(h, lin(L["o"], v.repeat(1, 2)), L["post_ln"], cfg.eps)
    want = ops.add(x2, lin(L["down"], ops.swiglu_forward(lin(L["gate"], n2), lin(L["up"], n2))))
    # the same roundings to bf16, but sums that meet in another order flip some of them
    assert (got.float() - want.float()).abs().max() <= 2.0 ** -7 * want.float().abs().max()
