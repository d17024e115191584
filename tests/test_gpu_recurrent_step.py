"""One token of the two recurrences with the state in 16-byte accesses, against the rule in 64 bits: key sizes from one row group per warp to eight, value sizes that end inside a block,
shared keys, both types; and sizes and addresses that keep the general kernel. Sums over dk in fp32."""
import pytest
import torch

import seq_ops as S
from helpers import check_status

pytestmark = pytest.mark.gpu


def _close(got, want, limit):
    d = (got.double() - want).abs().max() / want.abs().max()
    assert d < limit, float(d)


# the last three: dk not a multiple of 16, dv not of 4, dk above 128
@pytest.mark.parametrize("H,G,dk,dv", [(2, 1, 16, 4), (4, 2, 48, 36), (3, 3, 64, 32), (4, 4, 112, 72), (20, 20, 128, 128), (2, 2, 20, 8), (2, 1, 32, 6), (2, 2, 144, 16)])
def test_delta_rule(H, G, dk, dv):
    B = 3
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q, k = (r(B, G, dk) * dk ** -0.5 for _ in range(2))
    v, lg, beta, S0 = r(B, H, dv), -torch.rand(B, H, dk, generator=g, device="cuda") * 3, torch.rand(B, H, generator=g, device="cuda"), r(B, H, dk, dv)
    st = S0.clone()
    o = S.delta_rule(q.view(B, -1), k.view(B, -1), v.view(B, -1), lg.view(B, -1), beta, st, B, 1, H, G, dk, dv)
    check_status()
    qq, kk = (t.double().repeat_interleave(H // G, 1) for t in (q, k))
    s = torch.exp(lg.double())[..., None] * S0.double()
    u = beta.double()[..., None] * (v.double() - torch.einsum("bhkv,bhk->bhv", s, kk))
    s = s + kk[..., None] * u[:, :, None, :]
    _close(st, s, 3e-6)
    _close(o.view(B, H, dv), torch.einsum("bhkv,bhk->bhv", s, qq), 3e-6)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("lead", [0, 1])      # slices that begin one element further: the general kernel
@pytest.mark.parametrize("H,dk,dv", [(2, 16, 4), (4, 48, 36), (20, 128, 128), (2, 20, 8), (2, 32, 6)])
def test_decay_attention(dt, lead, H, dk, dv):
    B = 3
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    W = H * (2 * dk + dv) + 8
    proj = torch.randn(B, W, generator=g, device="cuda").to(dt)
    q, k, v = (proj[:, lead + a:lead + a + n] for a, n in ((0, H * dk), (H * dk, H * dk), (2 * H * dk, H * dv)))
    decay, S0 = torch.rand(H, generator=g, device="cuda"), torch.randn(B, H, dk, dv, generator=g, device="cuda")
    st = S0.clone()
    o = S.decay_attention(q, k, v, decay, st, B, 1, H, dk, dv)
    check_status()
    qq, kk, vv = (torch.nn.functional.silu(t.double()).reshape(B, H, -1) for t in (q, k, v))
    s = decay.double()[None, :, None, None] * S0.double() + kk[..., None] * vv[:, :, None, :]
    _close(st, s, 3e-6)
    _close(o.view(B, H, dv), torch.einsum("bhkv,bhk->bhv", s, qq), 3e-6)
