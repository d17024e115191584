"""Element-wise kernels with 16-byte accesses (csrc/layer_ops.cu, csrc/train_ops.cu) and the forms they leave to the 4-byte kernels, against the same
in 64 bits. bf16 intermediates and results bound the error: three roundings of 2^-9 forward, one of the result (2^-8 of it) backward, and fp32 sums
of n terms n 2^-24 of the sum of magnitudes."""
import pytest
import torch

import plz_ops as ops

pytestmark = pytest.mark.gpu


def rows(g, M, K, shift):
    """bf16 [M, K], 16-byte aligned rows (shift 0) or rows that start `shift` elements behind."""
    t = torch.randn(M, K + 16, generator=g, device="cuda").bfloat16()
    return t[:, shift:shift + K]


def turn(y, cos, sin, sign):
    lo, hi = y[..., :64], y[..., 64:]
    return torch.cat([lo * cos - sign * hi * sin, hi * cos + sign * lo * sin], -1)


@pytest.mark.parametrize("tokens,S,Hq,Hk,shift", [(1, 1, 1, 1, 0), (5, 5, 3, 2, 0), (77, 11, 32, 8, 0), (77, 11, 32, 8, 2), (4097, 4097, 5, 1, 0), (6000, 1000, 32, 8, 0)])
def test_qknorm_rope(tokens, S, Hq, Hk, shift):
    g = torch.Generator(device="cuda").manual_seed(tokens)
    xq, xk, dy = rows(g, tokens, Hq * 128, shift), rows(g, tokens, Hk * 128, shift), rows(g, tokens, Hq * 128, shift)
    w = (1 + 0.1 * torch.randn(128, generator=g, device="cuda")).bfloat16()
    cos, sin = ops.rope_tables(S)
    q, k = ops.qknorm_rope_forward2(xq, w, Hq, xk, None, Hk, cos, sin, S)
    dx, dw = ops.qknorm_rope_backward(xq, w, cos, sin, dy, Hq, S)
    at = torch.arange(tokens, device="cuda") % S
    c, s = cos.double()[at][:, None], sin.double()[at][:, None]
    for x, wt, H, y in ((xq, w.double(), Hq, q), (xk, 1.0, Hk, k)):
        v = x.double().reshape(tokens, H, 128)
        n = v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-6) * wt
        size = n.abs() + n.roll(64, -1).abs()
        assert bool(((y.double().view(tokens, H, 128) - turn(n, c, s, 1.0)).abs() <= 3 * 2.0 ** -8 * size).all())
    v, d = xq.double().reshape(tokens, Hq, 128), dy.double().reshape(tokens, Hq, 128)
    rs = torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-6)
    t = turn(d, c, s, -1.0)
    u = t * w.double()
    want = rs * (u - v * rs * (u * v * rs).mean(-1, keepdim=True))
    mag = rs * (u.abs() + v.abs() * rs * (u * v * rs).abs().mean(-1, keepdim=True))
    assert bool(((dx.double().view(tokens, Hq, 128) - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * mag).all())
    n = tokens * Hq
    assert bool(((dw.double() - (t * v * rs).sum((0, 1))).abs() <= n * 2.0 ** -24 * (t * v * rs).abs().sum((0, 1)) + 1e-6).all())


@pytest.mark.parametrize("M,K,shift,weighted", [(1, 8, 0, True), (3, 264, 0, False), (1001, 2560, 0, True), (1001, 2560, 2, True), (300, 8192, 0, True), (70, 8200, 0, True), (5, 258, 0, True)])
def test_rmsnorm_backward(M, K, shift, weighted):
    g = torch.Generator(device="cuda").manual_seed(K)
    x, dh = rows(g, M, K, shift), rows(g, M, K, shift)
    if shift == 0:
        x = x.contiguous()
    w = (1 + 0.1 * torch.randn(K, generator=g, device="cuda")).bfloat16() if weighted else None
    rstd = torch.rsqrt(x.float().square().mean(-1) + 1e-6)
    dx, dg = ops.rmsnorm_backward(x, dh, rstd, w)
    v, d, r = x.double(), dh.double(), rstd.double()[:, None]
    u = d * w.double() if weighted else d
    want = r * u - v * r ** 3 * (u * v).mean(-1, keepdim=True)
    mag = r * u.abs() + v.abs() * r ** 3 * (u * v).abs().mean(-1, keepdim=True)
    assert bool(((dx.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * mag).all())
    if weighted:
        assert bool(((dg.double() - (d * v * r).sum(0)).abs() <= (M + 4) * 2.0 ** -23 * (d * v * r).abs().sum(0) + 1e-6).all())


# the 16-byte forward takes 8192 rows (token, head) and more: quads of heads that are not full, and the sizes on either side of the line
@pytest.mark.parametrize("tokens,S,Hq,Hk,shift", [(911, 7, 7, 2, 0), (1023, 1023, 6, 2, 0), (1024, 64, 6, 2, 0), (1400, 3, 6, 1, 0)])
def test_qknorm_rope_many_rows(tokens, S, Hq, Hk, shift):
    test_qknorm_rope(tokens, S, Hq, Hk, shift)


# the 16-byte kernel from 64 rows or 4096 columns on: threads beyond the columns, an odd last row
@pytest.mark.parametrize("M,K,shift,weighted", [(64, 8, 0, True), (65, 264, 0, False), (63, 264, 0, True), (1, 4096, 0, True), (3, 4104, 0, True), (3, 4088, 0, True)])
def test_rmsnorm_backward_lines(M, K, shift, weighted):
    test_rmsnorm_backward(M, K, shift, weighted)
