"""Row-wise steps with the row in registers (csrc/seq_ops.cu: embedding, norm of picked rows, residual update with everything requested ahead) at the edges of
their widths, and the small-M product with palettes in shared memory or not (csrc/smallm_mma.cu), against the same in 64 bits. fp32 results of sums of
W squares: W 2^-24 relative; one bf16 rounding 2^-9 of the value where the output is bf16."""
import pytest
import torch

import plz_ops as ops
import seq_ops as S

pytestmark = pytest.mark.gpu


def rms(x, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def close(y, ref, W, mag=None):
    rel = (2.0 ** -8 if y.dtype == torch.bfloat16 else 0.0) + (W + 16) * 2.0 ** -24
    assert bool(((y.double() - ref).abs() <= rel * (ref.abs() if mag is None else mag) + 1e-30).all())


# one row, a few (everything ahead), more than two per SM; widths of the register forms, past them, not a multiple of four
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,W", [(1, 4), (3, 1000), (1, 2560), (500, 2560), (2, 3076), (300, 4096), (5, 4100), (297, 8192), (4, 2562)])
def test_rows(rows, W, dtype):
    g = torch.Generator(device="cuda").manual_seed(W)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    table, w, w2, vec = rnd(11, W).to(dtype), rnd(W), rnd(W), rnd(W)
    ids = torch.randint(0, 11, (rows,), generator=g, device="cuda")
    ids[-1] = 11                                                     # outside the table: a row of zeros
    e = torch.where((ids < 11)[:, None], table.double()[ids.clamp(max=10)] * 3.0, 0.0)
    x, xb, x2 = S.embed(table, ids, 3.0, copy=True)
    close(x, e, W), close(xb, e, W), close(x2, e, W)
    x, xb, _ = S.embed(table, ids, 3.0, w, 1.0, 1e-6)
    close(x, rms(e) * (w.double() + 1), W), close(xb, rms(e) * (w.double() + 1), W)
    idx = torch.randint(0, rows, (7,), generator=g, device="cuda")
    x = rnd(rows, W)
    close(S.rows_norm(x, idx, w, 0.5, 1e-6, dtype), rms(x.double()[idx]) * (w.double() + 0.5), W)
    y, add, out = rnd(rows, W).to(dtype), rnd(rows, W), torch.empty(rows, W, dtype=dtype, device="cuda")
    parts = [x.double(), 0.7 * rms(y.double()) * (w.double() + 1), add.double(), vec.double()]
    want, mag = sum(parts), sum(t.abs() for t in parts)
    S.stream_update(x, dtype, 1e-6, y, w, 0.7, 1.0, add, vec, w2, out)
    close(x, want, W, mag)
    # the second norm: its operand carries the error of x, its weight that of w2 + 1
    n = rms(want) * (w2.double() + 1)
    close(out, n, 2 * W, n.abs() + rms(want).abs() + (w2.double() + 1).abs() * mag * torch.rsqrt(want.square().mean(-1, keepdim=True)))


@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("M,N,K", [(1, 40, 512), (1, 2560, 9728), (16, 24, 2560), (9, 296, 5120)])
def test_small_m_palettes(M, N, K, shift):
    g = torch.Generator(device="cuda").manual_seed(N)
    idx = torch.randint(0, 4, (N, K), generator=g, device="cuda", dtype=torch.int8)
    pal = torch.randn(N * (K // 256) * 4 + shift, generator=g, device="cuda").bfloat16()[shift:].view(-1, 4)    # shift 4: 8-byte aligned only
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    W = torch.gather(pal.view(N, K // 256, 1, 4).expand(-1, -1, 256, -1).reshape(N, K, 4), 2, idx.long()[:, :, None])[:, :, 0].double()
    y = ops.hard_forward_smallm(ops.PackedWeight(ops.pack_indices(idx, n_major=True), pal, N, K, 1, 256), x)
    ref, mag = x.double() @ W.T, x.double().abs() @ W.abs().T
    assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + K * 2.0 ** -24 * mag).all())


# a warp per group (up to 256), a block per group, the widest register form, and the general kernel (wider, or rows that are not 16-byte aligned)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,groups,L,pitch", [(3, 20, 128, 0), (5, 3, 132, 4), (2, 9, 256, 0), (7, 2, 260, 0), (300, 1, 2560, 8), (2, 1, 3076, 0), (2, 1, 4100, 0), (4, 5, 30, 1)])
def test_norm_gate(rows, groups, L, pitch, dtype):
    g = torch.Generator(device="cuda").manual_seed(L)
    o, w = torch.randn(rows, groups * L, generator=g, device="cuda"), torch.randn(L, generator=g, device="cuda")
    gate = torch.randn(rows, groups * L + pitch, generator=g, device="cuda").to(dtype)[:, :groups * L]
    ref = rms(o.double().view(rows, groups, L)) * w.double() * torch.sigmoid(gate.double().reshape(rows, groups, L))
    close(S.norm_gate(o, gate, w, 1e-6, groups), ref.view(rows, -1), L + 64)


# query and key widths of both register forms, past them, and odd ones; the first layer writes the values that later ones mix in
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,n,qw,kw,vw", [(2, 3, 4096, 1024, 1024), (64, 1, 2048, 512, 256), (1, 300, 1028, 2052, 8), (2, 2, 4104, 128, 128), (1, 5, 130, 66, 34)])
def test_attn_prep(B, n, qw, kw, vw, dtype):
    g = torch.Generator(device="cuda").manual_seed(qw)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    proj, wq, wk, mix, cap = rnd(B * n, qw + kw + vw + 8).to(dtype), rnd(qw), rnd(kw), torch.tensor([0.3], device="cuda"), n + 7
    offs, first = (0, qw, qw + kw), rnd(B * n, vw).to(dtype)
    pos = torch.tensor([4], dtype=torch.int32, device="cuda")
    for write in (True, False):
        kc, vc, vf = (torch.zeros(B, cap, w, dtype=dtype, device="cuda") for w in (kw, vw, 1))
        vf = torch.zeros(B * n, vw, dtype=dtype, device="cuda") if write else first.clone()
        q = S.attn_prep(proj, offs, wq, wk, None if write else mix, vf, write, kc, vc, pos, B, n, 1e-6)
        p = proj.double()
        close(q, rms(p[:, :qw]) * wq.double(), qw)
        close(kc[:, 4:4 + n].reshape(B * n, kw), rms(p[:, qw:qw + kw]) * wk.double(), kw)
        v = p[:, qw + kw:qw + kw + vw]
        if write:
            assert torch.equal(vf, proj[:, qw + kw:qw + kw + vw]) and torch.equal(vc[:, 4:4 + n].reshape(B * n, vw), vf)
        else:
            lam = mix.double()
            close(vc[:, 4:4 + n].reshape(B * n, vw), (1 - lam) * v + lam * first.double(), 16, v.abs() + first.double().abs())
        assert not kc[:, :4].any() and not kc[:, 4 + n:].any() and not vc[:, :4].any() and not vc[:, 4 + n:].any()


def test_overlapped_rows():
    """Programmatic dependent launch on: kernels that may start under the one that writes their input read it only after that one has finished. The
    buffers come round again with other contents, so that a load that is too early is seen."""
    import plz_native as P
    g = torch.Generator(device="cuda").manual_seed(3)
    rows, W = 64, 2560
    table, w = torch.randn(500, W, generator=g, device="cuda").bfloat16(), torch.randn(W, generator=g, device="cuda")
    gate = torch.randn(rows, W, generator=g, device="cuda").bfloat16()
    ids = torch.randint(0, 500, (24, rows), generator=g, device="cuda")

    def chain(i):
        x, xb, _ = S.embed(table, ids[i], 2.0)
        a = S.norm_gate(x, gate, w, 1e-6, 1)
        b = S.norm_gate(x, gate, w[:128], 1e-6, 20)
        S.stream_update(x, torch.bfloat16, 1e-6, a, w, 0.7, 1.0, None, None, w, xb)
        return torch.cat([a, b, xb, S.rows_norm(x, None, w, 1.0, 1e-6, torch.bfloat16)])
    want = [chain(i) for i in range(24)]
    torch.cuda.synchronize()
    P.lib().plz_set_smallm_overlap(1)
    try:
        got = [chain(i) for i in range(24)]
    finally:
        P.lib().plz_set_smallm_overlap(0)
    assert all(torch.equal(a, b) for a, b in zip(want, got))


# the register forms start at 256 columns; beyond 4096 the update requests everything ahead for one row per SM only
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,W", [(2, 252), (3, 256), (1, 260), (150, 8192), (140, 4100)])
def test_rows_lines(rows, W, dtype):
    test_rows(rows, W, dtype)
