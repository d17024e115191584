"""Products on CTA pairs (csrc/lut_gemm_pair.cu, csrc/dense_gemm_pair.cu) with every tile width its plan chooses on 74 pairs, against the same product in 64 bits. One
bf16 rounding of the result bounds every element by 2^-8 of it; sums over K in fp32 add at most K 2^-24 of the sum of magnitudes."""
import pytest
import torch

import plz_ops as ops
import seq_ops as S

pytestmark = pytest.mark.gpu


def check(y, ref, mag, K):
    assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + K * 2.0 ** -24 * mag + 1e-30).all())


# tile widths 128, 160, 192 and 224 (in steps of 64 for the input gradient), 256 with ragged last columns; two waves of whole tiles and halves behind (19 x 4 tiles; 4 x 38, the last column
# tile of which is half outside); a wave of whole tiles only
@pytest.mark.parametrize("M,J,R,rank", [(256, 256, 128, 0), (1000, 2560, 192, 16), (1000, 3200, 128, 0), (900, 3904, 128, 8), (1024, 4544, 64, 0),
                                        (4800, 1024, 192, 16), (1000, 9664, 128, 0), (300, 1088, 320, 0), (2048, 2368, 128, 0)])
def test_tile_widths(M, J, R, rank):
    g = torch.Generator(device="cuda").manual_seed(M + J)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()

    def weight(N, K):
        idx = torch.randint(0, 4, (N, K), generator=g, device="cuda", dtype=torch.int8)
        pal = rnd(N * (K // 64), 4)
        W = torch.gather(pal.view(N, K // 64, 1, 4).expand(-1, -1, 64, -1).reshape(N, K, 4), 2, idx.long()[:, :, None])[:, :, 0].double()
        return ops.PackedWeight(ops.pack_indices(idx, n_major=True), pal, N, K, 1, 64), W
    # forward: J weight rows
    w, W = weight(J, R)
    x, bias = rnd(M, R), rnd(J)
    lora = (rnd(rank, R), rnd(J, rank), 0.5) if rank else None
    ref, mag = x.double() @ W.T, x.double().abs() @ W.abs().T
    y, t = ops.hard_forward(w, x, lora)
    if rank:
        ref, mag = ref + t.double() @ lora[1].double().T, mag + t.double().abs() @ lora[1].double().abs().T
    else:
        check(ops.hard_forward_bias(w, x, bias), ref + bias.double(), mag + bias.double().abs(), R)
    check(y, ref, mag, R + rank)
    # input gradient: J weight columns
    w, W = weight(R, J)
    lora = (rnd(rank, J), rnd(R, rank), 0.5) if rank else None
    ref, mag = x.double() @ W, x.double().abs() @ W.abs()
    out = torch.full((M, J + 16), 7.0, device="cuda", dtype=torch.bfloat16)       # nothing beside the result is written
    if rank:
        dx, dt = ops.backward_dx(w, x, lora)
        ref, mag = ref + dt.double() @ lora[0].double(), mag + dt.double().abs() @ lora[0].double().abs()
        ops.backward_dx_with_dt(w, x, lora, dt, out=out[:, 8:8 + J])
        check(out[:, 8:8 + J], ref, mag, R + rank)
        assert bool((out[:, :8] == 7).all()) and bool((out[:, 8 + J:] == 7).all())
    else:
        dx = ops.backward_dx(w, x)[0]
    check(dx, ref, mag, R + rank)


# the dense counterpart (csrc/dense_gemm_pair.cu): the same widths, gated outputs in steps of 64, reductions that end inside a stage or a block
@pytest.mark.parametrize("M,J,R,rank", [(256, 256, 128, 0), (1000, 2560, 200, 0), (1000, 2560, 192, 16), (1000, 3200, 72, 0), (900, 3904, 64, 64),
                                        (1024, 4544, 1000, 0), (4800, 1024, 192, 0), (1000, 9664, 128, 0), (300, 1088, 328, 0)])
def test_dense_tile_widths(M, J, R, rank):
    g = torch.Generator(device="cuda").manual_seed(M + J)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, bias = rnd(M, R), rnd(J, R), rnd(J)
    z, mag = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    if rank:
        lora = (rnd(rank, R), rnd(J, rank), 0.5)
        y, t = ops.dense_forward(w, x, lora)
        check(y, z + t.double() @ lora[1].double().T, mag + t.double().abs() @ lora[1].double().abs().T, R + rank)
    else:
        out = torch.full((M, J + 16), 7.0, device="cuda", dtype=torch.bfloat16)
        S.linear(x, w, out=out[:, 8:8 + J])
        check(out[:, 8:8 + J], z, mag, R)
        assert bool((out[:, :8] == 7).all()) and bool((out[:, 8 + J:] == 7).all())
        check(S.linear(x, w, bias), z + bias.double(), mag + bias.double().abs(), R)
        y, r = S.linear(x, w, act=S.ACT_RELU2), z.clamp(min=0)
        assert bool(((y.double() - r * r).abs() <= 2.0 ** -8 * r * r + (2 * r + 1) * (R * 2.0 ** -24 * mag) + 1e-30).all())
        w2 = (w * R ** -0.5).bfloat16()
        z, mag = x.double() @ w2.double().T, x.double().abs() @ w2.double().abs().T
        ref = torch.nn.functional.gelu(z[:, 0::2], approximate="tanh") * z[:, 1::2]
        # |d gelu| <= 1.13; each of the two factors carries R 2^-24 times the row's magnitude, the fast exp and divide 2^-20 of the gate
        slack = R * 2.0 ** -24 * (1.13 * mag[:, 0::2] * z[:, 1::2].abs() + mag[:, 1::2] * z[:, 0::2].abs()) + 2.0 ** -20 * (z[:, 0::2] * z[:, 1::2]).abs() + 1e-7
        assert bool(((S.linear(x, w2, act=S.ACT_GLU_GELU).double() - ref).abs() <= 2.0 ** -8 * ref.abs() + slack).all())
    # reduction over the rows of the matrix
    if R % 64 == 0:
        wt = rnd(R, J)
        lora = (rnd(rank, J), rnd(R, rank), 0.5) if rank else None
        dx, dt = ops.dense_backward_dx(wt, x, lora)
        ref, mag = x.double() @ wt.double(), x.double().abs() @ wt.double().abs()
        if rank:
            ref, mag = ref + dt.double() @ lora[0].double(), mag + dt.double().abs() @ lora[0].double().abs()
        check(dx, ref, mag, R + rank)
