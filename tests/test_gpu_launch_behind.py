"""Launches that start under the end of the kernel before: products, attention and row-wise kernels of prompts and training steps. None of them touches memory
ahead of its wait, so a chain through buffers that come round gives the bits of the same calls one at a time, a slow kernel ahead does not count against
their bounded waits, and a capture without the token chain's switch holds plain edges only."""
import ctypes as C

import pytest
import torch

import plz_native as P
import plz_ops as ops
import seq_ops as S

pytestmark = pytest.mark.gpu
H, HEADS, KV, D = 512, 4, 2, 128


def _given(M):
    g = torch.Generator(device="cuda").manual_seed(M)
    r = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device="cuda") * scale).bfloat16()
    idx = torch.randint(0, 4, (H, H), generator=g, device="cuda", dtype=torch.int8)
    w = ops.PackedWeight(ops.pack_indices(idx, n_major=True), r(H * H // 256, 4, scale=0.05).view(-1), H, H, 1, 256)
    lora = (r(16, H, scale=0.05), r(H, 16, scale=0.05), 2.0)
    return w, lora, r(H, H, scale=0.05), r(H), [r(M, H) for _ in range(6)]


def _chain(B, n, given, x, step):
    w, lora, wd, gain, _ = given
    done = lambda v: (step(), v)[1]
    h, rstd = done(ops.rmsnorm_forward(x, gain))
    q = done(ops.hard_forward(w, h, lora)[0])
    k = done(ops.dense_forward(wd, h, lora)[0])
    k, v = k[:, :KV * D].contiguous(), k[:, KV * D:].contiguous()
    o, lse = done(ops.attention_forward(q, k, v, B, n, HEADS, KV))
    act = done(ops.swiglu_forward(o, q))
    do = done(ops.add(act, x))
    dq, dk, dv = done(ops.attention_backward(q, k, v, o, do, lse, B, n, HEADS, KV))
    dx = done(ops.backward_dx(w, dq, lora)[0])
    dl = done(ops.backward_dw_hard(w, x, dx))
    dh, _ = done(ops.rmsnorm_backward(x, dx, rstd, gain))
    return [t.clone() for t in (o, dq, dk, dv, dx, dl, dh)]


@pytest.mark.parametrize("B,n", [(1, 128), (2, 256), (4, 640)])
def test_chain_has_the_bits_of_single_calls(B, n):
    given = _given(B * n)
    want = [_chain(B, n, given, x, torch.cuda.synchronize) for x in given[-1]]
    for _ in range(3):
        got = [_chain(B, n, given, x, lambda: None) for x in given[-1]]
        assert all(torch.equal(a, b) for p, q in zip(want, got) for a, b in zip(p[:5] + p[6:], q[:5] + q[6:]))
        assert all((p[5] - q[5]).abs().max() <= 1e-4 * p[5].abs().max() for p, q in zip(want, got))      # sums of 2^16 or fewer fp32 parts in any order
    P.device_status()


def test_slow_kernel_ahead():
    """One block that runs for two and a half seconds, longer than the bounded waits, ahead of every such launch."""
    slow = torch.ones(64, 40 << 20, device="cuda")
    w, lora, wd, gain, (x, y, *_) = _given(256)
    k = x[:, :KV * D].contiguous()
    o, lse = ops.attention_forward(y, k, k, 1, 256, HEADS, KV)
    calls = [lambda: ops.hard_forward(w, x, lora)[0], lambda: ops.dense_forward(wd, x)[0], lambda: ops.attention_forward(y, k, k, 1, 256, HEADS, KV)[0],
             lambda: ops.attention_backward(y, k, k, o, x, lse, 1, 256, HEADS, KV)[0], lambda: ops.weight_grad(x, y)]
    want = [c() for c in calls]
    for c, v in zip(calls, want):
        S.linear(slow, slow)
        assert (c().float() - v.float()).abs().max() <= 1e-5 * v.abs().max()       # the last: fp32 parts in any order
    P.device_status()


def test_captured_chain_has_plain_edges():
    given = _given(256)
    x = given[-1][0]
    run = lambda: ops.dense_forward(given[2], ops.hard_forward(given[0], ops.rmsnorm_forward(x, given[3])[0])[0])[0]
    want, graph = run(), torch.cuda.CUDAGraph(keep_graph=True)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        got = run()
    fn, n = C.CDLL("libcudart.so.12").cudaGraphGetEdges_v2, C.c_size_t(0)
    fn.argtypes = [C.c_void_p] * 5
    assert fn(graph.raw_cuda_graph(), None, None, None, C.byref(n)) == 0 and n.value >= 2
    a, b, data = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (C.c_uint8 * (8 * n.value))()
    assert fn(graph.raw_cuda_graph(), a, b, data, C.byref(n)) == 0
    assert all(data[8 * i + 2] == 0 for i in range(n.value))
    graph.instantiate()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


# products outside the token chain (few rows; at most 64 columns, walked by tiles or in clusters) do not let a kernel of the chain, which reads its matrix ahead of the wait, start
# before they have finished
@pytest.mark.parametrize("M,N", [(128, 1024), (64, 4096), (2048, 64), (16384, 32), (96, 16)])
def test_a_product_as_the_next_ones_matrix(M, N):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, wd, z = [r(M, 2560) for _ in range(4)], r(N, 2560), r(2, N)
    want = [S.linear(z, ops.dense_forward(wd, v)[0]) for v in x]
    torch.cuda.synchronize()
    P.lib().plz_set_smallm_overlap(1)
    try:
        got = [S.linear(z, ops.dense_forward(wd, v)[0]) for _ in range(5) for v in x]
    finally:
        P.lib().plz_set_smallm_overlap(0)
    P.device_status()
    assert all(torch.equal(a, b) for a, b in zip(got, want * 5))
