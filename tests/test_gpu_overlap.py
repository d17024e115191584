"""plz_set_smallm_overlap on: which launches may start under the kernel before them. Only the entry points of a token step read their weights that early; the
general products take matrices that the kernel right before may just have written."""
import ctypes as C
from contextlib import contextmanager

import pytest
import torch

import plz_native as P
import plz_ops as ops
import seq_ops as S

pytestmark = pytest.mark.gpu
N, K, R = 256, 512, 16


@contextmanager
def overlap():
    P.lib().plz_set_smallm_overlap(1)
    try:
        yield
    finally:
        P.lib().plz_set_smallm_overlap(0)


def _rnd(g, *s, scale=1.0):
    return (torch.randn(*s, generator=g, device="cuda") * scale).bfloat16()


def _given(M):
    g = torch.Generator(device="cuda").manual_seed(M)
    idx = torch.randint(0, 4, (N, K), generator=g, device="cuda", dtype=torch.int8)
    w = ops.PackedWeight(ops.pack_indices(idx, n_major=True), _rnd(g, N * K // 256, 4, scale=0.02).view(-1), N, K, 1, 256)
    return w, _rnd(g, M, K), _rnd(g, N, K, scale=0.02), (_rnd(g, R, K, scale=0.02), _rnd(g, N, R, scale=0.02), 2.0), _rnd(g, N)


def _early_launches(call):
    """Programmatic edges of a captured chain of a row-wise kernel and `call` (nothing runs)."""
    x, w = torch.ones(3, 256, device="cuda"), torch.ones(256, device="cuda")
    call(), torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with overlap(), torch.cuda.graph(graph):
        S.rows_norm(x, None, w, 0.0, 1e-6, torch.bfloat16)
        keep = call()
    fn = C.CDLL("libcudart.so.12").cudaGraphGetEdges_v2
    fn.argtypes = [C.c_void_p] * 5
    n = C.c_size_t(0)
    assert fn(graph.raw_cuda_graph(), None, None, None, C.byref(n)) == 0
    a, b, data = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (C.c_uint8 * (8 * n.value))()
    assert fn(graph.raw_cuda_graph(), a, b, data, C.byref(n)) == 0
    del keep
    return sum(data[8 * i + 2] == 1 for i in range(n.value))


@pytest.mark.parametrize("M", [1, 17, 64, 128])
def test_general_products_wait(M):
    w, x, W, lora, bias = _given(M)
    for call in (lambda: ops.hard_forward(w, x), lambda: ops.hard_forward(w, x, lora), lambda: ops.hard_forward_bias(w, x, bias),
                 lambda: ops.dense_forward(W, x), lambda: ops.dense_forward(W, x, lora), lambda: ops.lora_dt(lora, x[:, :N])):
        assert _early_launches(call) == 0
    if 1 < M <= 64:                          # the check sees such launches where there are some
        assert _early_launches(lambda: ops.hard_forward_smallm(w, x)) >= 1
        assert _early_launches(lambda: S.linear(x, W)) >= 1


@pytest.mark.parametrize("M", [17, 64, 128])
def test_matrix_of_the_kernel_before(M):
    """The matrix of a dense product is the output of another product of few rows, in a buffer that comes round with other contents."""
    g = torch.Generator(device="cuda").manual_seed(5)
    xs, a = [_rnd(g, M, K) for _ in range(16)], _rnd(g, K, K, scale=K ** -0.5)
    x = _rnd(g, M, K)
    buf = torch.empty(M, K, dtype=torch.bfloat16, device="cuda")[: M // 8 * 8]

    def run():
        out = []
        for v in xs:
            S.linear(v[: M // 8 * 8], a, out=buf)
            out.append(ops.dense_forward(buf, x)[0])
        torch.cuda.synchronize()
        return out
    want = run()
    with overlap():
        got = run()
    P.device_status()
    assert all(torch.equal(p, q) for p, q in zip(want, got))


def test_slow_kernel_before():
    """A launch that starts early does not count the time of a kernel ahead of it, here one block that runs for two and a half seconds, against its
    bounded waits (2 s)."""
    slow = torch.ones(64, 40 << 20, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(6)
    x, W = _rnd(g, 32, K), _rnd(g, 4096, K, scale=0.02)
    want = S.linear(x, W)
    with overlap():
        S.linear(slow, slow)
        got = S.linear(x, W)
    P.device_status()
    assert torch.equal(want, got)
