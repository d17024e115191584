"""Operations as one native call (csrc/torch_calls.cpp) against the general path through ctypes: the same bits for what both take, the same errors for what neither takes."""
import threading

import pytest
import torch

import fused_lut_linear_cuda as F
import palettized_linear as PL
import plz_native as P
import plz_ops as ops

pytestmark = pytest.mark.gpu


class _Never:
    def __getattr__(self, name):
        return lambda *a: None


@pytest.fixture
def general(monkeypatch):
    """Runs a function with every native call declining."""
    def run(f):
        with monkeypatch.context() as m:
            m.setattr(P, "calls", lambda: _Never())
            return f()
    return run


def _rnd(g, *s):
    return torch.randn(*s, generator=g, device="cuda").bfloat16()


def _weight(g, N, K, gs_n, gs_k):
    idx = torch.randint(0, 4, (N, K), generator=g, device="cuda", dtype=torch.int8)
    return ops.PackedWeight(ops.pack_indices(idx, n_major=True), _rnd(g, (N // gs_n) * (K // gs_k), 4), N, K, gs_n, gs_k)


# rows of the small kernels (whose sums meet in any order: one row per reduction group is exact at K = 256), of the few-row and of the large products; pitched rows
@pytest.mark.parametrize("M,pad", [(1, 0), (64, 8), (200, 0), (300, 16)])
@pytest.mark.parametrize("gs_n", [1, 256])
def test_same_bits(M, pad, gs_n, general):
    g = torch.Generator(device="cuda").manual_seed(M + gs_n)
    N, K = 512, 256
    w = _weight(g, N, K, gs_n, 256)
    x, dy, bias = _rnd(g, M, K + pad)[:, :K], _rnd(g, M, N + pad)[:, :N], _rnd(g, N)
    lg = torch.randn(N, K, 4, generator=g, device="cuda")
    planar = lg.permute(2, 1, 0).contiguous().half()
    noise = torch.randn(N, K, 4, generator=g, device="cuda")
    w2 = ops.PackedWeight(torch.zeros_like(w.packed), w.palette, N, K, gs_n, 256)
    calls = [lambda: ops.hard_forward(w, x)[0], lambda: ops.hard_forward_bias(w, x, bias), lambda: ops.hard_forward_bias(w, x, None), lambda: ops.backward_dx(w, dy)[0],
             lambda: ops.backward_dw_hard(w, x, dy), lambda: ops.col_sum(dy)]
    if M <= 64:
        calls.append(lambda: ops.hard_forward_smallm(w, x))
    for layout, t, z in (("nk4", lg, noise), ("4kn", planar, noise.permute(2, 1, 0).contiguous())):
        for nz in (None, "hash", z):
            calls.append(lambda layout=layout, t=t, nz=nz: ops.backward_dw_soft(w, x, dy, t, layout, noise=nz, tau=0.7, seed=9))
        calls.append(lambda layout=layout, t=t: (ops.soft_select(w2, t, layout, noise=z if layout == "4kn" else None), w2.packed.clone())[1])
    for i, f in enumerate(calls):
        got, want = f(), general(f)
        for a, b in zip(got if isinstance(got, tuple) else (got,), want if isinstance(want, tuple) else (want,)):
            assert a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride(), i
            # sums that atomics add up may round in another order
            assert torch.equal(a, b) or (a.dtype == torch.float32 and (a - b).abs().max() <= 1e-5 * b.abs().max()), i


@pytest.mark.parametrize("rank", [0, 16])
@pytest.mark.parametrize("shape", [(256,), (3, 256), (2, 40, 256), (300, 256)])
def test_eval_linear(rank, shape, general):
    g = torch.Generator(device="cuda").manual_seed(rank + len(shape))
    m = PL.PalettizedLinear(256, 512, rank=rank, lora_scale=2.0)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, generator=g, device="cuda"))
    m.extract_hard_indices()
    m.eval()
    x = _rnd(g, *shape)
    for z in (x, x.requires_grad_(True), torch.stack([x.detach()] * 2, -1)[..., 0]):
        a, b = m(z), general(lambda: m(z))
        assert torch.equal(a, b) and a.shape == b.shape and a.requires_grad == b.requires_grad


def test_what_is_refused(general):
    g = torch.Generator(device="cuda").manual_seed(1)
    w = _weight(g, 512, 256, 1, 256)
    x = _rnd(g, 80, 256)
    flat = ops.PackedWeight(w.packed.view(-1), w.palette, 512, 256, 1, 256)
    lg = torch.randn(512, 256, 4, device="cuda")
    bad = [lambda: ops.hard_forward(w, x.float()), lambda: ops.hard_forward(w, x[:, :128]), lambda: ops.hard_forward(w, x.t()), lambda: ops.hard_forward(w, x.cpu()),
           lambda: ops.hard_forward(flat, x), lambda: ops.hard_forward_smallm(w, x), lambda: ops.hard_forward_bias(w, x, torch.zeros(512, device="cuda")),
           lambda: ops.backward_dx(w, x), lambda: ops.backward_dw_hard(w, x, x), lambda: ops.col_sum(x.float()),
           lambda: ops.soft_select(w, lg, "nk4", tau=0.0), lambda: ops.soft_select(w, lg.double(), "nk4"), lambda: ops.soft_select(w, lg, "nk4", noise=lg.half()),
           lambda: ops.backward_dw_soft(w, x, _rnd(g, 80, 512), lg, "nk4", tau=-1.0)]
    m = PL.PalettizedLinear(256, 512, rank=8).eval()
    m.lora_A, m.lora_B = torch.nn.Parameter(m.lora_A.detach()[:0]), torch.nn.Parameter(m.lora_B.detach()[:, :0])
    bad.append(lambda: m(x[:4]))                # LoRA factors of rank 0
    for i, f in enumerate(bad):
        with pytest.raises(Exception) as a:
            f()
        with pytest.raises(Exception) as b:
            general(f)
        assert type(a.value) is type(b.value) and str(a.value) == str(b.value), i


# tensors without memory: what a transform hands to the function that it works on
@pytest.mark.parametrize("transform", [lambda f, x: torch.vmap(f)(torch.stack([x, x])), lambda f, x: torch.func.jvp(f, (x,), (torch.ones_like(x),)),
                                       lambda f, x: torch.func.grad(lambda z: f(z).float().sum())(x)], ids=["vmap", "jvp", "grad"])
def test_transforms_are_refused(transform, general):
    g = torch.Generator(device="cuda").manual_seed(3)
    w, w2 = _weight(g, 256, 256, 1, 256), _weight(g, 256, 256, 1, 256)
    lg = torch.randn(256, 256, 4, generator=g, device="cuda")
    plain, lora = (PL.PalettizedLinear(256, 256, rank=r).eval() for r in (0, 16))
    d = _rnd(g, 80, 256)
    fs = [lambda z: ops.hard_forward(w, z)[0], lambda z: ops.hard_forward_smallm(w, z), lambda z: ops.hard_forward_bias(w, z, None), lambda z: ops.hard_forward_bias(w, d, z[0]),
          lambda z: ops.backward_dx(w, z)[0], lambda z: ops.backward_dw_hard(w, z, d), lambda z: ops.backward_dw_hard(w, d, z), ops.col_sum,
          lambda z: ops.soft_select(w2, z.float()[:, :, None].expand(-1, -1, 4), "nk4"), lambda z: ops.backward_dw_soft(w, z, d, lg, "nk4")[0], plain, lora]
    for i, f in enumerate(fs):
        with pytest.raises(Exception) as a:
            transform(f, d)
        with pytest.raises(Exception) as b:
            general(lambda: transform(f, d))
        assert type(a.value) is type(b.value) and str(a.value) == str(b.value), i


def test_own_stream_thread_and_subclass(general):
    g = torch.Generator(device="cuda").manual_seed(2)
    w = _weight(g, 512, 256, 1, 256)
    x = _rnd(g, 200, 256)
    want = general(lambda: ops.hard_forward(w, x)[0])
    got = []

    def work():
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            assert P.stream_ptr() == s.cuda_stream
            torch.cuda._sleep(2000000)
            z = x * 1
            got.append(ops.hard_forward(w, z)[0])
        s.synchronize()
    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert torch.equal(got[0], want)

    class Sub(torch.Tensor):
        pass
    assert torch.equal(ops.hard_forward(w, x.as_subclass(Sub))[0], want)
    gr = torch.cuda.CUDAGraph()
    with torch.cuda.graph(gr):
        y = ops.hard_forward(w, x)[0]
    gr.replay()
    assert torch.equal(y, want)


def test_functions_under_autograd(general):
    g = torch.Generator(device="cuda").manual_seed(4)
    M, N, K = 300, 512, 256
    idx = torch.randint(0, 4, (K, N), generator=g, device="cuda", dtype=torch.int8)
    lg = torch.randn(4, K, N, generator=g, device="cuda").half()
    noise = torch.randn(4, K, N, generator=g, device="cuda")
    leaves = [_rnd(g, M, K), _rnd(g, N // 256, 4), _rnd(g, N)]
    dy = _rnd(g, M, N)

    def run():
        x, pal, b = (t.clone().requires_grad_(True) for t in leaves)
        y = F.fused_lut_linear(x, pal, idx, b, 256)
        soft = lg.clone().requires_grad_(True)
        z = F.fused_lut_linear_soft(x, pal, soft, b, 256, 1.0, noise=noise)
        return [y, z, *torch.autograd.grad(y, [x, pal, b], dy), *torch.autograd.grad(z, [x, pal, soft, b], dy)]
    for a, b in zip(run(), general(run)):
        assert a.dtype == b.dtype and (torch.equal(a, b) or (a.float() - b.float()).abs().max() <= 2.0 ** -7 * b.float().abs().max())
