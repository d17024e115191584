"""The C-ABI library builds, loads and exports every symbol include/plz.h declares.
No compute call is made here (there is no GPU): only argument validation that returns before any launch."""
import ctypes as C
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    txt = open(os.path.join(ROOT, "include", "plz.h")).read()
    txt = re.sub(r"/\*.*?\*/", "", txt, flags=re.S)
    return sorted(set(re.findall(r"\b(plz_[a-z0-9_]+)\s*\(", txt)))


def test_library_exports_every_declared_symbol(built_lib):
    lib = C.CDLL(built_lib)
    names = declared_symbols()
    assert len(names) >= 14
    for n in names:
        assert hasattr(lib, n), f"{n} is declared in plz.h but missing from libplz.so"


def test_binding_covers_the_header(built_lib):
    import plz_native as P
    assert sorted(P.SIGNATURES) == declared_symbols()
    assert P.lib().plz_version() >= 100


def test_argument_validation_without_gpu(built_lib):
    import plz_native as P
    lib = P.lib()
    # empty problems are accepted, null pointers and bad shapes are refused with a message
    assert lib.plz_pack_indices(None, 1, 1, 0, 0, None, 0, None) == 0
    assert lib.plz_pack_indices(None, 1, 1, 4, 64, None, 16, None) == 7  # PLZ_ERR_NULL
    w = P.Weight(256, 100, 1, 64, 0x1000, 32, 0x2000)   # K not a multiple of 64
    assert lib.plz_hard_fwd(C.byref(w), 0x10, 100, 8, None, None, 0x20, 256, None) == 1
    assert b"multiple of 64" in lib.plz_last_error()
    w = P.Weight(256, 256, 1, 256, 0x1001, 64, 0x2000)  # misaligned packed rows
    assert lib.plz_hard_fwd(C.byref(w), 0x10, 256, 8, None, None, 0x20, 256, None) == 2
    w = P.Weight(256, 256, 1, 256, 0x1000, 64, 0x2000)
    assert lib.plz_hard_fwd(C.byref(w), 0x10, 256, 0, None, None, 0x20, 256, None) == 0  # M == 0: nothing to do
    assert lib.plz_hard_fwd_smallm(C.byref(w), 0x10, 256, 65, 0x20, 256, None) == 1       # M > 64
    lo = P.Lora(12, 1.0, 0x10, 256, 0x20, 12)                                              # rank not a multiple of 8
    assert lib.plz_hard_fwd(C.byref(w), 0x10, 256, 8, C.byref(lo), 0x30, 0x20, 256, None) == 1
    lo = P.Lora(16, 1.0, 0x10, 256, 0x20, 16)
    assert lib.plz_hard_fwd(C.byref(w), 0x10, 256, 8, C.byref(lo), None, 0x20, 256, None) == 5  # no workspace
    # buffers to clear: count, sizes, alignment
    two = lambda *v: (C.c_void_p * 2)(*v)
    assert lib.plz_zero(None, None, 0, None) == 0 and lib.plz_zero(None, None, 5, None) == 1 and lib.plz_zero(None, None, 2, None) == 7
    assert lib.plz_zero(two(0x1000, 0x2000), (C.c_int64 * 2)(64, 6), 2, None) == 1
    assert lib.plz_zero(two(0x1000, 0x2008), (C.c_int64 * 2)(64, 64), 2, None) == 2
    assert lib.plz_zero(two(0x1000, None), (C.c_int64 * 2)(64, 64), 2, None) == 7
    # rows of the result that overlap, at few rows and at many, from packed and dense weights
    for M in (8, 100, 300):
        assert lib.plz_hard_fwd(C.byref(w), 0x1000, 256, M, None, None, 0x2000, 248, None) == 1 and b"pitch" in lib.plz_last_error()
        assert lib.plz_dense_fwd(0x1000, 256, 256, 256, 0x1000, 256, M, None, None, 0x2000, 248, None) == 1
    # attention backward: o must be aligned to 8 bytes (its row sums read it so)
    ptr = [0x1000] * 16
    assert lib.plz_attn_bwd(ptr[0], 128, ptr[1], 128, ptr[2], 128, 0x1004, ptr[3], 128, ptr[4], 1, 128, 1, 1, 128, 1.0, *ptr[5:9], None) == 2


def test_decode_step_is_checked_before_its_first_launch(built_lib):
    import torch
    import plz_native as P
    import plz_ops as ops
    lib, h, f = P.lib(), 256, 512
    lin = lambda n, k: [n, k, 1, 256, 0x1000, k // 4, 0x2000]
    layer = sum([lin(512, h), lin(128, h), lin(128, h), lin(h, 512), lin(f, h), lin(f, h), lin(h, f)], []) + [0x3000] * 6

    def call(B=2, layers=(layer, layer), **kw):
        rows = sum(layers, [])
        a = dict(B=B, T=5, n_layers=len(layers), hidden=h, intermediate=f, n_heads=4, n_kv_heads=1, head_dim=128, batch_stride=1280, tok_stride=128, embed=0x4000, ld_embed=h, vocab=7,
                 ids=0x5000, cos_row=0x6000, sin_row=0x7000, final_norm=0x8000, h=0x9000, h1=0xa000, ws=0xb000, ws_bytes=1 << 40, eps=1e-6)
        return lib.plz_decode_hidden(C.byref(P.Decode(**{**a, **kw})), (C.c_int64 * len(rows))(*rows), None)
    assert call(B=65) == 1 and b"64" in lib.plz_last_error()
    assert call(layers=(layer, layer[:-1] + [0])) == 7 and b"cache" in lib.plz_last_error()      # of the second layer
    assert call(layers=(layer[:2] + [1 << 32] + layer[3:], layer)) == 1
    assert call(hidden=1 << 32) == 1 and call(n_heads=1 << 32) == 1
    assert call(cos_row=None) == 7 and call(ids=None) == 7
    assert call(B=0) == 0
    # the binding: types and sizes of what it passes as bare pointers
    bf, embed, cache = torch.bfloat16, torch.zeros(7, h, dtype=torch.bfloat16), torch.zeros(0, 2, 8, 128, dtype=torch.bfloat16)
    tab, norm = torch.zeros(1, 64), torch.zeros(h, dtype=bf)

    def bind(cos=tab, last=norm):
        ops.decode_hidden(torch.zeros(2, dtype=torch.int64), embed, [], (), (), cache, cache, 1, last, cos, tab, 4, 1, f, 1e-6)
    for kw in ({"cos": tab.double()}, {"cos": tab[:, :32]}, {"last": norm.float()}, {"last": norm[:8]}):
        with pytest.raises(AssertionError):
            bind(**kw)
    with pytest.raises(P.PlzError):
        bind()


def test_ops_refuse_cpu_tensors(built_lib):
    import torch
    import fused_lut_linear_cuda as F
    x = torch.zeros(4, 256, dtype=torch.bfloat16)
    pal = torch.zeros(1, 4, dtype=torch.bfloat16)
    idx = torch.zeros(256, 256, dtype=torch.int8)
    with pytest.raises(RuntimeError):
        F.fused_lut_linear(x, pal, idx, None, 256)


def test_hot_kernels_do_not_spill():
    """Register spills in the pipelined GEMM kernels cost 15-20 % (measured once); keep them at zero.
    (The eight-stage narrow variant for outputs of up to 64 columns with a bias may spill a few bytes in its epilogue.)"""
    import build
    build.build(force=True)
    rep = build.spill_report()
    # lut_gemm_kernel<MT, BMODE, NARROW=false, FUSE=0> mangles to ...ELb0ELi0EE...; the other product kernels all count
    names = {"tn_gemm_kernel": 12, "lut_smallm_mma": 2, "lut_gemv_rows": 3, "lut_gemm_pair_kernel": 2, "dense_gemm_pair_kernel": 3, "narrow_gemm_kernel": 2, "turned_gemm_kernel": 3}
    hot = {k: v for k, v in rep.items() if ("lut_gemm_kernel" in k and "ELb0ELi0EE" in k) or any(n in k for n in names)}
    for n, least in names.items():
        assert sum(n in k for k in hot) >= least, n
    assert sum("lut_gemm_kernel" in k for k in hot) >= 7
    # decode attention holds a step of keys and values in 128 registers, four CTAs per SM: a few words of addresses may spill, no more
    assert all(v[0] <= 32 and v[1] <= 32 for k, v in rep.items() if "attn_decode_mma_kernel" in k)
    bad = {k: v for k, v in hot.items() if v[0] or v[1]}
    assert not bad, bad
