"""The native call module without a GPU: it loads, and declines tensors that are not on one, wrong types and wrong counts."""
import torch


def test_declines_what_it_does_not_take(built_lib):
    import plz_native as P
    c = P.calls()
    packed, pal, x = torch.zeros(8, 64, dtype=torch.uint8), torch.zeros(8, 4, dtype=torch.bfloat16), torch.zeros(2, 256, dtype=torch.bfloat16)
    w = (packed, pal, 8, 256, 1, 256)
    for args in ((c.hard_forward, *w, x), (c.hard_forward_smallm, *w, x), (c.hard_forward_bias, *w, x, None), (c.backward_dx, *w, x), (c.backward_dw_hard, *w, x, x),
                 (c.col_sum, x), (c.select_indices, *w, x, False, None, 1.0), (c.backward_dw_soft, *w, x, x, x, False, None, 1.0, 0, True, True),
                 (c.eval_linear, *w, x, None, None, 1.0)):
        f, rest = args[0], args[1:]
        assert f(*rest) is None
        assert f() is None and f(*(None for _ in rest)) is None and f(*(7 for _ in rest)) is None and f(*rest, 1) is None
        assert f(*(2 ** 80 for _ in rest)) is None


def test_host_numbers_are_not_frozen_into_a_graph(built_lib, monkeypatch):
    """While the stream is captured, numbers from the host go by the copy, which a capture refuses; a launch would replay these ones for good."""
    import plz_native as P
    import seq_ops as S

    def no_launch():
        raise AssertionError("launched")
    monkeypatch.setattr(P, "lib", no_launch)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    dst, v = torch.zeros(3, dtype=torch.int64), torch.arange(3)
    S.put(dst, v)
    assert torch.equal(dst, v) and torch.equal(S.on_device(v, "cpu"), v)


def test_module_is_rebuilt_for_another_torch_or_python(built_lib, monkeypatch):
    import sysconfig

    import build
    assert not build._calls_stale()
    with monkeypatch.context() as m:
        m.setattr(build.importlib.metadata, "version", lambda name: "0.0")
        assert build._calls_stale()
    with monkeypatch.context() as m:
        m.setattr(sysconfig, "get_config_var", lambda name: "cpython-00")
        assert build._calls_stale()
    assert not build._calls_stale()
