"""Token ids and row numbers that reach the device as kernel arguments: every count around a launch's 256, forms that go by a copy, and order behind queued work."""
import pytest
import torch

import seq_ops as S
from helpers import check_status

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1000, 4096, 4097])
def test_numbers_arrive(n):
    t = torch.randint(-2 ** 62, 2 ** 62, (n,), generator=torch.Generator().manual_seed(n))
    assert torch.equal(S.on_device(t, "cuda").cpu(), t)
    dst = torch.zeros(n + 2, dtype=torch.int64, device="cuda")
    S.put(dst[1:-1], t)
    assert torch.equal(dst.cpu(), torch.cat([torch.zeros(1, dtype=torch.int64), t, torch.zeros(1, dtype=torch.int64)]))
    check_status()


def test_other_forms():
    t = torch.arange(24).view(4, 6)
    for z in (t[:, ::2], t.t(), t.cuda(), t.int(), torch.empty(0, dtype=torch.int64), torch.tensor(5)):
        got = S.on_device(z, "cuda")
        assert got.is_cuda and got.dtype == z.dtype and torch.equal(got.cpu(), z.cpu())
    buf = torch.zeros(4, 1, dtype=torch.int64, device="cuda")
    for z in (torch.arange(4).view(4, 1), torch.arange(4, dtype=torch.int32).view(4, 1), torch.arange(4, device="cuda").view(4, 1), torch.tensor(7)):
        S.put(buf, z)
        assert torch.equal(buf.cpu(), z.cpu().long().expand(4, 1))


def test_in_the_order_of_the_stream():
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        buf = torch.zeros(3, dtype=torch.int64, device="cuda")
        seen = []
        for i in range(50):
            if i % 10 == 0:
                torch.cuda._sleep(1000000)
            v = torch.full((3,), i)
            S.put(buf, v)
            v.fill_(-1)                  # the host's tensor is free again at once
            seen.append(buf.clone())
    s.synchronize()
    assert torch.equal(torch.stack(seen).cpu(), torch.arange(50)[:, None].expand(50, 3))
