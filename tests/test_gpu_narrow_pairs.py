"""Packed products of few rows walk the reduction in pairs of 64-column blocks: odd and even numbers of blocks, a single one, the LoRA block as the second or
the first of the last pair, more pairs than slots, all paddings of the rows."""
import pytest
import torch

import plz_native as P
import plz_ops as ops
from helpers import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [3, 17, 33, 64, 128])
@pytest.mark.parametrize("blocks", [1, 2, 3, 5, 6, 7, 12, 29, 40])
@pytest.mark.parametrize("N,rank", [(136, 0), (136, 16), (2560, 16)])
def test_pairs_of_blocks(M, blocks, N, rank):
    K, g = 64 * blocks, torch.Generator(device="cuda").manual_seed(1000 * M + blocks)
    r = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device="cuda") * scale).bfloat16()
    idx = torch.randint(0, 4, (N, K), generator=g, device="cuda", dtype=torch.int8)
    w = ops.PackedWeight(ops.pack_indices(idx, n_major=True), r(N * blocks, 4).view(-1), N, K, 1, 64)
    x = r(M, K)
    lora = (r(rank, K, scale=K ** -0.5), r(N, rank), 2.0) if rank else None
    W = w.palette.view(N, blocks, 4).double().gather(2, idx.view(N, blocks, 64).long()).view(N, K)
    want = x.double() @ W.t()
    if rank:
        y, t = ops.hard_forward(w, x, lora)
        want = want + t.double() @ lora[1].double().t()
    else:
        y = ops.hard_forward_smallm(w, x) if M <= 64 else ops.hard_forward(w, x)[0]
    P.device_status()
    assert_close(y, want.float(), "y")
