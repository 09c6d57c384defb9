"""The tcgen05 attention of prompts gives the same bits each time: no row's result is read before its
last product, however far one warp of a tile runs ahead of another."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class Batch:
    def __init__(self, counts):
        row0 = [0]
        for c in counts:
            row0.append(row0[-1] + c)
        i32 = lambda v: torch.tensor(list(v), dtype=torch.int32, device=DEV)  # noqa: E731
        self.seq_slot, self.seq_start = i32(range(len(counts))), i32([0] * len(counts))
        self.seq_new, self.seq_row0 = i32(counts), i32(row0)
        self.max_new, self.max_context, self.is_decode = max(counts), max(counts), False


@pytest.mark.parametrize("weights", ["sigmoid", "softmax"])
@pytest.mark.parametrize("nq,nkv,d,window", [(16, 4, 128, 1024), (32, 32, 64, None)])
def test_the_same_bits_each_time(nq, nkv, d, window, weights):
    from reflex_b200 import ops

    counts = (2048, 65, 1000)
    g = torch.Generator(device=DEV).manual_seed(nq + d)
    batch, pages = Batch(counts), 32
    table = torch.arange(3 * pages, device=DEV, dtype=torch.int32).view(3, pages)
    k, v = (torch.randn((3 * pages, nkv, 64, d), generator=g, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn((sum(counts), nq * d), generator=g, device=DEV).bfloat16()
    bias = torch.full((nq,), -4.0, device=DEV)

    def once():
        if weights == "sigmoid":
            return ops.attention_sigmoid(q, k, v, table, 64, batch, nq, nkv, d, d, window, d ** -0.5, bias)
        return ops.attention(q, k, v, table, 64, batch, nq, nkv, d, window, d ** -0.5)

    first = once().clone()
    assert all(torch.equal(once(), first) for _ in range(100))
