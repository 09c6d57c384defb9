"""The faster forms of the true 32-bit kernels give the plain forms' bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from reflex_b200 import ops as o

    return o


def i32(v):
    return torch.tensor(list(v), dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("N,K", [(31, 64), (33, 68), (130, 4), (64, 132), (300, 2052), (4100, 96), (4801, 132)])
@pytest.mark.parametrize("R", [1, 2, 3, 4, 7, 8, 9, 16, 32, 33, 63, 64, 65, 129, 300, 2100])
def test_every_form_of_the_product_gives_the_same_bits(R, N, K):
    """Rows of a matrix whose start is off 16 bytes take the general form, one thread an element."""
    g = torch.Generator(device=DEV).manual_seed(R + N + K)
    x = torch.randn((R, K), generator=g, device=DEV)
    w = torch.randn((N, K), generator=g, device=DEV)
    apart = torch.empty(N * K + 1, device=DEV)[1:].view(N, K).copy_(w)
    assert apart.data_ptr() % 16 and apart.is_contiguous()
    y, plain = ops().linear(x, w), ops().linear(x, apart)
    assert torch.equal(y, plain)
    ref = x.double() @ w.double().t()
    assert ((y - ref).abs().max() / ref.abs().max()).item() < 5e-7 * K ** 0.5


def test_more_rows_than_a_grid_of_small_tiles_has():
    R, N, K = 32 * 65535 + 33, 4, 4
    x = torch.randn((R, K), generator=torch.Generator(device=DEV).manual_seed(1), device=DEV)
    w = torch.randn((N, K), generator=torch.Generator(device=DEV).manual_seed(2), device=DEV)
    apart = torch.empty(N * K + 1, device=DEV)[1:].view(N, K).copy_(w)
    assert torch.equal(ops().linear(x, w), ops().linear(x, apart))


class Batch:
    def __init__(self, counts, starts, slots):
        row0 = [0]
        for c in counts:
            row0.append(row0[-1] + c)
        self.seq_slot, self.seq_start, self.seq_new, self.seq_row0 = i32(slots), i32(starts), i32(counts), i32(row0)
        self.row_pos = i32([s + j for s, c in zip(starts, counts) for j in range(c)])
        self.row_slot = i32([sl for sl, c in zip(slots, counts) for _ in range(c)])
        self.max_new = max(counts)
        self.is_decode = all(c == 1 for c in counts)


@pytest.mark.parametrize("d", [32, 64, 128, 256])
@pytest.mark.parametrize("nq,nkv", [(4, 1), (6, 6), (40, 2)])
@pytest.mark.parametrize("window,keep_first,extras", [(None, 0, False), (33, 0, True), (40, 5, False), (70, 130, True)])
def test_attention_bits_are_the_plain_kernels(d, nq, nkv, window, keep_first, extras):
    """Prompts, a chunk of one and single rows over a shuffled page table; windows, kept first
    positions, sinks, slopes and a cap; pages beyond a sequence's end hold NaN."""
    g = torch.Generator(device=DEV).manual_seed(d + nq)
    counts, starts, slots = (70, 1, 33, 1), (0, 200, 129, 31), (2, 0, 3, 1)
    pages = 4 * 5
    k = torch.full((pages, nkv, 64, d), float("nan"), device=DEV)
    v = k.clone()
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).view(4, 5)
    for s, c, slot in zip(starts, counts, slots):
        for p in range(s + c):
            k[table[slot, p // 64], :, p % 64] = torch.randn((nkv, d), generator=g, device=DEV)
            v[table[slot, p // 64], :, p % 64] = torch.randn((nkv, d), generator=g, device=DEV)
    q = torch.randn((sum(counts), nq * d), generator=g, device=DEV)
    sink = torch.randn(nq, generator=g, device=DEV) if extras else None
    slopes = torch.rand(nq, generator=g, device=DEV) * 0.1 if extras else None
    b, cap, t = Batch(counts, starts, slots), 20.0 if extras else 0.0, table.to(torch.int32).to(DEV)
    got = ops().attention(q, k, v, t, 64, b, nq, nkv, d, window, d ** -0.5, sink, slopes, keep_first, cap)
    ref = ops().attention_plain(q, k, v, t, 64, b.row_pos, b.row_slot, nq, nkv, d, window, d ** -0.5, sink, slopes,
                                keep_first, cap)
    assert torch.isfinite(ref).all()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("page", [16, 32, 48, 96])  # 16 and 48: a tile of 32 keys lies in several pages
def test_attention_bits_with_pages_of_other_sizes(page):
    g = torch.Generator(device=DEV).manual_seed(page)
    nq, nkv, d, counts, starts, slots = 4, 2, 64, (70, 1, 33), (0, 100, 45), (2, 0, 1)
    per = 112 // page + 2
    k, v = (torch.randn((3 * per, nkv, page, d), generator=g, device=DEV) for _ in range(2))
    t = torch.randperm(3 * per, generator=torch.Generator().manual_seed(1)).view(3, per).to(torch.int32).to(DEV)
    q, b = torch.randn((sum(counts), nq * d), generator=g, device=DEV), Batch(counts, starts, slots)
    got = ops().attention_f32(q, k, v, t, page, b, nq, nkv, d, None, d ** -0.5)
    ref = ops().attention_plain(q, k, v, t, page, b.row_pos, b.row_slot, nq, nkv, d, None, d ** -0.5)
    assert torch.equal(got, ref)


@pytest.mark.parametrize("counts,starts", [((300, 40), (0, 0)), ((600,), (0,)), ((33, 65), (70, 0))])
@pytest.mark.parametrize("d", [32, 128, 256])
def test_attention_bits_with_one_block_an_sm_and_two(counts, starts, d):
    """The host's lengths decide how many blocks share an SM; a batch that does not say has two."""
    g = torch.Generator(device=DEV).manual_seed(d)
    nq, nkv, n = 8, 2, len(counts)
    per = max(s + c for s, c in zip(starts, counts)) // 64 + 1
    k, v = (torch.randn((n * per, nkv, 64, d), generator=g, device=DEV) for _ in range(2))
    t = torch.arange(n * per, dtype=torch.int32, device=DEV).view(n, per)
    q, b, got = torch.randn((sum(counts), nq * d), generator=g, device=DEV), Batch(counts, starts, range(n)), []
    for _ in range(2):
        got.append(ops().attention_f32(q, k, v, t, 64, b, nq, nkv, d, None, d ** -0.5))
        b.new_counts, b.starts = list(counts), list(starts)
    assert 0 < ops()._longest_blocks(b, nq, nkv, None)
    assert torch.equal(*got)
