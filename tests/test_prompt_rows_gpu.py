"""The elementwise kernels of prompts that take several rows, or several small parts, a thread: the same bits as the
forms for few rows, at the edges of their groups of rows and across sequences."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
COUNTS = (1, 2, 7, 8, 9, 100, 3, 131)  # 261 rows: the last group of four rows has one


def ops():
    from reflex_b200 import ops as o

    return o


def i32(v):
    return torch.tensor(list(v), dtype=torch.int32, device=DEV)


class Batch:
    def __init__(self, counts, slots):
        self.row_slot = i32([s for s, c in zip(slots, counts) for _ in range(c)])
        self.seq_slot, self.seq_new = i32(slots), i32(counts)


def piecewise(fn, counts):
    """fn(rows, batch) a sequence at a time: too few rows for the form under test."""
    out, r0 = [], 0
    for i, c in enumerate(counts):
        out.append(fn(slice(r0, r0 + c), Batch([c], [len(counts) - 1 - i])))
        r0 += c
    return [torch.cat(t) for t in zip(*out)]


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("channels,col0,ld,biases,act", [(1028, 4, 1040, True, "silu"), (12, 0, 16, False, None)])
def test_short_convolutions_of_several_rows(taps, channels, col0, ld, biases, act):
    g = torch.Generator(device=DEV).manual_seed(taps)
    R = lambda *s: torch.randn(s, generator=g, device=DEV)  # noqa: E731
    n = sum(COUNTS)
    proj, w, state = R(n, ld), R(taps, channels), R(len(COUNTS), (taps - 1) * channels + 4)
    b, cb = (R(channels), R(channels)) if biases else (None, None)

    def run(rows, batch):
        return ops().short_conv(proj[rows], col0, channels, b, w, cb, state, batch, also_bf16=True, activation=act)

    whole = run(slice(0, n), Batch(COUNTS, range(len(COUNTS) - 1, -1, -1)))
    for x, y in zip(whole, piecewise(run, COUNTS)):
        assert torch.equal(x, y)


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 2, 128, 128), (3, 1, 20, 36)])
@pytest.mark.parametrize("exact", [True, False])
def test_gated_delta_rows_of_prompts(taps, heads, kv_heads, dim, vdim, exact):
    g = torch.Generator(device=DEV).manual_seed(taps)
    R = lambda *s: torch.randn(s, generator=g, device=DEV)  # noqa: E731
    n, C = sum(COUNTS), 2 * kv_heads * dim + heads * vdim
    ld = C + 2 * heads + (-2 * heads) % 4
    proj, w, state = R(n, ld), R(taps, C), R(len(COUNTS), (taps - 1) * C + 8)
    bias, A = R(heads), -torch.rand(heads, generator=g, device=DEV)

    def run(rows, batch):
        return ops().gated_delta_prep(proj[rows], C, C + heads, w, state, batch, bias, A, 1e-6, dim ** -0.5, heads, kv_heads,
                                      dim, vdim, exact=exact)

    whole = run(slice(0, n), Batch(COUNTS, range(len(COUNTS) - 1, -1, -1)))
    for x, y in zip(whole, piecewise(run, COUNTS)):
        assert torch.equal(x, y)


@pytest.mark.parametrize("groups,size,shared", [(32, 64, False), (33, 64, True), (40, 128, True), (36, 68, False), (64, 4, False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gate", [None, "sigmoid", "silu"])
def test_norms_of_many_small_parts(groups, size, shared, dtype, gate):
    g = torch.Generator(device=DEV).manual_seed(size)
    R = lambda *s: torch.randn(s, generator=g, device=DEV)  # noqa: E731
    n, C = 16384 // groups + 3, groups * size
    x, w, z = R(n, C), R(size if shared else C), R(n, C + 12)

    def run(rows):
        kw = dict(gate=z[rows], gate_col=8, activation=gate) if gate else {}
        return ops().group_norm_gate(x[rows], w, 1e-5, groups, dtype, **kw)

    half = n // 2
    assert torch.equal(run(slice(0, n)), torch.cat([run(slice(0, half)), run(slice(half, n))]))


@pytest.mark.parametrize("rows", [5, 514])
@pytest.mark.parametrize("dim,vdim,rot", [(128, 128, 64), (36, 20, 24), (64, 64, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("writes", [True, False])
def test_rotated_rows_by_fours(rows, dim, vdim, rot, dtype, writes):
    g = torch.Generator(device=DEV).manual_seed(rows)
    nq, nkv, page, col0 = 6, 2, 64, 8
    wide = col0 + nq * dim + nkv * (dim + vdim) + 4
    proj = torch.randn((rows, wide), generator=g, device=DEV)
    other = torch.zeros((rows, wide + 1), device=DEV)  # an odd stride: an element a thread
    other[:, :wide] = proj
    pages = rows // page + 2
    table = torch.randperm(pages, generator=g, device=DEV).to(torch.int32).view(1, -1)
    pos, slot = i32(range(3, rows + 3)), i32([0] * rows)
    rotation = None
    if rot:
        denom = 10000.0 ** (torch.arange(rot // 2, device=DEV, dtype=torch.float32) * 2 / rot)
        rotation = type("R", (), dict(pairing="half", magnitude=1.0, denominators=denom, rotary_dim=rot))()
    got = []
    for p in (proj, other):
        kp, vp = torch.zeros((pages, nkv, page, dim), device=DEV, dtype=dtype), torch.zeros((pages, nkv, page, vdim), device=DEV, dtype=dtype)
        q = ops().sig_qkv_post(p, col0, rotation, pos, slot, kp, vp, table, page, nq, nkv, dim, vdim, writes, dtype)
        got.append((q, kp, vp))
    for x, y in zip(*got):
        assert torch.equal(x, y)
    assert got[0][0].abs().sum() > 0 and bool(got[0][2].abs().sum() > 0) == writes


@pytest.mark.parametrize("n", [4, 2048, 2052, 4100, 262147])  # the last one: an element a thread
def test_scaled_sums_by_fours(n):
    a, b = (torch.randn(n, generator=torch.Generator(device=DEV).manual_seed(s), device=DEV) for s in (1, 2))
    odd = torch.empty(n + 1, device=DEV)[1:].copy_(a)  # off 16 bytes: an element a thread
    ops().scaled_sum_(odd, b, 0.75, 0.55)
    assert torch.equal(ops().scaled_sum_(a, b, 0.75, 0.55), odd)
