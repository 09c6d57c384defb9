"""A decode step of the recurrences (csrc/state_step.cu) against their row-by-row walks, which are held to 64-bit
rules elsewhere.  The same products in sums of another order: at most 160 terms of 2^-24 each, 1e-5 of the
largest result."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = 1e-5


def ops():
    from reflex_b200 import ops as o

    return o


def i32(v):
    return torch.tensor(list(v), dtype=torch.int32, device=DEV)


class Batch:
    def __init__(self, slots, most=1):
        n = len(slots)
        self.seq_slot, self.seq_new, self.seq_row0, self.max_new = i32(slots), i32([1] * n), i32(range(n + 1)), most


def near(a, b):
    assert (a - b).abs().max() <= TOL * b.abs().max()


def compare(run, state, slots):
    """run(state, batch, exact): the walk serves a batch that says it may have more rows."""
    out = []
    for batch, exact in ((Batch(slots), False), (Batch(slots, 2), True)):
        s = state.clone()
        out.append((run(s, batch, exact), s))
    (a, s), (b, t) = out
    for x, y in zip(a, b):
        near(x, y)
    near(s, t)
    others = [i for i in range(state.shape[0]) if i not in slots]
    assert torch.equal(s[others], state[others])


SLOTS = [(2,), (3, 0, 4), tuple(range(79, -1, -1))]  # one, a few, and enough heads for a block each


def rand(g):
    return lambda *s: torch.randn(s, generator=g, device=DEV)


@pytest.mark.parametrize("slots", SLOTS)
@pytest.mark.parametrize("heads,groups,P,N", [(4, 2, 64, 128), (8, 1, 12, 20), (4, 4, 68, 8), (4, 1, 132, 64), (4, 2, 260, 100)])
def test_ssd_step(heads, groups, P, N, slots):
    R = rand(torch.Generator(device=DEV).manual_seed(P + N))
    n, inner = len(slots), heads * P
    xbc, proj, D, bias = R(n, inner + 2 * groups * N), R(n, inner + heads), R(heads), R(heads)
    A = -torch.rand(heads, device=DEV)
    compare(lambda s, b, exact: (ops().ssd_scan(xbc, proj, 0, inner, bias, A, D, s, 4, b, heads, P, N, groups, exact=exact),),
            R(max(slots) + 2, 4 + heads * P * N), slots)


@pytest.mark.parametrize("slots", SLOTS)
@pytest.mark.parametrize("heads,d", [(4, 64), (3, 4), (5, 36), (4, 32), (2, 72)])  # 72: the walk in either case
def test_delta_step(heads, d, slots):
    R = rand(torch.Generator(device=DEV).manual_seed(d))
    n, hd = len(slots), heads * d
    proj, wpre, wb, ab = R(n, 4 * hd), R(n, hd), R(hd), R(hd)
    compare(lambda s, b, exact: (ops().delta_rule(proj, 0, hd, 2 * hd, 3 * hd, wpre, wb, ab, 0.6, 1e-6, s, 8, b, heads, d,
                                                  exact=exact),), R(max(slots) + 2, 8 + hd * d), slots)


@pytest.mark.parametrize("slots", SLOTS)
@pytest.mark.parametrize("H,G,d,dv", [(4, 2, 128, 128), (3, 1, 64, 20), (4, 4, 12, 132), (2, 2, 100, 36), (2, 1, 160, 16)])
def test_gated_delta_step(H, G, d, dv, slots):
    R = rand(torch.Generator(device=DEV).manual_seed(d + dv))
    n = len(slots)
    qkv, gates = R(n, 2 * G * d + H * dv) * d ** -0.5, torch.rand((n, 2 * H), device=DEV)
    compare(lambda s, b, exact: (ops().gated_delta_scan(qkv, gates, s, 4, b, H, G, d, dv, exact=exact),),
            R(max(slots) + 2, 4 + H * d * dv), slots)


@pytest.mark.parametrize("slots", SLOTS)
@pytest.mark.parametrize("heads,dim,vdim", [(2, 128, 256), (3, 20, 196), (2, 100, 228), (2, 64, 64)])  # 64: the walk
def test_mlstm_step(heads, dim, vdim, slots):
    R = rand(torch.Generator(device=DEV).manual_seed(dim + vdim))
    n, io = len(slots), heads * (2 * dim + vdim)
    proj = R(n, io + 2 * heads + (-io - 2 * heads) % 4)
    bi, bf, floats = R(heads), R(heads), ops().mlstm_state_floats(dim, vdim)
    state = R(max(slots) + 2, heads, floats)
    state[..., dim * vdim + dim:] = state[..., -1:]  # one running number, held once per 64 columns
    compare(lambda s, b, exact: ops().mlstm_scan(proj, (0, heads * dim, 2 * heads * dim, io, io + heads), bi, bf, 15.0,
                                                 dim ** -0.5, b, s, heads, dim, vdim, max_rows=b.max_new, exact=exact),
            state, slots)


def test_infinite_values_stay_infinite_where_lanes_have_no_element():
    """Sizes that leave lanes of a column without an element: an infinite value among positive numbers gives its own
    results infinities, as walking does, and no NaN."""
    g = torch.Generator(device=DEV).manual_seed(2)
    R = lambda *s: torch.rand(s, generator=g, device=DEV)  # noqa: E731
    heads, d, n = 2, 36, 3
    hd, slots = heads * d, (2, 0, 1)

    def bad(row, at):
        row[:, at] = float("inf")
        return row

    def check(run, floats):
        out = []
        for batch, exact in ((Batch(slots), False), (Batch(slots, 2), True)):
            state = start[:, :floats].clone()
            out.append((run(state, batch, exact), state))
        for a, b in zip(*out):
            assert not a.isnan().any() and torch.equal(a.isinf(), b.isinf()) and a.isinf().any()

    start = R(3, hd * d)
    xbc, proj, one = bad(R(n, hd + 2 * d), 7), R(n, hd + heads), torch.ones(heads, device=DEV)
    check(lambda s, b, exact: ops().ssd_scan(xbc, proj, 0, hd, one, -one, one, s, 0, b, heads, d, d, 1, exact=exact), hd * d)
    rows, wpre, zero = bad(R(n, 4 * hd), 2 * hd + 7), R(n, hd), torch.zeros(hd, device=DEV)
    check(lambda s, b, exact: ops().delta_rule(rows, 0, hd, 2 * hd, 3 * hd, wpre, zero, zero, 0.6, 1e-6, s, 0, b, heads, d,
                                               exact=exact), hd * d)
