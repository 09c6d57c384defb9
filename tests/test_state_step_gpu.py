"""A decode step of the recurrences (csrc/state_step.cu) against their row-by-row walks and their rules in 64 bits.  The
same products in sums of another order: at most 160 terms of 2^-24 each, 1e-5 of the largest result.  In the 2-norm a
sum of four in each of 32 lanes, five meetings of lanes and a handful of factors, ten roundings of 2.5e-8 of the value
each, are 8e-8; NORM is twice that."""

import numpy as np
import pytest
import torch
from test_chunk_scan_gpu import delta_rule_rows, mlstm_rule, norm_off, ssd_rule

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = 1e-5
NORM = 1.6e-7


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


def up(t):
    return t.double().cpu().numpy()


def compare(run, state, slots, rule=None):
    """run(state, batch, exact): the walk serves a batch that says it may have more rows.  rule(sequence, its state):
    its results and the state after, in 64 bits."""
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
    if rule:
        refs = [rule(i, up(state[slot])) for i, slot in enumerate(slots)]
        for j, x in enumerate(a):
            assert norm_off(x, np.stack([r[j] for r in refs])) < NORM
        assert norm_off(s[list(slots)], np.stack([r[-1] for r in refs])) < NORM


SLOTS = [(2,), (3, 0, 4), tuple(range(79, -1, -1))]  # one, a few, and enough heads for a block each


def rand(g):
    return lambda *s: torch.randn(s, generator=g, device=DEV)


@pytest.mark.parametrize("slots", SLOTS)
@pytest.mark.parametrize("heads,groups,P,N", [(4, 2, 64, 128), (8, 1, 12, 20), (4, 4, 68, 8), (4, 1, 132, 64), (4, 2, 260, 100)])
def test_ssd_step(heads, groups, P, N, slots):
    R = rand(torch.Generator(device=DEV).manual_seed(P + N))
    n, inner = len(slots), heads * P
    xbc, proj, D, bias = R(n, inner + 2 * groups * N), R(n, inner + heads), R(heads), R(heads)
    A = -R(heads).abs()

    def rule(i, state):
        x, w = up(xbc[i:i + 1]), up(proj[i:i + 1])
        B, C = (x[:, o:o + groups * N].reshape(1, groups, N).repeat(heads // groups, 1) for o in (inner, inner + groups * N))
        dt, z = np.logaddexp(0.0, w[:, inner:] + up(bias)), w[0, :inner]
        y, S = ssd_rule(x[:, :inner].reshape(1, heads, P), B, C, dt, up(A), up(D), state[4:].reshape(heads, P, N))
        return y.ravel() * z / (1 + np.exp(-z)), np.concatenate([state[:4], S.ravel()])

    compare(lambda s, b, exact: (ops().ssd_scan(xbc, proj, 0, inner, bias, A, D, s, 4, b, heads, P, N, groups, exact=exact),),
            R(max(slots) + 2, 4 + heads * P * N), slots, rule)


@pytest.mark.parametrize("slots", SLOTS)
@pytest.mark.parametrize("heads,d", [(4, 64), (3, 4), (5, 36), (4, 32), (2, 72)])  # 72: the walk in either case
def test_delta_step(heads, d, slots):
    R = rand(torch.Generator(device=DEV).manual_seed(d))
    n, hd = len(slots), heads * d
    proj, wpre, wb, ab = R(n, 4 * hd), R(n, hd), R(hd), R(hd)

    def rule(i, state):
        sig = lambda x: 1 / (1 + np.exp(-x))  # noqa: E731
        r, k, v, a = up(proj[i]).reshape(4, 1, heads, d)
        w = np.exp(-0.6 * sig(up(wpre[i] + wb))).reshape(1, heads, d)
        y, S = delta_rule_rows(r, k, v, w, sig(a + up(ab).reshape(heads, d)), state[8:].reshape(heads, d, d), 1e-6)
        return y.ravel(), np.concatenate([state[:8], S.ravel()])

    compare(lambda s, b, exact: (ops().delta_rule(proj, 0, hd, 2 * hd, 3 * hd, wpre, wb, ab, 0.6, 1e-6, s, 8, b, heads, d,
                                                  exact=exact),), R(max(slots) + 2, 8 + hd * d), slots, rule)


@pytest.mark.parametrize("slots", SLOTS)
@pytest.mark.parametrize("H,G,d,dv", [(4, 2, 128, 128), (3, 1, 64, 20), (4, 4, 12, 132), (2, 2, 100, 36), (2, 1, 160, 16)])
def test_gated_delta_step(H, G, d, dv, slots):
    R = rand(torch.Generator(device=DEV).manual_seed(d + dv))
    n = len(slots)
    qkv, gates = R(n, 2 * G * d + H * dv) * d ** -0.5, torch.rand((n, 2 * H), device=DEV)

    def rule(i, state):
        row, (g, beta) = up(qkv[i]), up(gates[i]).reshape(2, H)
        q, k = row[:2 * G * d].reshape(2, G, d).repeat(H // G, 1)
        S = g[:, None, None] * state[4:].reshape(H, dv, d)
        S = S + (beta[:, None] * (row[2 * G * d:].reshape(H, dv) - (S * k[:, None]).sum(-1)))[:, :, None] * k[:, None]
        return (S * q[:, None]).sum(-1).ravel(), np.concatenate([state[:4], S.ravel()])

    compare(lambda s, b, exact: (ops().gated_delta_scan(qkv, gates, s, 4, b, H, G, d, dv, exact=exact),),
            R(max(slots) + 2, 4 + H * d * dv), slots, rule)


@pytest.mark.parametrize("slots", SLOTS)
@pytest.mark.parametrize("heads,dim,vdim", [(2, 128, 256), (3, 20, 196), (2, 100, 228), (2, 64, 64)])  # 64: the walk
def test_mlstm_step(heads, dim, vdim, slots):
    R = rand(torch.Generator(device=DEV).manual_seed(dim + vdim))
    n, io = len(slots), heads * (2 * dim + vdim)
    proj = R(n, io + 2 * heads + (-io - 2 * heads) % 4)
    bi, bf, floats = R(heads), R(heads), ops().mlstm_state_floats(dim, vdim)
    state = R(max(slots) + 2, heads, floats)
    state[..., dim * vdim + dim:] = state[..., -1:]  # one running number, held once per 64 columns

    def rule(i, old):
        row, cut = up(proj[i:i + 1]), lambda o, w: row[:, o:o + heads * w].reshape(1, heads, w)  # noqa: E731
        gi, gf = (15.0 * np.tanh((row[:, o:o + heads] + up(t)) / 15.0) for o, t in ((io, bi), (io + heads, bf)))
        y, den, S, nn, m = mlstm_rule(cut(0, dim) * dim ** -0.5, cut(heads * dim, dim), cut(2 * heads * dim, vdim), gi,
                                      -np.logaddexp(0.0, -gf), old[:, :dim * vdim].reshape(heads, dim, vdim),
                                      old[:, dim * vdim:dim * vdim + dim], old[:, -1])
        return y[0].ravel(), den[0], np.concatenate([S.reshape(heads, -1), nn, m[:, None].repeat(floats - dim * vdim - dim, 1)], 1)

    compare(lambda s, b, exact: ops().mlstm_scan(proj, (0, heads * dim, 2 * heads * dim, io, io + heads), bi, bf, 15.0,
                                                 dim ** -0.5, b, s, heads, dim, vdim, max_rows=b.max_new, exact=exact),
            state, slots, rule)


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
