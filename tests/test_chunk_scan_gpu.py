"""The recurrences that take a prompt's rows 64 at a time (csrc/chunk_scan.cuh)
against their row-by-row rules in 64 bits, at the edges of chunks and tiles.

Tolerance, of the largest result: sums of up to N + 64 <= 192 terms in 32 bits are off by at most
192 * 2^-24 = 1.2e-5; the weights' exponentials add a few units in the last place.  In the 2-norm roundings of
either sign mostly cancel: two sums of some 25 roundings of 0.3 units each, and as much for the weights, are 2.5e-7;
NORM is twice that, and a third of what products of operands rounded to 22 bits give."""

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = 2e-5
NORM = 5e-7


def ops():
    from reflex_b200 import ops as o

    return o


def i32(v):
    return torch.tensor(list(v), dtype=torch.int32, device=DEV)


@pytest.fixture(autouse=True)
def rules(monkeypatch):
    monkeypatch.setattr(ops(), "MLSTM_SIDE_BY_SIDE_MIN_ROWS", ops().MLSTM_SIDE_BY_SIDE_MIN_ROWS)


class Batch:
    def __init__(self, counts, slots):
        self.row0 = [0]
        for c in counts:
            self.row0.append(self.row0[-1] + c)
        self.seq_slot, self.seq_new, self.seq_row0 = i32(slots), i32(counts), i32(self.row0)
        self.max_new = max(counts)


def off(got, ref):
    got = got.double().cpu().numpy()
    return np.abs(got - ref).max() / np.abs(ref).max()


def norm_off(got, ref):
    return np.linalg.norm(got.double().cpu().numpy() - ref) / np.linalg.norm(ref)


def ssd_rule(x, B, C, dt, A, D, S):
    """x [T, H, P], B, C [T, H, N], dt [T, H], S [H, P, N]."""
    ys = []
    for t in range(x.shape[0]):
        S = np.exp(A * dt[t])[:, None, None] * S + (dt[t][:, None] * x[t])[:, :, None] * B[t][:, None, :]
        ys.append((S * C[t][:, None, :]).sum(-1) + D[:, None] * x[t])
    return np.stack(ys), S


@pytest.mark.parametrize("heads,groups,P,N", [(4, 2, 64, 128), (2, 1, 12, 20), (3, 3, 68, 8), (2, 2, 132, 100)])
@pytest.mark.parametrize("counts", [(64,), (65, 1, 63), (128, 0, 129), (200,)])
def test_ssd_in_chunks(heads, groups, P, N, counts, monkeypatch):
    monkeypatch.setattr(ops(), "SSD_CHUNK_MIN_ROWS", 1)
    rng = np.random.default_rng(heads * 100 + N + sum(counts))
    inner, R = heads * P, sum(counts)
    xbc = rng.standard_normal((R, inner + 2 * groups * N)).astype(np.float32)
    proj = rng.standard_normal((R, inner + heads + (-heads) % 4)).astype(np.float32)
    proj[:, inner:inner + heads] *= 3.0  # steps from near nothing to several
    A, D = -np.exp(rng.uniform(-2, 1, heads)).astype(np.float32), rng.standard_normal(heads).astype(np.float32)
    bias = rng.uniform(-0.5, 0.5, heads).astype(np.float32)
    slots = [3, 0, 5][:len(counts)]
    state = rng.standard_normal((6, 8 + heads * P * N)).astype(np.float32)
    dev = torch.from_numpy(state).to(DEV)
    to = lambda a: torch.from_numpy(a).to(DEV)  # noqa: E731
    b = Batch(counts, slots)
    out = ops().ssd_scan(to(xbc), to(proj), 0, inner, to(bias), to(A), to(D), dev, 8, b, heads, P, N, groups, exact=False)
    for i, (n, slot) in enumerate(zip(counts, slots)):
        rows = slice(b.row0[i], b.row0[i + 1])
        if not n:
            assert torch.equal(dev[slot].cpu(), torch.from_numpy(state[slot]))
            continue
        xd, pd = xbc[rows].astype(np.float64), proj[rows].astype(np.float64)
        x = xd[:, :inner].reshape(n, heads, P)
        rep = heads // groups
        Bm, Cm = (xd[:, inner + k * groups * N:inner + (k + 1) * groups * N].reshape(n, groups, N).repeat(rep, 1)
                  for k in (0, 1))
        dt = np.logaddexp(0.0, pd[:, inner:inner + heads] + bias)
        y, S = ssd_rule(x, Bm, Cm, dt, A.astype(np.float64), D.astype(np.float64),
                        state[slot, 8:].astype(np.float64).reshape(heads, P, N))
        z = pd[:, :inner]
        assert off(out[rows], y.reshape(n, inner) * z / (1 + np.exp(-z))) < TOL
        assert norm_off(out[rows], y.reshape(n, inner) * z / (1 + np.exp(-z))) < NORM
        assert off(dev[slot, 8:], S.ravel()) < TOL
        assert torch.equal(dev[slot, :8].cpu(), torch.from_numpy(state[slot, :8]))
    untouched = [s for s in range(6) if s not in slots]
    assert torch.equal(dev[untouched].cpu(), torch.from_numpy(state[untouched]))


def mlstm_rule(q, k, v, i, f, S, n, m):
    num, den = [], []
    for t in range(q.shape[0]):
        m2 = np.maximum(f[t] + m, i[t])
        a, b = np.exp(f[t] + m - m2), np.exp(i[t] - m2)
        S = a[:, None, None] * S + (b[:, None] * k[t])[:, :, None] * v[t][:, None, :]
        n = a[:, None] * n + b[:, None] * k[t]
        m = m2
        num.append((S * q[t][:, :, None]).sum(1))
        den.append(np.maximum(np.abs((n * q[t]).sum(-1)), np.exp(-m)) + 1e-6)
    return np.stack(num), np.stack(den), S, n, m


def mlstm_case(heads, dim, vdim, counts, slots, running, forget):
    """A step's rows and states; the slots in `running` go on from earlier rows, the others start."""
    rng = np.random.default_rng(heads + dim + sum(counts))
    R = sum(counts)
    i_off = heads * (2 * dim + vdim)
    f_off = i_off + heads
    ld = f_off + heads + (-(f_off + heads)) % 4
    proj = rng.standard_normal((R, ld)).astype(np.float32)
    proj[:, i_off:f_off + heads] *= 4.0  # gates that swing
    bi, bf = rng.standard_normal(heads).astype(np.float32), (rng.standard_normal(heads) + forget).astype(np.float32)
    state = np.zeros((max(slots) + 1, heads, ops().mlstm_state_floats(dim, vdim)), dtype=np.float32)
    for slot in running:
        state[slot, :, :dim * vdim + dim] = rng.standard_normal((heads, dim * vdim + dim))
        state[slot, :, dim * vdim + dim:] = rng.standard_normal(heads)[:, None]
    return proj, (0, heads * dim, 2 * heads * dim, i_off, f_off), bi, bf, state, Batch(counts, slots)


def mlstm_run(case, heads, dim, vdim, cap=12.0):
    proj, offsets, bi, bf, state, b = case
    ops().MLSTM_SIDE_BY_SIDE_MIN_ROWS = 1  # (the fixture above puts it back)
    to = lambda a: torch.from_numpy(a).to(DEV)  # noqa: E731
    dev = torch.from_numpy(state.copy()).to(DEV)
    num, den = ops().mlstm_scan(to(proj), offsets, to(bi), to(bf), cap, 0.25, b, dev, heads, dim, vdim,
                                max_rows=b.max_new, exact=False)
    return num, den, dev


def mlstm_check(case, got, heads, dim, vdim, cap=12.0):
    proj, (q_off, k_off, v_off, i_off, f_off), bi, bf, state, b = case
    num, den, dev = got
    for j, slot in enumerate(b.seq_slot.tolist()):
        n, rows = b.row0[j + 1] - b.row0[j], slice(b.row0[j], b.row0[j + 1])
        p = proj[rows].astype(np.float64)
        cut = lambda o, w: p[:, o:o + heads * w].reshape(n, heads, w)  # noqa: E731
        i = cap * np.tanh((p[:, i_off:i_off + heads] + bi) / cap)
        f = -np.logaddexp(0.0, -cap * np.tanh((p[:, f_off:f_off + heads] + bf) / cap))
        old = state[slot].astype(np.float64)
        rn, rd, S, nn, m = mlstm_rule(cut(q_off, dim) * 0.25, cut(k_off, dim), cut(v_off, vdim), i, f,
                                      old[:, :dim * vdim].reshape(heads, dim, vdim),
                                      old[:, dim * vdim:dim * vdim + dim], old[:, -1])
        assert off(num[rows], rn.reshape(n, -1)) < TOL and norm_off(num[rows], rn.reshape(n, -1)) < NORM
        assert off(den[rows], rd) < TOL
        new = dev[slot].double().cpu().numpy()
        assert (new[:, dim * vdim + dim:] == new[:, -1:]).all()
        scale = np.exp(new[:, -1] - m)  # the memory is relative to the number beside it
        assert np.abs(new[:, -1] - m).max() < 1e-5 * (1 + np.abs(m).max())
        assert off(torch.from_numpy(new[:, :dim * vdim] * scale[:, None]), S.reshape(heads, -1)) < TOL
        assert off(torch.from_numpy(new[:, dim * vdim:dim * vdim + dim] * scale[:, None]), nn) < TOL


@pytest.mark.parametrize("heads,dim,vdim", [(2, 128, 256), (3, 20, 12), (2, 64, 68), (4, 100, 130 - 2)])
@pytest.mark.parametrize("counts", [(64,), (65, 1, 127), (193,)])
def test_mlstm_in_chunks(heads, dim, vdim, counts):
    case = mlstm_case(heads, dim, vdim, counts, [3, 0, 5][:len(counts)], [3], 2.0)
    mlstm_check(case, mlstm_run(case, heads, dim, vdim), heads, dim, vdim)


def test_mlstm_with_more_blocks_than_the_chip_holds():
    """Heads that remember, running states, one long sequence before short ones: blocks of a head
    start long after others of it have ended, and still read the number the sequence came with."""
    heads, dim, vdim = 16, 128, 256
    case = mlstm_case(heads, dim, vdim, (450, 1, 64, 3, 65, 1, 17, 130), [3, 0, 5, 1, 7, 2, 4, 6], range(8), 5.0)
    first = mlstm_run(case, heads, dim, vdim)
    mlstm_check(case, first, heads, dim, vdim)
    for _ in range(20):
        assert all(torch.equal(a, b) for a, b in zip(mlstm_run(case, heads, dim, vdim), first))


def test_a_long_step_goes_through_a_bounded_scratch():
    """Memories of 64 heads of 256 x 128 for 37 chunks (310 MB) do not fit the scratch: rounds of rows,
    each going on from the state that the one before left; beside it a short sequence.  With
    decays near one a result is a sum over all rows; the walk it is compared with rounds 2,300 times,
    2300 * 2^-24 = 1.4e-4."""
    heads, groups, P, N, counts = 64, 2, 256, 128, (2300, 70)
    g = torch.Generator(device=DEV).manual_seed(4)
    R, inner = sum(counts), heads * P
    xbc = torch.randn((R, inner + 2 * groups * N), generator=g, device=DEV)
    proj = torch.randn((R, inner + heads), generator=g, device=DEV)
    A = -torch.rand(heads, generator=g, device=DEV) * 0.05  # slow decays: the first round's rows count in the second
    D, bias = torch.randn(heads, generator=g, device=DEV), torch.zeros(heads, device=DEV)
    assert ops().native.lib().rfx_ssd_chunk_floats(R, 2, 2300, heads, P, N) < 100 << 20
    got = []
    for exact in (True, False):
        state = torch.zeros((2, heads * P * N), device=DEV)
        y = ops().ssd_scan(xbc, proj, 0, inner, bias, A, D, state, 0, Batch(counts, [1, 0]), heads, P, N, groups, exact=exact)
        got.append((y, state))
    for a, b in zip(*got):
        assert ((a - b).abs().max() / a.abs().max()).item() < 1.4e-4
    assert math.isfinite(got[1][0].sum().item())


def delta_rule_rows(r, k, v, w, a, S, eps):
    """All [T, H, d]; S [H, value, key].  Both terms read the old S."""
    out = []
    for t in range(r.shape[0]):
        u = k[t] / np.sqrt((k[t] ** 2).sum(-1, keepdims=True) + eps)
        seen = (S * u[:, None, :]).sum(-1)
        S = S * w[t][:, None, :] - seen[:, :, None] * (a[t] * u)[:, None, :] + v[t][:, :, None] * k[t][:, None, :]
        out.append((S * r[t][:, None, :]).sum(-1))
    return np.stack(out), S


def delta_case(counts, rate, eps):
    heads, d = 3, 64
    hd, R = heads * d, sum(counts)
    rng = np.random.default_rng(sum(counts))
    proj = rng.standard_normal((R, 4 * hd)).astype(np.float32)
    wpre = (3 * rng.standard_normal((R, hd))).astype(np.float32)
    wb, ab = rng.standard_normal(hd).astype(np.float32), rng.standard_normal(hd).astype(np.float32)
    slots = [3, 0, 5][:len(counts)]
    state = rng.standard_normal((6, 4 + hd * d)).astype(np.float32)
    dev = torch.from_numpy(state.copy()).to(DEV)
    to = lambda x: torch.from_numpy(x).to(DEV)  # noqa: E731
    b = Batch(counts, slots)
    out = ops().delta_rule(to(proj), 0, hd, 2 * hd, 3 * hd, to(wpre), to(wb), to(ab), rate, eps, dev, 4, b, heads, d,
                           exact=False)
    for i, (n, slot) in enumerate(zip(counts, slots)):
        if not n:
            assert torch.equal(dev[slot].cpu(), torch.from_numpy(state[slot]))
            continue
        rows = slice(b.row0[i], b.row0[i + 1])
        r, k, v, a = (proj[rows, o * hd:(o + 1) * hd].astype(np.float64).reshape(n, heads, d) for o in range(4))
        sig = lambda x: 1 / (1 + np.exp(-x))  # noqa: E731
        w = np.exp(-rate * sig((wpre[rows].astype(np.float64) + wb).reshape(n, heads, d)))
        ref, S = delta_rule_rows(r, k, v, w, sig(a + ab.astype(np.float64).reshape(heads, d)),
                                 state[slot, 4:].astype(np.float64).reshape(heads, d, d), eps)
        assert off(out[rows], ref.reshape(n, hd)) < TOL and (rate > 1 or norm_off(out[rows], ref.reshape(n, hd)) < NORM)
        assert off(dev[slot, 4:], S.ravel()) < TOL
        assert torch.equal(dev[slot, :4].cpu(), torch.from_numpy(state[slot, :4]))
    untouched = [s for s in range(6) if s not in slots]
    assert torch.equal(dev[untouched].cpu(), torch.from_numpy(state[untouched]))


@pytest.mark.parametrize("rate", [math.exp(-0.5), 2.0, 0.0, 2.5])  # 2.5: beyond the chunks' range, the walk
@pytest.mark.parametrize("counts", [(32,), (33, 1, 31), (64, 0, 97), (160,)])
def test_delta_rule_in_chunks(counts, rate, monkeypatch):
    monkeypatch.setattr(ops(), "DELTA_CHUNK_MIN_ROWS", 1)
    delta_case(counts, rate, 1e-6)


def test_delta_rule_in_chunks_without_an_epsilon(monkeypatch):
    """Rows that a last chunk does not have bring nothing: their key has no length to divide by."""
    monkeypatch.setattr(ops(), "DELTA_CHUNK_MIN_ROWS", 1)
    delta_case((33, 1, 31), 0.5, 0.0)


def test_a_long_delta_step_goes_through_a_bounded_scratch():
    heads, d, counts = 64, 64, (5000, 70)
    g = torch.Generator(device=DEV).manual_seed(5)
    R, hd = sum(counts), heads * d
    proj = torch.randn((R, 4 * hd), generator=g, device=DEV)
    wpre = torch.randn((R, hd), generator=g, device=DEV) - 6.0  # slow decays
    zero = torch.zeros(hd, device=DEV)
    assert ops().native.lib().rfx_delta_rule_chunk_floats(R, 2, 5000, heads) < 80 << 20
    got = []
    for exact in (True, False):
        state = torch.zeros((2, hd * d), device=DEV)
        y = ops().delta_rule(proj, 0, hd, 2 * hd, 3 * hd, wpre, zero, zero, math.exp(-0.5), 1e-6, state, 0,
                             Batch(counts, [1, 0]), heads, d, exact=exact)
        got.append((y, state))
    for a, b in zip(*got):  # the removal forgets what 32 rows back added: no sum over all rows here
        assert ((a - b).abs().max() / a.abs().max()).item() < TOL


def test_many_sequences_go_through_a_bounded_scratch(monkeypatch):
    """121 chunks of 64 heads of 256 x 128 where the scratch holds 31, and 260 of the delta rule's of 64 heads where it
    holds 95: rounds of sequences, the longest of them in several; against the walk, a short sum's roundings apart."""
    monkeypatch.setattr(ops(), "DELTA_CHUNK_MIN_ROWS", 1)
    heads, groups, P, N = 64, 2, 256, 128
    counts = [120 + (i * 7) % 30 for i in range(39)] + [700]
    g = torch.Generator(device=DEV).manual_seed(6)
    R, inner = sum(counts), heads * P
    xbc = torch.randn((R, inner + 2 * groups * N), generator=g, device=DEV)
    proj = torch.randn((R, inner + heads), generator=g, device=DEV)
    A, D = -torch.rand(heads, generator=g, device=DEV) - 0.5, torch.randn(heads, generator=g, device=DEV)
    bias, start = torch.zeros(heads, device=DEV), torch.randn((40, heads * P * N), generator=g, device=DEV)
    slots = [(i * 11) % 40 for i in range(40)]
    got = []
    for exact in (True, False):
        state = start.clone()
        y = ops().ssd_scan(xbc, proj, 0, inner, bias, A, D, state, 0, Batch(counts, slots), heads, P, N, groups, exact=exact)
        got.append((y, state))
    for a, b in zip(*got):
        assert ((a - b).abs().max() / a.abs().max()).item() < 2 * TOL
    hd = heads * 64
    proj, wpre = torch.randn((R, 4 * hd), generator=g, device=DEV), torch.randn((R, hd), generator=g, device=DEV)
    zero, got = torch.zeros(hd, device=DEV), []
    for exact in (True, False):
        state = start[:, :hd * 64].clone()
        y = ops().delta_rule(proj, 0, hd, 2 * hd, 3 * hd, wpre, zero, zero, math.exp(-0.5), 1e-6, state, 0,
                             Batch(counts, slots), heads, 64, exact=exact)
        got.append((y, state))
    for a, b in zip(*got):
        assert ((a - b).abs().max() / a.abs().max()).item() < 2 * TOL


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_row_that_is_not_finite_does_not_reach_earlier_rows(bad):
    """An element of v at row 70 spoils its own column from there on, one of k every result from there on, and
    neither anything before: rows 64 to 69 share its chunk, 68 and 69 its four."""
    heads, groups, P, N, T = 4, 2, 64, 128, 200
    g = torch.Generator(device=DEV).manual_seed(9)
    inner, b = heads * P, Batch([T], [0])
    xbc = torch.randn((T, inner + 2 * groups * N), generator=g, device=DEV)
    proj = torch.randn((T, inner + heads), generator=g, device=DEV)
    A, D, bias = -torch.ones(heads, device=DEV), torch.zeros(heads, device=DEV), torch.zeros(heads, device=DEV)

    def ssd(x):
        state = torch.zeros((1, heads * P * N), device=DEV)
        return ops().ssd_scan(x, proj, 0, inner, bias, A, D, state, 0, b, heads, P, N, groups, exact=False), state

    clean, clean_state = ssd(xbc)
    for column in (P + 5, inner + 3):  # element 5 of head 1's v; element 3 of the first group's k
        x = xbc.clone()
        x[70, column] = bad
        y, state = ssd(x)
        hit = torch.zeros(inner, dtype=torch.bool, device=DEV)
        hit[P + 5 if column < inner else slice(0, heads // groups * P)] = True
        assert torch.equal(y[:70], clean[:70]) and torch.equal(y[:, ~hit], clean[:, ~hit])
        assert not torch.isfinite(y[70:, hit]).any()
        assert torch.equal(state.view(inner, N)[~hit], clean_state.view(inner, N)[~hit])
    case = mlstm_case(2, 128, 256, (T,), [0], [0], 2.0)
    num, den, _ = mlstm_run(case, 2, 128, 256)
    case[0][70, 2 * 2 * 128 + 256 + 100] = bad  # element 100 of head 1's v
    num2, den2, _ = mlstm_run(case, 2, 128, 256)
    hit = torch.zeros(512, dtype=torch.bool, device=DEV)
    hit[256 + 100] = True
    assert torch.equal(num2[:70], num[:70]) and torch.equal(num2[:, ~hit], num[:, ~hit]) and torch.equal(den, den2)
    assert not torch.isfinite(num2[70:, hit]).any()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_row_that_is_not_finite_does_not_reach_earlier_rows_of_the_delta_rule(bad, monkeypatch):
    """An element of v at row 70 spoils its own column from there on; one of k or of the decay its head's results:
    from row 70 on, and nothing of rows 64 to 69 before it in its chunk."""
    monkeypatch.setattr(ops(), "DELTA_CHUNK_MIN_ROWS", 1)
    heads, d, T = 2, 64, 100
    hd, b = heads * d, Batch([T], [0])
    g = torch.Generator(device=DEV).manual_seed(10)
    proj, wpre = torch.randn((T, 4 * hd), generator=g, device=DEV), torch.randn((T, hd), generator=g, device=DEV)
    zero = torch.zeros(hd, device=DEV)

    def run(p, w):
        state = torch.zeros((1, hd * d), device=DEV)
        return ops().delta_rule(p, 0, hd, 2 * hd, 3 * hd, w, zero, zero, 0.6, 1e-6, state, 0, b, heads, d, exact=False), state

    clean, clean_state = run(proj, wpre)
    for part in ("v", "k", "decay"):
        p, w = proj.clone(), wpre.clone()
        if part == "decay":
            w[70, 67] = float("nan")
        else:
            p[70, (2 * hd if part == "v" else hd) + 67] = bad
        y, state = run(p, w)
        hit = torch.zeros(hd, dtype=torch.bool, device=DEV)
        hit[67 if part == "v" else slice(64, 128)] = True
        assert torch.equal(y[:70], clean[:70]) and torch.equal(y[:, ~hit], clean[:, ~hit]), part
        assert not torch.isfinite(y[71:, hit]).any(), part
        assert torch.equal(state.view(hd, d)[~hit], clean_state.view(hd, d)[~hit]), part


def plain_ssd(x, B, C, S, A, step):
    """Step sizes of `step` (32 and more is its own softplus) and a gate of 32 (its own silu): results and memory of the
    chunks, and 64-bit ones by rows.  x [T, H, P], B, C [T, G, N], S [H, P, N]."""
    (T, H, P), (G, N) = x.shape, B.shape[1:]
    proj = torch.full((T, H * P + H), 32.0, device=DEV)
    proj[:, H * P:] = step
    state, zero = S.reshape(1, -1).clone(), torch.zeros(H, device=DEV)
    xbc = torch.cat([t.reshape(T, -1) for t in (x, B, C)], 1).contiguous()
    y = ops().ssd_scan(xbc, proj, 0, H * P, zero, A, zero, state, 0, Batch([T], [0]), H, P, N, G, exact=False)
    up = lambda t: t.double().cpu().numpy()  # noqa: E731
    dt = np.full((T, H), step if step >= 32 else np.log1p(np.exp(step)))
    ref, ref_S = ssd_rule(up(x), up(B).repeat(H // G, 1), up(C).repeat(H // G, 1), dt, up(A), np.zeros(H), up(S))
    return y.view(T, H, P), 32 * ref, state.view(H, P, N), ref_S


@pytest.mark.parametrize("N", [16, 24, 64, 100, 128])
@pytest.mark.parametrize("decay", [0.0, 1.0])
def test_sums_that_32_bits_hold_are_exact(N, decay):
    """Small whole numbers and steps of 32: without a decay all sums are whole numbers below 2^24; with one every row
    forgets what was before it (e^-32), which leaves one product an element."""
    H, G, P, T = 4, 2, 64, 200
    g = torch.Generator(device=DEV).manual_seed(N)
    whole = lambda *s: torch.randint(-3, 4, s, generator=g, device=DEV).float()  # noqa: E731
    y, ref, state, ref_S = plain_ssd(whole(T, H, P), whole(T, G, N), whole(T, G, N), whole(H, P, N),
                                     torch.full((H,), -decay, device=DEV), 32.0)
    tiny = 1e-9 if decay else 0.0  # beside what e^-32 leaves of the rows before
    assert np.abs(y.double().cpu().numpy() - ref).max() <= tiny * np.abs(ref).max()
    assert np.abs(state.double().cpu().numpy() - ref_S).max() <= tiny * np.abs(ref_S).max()


@pytest.mark.parametrize("N", [16, 64, 128])
def test_sums_of_one_sign_lean_to_neither_side(N):
    """51,200 results of either rounding: what is off on average is far less than one rounding's 2^-25 of the value, and
    a quarter of that is allowed for what the tensor core cuts off."""
    H, G, P, T = 4, 2, 64, 200
    g = torch.Generator(device=DEV).manual_seed(N)
    pos = lambda *s: torch.rand(s, generator=g, device=DEV)  # noqa: E731
    y, ref, state, ref_S = plain_ssd(pos(T, H, P), pos(T, G, N), pos(T, G, N), pos(H, P, N),
                                     torch.full((H,), -0.25, device=DEV), 0.5)
    for got, want in ((y, ref), (state, ref_S)):
        d = got.double().cpu().numpy() - want
        assert abs(d.sum()) / want.sum() < 3e-8 and np.linalg.norm(d) / np.linalg.norm(want) < 1e-7


def test_a_weight_is_one_exponential(monkeypatch):
    """k and v of unit vectors and q of ones leave every weight on its own in the results, 32 e^(A (dt_s+1 + .. + dt_t)).
    A rounding is off by 2.5e-8 of the value in the mean square, an exponential by a third more; two exponentials and
    their product by 5e-8 (4.8e-8 were measured, 3.4e-8 with one)."""
    monkeypatch.setattr(ops(), "SSD_CHUNK_MIN_ROWS", 1)
    H, T = 16, 64
    g = torch.Generator(device=DEV).manual_seed(3)
    eye = torch.eye(T, device=DEV)
    x, B, C = eye.view(T, 1, T).repeat(1, H, 1), eye.view(T, 1, T), torch.ones((T, 1, T), device=DEV)
    A = -torch.rand(H, generator=g, device=DEV) * 8e-5 - 4e-5  # exponents down to -0.25
    y, ref, _, _ = plain_ssd(x, B, C, torch.zeros((H, T, T), device=DEV), A, 32.0)
    t, s = torch.meshgrid(torch.arange(T), torch.arange(T), indexing="ij")
    apart = (t // 16 > s // 16).numpy()
    d = (y.double().cpu().numpy() / np.where(ref, ref, 1.0) - 1.0).transpose(0, 2, 1)[apart]
    assert np.sqrt((d * d).mean()) < 4e-8


def test_gates_of_all_sizes_as_a_decode_step_has_them(monkeypatch):
    """silu(z) from -inf to inf and where e^-z overflows: the rows of a prompt (the results before the gate are 128
    everywhere) and as many sequences of one row, the same operations on the same numbers."""
    monkeypatch.setattr(ops(), "SSD_CHUNK_MIN_ROWS", 2)
    H, G, P, N, T = 4, 2, 64, 16, 64
    z = torch.cat([torch.linspace(-120, 120, H * P - 6, device=DEV),
                   torch.tensor([-float("inf"), float("inf"), float("nan"), -3e38, 3e38, -0.0], device=DEV)])
    proj = torch.cat([z, torch.full((H,), 32.0, device=DEV)]).repeat(T, 1).contiguous()
    xbc, zero = torch.ones((T, H * P + 2 * G * N), device=DEV), torch.zeros(H, device=DEV)
    xbc[:, H * P:] = 0.5
    forget = torch.full((H,), -64.0, device=DEV)  # e^-2048: a row has no other before it
    pre = []
    for counts in ((T,), (1,) * T):
        b = Batch(counts, range(len(counts)))
        state = torch.zeros((len(counts), H * P * N), device=DEV)
        pre.append(ops().ssd_scan(xbc, proj, 0, H * P, zero, forget, zero, state, 0, b, H, P, N, G, exact=False))
    assert torch.equal(pre[0].isnan(), pre[1].isnan())
    assert torch.equal(pre[0].nan_to_num(7.0), pre[1].nan_to_num(7.0))


def test_memories_that_grow_beyond_32_bits_are_infinite():
    """e^128 a row, positive numbers throughout: infinity, as by rows, and no NaN."""
    H, G, P, N, T = 4, 2, 64, 16, 130
    one = lambda *s: torch.ones(s, device=DEV)  # noqa: E731
    y, _, state, _ = plain_ssd(one(T, H, P), one(T, G, N), one(T, G, N), one(H, P, N), 4.0 * one(H), 32.0)
    assert bool((y == math.inf).all()) and bool((state == math.inf).all())


@pytest.mark.parametrize("N", [24, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 1e30])
def test_numbers_no_part_holds_in_q_and_in_the_memory(N, bad):
    """An element of q reaches its row's results in its group's heads; one of the memory that a sequence comes with its own
    column's; all others keep their bits.  1e30 is finite and counts as it is."""
    H, G, P, T = 4, 2, 64, 200
    g = torch.Generator(device=DEV).manual_seed(11)
    draw = lambda *s: torch.randn(s, generator=g, device=DEV)  # noqa: E731
    x, B, C, S = draw(T, H, P), draw(T, G, N), draw(T, G, N), draw(H, P, N)
    A = torch.full((H,), -0.01, device=DEV)
    y, _, state, _ = plain_ssd(x, B, C, S, A, 0.5)
    for where in ("q", "memory"):
        C2, S2 = C.clone(), S.clone()
        hit, moved = torch.zeros((T, H, P), dtype=torch.bool, device=DEV), torch.zeros((H, P, N), dtype=torch.bool, device=DEV)
        if where == "q":
            C2[70, 1, 3] = bad
            hit[70, 2:] = True
        else:
            S2[1, 5, 7] = bad
            hit[:, 1, 5] = True
            moved[1, 5, 7] = True
        y2, ref, state2, ref_S = plain_ssd(x, B, C2, S2, A, 0.5)
        assert torch.equal(y2[~hit], y[~hit]) and torch.equal(state2[~moved], state[~moved])
        if math.isfinite(bad):
            for got, want in ((y2, ref), (state2, ref_S)):
                assert off(got, want) < TOL
        else:
            assert not y2[hit].isfinite().any() and not state2[moved].isfinite().any()


@pytest.mark.parametrize("huge", [3.3895e38, 3.395e38])  # bfloat16's largest number holds the first, not the second
@pytest.mark.parametrize("N", [24, 128])
def test_numbers_beyond_bfloat16s_range_count_as_they_are(huge, N):
    """One element of v near the end of 32 bits' range, with k and q small enough for finite results."""
    heads, groups, P, T = 4, 1, 64, 200
    g = torch.Generator(device=DEV).manual_seed(5)
    inner, b = heads * P, Batch([T], [0])
    xbc = torch.randn((T, inner + 2 * groups * N), generator=g, device=DEV)
    xbc[:, inner:] *= 1e-3
    proj = torch.randn((T, inner + heads), generator=g, device=DEV)
    A, D, bias = -torch.ones(heads, device=DEV), torch.zeros(heads, device=DEV), torch.zeros(heads, device=DEV)

    def ssd(x):
        state = torch.zeros((1, heads * P * N), device=DEV)
        return ops().ssd_scan(x, proj, 0, inner, bias, A, D, state, 0, b, heads, P, N, groups, exact=False), state

    clean, clean_state = ssd(xbc)
    xbc[70, P + 5] = huge
    y, state = ssd(xbc)
    hit = torch.zeros(inner, dtype=torch.bool, device=DEV)
    hit[P + 5] = True
    assert torch.equal(y[:70], clean[:70]) and torch.equal(y[:, ~hit], clean[:, ~hit])
    assert torch.equal(state.view(inner, N)[~hit], clean_state.view(inner, N)[~hit])
    x64, p64 = xbc.double().cpu().numpy(), proj.double().cpu().numpy()
    dt = np.log1p(np.exp(p64[:, inner:]))
    B, C = (x64[:, o:o + N].reshape(T, 1, N).repeat(heads, 1) for o in (inner, inner + N))
    ref, S = ssd_rule(x64[:, :inner].reshape(T, heads, P), B, C, dt, -np.ones(heads), np.zeros(heads), np.zeros((heads, P, N)))
    z = p64[:, P + 5]
    assert off(y[:, P + 5], ref[:, 1, 5] * z / (1 + np.exp(-z))) < TOL
    assert off(state.view(heads, P, N)[1, 5], S[1, 5]) < TOL
