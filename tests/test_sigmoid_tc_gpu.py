"""Attention with sigmoid weights on the tcgen05 kernel (csrc/attention_prefill_tc.cu) against its rule in 64 bits.

Tolerance, of the largest result: a weight is rounded to bfloat16 (2^-9 of it) and so is the result, as in the
mma.sync form, whose bound stands beside its own test: 1.5e-2."""

import math

import pytest
import torch
from test_kegasun_gpu import FakeBatch, ops, relerr
from test_zelinex_gpu import _paged_kv, _sigmoid_ref, f32

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def call(fn, q, kp, vp, table, b, nq, nkv, d, window, scale, bias):
    return fn(q, kp, vp, table, 64, b.seq_slot, b.seq_start, b.seq_new, b.seq_row0, b.max_new, nq, nkv, d, window, scale,
              bias)


def batch_of(seqs, slots):
    b = FakeBatch([[0] * n for _, n in seqs], slots, [s for s, _ in seqs])
    b.max_new, b.max_context = max(n for _, n in seqs), max(s + n for s, n in seqs)
    b.is_decode = b.max_new == 1
    return b


@pytest.mark.parametrize("nq,nkv,d,seqs,window", [
    (4, 2, 64, [(0, 70), (130, 3), (0, 1)], 20),
    (2, 1, 64, [(0, 200), (63, 2), (133, 3)], 70),          # portions after earlier rows
    (6, 2, 128, [(0, 300), (328, 4)], 150),                 # three heads: no divisor of a tile's 128 rows
    (7, 1, 64, [(0, 129), (64, 65)], 64),                   # seven; a window of a page
    (8, 2, 128, [(200, 40), (500, 1), (63, 1), (0, 90)], 33),  # decode rows beside prompts
    (3, 3, 128, [(0, 140)], 128),
    (12, 3, 64, [(0, 260), (5, 1)], None),                  # every earlier key
    (6, 1, 128, [(0, 5), (64, 1), (127, 2)], 1),            # the token itself alone
    (16, 1, 64, [(500, 1), (63, 1), (64, 1), (0, 2)], 200),
    (1, 1, 128, [(1, 127), (0, 64), (63, 65)], None),
])
@pytest.mark.parametrize("with_bias", [True, False])
def test_against_the_rule(nq, nkv, d, seqs, window, with_bias):
    """Pages scattered, NaN in every row that no sequence has; a bias of its own for each head."""
    g = torch.Generator().manual_seed(nq * 100 + d)
    slots, table, kp, vp, ks, vs = _paged_kv([s + n for s, n in seqs], nkv, d, d, torch.bfloat16, g)
    R = sum(n for _, n in seqs)
    q = torch.randn(R, nq, d, generator=g)
    bias = (torch.randn(nq, generator=g) * 2 - 1).double() * (1 if with_bias else 0)
    scale = 1.5 / math.sqrt(d)
    ref = _sigmoid_ref(q, ks, vs, seqs, scale, window, bias.numpy(), torch.bfloat16)
    out = call(ops().attention_sigmoid_tc, q.bfloat16().reshape(R, nq * d).to(DEV), kp.to(DEV), vp.to(DEV), table.to(DEV),
               batch_of(seqs, slots), nq, nkv, d, window, scale, f32(bias) if with_bias else None)
    assert relerr(out.reshape(R, nq, d), ref) < 1.5e-2
    ops().check_device_errors(DEV)


@pytest.mark.parametrize("d", [64, 128])
def test_a_key_that_stands_out_just_inside_and_just_outside_the_window(d):
    """Every key weighs next to nothing (a bias of -12) but one, at position 100: a window that is one token off
    shows as a whole value."""
    nq, nkv, window, T = 4, 2, 77, 260
    g = torch.Generator().manual_seed(9)
    k, v = torch.randn(T, nkv, d, generator=g) * 0.05, torch.randn(T, nkv, d, generator=g)
    k[100], v[100] = 0.0, 50.0
    k[100, :, 3] = 8.0
    q = torch.randn(T, nq, d, generator=g) * 0.05
    q[:, :, 3] = 4.0
    pages = (T + 63) // 64
    kp, vp = torch.zeros(pages, nkv, 64, d), torch.zeros(pages, nkv, 64, d)
    for p in range(T):
        kp[p // 64, :, p % 64], vp[p // 64, :, p % 64] = k[p], v[p]
    table = torch.arange(pages, dtype=torch.int32, device=DEV).reshape(1, pages)
    out = call(ops().attention_sigmoid_tc, q.bfloat16().reshape(T, nq * d).to(DEV), kp.bfloat16().to(DEV),
               vp.bfloat16().to(DEV), table, batch_of([(0, T)], [0]), nq, nkv, d, window, 1.0, f32([-12.0] * nq))
    biggest = out.float().abs().amax(1).tolist()
    for i, m in enumerate(biggest):
        inside = 100 <= i <= 100 + window - 1
        assert (m > 45.0) == inside and (inside or m < 1.0), (i, m)


def test_a_step_the_kernel_refuses_goes_to_the_other_form(monkeypatch):
    g = torch.Generator().manual_seed(3)
    seqs, nq, nkv, d = [(0, 70)], 4, 2, 64
    slots, table, kp, vp, _, _ = _paged_kv([70], nkv, d, d, torch.bfloat16, g)
    q, b = torch.randn(70, nq * d, generator=g).bfloat16().to(DEV), batch_of(seqs, slots)
    kp, vp, table, lib = kp.to(DEV), vp.to(DEV), table.to(DEV), ops().native.lib()

    class Refuses:
        def __getattr__(self, name):
            return (lambda *a: ops().native.ERR_UNSUPPORTED) if name == "rfx_attention_sigmoid_tc" else getattr(lib, name)

    monkeypatch.setattr(ops().native, "lib", Refuses)
    got = ops().attention_sigmoid(q, kp, vp, table, 64, b, nq, nkv, d, d, 40, 0.125, None)
    bias = torch.zeros(nq, device=DEV)
    assert torch.equal(got, ops().attention_sigmoid_mma(q, kp, vp, table, 64, b.seq_slot, b.seq_start, b.seq_new, b.seq_row0,
                                                        b.max_new, nq, nkv, d, d, 40, 0.125, bias))
