"""A decode step of the selective scan in one launch (csrc/mamba_step.cu) against the launches it
stands for, several steps one after another in slots that are not in order.

Both round the filtered row and the low-rank vector to bfloat16; their 32-bit sums differ in order, so
a rounding may fall the other way now and then (2^-8 of one of `rank` terms)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from reflex_b200 import ops as o

    return o


class Batch:
    def __init__(self, slots):
        self.row_slot = self.seq_slot = torch.tensor(slots, dtype=torch.int32, device=DEV)
        self.seq_row0 = torch.arange(len(slots) + 1, dtype=torch.int32, device=DEV)
        self.max_new = 1


class Ctx:
    pass


@pytest.mark.parametrize("C,N,rank,taps,taken", [(512, 16, 8, 4, True), (1024, 4, 64, 2, True), (3072, 32, 96, 4, True),
                                                 (2048, 16, 64, 1, True), (8192, 16, 256, 4, False), (520, 16, 8, 4, False),
                                                 (1024, 12, 8, 4, False)])
@pytest.mark.parametrize("rows", [1, 3, 8])
def test_a_step_in_one_launch(C, N, rank, taps, taken, rows, monkeypatch):
    from reflex_b200.config.spec import MixerSpec
    from reflex_b200.parts.selective_scan import SelectiveScan

    W, dt = 64, torch.bfloat16
    g = torch.Generator(device=DEV).manual_seed(C + N + rows)
    spec = MixerSpec("selective_scan", W, params=(("inner", C), ("state", N), ("dt_rank", rank), ("taps", taps)))
    part = SelectiveScan(spec, dt, DEV)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)  # noqa: E731
    part.bind({"in_proj": rnd(2 * C, W) * 0.1, "conv": rnd(C, taps) * 0.4, "conv_bias": rnd(C) * 0.2,
               "x_proj": rnd(rank + 2 * N, C) * 0.03, "dt_proj": rnd(C, rank) * 0.1, "dt_bias": rnd(C) * 0.3,
               "A_log": rnd(C, N) * 0.3, "D": rnd(C), "o_proj": rnd(W, C) * 0.03})
    slots = [5, 0, 3, 8, 1, 7, 2, 6][:rows]
    states = [rnd(9, (taps - 1) * C + C * N) for _ in range(1)] * 2
    states = [states[0].clone(), states[0].clone()]
    start = states[0].clone()
    calls = []
    whole = ops().mamba_step
    monkeypatch.setattr(ops(), "mamba_step", lambda *a: calls.append(whole(*a)) or calls[-1])
    for _ in range(3):
        x = rnd(rows, W).to(dt)
        outs = []
        for limit, state in zip((8, 0), states):
            monkeypatch.setattr(ops(), "MAMBA_STEP_MAX_ROWS", limit)
            ctx = Ctx()
            ctx.batch, ctx.state = Batch(slots), state
            outs.append(part.forward(x, ctx).double())
        assert (calls[-2] is not None) == taken and calls[-1] is None
        assert ((outs[0] - outs[1]).norm() / outs[1].norm()).item() < 4e-3
        n = (taps - 1) * C
        assert torch.equal(states[0][:, :n], states[1][:, :n])
        a, b = states[0][slots, n:].double(), states[1][slots, n:].double()
        assert ((a - b).norm() / b.norm()).item() < 1e-3
    idle = [s for s in range(9) if s not in slots]
    assert torch.equal(states[0][idle], start[idle])
