"""The experts' products for a few rows (csrc/moe_gemm.cu) against 64-bit formulas.

Inputs are bfloat16 exactly; sums are 32-bit (K 2^-24 of the terms' size at worst), the activation is
rounded to bfloat16 once before the second product (2^-9 each, averaged over the sum)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from reflex_b200 import ops as o

    return o


def act64(kind, g, u):
    if kind == "relu2":
        return g.clamp(min=0) ** 2
    if kind == "silu":
        return g * torch.sigmoid(g)
    if kind == "swiglu":
        return g * torch.sigmoid(g) * u
    g, u = g.clamp(max=0.7), u.clamp(-0.7, 0.7)
    return g * torch.sigmoid(1.5 * g) * (u + 1)


def check(x, up, down, ids, wts, kind, by_input, placed, bound=3e-3):
    R, ff, gated = x.shape[0], down.shape[2], kind in ("glu_clamped", "swiglu")
    got = ops().moe_experts(x, up, down, ids, wts, activation=kind, weight_input=by_input, alpha=1.5, limit=0.7,
                            placed=placed)
    ref = torch.zeros(x.shape, dtype=torch.float64, device=DEV)
    for r in range(R):
        for k in range(ids.shape[1]):
            e, w = int(ids[r, k]), wts[r, k].double()
            row = (x[r].float() * wts[r, k]).bfloat16().double() if by_input else x[r].double()
            h = up[e].double() @ row
            y = down[e].double() @ act64(kind, h[:ff], h[ff:] if gated else None)
            ref[r] += y if by_input else w * y
    assert ((got - ref).norm() / ref.norm()).item() < bound  # 2^-9 = 2e-3 an activation, uniform: 1.1e-3 rms


def weights(g, E, width, ff, kind):
    gated = kind in ("glu_clamped", "swiglu")
    up = (torch.randn((E, ff * (2 if gated else 1), width), generator=g, device=DEV) * 0.1).bfloat16()
    return up, (torch.randn((E, width, ff), generator=g, device=DEV) * 0.1).bfloat16()


@pytest.mark.parametrize("kind", ["relu2", "silu", "glu_clamped", "swiglu"])
@pytest.mark.parametrize("R,E,top,width,ff", [(2, 8, 1, 64, 8), (5, 3, 2, 40, 72), (16, 16, 4, 136, 200),
                                              (17, 4, 3, 264, 128), (33, 40, 2, 128, 64), (64, 2, 2, 512, 136)])
def test_a_few_rows_through_their_experts(R, E, top, width, ff, kind):
    g = torch.Generator(device=DEV).manual_seed(R + E)
    x = torch.randn((R, width), generator=g, device=DEV).bfloat16()
    up, down = weights(g, E, width, ff, kind)
    # the first expert is never chosen where there are others enough
    scores = torch.randn((R, E), generator=g, device=DEV)
    if E > top:
        scores[:, 0] = -100.0
    ids, wts, placed = ops().moe_route(scores, None, top, place=True)
    for by_input in (False, True):
        check(x, up, down, ids, wts, kind, by_input, placed)
    ops().check_device_errors(DEV)


@pytest.mark.parametrize("kind", ["relu2", "swiglu"])
@pytest.mark.parametrize("R,E,top,width,ff", [(9, 3, 4, 712, 200), (20, 2, 3, 136, 72), (40, 5, 3, 264, 136),
                                              (64, 3, 4, 64, 520)])
def test_rows_that_name_an_expert_several_times(R, E, top, width, ff, kind):
    """Expert 1 has R top rows or nearly so: more than the boxes of 16, 32 or 64 that R alone would ask for."""
    g = torch.Generator(device=DEV).manual_seed(R + E)
    x = torch.randn((R, width), generator=g, device=DEV).bfloat16()
    up, down = weights(g, E, width, ff, kind)
    ids = torch.ones((R, top), dtype=torch.int32, device=DEV)
    ids[R // 2, 0] = 0
    wts = torch.rand((R, top), generator=g, device=DEV)
    check(x, up, down, ids, wts, kind, False, None)
    ops().check_device_errors(DEV)


@pytest.mark.parametrize("why", ["off 16 bytes", "not contiguous", "refused"])
def test_experts_the_kernel_does_not_take_go_through_the_library(why, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(7)
    R, E, top, width, ff = 6, 4, 2, 64, 72
    x = torch.randn((R, width), generator=g, device=DEV).bfloat16()
    up, down = weights(g, E, width, ff, "swiglu")
    ids, wts, placed = ops().moe_route(torch.randn((R, E), generator=g, device=DEV), None, top, place=True)
    monkeypatch.setattr(ops(), "_GROUPED_MM", [False, False])  # one library product an expert: takes any operands
    if why == "off 16 bytes":
        down = torch.empty(down.numel() + 1, dtype=down.dtype, device=DEV)[1:].view(down.shape).copy_(down)
    elif why == "not contiguous":
        wide = torch.empty((E, 2 * ff, width + 8), dtype=up.dtype, device=DEV)
        wide[:, :, :width] = up
        up = wide[:, :, :width]
    else:
        lib = ops().native.lib()

        class Refuses:
            def __getattr__(self, name):
                return (lambda *a: ops().native.ERR_UNSUPPORTED) if name == "rfx_moe_gemm" else getattr(lib, name)

        monkeypatch.setattr(ops().native, "lib", Refuses)
    # the library's up product is rounded to bfloat16 too: gate, up and activation, at most 2^-9 each
    check(x, up, down, ids, wts, "swiglu", False, placed, bound=6e-3)


def test_a_captured_step_of_experts_off_16_bytes_waits_for_nobody(monkeypatch):
    """Without a grouped product that takes them, a captured step is the one expert a row form."""
    g = torch.Generator(device=DEV).manual_seed(8)
    R, E, top, width, ff = 4, 4, 2, 64, 40
    x = torch.randn((R, width), generator=g, device=DEV).bfloat16()
    up, down = weights(g, E, width, ff, "silu")
    up = torch.empty(up.numel() + 4, dtype=up.dtype, device=DEV)[4:].view(up.shape).copy_(up)
    assert up.data_ptr() % 16 == 8
    ids, wts = ops().moe_route(torch.randn((R, E), generator=g, device=DEV), None, top)
    monkeypatch.setattr(ops(), "_GROUPED_MM", [False, False])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops().moe_experts(x, up, down, ids, wts, activation="silu")
    graph.replay()
    eager = ops().moe_experts(x, up, down, ids, wts, activation="silu")
    assert ((out - eager).norm() / eager.norm()).item() < 5e-3
