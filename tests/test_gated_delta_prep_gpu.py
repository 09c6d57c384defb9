"""The products between a chunk's rows of the gated delta rule (csrc/gated_delta_chunk.cu) against 64 bits.

Bound, 2-norm: sums of sixteen 32-bit multiply-adds, eight of them added up, some 1e-7; the decays' products and the
substitution add as much again.  Products of operands rounded to 22 bits are 1e-6 off."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
CH, TLD, COEF = 16, 24, 2 * 16 * 24 + 2 * 16 + 4


@pytest.mark.parametrize("H,G,d", [(4, 2, 128), (2, 2, 64), (9, 1, 40), (2, 1, 256), (1, 1, 4)])
@pytest.mark.parametrize("counts", [(16,), (33, 1, 47)])
def test_chunk_coefficients(H, G, d, counts):
    from reflex_b200 import ops

    rng = np.random.default_rng(H + d + len(counts))
    dv, R, S = 16, sum(counts), len(counts)
    qkv = rng.standard_normal((R, 2 * G * d + H * dv)).astype(np.float32)
    qkv[:, :2 * G * d] /= np.sqrt(d)
    gates = np.concatenate([np.exp(-rng.uniform(0, 1, (R, H))), rng.uniform(0, 1, (R, H))], 1).astype(np.float32)
    row0 = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    to = lambda a: torch.from_numpy(a).to(DEV)  # noqa: E731
    lib = ops.native.lib()
    coef = torch.zeros(int(lib.rfx_gated_delta_chunk_floats(R, S, H)), device=DEV)
    x, g, r0 = to(qkv), to(gates), to(row0)
    st = lib.rfx_gated_delta_chunk_prep(x.data_ptr(), g.data_ptr(), r0.data_ptr(), S, coef.data_ptr(), H, G, d, dv,
                                        max(counts), ops._stream())
    assert st == 0
    got = coef.double().cpu().numpy().reshape(-1, H, COEF)
    q, k = (qkv[:, o * G * d:(o + 1) * G * d].astype(np.float64).reshape(R, G, d) for o in (0, 1))
    for s, n in enumerate(counts):
        for c in range((n + CH - 1) // CH):
            rows = slice(row0[s] + c * CH, row0[s] + min(n, (c + 1) * CH))
            m = rows.stop - rows.start
            for h in range(H):
                decay, beta = gates[rows, h].astype(np.float64), gates[rows, H + h].astype(np.float64)
                run = np.cumprod(decay)
                ratio = np.tril(run[:, None] / run[None, :])
                kk, qk = (a[rows, h // (H // G)] @ k[rows, h // (H // G)].T for a in (k, q))
                T = np.linalg.solve(np.eye(m) + beta[:, None] * np.tril(ratio * kk, -1), np.diag(beta))
                place = got[row0[s] // CH + s + c, h]
                for at, ref in ((0, T), (CH * TLD, ratio * qk)):
                    have = place[at:at + CH * TLD].reshape(CH, TLD)[:m, :m]
                    assert np.linalg.norm(have - ref) / np.linalg.norm(ref) < 5e-7
                assert np.abs(place[2 * CH * TLD:2 * CH * TLD + m] / run - 1).max() < 2e-6
