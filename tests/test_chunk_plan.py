"""The scratch of the chunked recurrences (csrc/chunk_plan.cuh): about 256 MB at most whatever the lengths, never
more than all chunks at once take, nothing for a step without rows."""

import pytest

BUDGET = 64 << 20  # floats


def sizes():
    from reflex_b200.ops import native

    lib = native.lib()
    return [(64, lambda R, S, m: lib.rfx_ssd_chunk_floats(R, S, m, 32, 64, 128)),
            (64, lambda R, S, m: lib.rfx_mlstm_chunks_floats(R, S, m, 16, 128, 256)),
            (32, lambda R, S, m: lib.rfx_delta_rule_chunk_floats(R, S, m, 64))]


@pytest.mark.parametrize("lengths", [[17], [2048], [100000], [500] * 100, [4000] + [64] * 63, [5000, 70], [1] * 3000,
                                     [65] * 1000 + [9000], [200000, 1, 1, 64]])
def test_bounded_and_never_more_than_one_round(lengths):
    R, S, most = sum(lengths), len(lengths), max(lengths)
    for L, floats in sizes():
        one = floats(1, 1, 1)  # a chunk's
        assert 0 < floats(R, S, most) <= min(max(BUDGET, one), (R // L + S) * one)
        assert floats(R, S, most) == (R // L + S) * one or floats(R, S, most) > BUDGET // 3  # rounds use what they may


def test_nothing_for_a_step_without_rows():
    for _, floats in sizes():
        assert floats(0, 1, 0) == floats(0, 0, 0) == floats(0, 2, 64) == floats(10, 0, 10) == 0
