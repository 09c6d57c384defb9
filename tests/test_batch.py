"""The step's descriptors on the host: packing, field alignment, the decode
context bucket, and the decode split choice (pure arithmetic, no GPU)."""

from reflex_b200.engine.batch import decode_context_bucket, layout, pack_host


def test_pack_host_lays_out_rows_and_wanted_places():
    tokens = [[5, 6, 7], [9], [1, 2]]
    words, offs, new_counts, row0, want_rows = pack_host(tokens, [4, 0, 2], [10, 0, 63], [[0, 2], [], [1]])
    assert new_counts == [3, 1, 2] and row0 == [0, 3, 4, 6] and want_rows == [0, 2, 5]

    def field(name):
        p, n = offs[name]
        return words[p:p + n].tolist()

    assert field("tokens") == [5, 6, 7, 9, 1, 2]
    assert field("row_pos") == [10, 11, 12, 0, 63, 64]
    assert field("row_slot") == [4, 4, 4, 0, 2, 2]
    assert field("seq_slot") == [4, 0, 2] and field("seq_start") == [10, 0, 63]
    assert field("seq_new") == [3, 1, 2] and field("seq_row0") == [0, 3, 4, 6]
    assert field("want_rows") == [0, 2, 5]
    # every field starts on 16 bytes (kernels read them with wide loads; TMA needs it)
    assert all(p % 4 == 0 for p, _ in offs.values())
    assert len(words) == layout(6, 3, 3)[1]


def test_decode_context_bucket_rounds_up_and_never_down():
    last = 0
    for ctx in range(1, 70000, 37):
        b = decode_context_bucket(ctx)
        assert b >= ctx and b % 64 == 0 and b >= last
        last = b
    assert decode_context_bucket(1) == 256 and decode_context_bucket(256) == 256
    assert decode_context_bucket(257) == 512 and decode_context_bucket(2048) == 2048
    assert decode_context_bucket(2049) == 4096 and decode_context_bucket(4097) == 8192


def test_decode_splits_grow_with_context_and_shrink_with_batch():
    from reflex_b200.ops import decode_splits

    for rows in (1, 8, 64):
        picks = [decode_splits(rows, 32, 8, pages) for pages in (1, 4, 16, 64, 256)]
        assert picks == sorted(picks) and picks[0] == 1
    for pages in (12, 64, 256):
        picks = [decode_splits(rows, 32, 8, pages) for rows in (1, 8, 64, 256)]
        assert picks == sorted(picks, reverse=True)
        assert all(1 <= s <= 64 and s <= pages for s in picks)


def test_which_batches_give_the_32_bit_attention_an_sm_a_block():
    """The work in blocks as long as the longest: half of a new prompt's blocks, nearly all of a continued one's; nothing
    where blocks do not differ in length or the host does not say."""
    from types import SimpleNamespace as B

    from reflex_b200.ops import _longest_blocks as f

    assert f(B(new_counts=[512], starts=[0]), 8, 2, None) == 128
    assert 200 < f(B(new_counts=[512], starts=[800]), 8, 2, None) < 256
    assert 140 < f(B(new_counts=[155, 311, 235], starts=[0, 0, 0]), 8, 2, None) < 151
    assert f(B(new_counts=[64], starts=[0]), 40, 2, 64) == 2 * 2 * 32  # two heads' blocks of sixteen and four, a row each
    for b, window in ((B(new_counts=[1] * 64, starts=[1000] * 64), None), (B(new_counts=[4, 4], starts=[0, 9]), None),
                      (B(new_counts=[512], starts=[0]), 100), (B(), None), (B(new_counts=[], starts=[]), None)):
        assert f(b, 8, 2, window) == 0
    assert f(B(new_counts=[512], starts=[0]), 8, 3, None) == 0 and f(B(new_counts=[512], starts=[0]), 8, 0, None) == 0
