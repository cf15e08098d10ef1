"""How decode attention shares a sequence's keys among CTAs: the rule on the host."""
import itertools

from idrak_b200.ops.decode import DECODE_CTAS, DECODE_TILE, key_shares


def test_shares_are_bounded():
    for seqs, kv_heads, longest, window, sms in itertools.product(
            (1, 2, 7, 16, 64, 150, 256, 1000, 3000), (1, 3, 8, 32),
            (0, 1, 127, 128, 129, 256, 257, 1024, 4096, 32768, 131072, 1 << 20), (0, 1, 300, 4096), (148, 20)):
        splits, min_keys = key_shares(seqs, kv_heads, longest, window, sms)
        heads, span = seqs * kv_heads, min(longest, window + DECODE_TILE) if window else longest
        assert 1 <= splits <= 64 and min_keys % 128 == 0 and 128 <= min_keys <= 4096
        assert splits == 1 or heads * splits <= DECODE_CTAS                   # partial results and launched CTAs
        assert (splits - 1) * min_keys < max(span, 1)                         # no share that even the longest leaves empty
        if 1 < splits and heads <= sms // 4 and span <= 8192:
            assert heads * splits <= 3 * sms                                  # all there together


def test_large_batches_and_windows():
    assert key_shares(256, 8, 32768) == (8, 2048)                             # 136 MB of partial results without the bound
    assert key_shares(64, 8, 4096) == (4, 1024) and key_shares(1, 8, 512) == (4, 128)
    assert key_shares(1, 8, 32768, 256) == (3, 128)                           # 288 keys, whatever the bound on the length
    assert key_shares(200, 2, 512) == (1, 1024) and key_shares(16, 8, 4096) == (8, 512)
