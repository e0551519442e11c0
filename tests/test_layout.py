"""Sizes of datasets: from the ln n! table on, a dataset holds at least the 131072 entries that the
genotype-split search could look up by two 16-bit counts, whatever the counts (a bounded wait that expires can
leave wrong ones); larger datasets are no larger for it."""
import epik2


def test_the_table_can_be_read_for_any_two_16_bit_counts():
    L = epik2.library()
    for s, m in ((1, 1), (100, 3), (2048, 128), (800, 70), (131070, 3)):
        assert L.epik2_replicate_bytes(s, m) >= 4 * 131072
        assert epik2.dataset_bytes(s, m) >= s * m + 4 * 131072


def test_larger_datasets_hold_their_buffers_only():
    s, m = 16384, 4096
    pad = lambda n: -(-n // 256) * 256
    parts = [s * m, 4 * (s + 2), 4 * s, 8 * (s // 32 + 1) * m, 16 * m, 16 * 2 * (m * (m - 1) // 2), 8 * (s + 2)]
    assert epik2.dataset_bytes(s, m) == sum(pad(n) for n in parts)
