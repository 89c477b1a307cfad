"""The serving loop's bound on a file's memory needs no GPU: layouts from the header alone, a
frequency table in place of the header's band, both orders of the band."""
import numpy as np

from astroflow_b200.serve import workspace_bound


def bound(fch1=1000.0, foff=0.125, n=1 << 17, c=4096, bits=8, ndm=6001, **kw):
    return workspace_bound(n, c, bits, 4.9e-5, fch1, foff, ndm, dict(dm_low=0.0, dm_high=3000.0, dm_step=0.5, **kw))


def test_folded_chunks_count_words_up_to_the_largest_delay():
    # 4096 channels x (a quarter of the chunk and 141,000 samples of delay, at most the chunk)
    assert bound() > 4096 * 4 * (1 << 17)
    short = bound(n=1 << 20)
    assert 4096 * 4 * ((1 << 18) + 140000) < short - (2 << 30) < 4096 * 4 * ((1 << 18) + 200000)


def test_frequency_tables_and_descending_bands():
    table = 1000.0 + 0.125 * np.arange(4096)
    assert bound(fch1=0.0, foff=0.0, freq_table=table) == bound(fch1=1000.0 + 0.125 * 4095, foff=-0.125)
    assert bound(fch1=0.0, foff=0.0) > 0  # no band at all: the plan itself refuses it


def test_small_files_reserve_little():
    assert bound(n=2000, c=64, ndm=50) < 200 << 20
