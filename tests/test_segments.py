"""Segments of the executors that march (csrc/segments.h), against a search over every number of segments.  No GPU needed."""
import random
import time

from tile_fusion_b200 import _lib


def _cost(n, columns, resident, lead, length):
    segs = -(-n // length)
    return -(-columns * segs // resident) * (length + lead)


def test_no_better_number_of_segments(built_lib):
    L = _lib.lib()
    rng = random.Random(1)
    for _ in range(1000):
        n, columns, resident = rng.randint(1, 700), rng.choice((1, 2, 3, 7, 40, 5000)), rng.choice((1, 5, 148, 296, 1776))
        for lead, least in ((3, 1), (4, 4)):
            lens = [n] + [-(-n // k) for k in range(2, n + 1) if -(-n // k) >= least]
            got = L.tf_segment_preview(n, columns, resident, lead, least)
            assert got in lens
            assert _cost(n, columns, resident, lead, got) == min(_cost(n, columns, resident, lead, x) for x in lens)


def test_search_is_short(built_lib):
    """It runs in front of every launch: a thin band of 2^31 rows, lines by the million, a single worker."""
    L = _lib.lib()
    t = time.perf_counter()
    for n, columns, resident in ((1 << 25, 1, 296), (1 << 25, 8, 148), (5_000_000, 37, 1184), (5_000_000, 1, 1), (1 << 25, 1, 1 << 25)):
        for lead, least in ((3, 1), (4, 4)):
            assert 1 <= L.tf_segment_preview(n, columns, resident, lead, least) <= n
    assert time.perf_counter() - t < 0.01
