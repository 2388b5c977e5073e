"""The wave schedules that renderers take: mlpsp_wave_schedule covers every list, engine.WaveSchedule keeps doing so."""
import itertools

import numpy as np
import pytest

from mlp_splatting_b200 import _lib as L
from mlp_splatting_b200.engine import WaveSchedule

SIZES = [(1, 1), (128, 96), (173, 174), (320, 240), (957, 541), (1920, 1080)]


@pytest.mark.parametrize("hidden, precision, views, caller_lists", [(32, 1, 1, False), (64, 1, 4, False), (32, 0, 1, True)])
@pytest.mark.parametrize("capacity", [1, 40, 1536, 2560])
def test_every_schedule_reaches_the_end_of_the_lists(hidden, precision, views, caller_lists, capacity):
    for size, n in itertools.product(SIZES, (0, 1, 2_000, 500_000)):
        _walk(size, n, hidden, precision, views, caller_lists, capacity)


def _walk(size, n, hidden, precision, views, caller_lists, capacity):
    s = WaveSchedule(*size, capacity, views)
    words = np.zeros(L.STATUS_WORDS, np.int32)

    def check():
        given, _ = s.get(n, hidden, precision, caller_lists)
        assert 1 <= len(given) <= L.MAX_WAVES and all(1 <= w for w in given)
        # the last window is stretched to the capacity and, like every window, holds at most 2,048 candidates
        before = sum(given[:-1])
        assert before < capacity and capacity - before <= 2048 and max(given[:-1], default=1) <= 2048
        return list(given)

    first = check()
    assert sum(first) == capacity
    for used, tiles, longest in itertools.product(range(0, len(first) + 1), (0, 1, 10_000), (1, capacity)):
        words[L.ST_WAVES], words[L.ST_LAST_TILES], words[L.ST_MAX_TILE_LEN] = min(used, len(s.given)), tiles, longest
        s.adapt(words)
        check()


def test_a_frame_that_goes_further_brings_the_full_schedule_back():
    s = WaveSchedule(1200, 680, 1536)
    full = list(s.get(100_000, 32, 1)[0])
    words = np.zeros(L.STATUS_WORDS, np.int32)

    def frame(used, tiles):
        words[L.ST_WAVES], words[L.ST_LAST_TILES], words[L.ST_MAX_TILE_LEN] = used, tiles, 1200
        s.adapt(words)
        return s.get(100_000, 32, 1)

    assert frame(2, 9_000) == (full[:2] + [1536], True)       # most tiles came to the second wave: it stays a wave of its own
    assert frame(2, 9_000) == (full[:2] + [1536], True)
    assert frame(2, 3) == (full[:1] + [1536], False)          # three tiles: the second wave takes the rest of their lists
    assert frame(2, 3) == (full[:1] + [1536], False)
    assert frame(2, 9_000) == (full, False)
    assert frame(len(full), 9_000) == (full, False)
    assert s.get(100_001, 32, 1) == (full, False)             # another scene starts over
