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


def _words(waves=1, evaluated=0, composited=0, kept=0, tiles=0, longest=1536):
    w = np.zeros(L.STATUS_WORDS, np.int32)
    w[L.ST_WAVES], w[L.ST_LAST_TILES], w[L.ST_MAX_TILE_LEN], w[L.ST_PAIRS_KEPT] = waves, tiles, longest, kept
    for word, v in ((L.ST_RECORDS_LO, evaluated), (L.ST_USED_LO, composited)):
        w[word:word + 2] = np.array([v], np.uint64).view(np.int32)
    return w


@pytest.mark.parametrize("kinds", [[(2_000, 32, 1, False), (2_000, 32, 1, True)],          # own and given lists
                                   [(100_000, 32, 1, False), (100_000, 32, 0, False)],     # binary16 and its FP32 fallback
                                   [(100_000, 32, 1, False), (3_000, 64, 1, False)]])      # two scenes
def test_calls_of_two_kinds_keep_what_each_has_learned(kinds):
    s = WaveSchedule(640, 480, 1536)
    learned = []
    for kind in kinds:
        full = list(s.get(*kind)[0])
        s.adapt(_words(waves=2, tiles=5_000))
        assert s.get(*kind) == (full[:2] + [1536], True)
        learned.append(s.get(*kind))
    for _ in range(3):
        for kind, want in zip(kinds, learned):
            assert s.get(*kind) == want
    # a few more primitives, the same windows: the same kind
    assert s.get(kinds[-1][0] + 3, *kinds[-1][1:]) == learned[-1]


def test_the_number_of_kinds_is_bounded():
    s = WaveSchedule(640, 480, 1536)
    for n in range(1_000, 400_000, 700):
        s.get(n, 32, n % 2)
    assert len(s._kinds) <= s.KINDS and len(s._calls) <= 4 * s.KINDS


@pytest.mark.parametrize("precision, vain", [(1, 1_500_000), (0, 400_000)])
def test_deep_overlap_gets_shorter_windows_and_gives_them_back(precision, vain):
    s = WaveSchedule(140, 100, 1536)
    one = list(s.get(3_000, 32, precision)[0])
    assert one == [1536]
    s.adapt(_words(evaluated=200_000 + vain, composited=200_000, kept=30_000))
    several = list(s.get(3_000, 32, precision)[0])
    assert len(several) > 1 and several[0] < 512 and sum(several) >= 1536
    sizes = [several[0]]
    for _ in range(8):              # and shorter yet while that is not enough, down to 32
        s.adapt(_words(waves=2, evaluated=200_000 + vain, composited=200_000, kept=30_000))
        given, _ = s.get(3_000, 32, precision)
        assert sum(given) >= 1536 and 1536 - sum(given[:-1]) <= 2048
        sizes.append(s.default[0])
    assert sizes[-1] == 32 and all(b <= a for a, b in zip(sizes, sizes[1:]))
    for _ in range(8):              # little in vain: longer again, but not one window while the lists could fill it
        s.adapt(_words(waves=2, evaluated=210_000, composited=200_000, kept=30_000))
    assert s.default == several
    s.adapt(_words(waves=2, evaluated=210_000, composited=200_000, kept=7_000))
    assert s.get(3_000, 32, precision) == (one, False)


def test_windows_that_help_are_kept():
    s = WaveSchedule(200, 150, 1536)
    assert s.get(1_500, 32, 1)[0] == [1536]
    vain = {0: 2_100_000, 1: 900_000, 2: 290_000}       # by how often the windows were halved: each is a third of the last
    seen = []
    for _ in range(12):
        level = s._now.level
        seen.append(level)
        s.adapt(_words(waves=3, evaluated=700_000 + vain[level], composited=700_000, kept=60_000))
    assert seen == [0, 1] + [2] * 10


def test_ordinary_ratios_leave_the_windows_alone():
    s = WaveSchedule(1200, 680, 1536)
    full = list(s.get(100_000, 32, 1)[0])
    s.adapt(_words(waves=len(full), evaluated=11_300_000, composited=7_800_000, tiles=9_000))       # 3.5 M in vain, 1.45 times
    assert s.get(100_000, 32, 1) == (full, False)
    small = WaveSchedule(128, 96, 1536)
    assert small.get(500, 32, 1) == ([1536], False)
    small.adapt(_words(evaluated=400_000, composited=187_000))      # 2.1 times, but few: another wave costs more
    assert small.get(500, 32, 1) == ([1536], False)


@pytest.mark.parametrize("precision, few, many", [(1, 100_000, 100_001), (0, 30_000, 30_001)])
def test_one_window_is_not_for_long_given_lists(precision, few, many):
    s = WaveSchedule(140, 100, 2048)
    assert s.get(3_000, 32, precision, True, few)[0] == [2048]
    assert len(s.get(3_000, 32, precision, True, many)[0]) > 1
    assert s.get(3_000, 32, precision)[0] == [2048]
