"""The shipped tuning table (no GPU): each class and key type holds the
configuration that the tuner picks by the table's own timings."""
import pytest

pytest.importorskip("torch")

from apsep_gb300 import _lib, autotune  # noqa: E402


@pytest.mark.parametrize("dtype", ["int32", "float32"])
def test_choices_follow_the_timings(dtype):
    table = autotune.load()
    entries = table.by_dtype.get(dtype, table.entries)
    timings = table.timings[dtype]
    assert sorted(map(int, timings)) == sorted(entries)
    for c, cfg in entries.items():
        us = {int(k): v for k, v in timings[str(c)].items()}
        assert sorted(us) == list(range(_lib.NUM_CONFIGS)), c
        assert us[cfg] <= 1.005 * min(us.values()) and cfg == autotune.pick(us), (dtype, c, cfg, us)


def test_pick():
    assert autotune.pick({0: 10.0, 2: 9.96, 4: 12.0}) == 0  # as good as the fastest
    assert autotune.pick({0: 10.1, 2: 9.96, 4: 12.0}) == 2
    assert autotune.pick({1: 13.43, 4: 13.38, 5: 13.7}) == 4 and autotune.pick({5: 1.0}) == 5
    assert sorted(autotune._PREFERENCE) == list(range(_lib.NUM_CONFIGS))


def test_classes_are_timed_at_lengths_of_their_own():
    for c in range(8, 31):
        for n in autotune.class_sizes(c):
            assert autotune.size_class(n) == c and n <= _lib.MAX_KEYS
