"""Which of the two kernels of the same bits a decode or verify step of the delta rule goes to."""
import pytest

from ferrite_b200._ext import load


# segment lengths, heads (key, value, width), the one that was faster on B200 with both times (us: kernel for single rows, kernel of several rows)
@pytest.mark.parametrize("ns,heads,sliced", [
    ([17], (16, 16, 128), True),                  # 33.4, 10.7
    ([2], (16, 16, 128), True),                   # 6.4, 4.8
    ([17] * 4, (16, 16, 128), True),              # 33.6, 21.0
    ([1] * 7 + [17], (16, 16, 128), True),        # 34.1, 23.8
    ([2] * 8, (16, 16, 128), False),              # 7.1, 18.7
    ([5] * 8, (16, 16, 128), False),              # 12.6, 23.5
    ([2] * 24, (16, 16, 128), False),             # 22.7, 58.5
    ([1] * 23 + [2], (16, 16, 128), False),       # 18.7, 54.6
    ([1] * 24, (16, 16, 128), False),             # 15.0, 44
    ([5] * 8, (16, 32, 128), False),              # 26.0, 28.5
    ([17] * 8, (16, 32, 128), True),              # 71.8, 52.4
    ([2] * 24, (8, 8, 64), False),                # 5.8, 14.1
    ([17] * 24, (8, 8, 64), True),                # 30.7, 26.9
    ([5] * 8, (2, 16, 128), False),               # 12.4, 19.9
    ([17], (2, 16, 128), True),                   # 33.4, 20.1
    ([17], (1, 16, 128), False)])                 # sixteen heads to a key head: no cluster holds them
def test_segments_of_several_rows(ns, heads, sliced):
    C = load()
    assert C.gdn_step_sliced(len(ns), sum(ns), max(ns), *heads) == sliced
    if len(set(ns)) == 1:                         # the longest segment is not known: as if all were alike
        assert C.gdn_step_sliced(len(ns), sum(ns), 0, *heads) == sliced


def test_single_rows():
    """Slices that fill a wave of CTAs and no more."""
    C = load()
    assert [C.gdn_step_sliced(n, n, 1, 16, 16, 128) for n in (1, 2, 3, 24)] == [True, True, False, False]
    assert not C.gdn_step_sliced(1, 1, 1, 8, 8, 128)
