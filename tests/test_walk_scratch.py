"""The walk's scratch holds every wave setting (no GPU needed).

A pass's scratch is laid out from the list's capacity for the widest wave
(592 segments on 148 SMs).  A slightly narrower wave can take more segment
records than that one: it goes over to ramped segments, with spare waves, or
needs one wave more, a few channels earlier.
"""

from __future__ import annotations

import ctypes

import pytest

from fauxice_b200 import _lib

WIDEST = 592
CHUNK = 256
WAVE = 18  # most chunks per segment on average


def _records(channels: int, segments: int) -> tuple[int, int]:
    used, reserved = ctypes.c_int64(), ctypes.c_int64()
    assert _lib.load().fx_walk_segments(channels, segments, ctypes.byref(used),
                                        ctypes.byref(reserved)) == 0
    return used.value, reserved.value


# the least list, the ends of the even segments and of one, two and five waves of the
# widest and of narrower waves, and lists of a 2^30-pixel frame
@pytest.mark.parametrize("channels", sorted(
    {1, 65536, 605000, 605734, 3 << 30}
    | {4 * s * CHUNK + d for s in (148, 588, 591, WIDEST) for d in (-CHUNK, 0, 1)}
    | {k * s * WAVE * CHUNK + d for k in (1, 2, 5) for s in (148, 590, 591, WIDEST)
       for d in (0, 1)}))
def test_no_wave_needs_more_records_than_the_scratch_holds(channels):
    for segments in range(WIDEST + 2):
        used, reserved = _records(channels, segments)
        assert 0 < used <= reserved, segments


def test_a_narrower_wave_can_need_more_records_than_the_widest():
    assert _records(605000, 591)[0] > _records(605000, WIDEST)[0]


def test_bad_arguments_are_refused():
    lib, n = _lib.load(), ctypes.byref(ctypes.c_int64())
    assert lib.fx_walk_segments(0, 0, n, n) == 1
    assert lib.fx_walk_segments(1, -1, n, n) == 1
    assert lib.fx_walk_segments(1, 0, None, n) == 1
