"""The emit kernel's site writer on the host (no GPU needed).

fx_write_site is the code k_apply runs for every attempted site.  Its values,
draws and state are those of the reference's writer (reconstruction.py:916-982
with dither.py:59-104, restated here), and a classification or a walk bit that
says other draws than the ones made is reported.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from fauxice_b200 import _lib
from fauxice_b200.profile import DEFAULT_PROFILE

INTERNAL = 16  # FX_ERR_INTERNAL
NORMALIZATION = float.fromhex("0x1.fffffep-25")
PARAMS = DEFAULT_PROFILE.hot_path_parameters().to_c()
LOW, HIGH = float(PARAMS.dither_low), float(PARAMS.dither_high)


def _delta(value, scale, state):
    """(delta, state): conditional_dither_delta."""

    cand = float(np.float32(value))
    if not LOW < HIGH or not LOW < cand < HIGH:
        return 0.0, state
    width = HIGH - LOW
    envelope = ((HIGH - cand) * (cand - LOW)) * (4.0 / (width * width))
    span = float(np.float32(float(np.float32(scale)) * cand))
    state = (125 * state + 1) & 0xFFFFFF
    d = envelope * (0.0 + ((state + 1) * NORMALIZATION - 0.5) * span)
    return (d if LOW < cand + d < HIGH else 0.0), state


def _write(cand, orig, floor, state):
    """(values, draws per channel, state): write_reconstructed_pixel."""

    if not all(np.isfinite(c) and c > 0.0 for c in cand):
        return list(orig), [0, 0, 0], state
    values, draws = [], []
    for c in range(3):
        first, after = _delta(cand[c], PARAMS.dither_scales[c], state)
        made, state = int(after != state), after
        if floor and cand[c] + first <= float(orig[c]):
            values.append(orig[c])
        else:
            d = first
            if floor:
                d, after = _delta(cand[c], PARAMS.dither_scales[c], state)
                made, state = made + int(after != state), after
            values.append(np.float32(cand[c] + d))
        draws.append(made)
    return values, draws, state


def _call(cand, orig, floor, meta, redraw, state):
    c, o, values = np.array(cand, np.float64), np.array(orig, np.float32), np.zeros(3, np.float32)
    s, draws = ctypes.c_uint32(state), ctypes.c_int32()
    rc = _lib.load().fx_write_site(ctypes.byref(PARAMS), int(floor), _lib.ptr(c), _lib.ptr(o), meta,
                                   redraw, ctypes.byref(s), _lib.ptr(values), ctypes.byref(draws))
    return rc, values, draws.value, s.value


def _site(seed):
    rng = np.random.default_rng(seed)
    orig = rng.uniform(3e4, 6.2e4, 3).astype(np.float32)
    cand = orig * (1.0 + rng.normal(0.0, 0.004, 3))
    if seed % 5 == 1:
        cand[rng.integers(3)] = rng.choice([LOW, HIGH, 0.5 * LOW, 70000.0])  # no draw
    if seed % 17 == 2:
        cand[rng.integers(3)] = rng.choice([0.0, -3.0, np.nan, np.inf])  # not valid
    return cand, orig, bool(seed % 3), int(rng.integers(1 << 24))


@pytest.mark.parametrize("block", range(4))
def test_sites_are_written_as_the_reference_writes_them(block):
    seen = set()
    for seed in range(500 * block, 500 * (block + 1)):
        cand, orig, floor, state = _site(seed)
        values, draws, after = _write(cand, orig, floor, state)
        ambiguous = seed % 2  # channels with draws as code 3 and a bit, or as their draws
        meta, redraw, bit = 0x80, 0, 0
        for c, n in enumerate(draws):
            if ambiguous and n:
                meta |= 3 << (2 * c)
                redraw |= (n - 1) << bit
                bit += 1
            else:
                meta |= n << (2 * c)
        got = _call(cand, orig, floor, meta, redraw, state)
        assert got[0] == 0
        assert got[1].tobytes() == np.array(values, np.float32).tobytes()
        assert got[2:] == (sum(draws), after)
        seen.update(draws)
        # a wrong bit, or a wrong class, of each channel
        for k in range(bit):
            assert _call(cand, orig, floor, meta, redraw ^ (1 << k), state)[0] == INTERNAL
        for c, n in enumerate(draws):
            for wrong in {0, 1, 2} - {n}:
                other = meta & ~(3 << (2 * c)) | wrong << (2 * c)
                keep = redraw
                if (meta >> (2 * c)) & 3 == 3:  # its bit leaves the word
                    at = sum((meta >> (2 * j)) & 3 == 3 for j in range(c))
                    keep = (redraw & ((1 << at) - 1)) | (redraw >> (at + 1) << at)
                assert _call(cand, orig, floor, other, keep, state)[0] == INTERNAL
    assert seen == {0, 1, 2}


def test_null_arguments_are_refused():
    assert _lib.load().fx_write_site(None, 1, None, None, 0, 0, None, None, None) == 1
