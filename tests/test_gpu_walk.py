"""The writer's window walk at the edges of its segment layouts.

Chains from a few channels (one lane walks them) over even segment lengths to
several waves of ramped ones, with windows that hold every entry count and
windows that miss most of them, in one group of segments and in several: the
draws, and with them every output value, equal the oracle's.
"""

from __future__ import annotations

import functools

import numpy as np
import pytest

import cases
from _helpers import make_job
from fauxice_b200 import _lib, engine
from fauxice_b200.engine import process_b200
from oracle import oracle as ox

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _case(h: int, w: int, spec: str):
    main, prepass = cases.generated(41, h, w, spec)
    return make_job(main, prepass), ox.process(main, prepass)


@pytest.mark.parametrize("h, w, spec", [(16, 24, "native"), (24, 40, "native"), (40, 64, "heavy"),
                                        (61, 64, "native"), (200, 333, "heavy"),
                                        (517, 611, "heavy")])
@pytest.mark.parametrize("wave, sigmas", [(0, 4.5), (1, 4.5), (2, 0.0), (3, 4.5), (25, 0.0),
                                          (64, 4.5), (64, 0.5)])
def test_every_layout_draws_as_the_oracle(h, w, spec, wave, sigmas):
    job, expected = _case(h, w, spec)
    ctx, lib = engine.context(), _lib.load()
    assert lib.fx_set_walk_wave(ctx.handle, wave) == 0
    assert lib.fx_set_walk_window(ctx.handle, sigmas) == 0
    try:
        result = process_b200(job)
    finally:
        assert lib.fx_set_walk_wave(ctx.handle, 0) == 0
        assert lib.fx_set_walk_window(ctx.handle, 4.5) == 0
    assert np.array_equal(result.output_rgb16, expected.output_rgb16)
    assert result.replay.public_rng_advances == expected.public_rng_advances
    assert result.replay.final_rng_state == expected.final_rng_state


# lists of 605,000 channels: waves just below the widest take more segment records than
# the widest; windows of 16 sigma keep more survivors than the pool of kept lists holds,
# and windows of 0 sigma end wave after wave early
@pytest.mark.parametrize("wave, sigmas", [(588, 4.5), (591, 4.5), (591, 16.0), (0, 16.0),
                                          (300, 0.0), (591, 0.0)])
def test_waves_near_the_widest_draw_as_the_oracle(wave, sigmas):
    job, expected = _case(1094, 1100, "native")
    ctx, lib = engine.context(), _lib.load()
    assert lib.fx_set_list_capacity(ctx.handle, 605000) == 0
    assert lib.fx_set_walk_wave(ctx.handle, wave) == 0
    assert lib.fx_set_walk_window(ctx.handle, sigmas) == 0
    try:
        result = process_b200(job)
    finally:
        assert lib.fx_set_list_capacity(ctx.handle, 0) == 0
        assert lib.fx_set_walk_wave(ctx.handle, 0) == 0
        assert lib.fx_set_walk_window(ctx.handle, 4.5) == 0
    assert np.array_equal(result.output_rgb16, expected.output_rgb16)
    assert result.replay.public_rng_advances == expected.public_rng_advances
    assert result.replay.final_rng_state == expected.final_rng_state


@pytest.mark.parametrize("h, w, spec", [(61, 64, "native"), (200, 333, "heavy"),
                                        (517, 611, "heavy"), (300, 411, "native")])
def test_serial_walk_draws_as_the_oracle(h, w, spec):
    """One lane walks the whole chain (rows of 32 channels and a remainder)."""

    job, expected = _case(h, w, spec)
    ctx, lib = engine.context(), _lib.load()
    assert lib.fx_set_parallel_walk(ctx.handle, 0) == 0
    try:
        result = process_b200(job)
    finally:
        assert lib.fx_set_parallel_walk(ctx.handle, 1) == 0
    assert np.array_equal(result.output_rgb16, expected.output_rgb16)
    assert result.replay.public_rng_advances == expected.public_rng_advances
    assert result.replay.final_rng_state == expected.final_rng_state
