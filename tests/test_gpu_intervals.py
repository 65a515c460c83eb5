"""Copy intervals of RNG-dependent channels beyond the profile's dither.

The profile's amplitudes keep every delta inside the dither bounds, so the
floor test alone decides.  With larger amplitudes and tighter bounds the delta
leaves them on some states and a channel's copy set gets up to three
breakpoints and two intervals; sizes around the units of 256 sites and the
segments of 1024 that list the channels (6 w + h w sites; units of 64 on the
smaller frames).
"""

from __future__ import annotations

import numpy as np
import pytest

import cases
from fauxice_b200 import _lib, engine
from fauxice_b200.profile import DEFAULT_PROFILE, NIKON_PE_INITIAL_STATE
from oracle import oracle as ox

pytestmark = pytest.mark.gpu

BOUNDS = ox.dither_bounds(ox.tables()[0])


@pytest.mark.parametrize("h, w", [(16, 16), (74, 16), (58, 16), (26, 40), (57, 65), (130, 211),
                                  (620, 651)])
@pytest.mark.parametrize("scales, margin", [
    ((0.015, 0.025, 0.015), 0.0), ((0.4, 0.9, 2.0), 0.0), ((30.0, 4.0, 300.0), 0.0),
    ((0.02, 1.5, 8.0), 0.05), ((1e-7, 1e-12, 1e5), 0.02)])
def test_wide_dither_draws_as_the_oracle(h, w, scales, margin):
    main, _ = cases.generated(43, h, w, "heavy")
    low, high = BOUNDS
    low, high = (float(np.float32(v)) for v in (low + margin * (high - low),
                                                high - margin * (high - low)))
    scales = tuple(float(np.float32(v)) for v in scales)
    stages = ox.stage_table(ox.producer_rows(main))
    expected = ox.replay(main, stages, ox.Params(dither_scales=scales, dither_low=low,
                                                 dither_high=high))
    params = DEFAULT_PROFILE.hot_path_parameters().to_c()
    params.dither_scales[:] = scales
    params.dither_low, params.dither_high = low, high
    got = engine.run_frame(engine.context(), main, params, stages.astype(_lib.STAGE_DTYPE),
                           NIKON_PE_INITIAL_STATE, True)
    assert np.array_equal(got.output, expected.output_rgb16)
    assert np.array_equal(got.changed.astype(bool), expected.changed_mask)
    assert got.counters.public_advances == expected.public_rng_advances
    assert got.counters.final_state == expected.final_rng_state
