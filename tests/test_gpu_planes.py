"""The score planes at the edges of a warp's 128 padded columns."""

from __future__ import annotations

import numpy as np
import pytest

import cases
from fauxice_b200 import _lib, engine
from fauxice_b200.profile import DEFAULT_PROFILE, NIKON_PE_INITIAL_STATE
from oracle import oracle as ox

pytestmark = pytest.mark.gpu


# padded column = column + 5, 128 per warp and 512 per block
@pytest.mark.parametrize("minimum", [True, False])
@pytest.mark.parametrize("visible", [0, 1, 2])
@pytest.mark.parametrize("w", [9, 122, 123, 124, 125, 251, 506, 507, 508, 635])
def test_planes_match_the_oracle(w, visible, minimum):
    h = 9
    main, _ = cases.generated(59, h, w, "heavy")
    stages = ox.stage_table(ox.producer_rows(main))
    stages["alpha"][5] = 1.0  # a row with the configured replacement
    stages["replacement"][5] = 41000.0
    stages["replacement_valid"][5] = 1
    expected = ox.replay(main, stages, ox.Params(horizontal_minimum=minimum,
                                                 visible_channel=visible))
    params = DEFAULT_PROFILE.hot_path_parameters().to_c()
    params.horizontal_minimum = int(minimum)
    params.visible_channel = visible
    got = engine.run_frame(engine.context(), main, params, stages.astype(_lib.STAGE_DTYPE),
                           NIKON_PE_INITIAL_STATE, True)
    assert np.array_equal(got.score, expected.score_plane)
    assert np.array_equal(got.output, expected.output_rgb16)
    assert got.counters.final_state == expected.final_rng_state
