"""The hidden startup stages at the edges of their 32-column blocks."""

from __future__ import annotations

import numpy as np
import pytest

import cases
from fauxice_b200 import _lib, engine
from fauxice_b200.profile import DEFAULT_PROFILE, NIKON_PE_INITIAL_STATE
from oracle import oracle as ox

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cross", [True, False])
@pytest.mark.parametrize("h, w", [(16, 12), (9, 31), (12, 32), (16, 33), (11, 36), (13, 65),
                                  (10, 97)])
def test_startup_stages_match_the_oracle(h, w, cross):
    main, _ = cases.generated(53, h, w, "heavy")
    stages = ox.stage_table(ox.producer_rows(main))
    expected = ox.replay(main, stages, ox.Params(cross_neighbor=cross))
    params = DEFAULT_PROFILE.hot_path_parameters().to_c()
    params.cross_neighbor = int(cross)
    got = engine.run_frame(engine.context(), main, params, stages.astype(_lib.STAGE_DTYPE),
                           NIKON_PE_INITIAL_STATE, True)
    assert tuple(got.counters.startup_attempted) == tuple(expected.startup_attempted)
    assert tuple(got.counters.startup_advances) == tuple(expected.startup_advances)
    assert got.counters.startup_final_state == expected.startup_final_state
    assert np.array_equal(got.output, expected.output_rgb16)
    assert got.counters.final_state == expected.final_rng_state
