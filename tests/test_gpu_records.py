"""Feature records that are not finite.

A band of rows whose auxiliary values are near the binary32 limit overflows
the column sums around it; a pixel that reads such a record is refused, and
one out of reach is not.
"""

from __future__ import annotations

import numpy as np
import pytest

import cases
from fauxice_b200 import _lib, engine
from fauxice_b200.profile import DEFAULT_PROFILE, NIKON_PE_INITIAL_STATE
from oracle import oracle as ox

pytestmark = pytest.mark.gpu


def _job(first: int, rows: int, offset: float):
    main, _ = cases.generated(47, 48, 70, "heavy")
    stages = ox.stage_table(ox.producer_rows(main))
    stages["offset"][first:first + rows] = offset
    return main, stages


@pytest.mark.parametrize("tile", [8, 16])
@pytest.mark.parametrize("first, rows, offset, refused", [
    (20, 9, -3e38, True), (20, 9, 3e38, False), (20, 9, -1e30, False), (20, 1, 1e30, False)])
def test_records_that_overflow_are_refused(first, rows, offset, refused, tile):
    main, stages = _job(first, rows, offset)
    params = DEFAULT_PROFILE.hot_path_parameters().to_c()
    ctx, lib = engine.context(), _lib.load()
    assert lib.fx_set_stencil_tile(ctx.handle, tile) == 0
    try:
        if refused:
            with pytest.raises(ox.OracleError, match="status 5"):
                ox.replay(main, stages)
            with pytest.raises(Exception, match="combiner inputs must be finite"):
                engine.run_frame(ctx, main, params, stages.astype(_lib.STAGE_DTYPE),
                                 NIKON_PE_INITIAL_STATE, True)
            return
        expected = ox.replay(main, stages)
        got = engine.run_frame(ctx, main, params, stages.astype(_lib.STAGE_DTYPE),
                               NIKON_PE_INITIAL_STATE, True)
    finally:
        assert lib.fx_set_stencil_tile(ctx.handle, 0) == 0
    assert np.array_equal(got.output, expected.output_rgb16)
    assert got.counters.public_advances == expected.public_rng_advances
    assert got.counters.final_state == expected.final_rng_state
