"""Producer records over the row blockings: frame heights that give a block
one to five 8-row blocks, and more than one wave of blocks, each with a short
last block, widths with partial tiles and cells, and dark IR samples that
fail cells: all four record fields equal the oracle's."""

from __future__ import annotations

import numpy as np
import pytest

from fauxice_b200 import _lib, engine
from oracle import oracle as ox

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h, w", [(5, 8), (9, 63), (1183, 64), (1187, 65), (2371, 73), (3560, 131),
                                  (4741, 40), (5923, 24), (8190, 17)])
@pytest.mark.parametrize("dark", [0.0, 0.002, 0.4])
def test_rows_match_the_oracle(h, w, dark):
    rng = np.random.default_rng(h + w)
    px = rng.integers(0, 65536, size=(h, w, 4), dtype=np.uint16)
    px[..., 3] = rng.integers(8849, 65536, size=(h, w))
    px[..., 3][rng.random((h, w)) < dark] = 8847  # the last failing value
    ctx = engine.context()
    rows = [np.empty(h, np.float32) for _ in range(4)]
    rc = _lib.load().fx_producer_rows(ctx.handle, _lib.ptr(px), h, w, *(_lib.ptr(r) for r in rows))
    assert rc == 0, ctx._error(ctx.handle)
    expected = ox.producer_rows(px)
    for got, name in zip(rows, ("p1", "p2", "mean_vis", "mean_ir")):
        assert np.array_equal(got.view(np.uint32), expected[name].view(np.uint32)), name
