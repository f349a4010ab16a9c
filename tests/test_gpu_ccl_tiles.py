"""Labelling at tile borders: whole tiles of one plate beside mixed ones, borders along, across and a cell off
the 32 x 32 tiles, tiles of one row or one column, and worlds that wrap inside a tile.  Labels are whole
numbers and equal the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import master_thesis_gb300 as T
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [T.CCL_4, T.CCL_8, T.CCL_REF8])
@pytest.mark.parametrize("W,H", [(32, 32), (33, 65), (65, 33), (1, 70), (70, 1), (2, 2), (96, 64), (97, 130), (31, 200),
                                 (224, 161)])
@pytest.mark.parametrize("kind", ["one", "blocks", "diagonal", "sparse", "columns", "few"])
def test_tile_borders(kind, W, H, mode):
    y, x = np.mgrid[0:H, 0:W]
    rng = np.random.default_rng(W * 1000 + H)
    ids = {"one": np.full((H, W), 7), "blocks": (x // 33 + 2 * (y // 31)) % 3, "diagonal": (x + y) // 37 % 2,
           "sparse": rng.random((H, W)) < 0.004, "columns": x // 32 % 2 + 2 * (rng.random((H, W)) < 0.01),
           "few": rng.integers(0, 2, ((H + 2) // 3, (W + 2) // 3)).repeat(3, 0).repeat(3, 1)[:H, :W]}[kind]
    ids = np.ascontiguousarray(ids).astype(np.uint8)
    with T.World(T.baseline_settings(), W, H, seed=1) as w:
        w.upload(T.FIELD_PLATE_ID, ids)
        w.ccl(mode)
        np.testing.assert_array_equal(w.download(T.FIELD_LABELS), O.ccl(ids, mode))
