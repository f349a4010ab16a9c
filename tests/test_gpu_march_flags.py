"""The hydraulic march on a world whose blocks take long pieces of a strip, with cells outside the packed ranges far
apart in a piece: every flagged segment of chunks runs again in scalar form, and the rows between stay packed.  Bit for
bit as the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import master_thesis_gb300 as T
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(2048, 4096), (2047, 4099)])
@pytest.mark.parametrize("iters", [1, 2])
@pytest.mark.parametrize("cells", [3, 60, 3000])
def test_cells_outside_the_ranges_far_apart(cells, iters, W, H):
    s = T.baseline_settings()
    s.step.hydraulicTile = 9
    rng = np.random.default_rng(cells)
    h = rng.normal(0.2, 0.1, (H, W)).astype(np.float32)
    water = np.abs(rng.normal(0, 0.05, (H, W))).astype(np.float32)
    sed = np.abs(rng.normal(0, 0.01, (H, W))).astype(np.float32)
    flux = np.abs(rng.normal(0, 0.01, (H, W, 4))).astype(np.float32)
    h[rng.integers(0, H, cells), rng.integers(0, W, cells)] = 3e24
    with T.World(s, W, H, seed=1000) as w:
        for f, a in ((T.FIELD_HEIGHT, h), (T.FIELD_WATER, water), (T.FIELD_SEDIMENT, sed), (T.FIELD_FLUX, flux)):
            w.upload(f, a)
        w.hydraulic(iters, 0.02)
        want = O.hydraulic(h, water, sed, flux, iters, 0.02, 1000, s)
        for name, f, v in zip(("height", "water", "sediment", "flux"),
                              (T.FIELD_HEIGHT, T.FIELD_WATER, T.FIELD_SEDIMENT, T.FIELD_FLUX), want):
            np.testing.assert_array_equal(w.download(f).view(np.uint32), v.view(np.uint32), err_msg=name)
