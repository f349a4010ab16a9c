"""Cells without a plate (id 255) beside plates in motion, with plate dynamics: their arrivals bring no friction and
nothing else changes, so heights, ids and marks of the resolve are those of the same world without dynamics."""
from __future__ import annotations

import numpy as np
import pytest

import master_thesis_gb300 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(64, 48), (131, 70)])
@pytest.mark.parametrize("uplift", [T.UPLIFT_NONE, T.UPLIFT_GAUSSIAN])
def test_dynamics_beside_cells_without_a_plate(uplift, W, H):
    got = []
    for dynamics in (T.PLATE_DYNAMICS_REFERENCE, 0):
        s = T.baseline_settings()
        s.step.plateDynamics, s.step.upliftMode = dynamics, uplift
        s.kernel.minCollisionSize, s.kernel.collisionTypeUpdateCooldown = 2, 1
        with T.World(s, W, H, seed=3) as w:
            w.init_synthetic(6, 4.0, 9)
            ids = w.download(T.FIELD_PLATE_ID)
            rng = np.random.default_rng(W)
            ids[rng.random((H, W)) < 0.3] = 255
            ids[: H // 4] = 255
            w.upload(T.FIELD_PLATE_ID, ids)
            w.collide()
            w.resolve()
            w.check()
            got.append([w.download(f) for f in (T.FIELD_COLLISION, T.FIELD_HEIGHT, T.FIELD_PLATE_ID, T.FIELD_DIV_BITMAP)])
            w.finish()
            w.check()
            assert np.isfinite(w.plate_dynamics()["frictionLoss"]).all()
    assert (got[0][0] > 0xFF).any()  # convergent cells
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
