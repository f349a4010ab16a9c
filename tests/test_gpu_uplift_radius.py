"""Gaussian uplift of radius 0: the centre tap alone, upliftAmount on every convergent cell.  The heights equal the
oracle's bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import master_thesis_gb300 as T
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(64, 16), (129, 65)])
@pytest.mark.parametrize("amount,sigma", [(0.01, 1.5), (-0.25, 0.5), (0.01, 0.0)])
@pytest.mark.parametrize("dynamics", [0, T.PLATE_DYNAMICS_REFERENCE])
def test_radius_0(dynamics, amount, sigma, W, H):
    s = T.baseline_settings()
    s.step.hydraulicIterations = s.step.thermalIterations = 0
    s.step.upliftRadius, s.step.upliftAmount, s.step.upliftSigma = 0, amount, sigma
    s.step.plateDynamics = dynamics
    with T.World(s, W, H, seed=3) as w:
        w.init_synthetic(6, 4.0, 9)
        h = w.download(T.FIELD_HEIGHT)
        h[::5, ::3] = -0.0
        w.upload(T.FIELD_HEIGHT, h)
        o = O.OracleWorld(s, h, w.download(T.FIELD_PLATE_ID), w.plates(), 3)
        for _ in range(2):
            w.step(1)
            o.step(1)
            assert (o.word > 0xFF).any()
            got = w.download(T.FIELD_HEIGHT)
            ok = ~np.isnan(o.h)
            np.testing.assert_array_equal(got, o.h)
            np.testing.assert_array_equal(got.view(np.uint32)[ok], o.h.view(np.uint32)[ok])
