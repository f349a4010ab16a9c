"""Pipe lengths and steps that the packed flux does not take (a length outside [2^-32, 2^32], a negative step): the
tiles run the flux in scalar form, and the marching variants the tiles.  Fused and split path, odd and even widths,
operands outside the packed flow's ranges too.  Bit for bit as the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import master_thesis_gb300 as T
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,dt", [(1e-12, 0.02), (-1000.0, 0.02), (1e12, 0.02), (0.0, 0.02), (1000.0, -0.02),
                                       (-1000.0, 0.5), (1000.0, -0.5)])
@pytest.mark.parametrize("W,H,iters", [(57, 25, 2), (120, 33, 3), (61, 4, 1)])
@pytest.mark.parametrize("tile", [0, 1, 2, 4, 5, 7, 9])
@pytest.mark.parametrize("kind", ["plain", "huge"])
def test_scalar_flux(kind, tile, W, H, iters, length, dt):
    s = T.baseline_settings()
    s.step.hydraulicTile = tile
    s.kernel.hydrationPipeLength = length
    rng = np.random.default_rng(W * 131 + H)
    h = rng.normal(0.2, 0.1, (H, W)).astype(np.float32)
    water = np.abs(rng.normal(0, 0.2, (H, W))).astype(np.float32)
    sed = np.abs(rng.normal(0, 0.05, (H, W))).astype(np.float32)
    flux = np.abs(rng.normal(0, 0.02, (H, W, 4))).astype(np.float32)
    if kind == "huge":
        h[rng.random((H, W)) < 0.02] = 3e24
        flux[rng.random((H, W)) < 0.02] *= 400
    with T.World(s, W, H, seed=1000) as w:
        for f, a in ((T.FIELD_HEIGHT, h), (T.FIELD_WATER, water), (T.FIELD_SEDIMENT, sed), (T.FIELD_FLUX, flux)):
            w.upload(f, a)
        w.hydraulic(iters, dt)
        want = O.hydraulic(h, water, sed, flux, iters, dt, 1000, s)
        for name, f, v in zip(("height", "water", "sediment", "flux"),
                              (T.FIELD_HEIGHT, T.FIELD_WATER, T.FIELD_SEDIMENT, T.FIELD_FLUX), want):
            got, v = w.download(f), v.reshape(w.download(f).shape)
            np.testing.assert_array_equal(got, v, err_msg=name)
            ok = ~np.isnan(v)  # and the signs of zeros
            np.testing.assert_array_equal(got.view(np.uint32)[ok], v.view(np.uint32)[ok], err_msg=name)
