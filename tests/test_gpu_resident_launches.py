"""Worlds of a few blocks, whose launches are resident several at a time: long runs of sub-iterations and
iterations in one call, each kernel reading what the ones ahead of it wrote on the same SMs.  Bit for bit as the
oracle."""
from __future__ import annotations

import numpy as np
import pytest

import master_thesis_gb300 as T
import oracle as O

pytestmark = pytest.mark.gpu


def fields(W, H):
    rng = np.random.default_rng(W * 7 + H)
    h = rng.normal(0.2, 0.1, (H, W)).astype(np.float32)
    water = np.abs(rng.normal(0, 0.05, (H, W))).astype(np.float32)
    sed = np.abs(rng.normal(0, 0.01, (H, W))).astype(np.float32)
    flux = np.abs(rng.normal(0, 0.01, (H, W, 4))).astype(np.float32)
    return h, water, sed, flux


@pytest.mark.parametrize("W,H", [(64, 64), (250, 33), (117, 70)])
@pytest.mark.parametrize("tile,iters", [(9, 200), (9, 201), (1, 200), (4, 200), (6, 60)])
def test_many_sub_iterations(W, H, tile, iters):
    s = T.baseline_settings()
    s.step.hydraulicTile = tile
    h, water, sed, flux = fields(W, H)
    want = O.hydraulic(h, water, sed, flux, iters, 0.02, 1000, s)
    with T.World(s, W, H, seed=1000) as w:
        for f, a in ((T.FIELD_HEIGHT, h), (T.FIELD_WATER, water), (T.FIELD_SEDIMENT, sed), (T.FIELD_FLUX, flux)):
            w.upload(f, a)
        w.hydraulic(iters, 0.02)
        for name, f, v in zip(("height", "water", "sediment", "flux"),
                              (T.FIELD_HEIGHT, T.FIELD_WATER, T.FIELD_SEDIMENT, T.FIELD_FLUX), want):
            np.testing.assert_array_equal(w.download(f).view(np.uint32), v.view(np.uint32), err_msg=name)


@pytest.mark.parametrize("W,H", [(64, 64), (250, 33), (117, 70)])
@pytest.mark.parametrize("tile", [1, 2, 3, 4, 5])
def test_many_thermal_iterations(W, H, tile):
    s = T.baseline_settings()
    s.step.thermalTile = tile
    h = fields(W, H)[0]
    with T.World(s, W, H, seed=1000) as w:
        w.upload(T.FIELD_HEIGHT, h)
        w.thermal(200)
        np.testing.assert_array_equal(w.download(T.FIELD_HEIGHT).view(np.uint32),
                                      O.thermal(h, 200, s).reshape(H, W).view(np.uint32))
