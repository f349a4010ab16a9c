"""Worlds with one very long side: every tile of a phase's work list is there, and the erosion phases reach
every row and column."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import master_thesis_gb300 as T
import oracle as O

# tiles: 56 x 4 (the fewest rows of a tile), 56 x 8, 52 x 9, 60 x 24, 32 x 32 (the fewest columns)
TILES = [(56, 4), (56, 8), (52, 9), (60, 24), (32, 32)]


@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("W,H", [(1, 262144), (1, 262145), (16, 600000), (1, 1 << 24), (1 << 24, 3), (4194305, 1), (300, 200)])
@pytest.mark.parametrize("world", [0, 15, 16, 1023])
def test_work_list_covers_the_world(world, W, H, tile):
    bad = C.c_ulonglong(1)
    assert T.lib().tecto_selftest_tiles(W, H, world, *tile, C.byref(bad)) == 0
    assert bad.value == 0


def test_work_list_arguments():
    bad = C.c_ulonglong()
    f = T.lib().tecto_selftest_tiles
    assert f(0, 1, 0, 56, 4, C.byref(bad)) == -1 and f(1 << 20, 1 << 20, 0, 56, 4, C.byref(bad)) == -1
    assert f(1 << 15, 1 << 15, 0, 1, 1, C.byref(bad)) == -1 and f(4, 4, 0, 1 << 20, 4, C.byref(bad)) == -1
    assert f(4, 4, 1024, 56, 4, C.byref(bad)) == -1 and f(4, 4, 0, 0, 4, C.byref(bad)) == -1 and f(4, 4, 0, 56, 4, None) == -1


def check(W, H, tile, thermal_tile, iters, dt):
    s = T.baseline_settings()
    s.step.hydraulicTile, s.step.thermalTile = tile, thermal_tile
    rng = np.random.default_rng(W + H)
    h = rng.normal(0.2, 0.1, (H, W)).astype(np.float32)
    water = np.abs(rng.normal(0, 0.05, (H, W))).astype(np.float32)
    sed = np.abs(rng.normal(0, 0.01, (H, W))).astype(np.float32)
    flux = np.abs(rng.normal(0, 0.01, (H, W, 4))).astype(np.float32)
    with T.World(s, W, H, seed=1000) as w:
        for f, a in ((T.FIELD_HEIGHT, h), (T.FIELD_WATER, water), (T.FIELD_SEDIMENT, sed), (T.FIELD_FLUX, flux)):
            w.upload(f, a)
        w.hydraulic(iters, dt)
        want = O.hydraulic(h, water, sed, flux, iters, dt, 1000, s)
        for name, f, v in zip(("height", "water", "sediment", "flux"),
                              (T.FIELD_HEIGHT, T.FIELD_WATER, T.FIELD_SEDIMENT, T.FIELD_FLUX), want):
            np.testing.assert_array_equal(w.download(f).view(np.uint32), v.view(np.uint32), err_msg=name)
        w.thermal(2)
        np.testing.assert_array_equal(w.download(T.FIELD_HEIGHT).view(np.uint32),
                                      O.thermal(want[0], 2, s).reshape(H, W).view(np.uint32))


# more tile rows than 16 bits hold, for one sub-iteration (56 x 8) and for two (52 x 12); and more
# tile columns (52 and 56 wide)
@pytest.mark.gpu
@pytest.mark.parametrize("W,H,tile,iters,dt", [(3, 270000, 7, 1, 0.02), (2, 530000, 1, 1, 0.02), (2, 530000, 2, 1, 0.5), (2, 800000, 2, 2, 0.02),
                                               (2, 600000, 1, 2, 0.02), (2, 600000, 0, 3, 0.02), (3700000, 2, 4, 2, 0.02),
                                               (3700000, 2, 9, 1, 0.02), (2, 1060000, 4, 1, 0.02)])
def test_more_tiles_a_side_than_16_bits(W, H, tile, iters, dt):
    check(W, H, tile, 4, iters, dt)


# positions above 2^22, where the fused kernels' floors would end: the tiles, the march, and two at once
@pytest.mark.gpu
@pytest.mark.parametrize("W,H,tile,iters", [(4250000, 2, 4, 2), (4250000, 2, 7, 1), (2, 4250000, 9, 2), (4194304, 4, 9, 1),
                                            (4, 4194250, 0, 2)])
def test_sides_above_two_to_the_22(W, H, tile, iters):
    check(W, H, tile, 0, iters, 0.02)
