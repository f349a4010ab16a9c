"""The packed marching kernels (hydraulicTile 9, thermalTile 5) at the edges of their packed arithmetic.

Inside them the variant tests compare it with the oracle; here the operands leave them (quotients of tiny
or huge operands, the velocity clamp, a negative step, a pipe length that the fast quotients do not take),
so that rows run a second time in the scalar form.  Every field equals the oracle's bit for bit: the
same IEEE operations in the same order.  The thermal march has three forms by its parameters, and runs a
piece again where a slope sum is above 2^32.
"""
from __future__ import annotations

import numpy as np
import pytest

import master_thesis_gb300 as T
import oracle as O

pytestmark = pytest.mark.gpu


def fields(kind, W, H):
    rng = np.random.default_rng(W * 131 + H)
    f32 = np.float32
    h = rng.normal(0.2, 0.1, (H, W)).astype(f32)
    water = np.abs(rng.normal(0, 0.2, (H, W))).astype(f32)
    sed = np.abs(rng.normal(0, 0.05, (H, W))).astype(f32)
    flux = np.abs(rng.normal(0, 0.02, (H, W, 4))).astype(f32)
    at = rng.random((H, W)) < 0.02
    if kind == "tiny":  # level ground, differences and fluxes far below 2^-90, some subnormal
        h[:] = 0
        water = (water * 1e-36).astype(f32)
        flux = (flux * f32(1e-35)).astype(f32)
        water[at] = 0
    elif kind == "huge":
        h[at] = f32(3e24)
        water[rng.random((H, W)) < 0.02] = f32(8e20)
    elif kind == "clamp":  # shallow water between strong fluxes: velocities above 50 cells a second
        water = (water * f32(0.01)).astype(f32)
        flux[at] *= f32(400)
    elif kind == "flat":  # zero slopes, zero fluxes, zero quotients of both signs
        h[:] = f32(0.25)
        flux[:] = 0
        water[~at] = 0
    return h, water, sed, flux


@pytest.mark.parametrize("W,H", [(124, 37), (61, 23), (250, 9), (122, 4)])
@pytest.mark.parametrize("kind", ["tiny", "huge", "clamp", "flat", "backward", "short_pipe"])
def test_operands_outside_the_packed_ranges(kind, W, H):
    s = T.baseline_settings()
    s.step.hydraulicTile = 9
    dt = -0.02 if kind == "backward" else 0.02
    if kind == "short_pipe":
        s.kernel.hydrationPipeLength = 1e-12
    h, water, sed, flux = fields(kind, W, H)
    with T.World(s, W, H, seed=1000) as w:
        for f, a in ((T.FIELD_HEIGHT, h), (T.FIELD_WATER, water), (T.FIELD_SEDIMENT, sed), (T.FIELD_FLUX, flux)):
            w.upload(f, a)
        w.hydraulic(3, dt)
        want = O.hydraulic(h, water, sed, flux, 3, dt, 1000, s)
        for name, f, v in zip(("height", "water", "sediment", "flux"),
                              (T.FIELD_HEIGHT, T.FIELD_WATER, T.FIELD_SEDIMENT, T.FIELD_FLUX), want):
            np.testing.assert_array_equal(w.download(f), v.reshape(w.download(f).shape), err_msg=f"{kind} {name}")


# (threshold angle, amplitude, strength): the packed form with the amplitude folded in, the packed form,
# the scalar form for a threshold below 2^-32
@pytest.mark.parametrize("thr,A,S", [(0.01, 0.5, 1.0), (0.01, 2.0**-9, 1.0), (0.01, 0.3, 1.0), (0.01, 0.5, 0.7),
                                     (1e-12, 0.5, 1.0)])
@pytest.mark.parametrize("W,H", [(64, 7), (60, 1), (61, 50), (122, 2), (187, 33)])
@pytest.mark.parametrize("kind", ["rough", "flat", "huge"])
def test_thermal_march_forms(kind, W, H, thr, A, S):
    s = T.baseline_settings()
    s.step.thermalTile = 5
    s.kernel.thermalThresholdAngle, s.kernel.thermalCellSize = thr, 1.0
    s.kernel.thermalErosionAmplitude, s.kernel.thermalErosionStrength = A, S
    rng = np.random.default_rng(W * 17 + H)
    h = rng.normal(0, 0.1, (H, W)).astype(np.float32)
    if kind == "flat":  # zeros of both signs, a few peaks
        h = np.where(rng.random((H, W)) < 0.1, h, np.where(rng.random((H, W)) < 0.5, 0.0, -0.0)).astype(np.float32)
    elif kind == "huge":
        h[rng.random((H, W)) < 0.01] = 3e10
    with T.World(s, W, H, seed=1000) as w:
        w.upload(T.FIELD_HEIGHT, h)
        w.thermal(3)
        got, want = w.download(T.FIELD_HEIGHT), O.thermal(h, 3, s).reshape(H, W)
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("W,H,iters", [(5, 3, 2), (3, 40, 4), (113, 4, 2), (112, 61, 2), (225, 9, 5), (49, 130, 2),
                                       (160, 33, 4), (1001, 47, 2), (116, 21, 2), (117, 21, 2), (52, 70, 2), (53, 70, 2)])
@pytest.mark.parametrize("kind", ["tiny", "clamp", "huge"])
def test_two_sub_iterations_in_one_march(kind, W, H, iters):
    """Two sub-iterations share a march where its narrower strips are not many more than 120-column ones:
    pieces of a few rows, strips of one column and narrower than half a block, worlds that wrap within a
    halo, odd widths, operands that send rows through the scalar form in the first or the second of two, and
    an odd number left over.  Bit for bit as the oracle."""
    s = T.baseline_settings()
    s.step.hydraulicTile = 9
    h, water, sed, flux = fields(kind, W, H)
    with T.World(s, W, H, seed=1000) as w:
        for f, a in ((T.FIELD_HEIGHT, h), (T.FIELD_WATER, water), (T.FIELD_SEDIMENT, sed), (T.FIELD_FLUX, flux)):
            w.upload(f, a)
        w.hydraulic(iters, 0.02)
        want = O.hydraulic(h, water, sed, flux, iters, 0.02, 1000, s)
        for name, f, v in zip(("height", "water", "sediment", "flux"),
                              (T.FIELD_HEIGHT, T.FIELD_WATER, T.FIELD_SEDIMENT, T.FIELD_FLUX), want):
            np.testing.assert_array_equal(w.download(f).view(np.uint32), v.view(np.uint32), err_msg=name)


@pytest.mark.parametrize("W,H,iters", [(5, 3, 2), (3, 40, 3), (51, 9, 2), (52, 10, 2), (53, 25, 4), (105, 29, 2),
                                       (104, 41, 3), (7, 130, 2)])
@pytest.mark.parametrize("tile", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("kind", ["tiny", "clamp", "huge"])
def test_two_sub_iterations_on_one_tile(kind, tile, W, H, iters):
    """As above on tiles: one cell less and more than a tile, worlds that wrap within a halo, tiles that run
    again in the scalar form, and an odd number left over."""
    s = T.baseline_settings()
    s.step.hydraulicTile = tile
    h, water, sed, flux = fields(kind, W, H)
    with T.World(s, W, H, seed=1000) as w:
        for f, a in ((T.FIELD_HEIGHT, h), (T.FIELD_WATER, water), (T.FIELD_SEDIMENT, sed), (T.FIELD_FLUX, flux)):
            w.upload(f, a)
        w.hydraulic(iters, 0.02)
        want = O.hydraulic(h, water, sed, flux, iters, 0.02, 1000, s)
        for name, f, v in zip(("height", "water", "sediment", "flux"),
                              (T.FIELD_HEIGHT, T.FIELD_WATER, T.FIELD_SEDIMENT, T.FIELD_FLUX), want):
            np.testing.assert_array_equal(w.download(f).view(np.uint32), v.view(np.uint32), err_msg=name)


@pytest.mark.parametrize("W,H", [(59, 8), (60, 17), (61, 25), (121, 33), (2, 5), (1, 40)])
@pytest.mark.parametrize("tile", [1, 3, 4, 5, 7, 9])
@pytest.mark.parametrize("kind", ["tiny", "clamp", "huge"])
def test_split_path_tiles(kind, tile, W, H):
    """The split path's narrower halo: one column and row less and more than its tiles, worlds that wrap within
    it, and tiles that run again in the scalar form.  dt 0.5 lets the transport reach 25 cells."""
    s = T.baseline_settings()
    s.step.hydraulicTile = tile
    h, water, sed, flux = fields(kind, W, H)
    with T.World(s, W, H, seed=1000) as w:
        for f, a in ((T.FIELD_HEIGHT, h), (T.FIELD_WATER, water), (T.FIELD_SEDIMENT, sed), (T.FIELD_FLUX, flux)):
            w.upload(f, a)
        w.hydraulic(3, 0.5)
        want = O.hydraulic(h, water, sed, flux, 3, 0.5, 1000, s)
        for name, f, v in zip(("height", "water", "sediment", "flux"),
                              (T.FIELD_HEIGHT, T.FIELD_WATER, T.FIELD_SEDIMENT, T.FIELD_FLUX), want):
            np.testing.assert_array_equal(w.download(f).view(np.uint32), v.view(np.uint32), err_msg=name)
