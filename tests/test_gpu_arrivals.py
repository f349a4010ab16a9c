"""Arrival words, collision evidence and the resolve at dense, ragged and far-moving arrivals.

Blocks of arrivals lie in one world or over several, runs of one to many arrivals cross their ends, and
destinations without arrivals form gaps from one cell to whole rows of worlds, at a world's start and end.
Salt-and-pepper plates give every cell a class of its own, so that the resolve's lists of divergent and
convergent cells fill up.  Words, ids, bitmaps and marks are whole numbers, and the heights come from the same IEEE
operations in the same order: everything equals the oracle exactly.
"""
from __future__ import annotations

import numpy as np
import pytest

import master_thesis_gb300 as T
import oracle as O

pytestmark = pytest.mark.gpu

SMALL = [(61, 23)]                                    # one position a thread
SPREAD = [(33, 17), (3, 2), (64, 64), (7, 300), (129, 65)]
LARGE = [(1001, 521), (33, 17), (64, 64), (5, 3), (130, 70)]  # 2^19 cells and more: four a thread


@pytest.mark.parametrize("shapes", [SMALL, SPREAD, LARGE])
@pytest.mark.parametrize("kind", ["noise", "far", "stripes"])
@pytest.mark.parametrize("radius", [None, 3, 8])
def test_arrivals_match_oracle(kind, shapes, radius):
    if shapes is LARGE and radius == 8:
        pytest.skip("the largest batch at two radii")
    s = T.baseline_settings()
    s.step.hydraulicIterations = 0
    s.step.thermalIterations = 0
    if radius is None:
        s.step.upliftMode = T.UPLIFT_NONE
    else:
        s.step.upliftRadius = radius
    s.kernel.minCollisionSize = 2
    s.kernel.collisionTypeUpdateCooldown = 1
    worlds, oracles = [], []
    for i, (W, H) in enumerate(shapes):
        w = T.World(s, W, H, seed=1000 + i)
        w.init_synthetic(7, 150.0 if kind == "far" else 6.0, 5 + i)
        ids = w.download(T.FIELD_PLATE_ID)
        rng = np.random.default_rng(i)
        if kind == "noise":
            ids = rng.integers(0, 7, (H, W)).astype(np.uint8)
        elif kind == "stripes":
            ids = np.broadcast_to((np.arange(W) // 3 % 7).astype(np.uint8), (H, W)).copy()
        w.upload(T.FIELD_PLATE_ID, ids)
        worlds.append(w)
        oracles.append(O.OracleWorld(s, w.download(T.FIELD_HEIGHT), ids, w.plates(), 1000 + i))
    b = T.Batch() if len(worlds) > 1 else None
    if b:
        for w in worlds:
            b.add(w)
    for step in range(2):
        if b:
            b.step(1)
        else:
            worlds[0].step(1)
        for i, (w, o) in enumerate(zip(worlds, oracles)):
            o.step(1)
            for name, f, want in (("words", T.FIELD_COLLISION, o.word), ("ids", T.FIELD_PLATE_ID, o.id),
                                  ("height", T.FIELD_HEIGHT, o.h), ("types", T.FIELD_TYPE_BITMAP, o.bitmap),
                                  ("divergence", T.FIELD_DIV_BITMAP, o.div), ("accretion", T.FIELD_ACCRETION, o.acc)):
                np.testing.assert_array_equal(w.download(f).ravel(), want.ravel(),
                                              err_msg=f"{name} of {shapes[i]}, step {step}")
    if b:
        b.check()
        b.close()
    for w in worlds:
        w.close()
