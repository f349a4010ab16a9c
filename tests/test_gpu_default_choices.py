"""Which kernels a call runs where its settings leave the choice to the engine, seen by the launches it makes."""
from __future__ import annotations

import pytest

import master_thesis_gb300 as T

pytestmark = pytest.mark.gpu


def launches(W, H, s, call):
    with T.World(s, W, H, seed=1) as w:
        w.init_synthetic(4, 1.0, 1)
        before = w.launches
        call(w)
        return w.launches - before


# the march takes one iteration a launch, the tiles of variant 4 two
@pytest.mark.parametrize("thr,A,S,march", [(0.01, 0.5, 1.0, True), (0.01, 0.3, 0.7, True), (0.0, 0.5, 1.0, False),
                                           (1e-12, 0.5, 1.0, False), (0.01, -0.5, 1.0, False)])
def test_thermal_march_from_a_million_cells_in_its_packed_forms(thr, A, S, march):
    s = T.baseline_settings()
    s.kernel.thermalThresholdAngle, s.kernel.thermalCellSize = thr, 1.0
    s.kernel.thermalErosionAmplitude, s.kernel.thermalErosionStrength = A, S
    assert launches(1100, 1000, s, lambda w: w.thermal(10)) == (10 if march else 5)


# rain, then two sub-iterations a launch (variant 4) or one (variant 7 has no form for two)
@pytest.mark.parametrize("W,H,tile,count", [(400, 400, 7, 3), (362, 362, 7, 5), (400, 400, 4, 3)])
def test_short_tiles_run_in_small_batches_only(W, H, tile, count):
    s = T.baseline_settings()
    s.step.hydraulicTile = tile  # dt 0.02: not the split path
    assert launches(W, H, s, lambda w: w.hydraulic(4, 0.02)) == count
