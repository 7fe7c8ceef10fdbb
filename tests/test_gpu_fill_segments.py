"""Hole fill by 32-pixel segments (the neighbouring segments loaded with the own one) against the per-pixel walk
(the form that counts telemetry): the final map bit for bit, at gaps around one and two segments, widths
around segment borders and frames with wide holes."""
import numpy as np
import pytest

from helpers import same_bits, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap", [0, 1, 31, 33, 64, 200])
@pytest.mark.parametrize("w", [1, 31, 32, 33, 64, 65, 97, 300])
def test_segments_equal_walk(apg, gap, w):
    h, dmax = 24, 16
    L, R = synth(w, h, dmax, lo=0, hi=max(1, min(dmax, w) - 2), patch=0.3, seed=17)
    R = np.where(np.random.default_rng(w).random((h, 1)) < 0.5, R, np.uint8(90))  # rows of the right image blank: long holes
    for mode, shadow in ((1, apg.InpaintMethod.Legacy), (1, apg.InpaintMethod.ShadowReclass)):
        e = apg.Engine(apg.config_from_mode(mode, dmax, 0, max_fill_gap=gap))
        maps = []
        for telemetry in (False, True):
            with apg.ExperimentalInpaintScope(shadow, 32 if shadow == apg.InpaintMethod.Legacy else gap, collect_telemetry=telemetry):
                maps.append(e.process(L, R)["disparity"])
        e.close()
        assert same_bits(maps[0], maps[1])
