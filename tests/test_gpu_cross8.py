"""Cross aggregation over byte volumes (the default where every cost is below 255) against the 16-bit
kernels (tuning cost8 = 1): the aggregated volume bit for bit (integers; tolerance 0).  Shapes: heights
around the row segments and four-row chunks, widths around a block's columns, arms from 1 to the longest
the byte form takes and one past it, ranges that leave padded disparities, start below zero or come from
the prior or the hierarchical pass."""
import numpy as np
import pytest

from helpers import same_bits, synth

pytestmark = pytest.mark.gpu

CASES = [
    (1, 65, 31, 64, 0, {}), (1, 63, 32, 64, 0, {}), (1, 64, 33, 50, 0, {}), (1, 129, 130, 128, 0, {}),
    (1, 140, 257, 100, 0, {}), (1, 200, 65, 192, 0, {}), (1, 259, 35, 256, 0, {}), (1, 5, 70, 64, 0, {}),
    (1, 90, 1, 64, 0, {}), (1, 1, 90, 16, 0, {}), (1, 150, 40, 130, 9, {}), (1, 150, 70, 60, -7, {}),
    (1, 220, 40, 180, -20, {}), (1, 128, 96, 64, 0, {"hier_enable": 1}), (1, 192, 96, 200, 0, {"hier_enable": 1}),
    (2, 160, 96, 64, 0, {}), (2, 200, 64, 250, 0, {}),
    (1, 90, 70, 64, 0, {"max_arm_length": 1}), (1, 90, 70, 64, 0, {"max_arm_length": 17, "color_threshold": 255}),
    (1, 90, 70, 64, -3, {"max_arm_length": 17, "color_threshold": 255}),
    (1, 90, 70, 64, 0, {"max_arm_length": 18, "color_threshold": 255}),
    (1, 90, 70, 64, 0, {"census_type": 0}), (1, 90, 70, 64, 0, {"agg_iterations": 2}),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"m{c[0]}_{c[1]}x{c[2]}_d{c[4]}..{c[3]}_{'_'.join(map(str, c[5].values())) or 'preset'}")
def test_byte_aggregation_equals_16_bit(apg, case):
    mode, w, h, dmax, dmin, over = case
    L, R = synth(w, h, dmax, lo=max(0, dmin), hi=max(1, min(dmax, w) - 2), patch=0.2, seed=43)
    cfg = apg.config_from_mode(mode, dmax, dmin, **over)
    vols = []
    for cost8 in (0, 1):
        e = apg.Engine(cfg)
        e.set_tuning("cost8", cost8)
        e.process(L, R)
        vols.append(e.dump("cost_agg"))
        e.close()
    assert same_bits(vols[0], vols[1]), np.argwhere(vols[0] != vols[1])[:3]
