"""The byte sweeps (two scanlines per warp, one byte per voxel and direction) against the 16-bit sweeps
(tuning cost8 = 1) and the oracle: bit-identical maps and final path sums (integers; tolerance 0).

Shapes sit at the edges of the kernels' division of work: an odd number of scanlines (a warp with one),
one row, one column, lengths around the 8-, 16- and 32-step blocks, each padded range with and without
padded disparities, ranges that start below and above zero, per-pixel ranges (hierarchical, prior), both
path counts, penalties whose pairwise sums leave a byte, and the largest penalty the sweeps take."""
import numpy as np
import pytest

from helpers import same_bits, synth, to_oracle

pytestmark = pytest.mark.gpu
MAPS = ("disparity", "confidence", "invalid_reason", "reliable_mask")

CASES = [
    # mode, w, h, dmax, dmin, overrides
    (1, 97, 61, 64, 0, {}),
    (1, 65, 33, 40, 0, {}),
    (1, 160, 120, 64, 0, {"paths": 8}),
    (0, 131, 47, 64, 0, {}),
    (0, 201, 49, 128, 0, {}),
    (1, 200, 31, 100, -6, {}),
    (1, 210, 64, 192, 0, {}),
    (0, 251, 33, 170, 0, {}),
    (1, 260, 40, 180, 8, {"paths": 8}),
    (1, 301, 35, 256, 0, {}),
    (0, 300, 64, 256, 0, {"paths": 8}),
    (0, 64, 1, 48, 0, {}),
    (0, 1, 50, 16, 0, {}),
    (1, 17, 16, 130, 0, {}),
    (1, 150, 80, 64, 0, {"hier_enable": 1}),
    (0, 180, 80, 128, 0, {"hier_enable": 1}),
    (2, 160, 96, 64, 0, {}),
    (2, 200, 80, 190, 0, {}),
    (1, 140, 70, 128, 0, {"P1": 60, "P2_base": 200}),
    (1, 140, 70, 192, 0, {"P1": 100, "P2_base": 255, "paths": 8}),
    (1, 120, 60, 64, 0, {"P1": 0, "P2_base": 1, "adaptive_penalties": 0}),
    # more chains than the first sweep keeps on the device at once; last sweeps on one warp per pair
    (0, 700, 1500, 130, 0, {}),
    (0, 320, 800, 200, 0, {"paths": 8}),
    (0, 1930, 60, 150, 0, {}),
    (0, 1930, 45, 250, 0, {}),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"m{c[0]}_{c[1]}x{c[2]}_d{c[4]}..{c[3]}_{'_'.join(c[5]) or 'preset'}")
def test_byte_sweeps_equal_16_bit_sweeps(apg, O, case):
    mode, w, h, dmax, dmin, over = case
    L, R = synth(w, h, dmax, patch=0.2 if mode == 2 else 0.0, seed=31)
    cfg = apg.config_from_mode(mode, dmax, dmin, **over)
    outs = []
    for cost8 in (0, 1):
        for debug in (0, apg.DEBUG_KEEP_SUM):
            e = apg.Engine(cfg, debug=debug)
            e.set_tuning("cost8", cost8)
            o = e.process(L, R)
            if debug:
                for k in ("sgm_sum", "best", "second", "disp_wta"):
                    o[k] = e.dump(k)
            e.close()
            outs.append(o)
    for o in outs[1:]:
        for k in MAPS:
            assert same_bits(o[k], outs[0][k]), k
    for k in ("sgm_sum", "best", "second", "disp_wta"):
        assert same_bits(outs[1][k], outs[3][k]), k
    if not over.get("hier_enable"):
        want = O.pipeline(to_oracle(O, cfg), L, R)
        for k in MAPS:
            assert same_bits(outs[0][k], want[k]), k
