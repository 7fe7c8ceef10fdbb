"""The pixel-run cost kernel's tile widths without aggregation: frames large enough that a block walks several
tiles (long runs, a padded last tile, ranges below zero and off the 64 grid, per-pixel ranges) against the
column-tile kernel, bit for bit (integer costs; the right-image map shares its final arithmetic)."""
import pytest

from helpers import same_bits, synth

pytestmark = pytest.mark.gpu

CASES = [(0, 1920, 320, 256, 0, {}), (0, 1537, 620, 60, -5, {}), (0, 769, 900, 128, 0, {}), (0, 1281, 500, 190, 3, {}),
         (0, 31, 1500, 64, 0, {}), (2, 1000, 420, 100, 0, {"agg_enable": 0, "refine_enable": 0})]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"m{c[0]}_{c[1]}x{c[2]}_d{c[4]}..{c[3]}")
def test_wide_tiles_equal_column_tiles(apg, case):
    mode, w, h, dmax, dmin, over = case
    L, R = synth(w, h, dmax, lo=max(0, dmin), hi=max(1, min(dmax, w) - 2), patch=0.1, seed=61)
    got = []
    for kernel in (0, 1):
        e = apg.Engine(apg.config_from_mode(mode, dmax, dmin, **over), debug=apg.DEBUG_RAW_COST)
        e.set_tuning("cost_kernel", kernel)
        e.process(L, R)
        got.append((e.dump("cost_raw"), e.dump("disp_right")))
        e.close()
    assert same_bits(got[0][0], got[1][0])
    assert same_bits(got[0][1], got[1][1])


# ranges from the coarse pass and from the prior: runs of narrow ranges (64 disparities and less), of wide ones,
# tiles of both; a range start off the four-word grid and near the end of the range
NARROW = [(1, 1000, 260, 250, 0, {"hier_enable": 1}), (1, 333, 200, 130, -6, {"hier_enable": 1}),
          (1, 640, 130, 190, 0, {"hier_enable": 1, "max_arm_length": 3}), (2, 700, 200, 256, 0, {"refine_enable": 0}),
          (2, 530, 140, 120, 9, {"refine_enable": 0})]


@pytest.mark.parametrize("case", NARROW, ids=lambda c: f"m{c[0]}_{c[1]}x{c[2]}_d{c[4]}..{c[3]}_{len(c[5])}")
def test_narrow_runs_equal_column_tiles(apg, case):
    mode, w, h, dmax, dmin, over = case
    L, R = synth(w, h, dmax, lo=max(0, dmin), hi=max(1, min(dmax, w) - 2), patch=0.1, seed=62)
    got = []
    for kernel in (0, 1):
        e = apg.Engine(apg.config_from_mode(mode, dmax, dmin, **over))
        e.set_tuning("cost_kernel", kernel)
        e.set_tuning("cost8", 1)  # 16-bit volumes in both
        e.process(L, R)
        got.append((e.dump("cost_agg"), e.dump("disp_right")))
        e.set_tuning("cost8", 0)
        if kernel == 0:
            e.process(L, R)
            got.append((e.dump("cost_agg"), e.dump("disp_right")))
        e.close()
    for other in got[1:]:
        assert same_bits(got[0][0], other[0])
        assert same_bits(got[0][1], other[1])
