"""The refiner on frames whose rows are longer than one block's shared memory holds (five bytes a column beside
some 40 KB: about 38,000 columns, 40,000 with the 64-bit census), which take a pass in runs of columns: the
maps equal the oracle's, bit for bit (tolerance 0).  One band, two bands and bands of several clusters; both
censuses; the window in shared memory and through L1; widths around the split."""
import pytest

from helpers import same_bits, synth, to_oracle

pytestmark = pytest.mark.gpu
MAPS = ("disparity", "confidence", "invalid_reason", "reliable_mask")


@pytest.mark.parametrize("w,h,dmax,dmin,over,window", [
    (40001, 3, 16, 0, {}, 0),
    (39990, 35, 12, 0, {}, 0),
    (38777, 40, 14, -5, {}, 1),
    (40510, 33, 10, 0, {"census_type": 0}, 0),
    (38720, 265, 6, 0, {"agg_enable": 0, "paths": 4}, 0),
])
def test_wide_frames_match_oracle(apg, O, w, h, dmax, dmin, over, window):
    L, R = synth(w, h, dmax, lo=max(0, dmin), patch=0.25, seed=67)
    cfg = apg.config_from_mode(2, dmax, dmin, **over)
    e = apg.Engine(cfg)
    e.set_tuning("refine_window", window)
    got = e.process(L, R)
    ref = e.dump("disp_refined")
    e.close()
    want = O.pipeline(to_oracle(O, cfg), L, R, stages=True)
    assert same_bits(ref, want["disp_refined"])
    for k in MAPS:
        assert same_bits(got[k], want[k]), k
