"""The refiner on frames of more bands of 32 rows than fit on the device at once (five blocks of some 40 KB an SM:
740 bands, 23,680 rows; seven with the 64-bit census: 33,152), which take a pass in groups of bands: the maps
equal the oracle's, bit for bit (tolerance 0).  Two groups with one band in the last, three groups, both
censuses, and a frame whose last row is a band of its own."""
import pytest

from helpers import same_bits, synth, to_oracle

pytestmark = pytest.mark.gpu
MAPS = ("disparity", "confidence", "invalid_reason", "reliable_mask")


@pytest.mark.parametrize("w,h,dmax,dmin,over", [
    (24, 23700, 8, 0, {}),
    (40, 24001, 12, -3, {"paths": 4}),
    (17, 47400, 6, 0, {"paths": 4}),
    (20, 33300, 8, 0, {"census_type": 0, "paths": 4}),
])
def test_tall_frames_match_oracle(apg, O, w, h, dmax, dmin, over):
    L, R = synth(w, h, dmax, lo=max(0, dmin), patch=0.25, seed=71)
    cfg = apg.config_from_mode(2, dmax, dmin, **over)
    e = apg.Engine(cfg)
    got = e.process(L, R)
    ref = e.dump("disp_refined")
    e.close()
    want = O.pipeline(to_oracle(O, cfg), L, R, stages=True)
    assert same_bits(ref, want["disp_refined"])
    for k in MAPS:
        assert same_bits(got[k], want[k]), k
