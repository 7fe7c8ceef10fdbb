"""The refiner's band wavefront at the edges of its division of work, against the oracle, bit for bit
(tolerance 0): bands in one and several thread-block clusters, a last band of one row, images narrower
than a band's lanes, column counts around the eight-column hand-over, the 64-bit census (left images in
48-byte records), and the forms of the right-image window (shared memory, and global loads on request
or for ranges the window does not hold)."""
import numpy as np
import pytest

from helpers import same_bits, synth, to_oracle

pytestmark = pytest.mark.gpu
MAPS = ("disparity", "confidence", "invalid_reason", "reliable_mask")


@pytest.mark.parametrize("w,h,dmax,dmin,over,window", [
    (64, 256, 24, 0, {}, 0),       # 8 bands: one cluster
    (97, 300, 32, 0, {}, 0),       # 10 bands: two clusters
    (40, 545, 24, 0, {}, 0),       # 18 bands, the last of one row
    (17, 290, 12, 0, {}, 0),       # narrower than a band's 32 lanes
    (71, 100, 20, 0, {}, 0), (72, 100, 20, 0, {}, 0), (73, 100, 20, 0, {}, 0),
    (90, 280, 16, -8, {}, 0),
    (96, 300, 32, 0, {}, 1),       # the window read through L1
    (80, 290, 24, 0, {"census_type": 0}, 0),
    (520, 40, 500, 0, {"agg_enable": 0}, 0),
])
def test_refiner_bands_match_oracle(apg, O, w, h, dmax, dmin, over, window):
    L, R = synth(w, h, dmax, patch=0.25, seed=41)
    cfg = apg.config_from_mode(2, dmax, dmin, **over)
    e = apg.Engine(cfg)
    e.set_tuning("refine_window", window)
    got = [e.process(L, R) for _ in range(2)]  # the second frame on the same buffers
    ref = e.dump("disp_refined")
    e.close()
    want = O.pipeline(to_oracle(O, cfg), L, R, stages=True)
    assert same_bits(ref, want["disp_refined"])
    for k in MAPS:
        assert same_bits(got[0][k], want[k]) and same_bits(got[1][k], want[k]), k
