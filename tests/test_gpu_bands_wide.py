"""Host frames in row bands over the byte sweeps where the test of small frames does not reach: frames so wide
that a band's sweep runs one warp per pair of columns (some 1,500 columns at 256 padded disparities, 1,800 at
128 and 192, 3,600 at 64), the default number of bands on frames that take several, and an experimental scope.
Maps equal those of one sweep, bit for bit (tolerance 0), and the oracle's where stated."""
import pytest

from helpers import same_bits, synth, to_oracle

pytestmark = pytest.mark.gpu
MAPS = ("disparity", "confidence", "invalid_reason", "reliable_mask")


def _run(apg, cfg, L, R, bands):
    e = apg.Engine(cfg)
    e.set_tuning("host_bands", bands)
    out = e.process(L, R)
    e.close()
    return out


@pytest.mark.parametrize("mode,w,h,dmax,over", [
    (0, 1931, 257, 256, {}), (1, 1921, 260, 250, {}), (0, 1999, 289, 128, {}), (1, 2101, 256, 100, {}),
    (0, 1801, 300, 192, {}), (0, 3601, 257, 64, {}), (1, 1921, 257, 256, {"P1": 60, "P2_base": 200}),
])
def test_wide_frames_in_bands(apg, mode, w, h, dmax, over):
    L, R = synth(w, h, dmax, cells=8, hi=dmax - 8, seed=77)
    cfg = apg.config_from_mode(mode, dmax, 0, **over)
    want = _run(apg, cfg, L, R, 1)
    for bands in (0, 2, 5):
        got = _run(apg, cfg, L, R, bands)
        for k in MAPS:
            assert same_bits(got[k], want[k]), (bands, k)


@pytest.mark.parametrize("mode,w,h,dmax,bands", [(0, 384, 300, 128, 4), (1, 352, 289, 192, 3), (0, 811, 700, 64, 0)])
def test_bands_match_oracle(apg, O, mode, w, h, dmax, bands):
    L, R = synth(w, h, dmax, cells=6, hi=dmax - 8, seed=78)
    cfg = apg.config_from_mode(mode, dmax)
    got = _run(apg, cfg, L, R, bands)
    want = O.pipeline(to_oracle(O, cfg), L, R)
    for k in MAPS:
        assert same_bits(got[k], want[k]), k


def test_bands_under_experimental_scope(apg):
    L, R = synth(640, 360, 128, cells=8, seed=79)
    cfg = apg.config_from_mode(1, 128)
    outs = []
    for bands in (4, 1):
        with apg.ExperimentalSubpixelScope(2, 0.3):
            outs.append(_run(apg, cfg, L, R, bands))
    for k in MAPS:
        assert same_bits(outs[0][k], outs[1][k]), k
