"""Sub-pixel telemetry at odd widths against the oracle.  The byte sweeps run two scanlines per warp; an odd
number of columns leaves the last warp one, whose pixels count once.  The counters are whole numbers
(tolerance 0); the sum of shifts is added in another order (relative 1e-12).  Shapes: both forms of the last
sweep (two warps per pair up to some 1,500 columns at 256 padded disparities, one beyond), both path counts,
and a hierarchical frame whose half width is odd."""
import pytest

from helpers import synth, to_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture
def oracle_scope(O):
    yield
    O.set_experimental()


@pytest.mark.parametrize("mode,w,h,dmax,over", [
    (1, 161, 96, 48, {}), (0, 97, 33, 64, {}), (0, 1, 40, 16, {}), (1, 201, 40, 128, {"paths": 8}),
    (0, 211, 40, 192, {}), (0, 1931, 24, 250, {}), (1, 162, 96, 48, {"hier_enable": 1}),
])
def test_telemetry_counts_each_pixel_once(apg, O, oracle_scope, mode, w, h, dmax, over):
    L, R = synth(w, h, dmax, hi=max(1, min(dmax, w) - 2), patch=0.25, seed=61)
    cfg = apg.config_from_mode(mode, dmax, **over)
    O.set_experimental(2, 0.0, 0, 32, sp_telemetry=True, ip_telemetry=True)
    O.pipeline(to_oracle(O, cfg), L, R)
    want, _ = O.get_telemetry()
    e = apg.Engine(cfg)
    with apg.ExperimentalSubpixelScope(2, 0.0, collect_telemetry=True), \
            apg.ExperimentalInpaintScope(0, 32, collect_telemetry=True):
        e.process(L, R)
        got = apg.ExperimentalSubpixelScope.current_telemetry()
    e.close()
    for k, v in want.items():
        assert getattr(got, k) == (pytest.approx(v, rel=1e-12) if k == "sum_abs_delta" else v), k
