"""The right-image disparity map asked for after a frame: where the frame wrote the map (stages kept, the
refiner), the dump is that map and starts no kernel; where it did not, one kernel writes it from the keys.
Both give the same bits (tolerance 0)."""
import pytest

from helpers import same_bits, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,w,h,dmax,over", [(0, 131, 47, 64, {}), (1, 131, 47, 64, {}), (2, 131, 47, 64, {})])
def test_the_frames_own_map_is_dumped(apg, mode, w, h, dmax, over):
    L, R = synth(w, h, dmax, patch=0.2, seed=37)
    cfg = apg.config_from_mode(mode, dmax, 0, **over)
    maps = []
    for debug, refine in ((apg.DEBUG_RAW_COST, 0), (0, 0), (0, 1)):
        cfg.refine_enable = refine
        e = apg.Engine(cfg, debug=debug)
        e.process(L, R)
        before = apg.kernel_launch_count()
        maps.append(e.dump("disp_right"))
        assert apg.kernel_launch_count() - before == (0 if debug or refine else 1)
        e.close()
    assert same_bits(maps[0], maps[1]) and same_bits(maps[0], maps[2])
