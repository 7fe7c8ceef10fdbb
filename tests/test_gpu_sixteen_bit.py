"""The 16-bit sweeps, which penalties past a byte, more than 256 disparities, several aggregation passes and very
large frames take: the forms that presets no longer reach, against each other and the oracle, bit for bit
(tolerance 0)."""
import pytest

from helpers import same_bits, synth, to_oracle

pytestmark = pytest.mark.gpu
MAPS = ("disparity", "confidence", "invalid_reason", "reliable_mask")


@pytest.mark.parametrize("mode,w,h,dmax,dmin,over,cost8", [
    (0, 301, 47, 256, 0, {}, 0), (1, 301, 65, 250, 0, {}, 0), (1, 200, 33, 220, -9, {}, 0),
    (0, 300, 40, 256, 0, {"paths": 8}, 0), (2, 280, 48, 200, 0, {}, 0), (0, 17, 9, 250, 0, {}, 0),
    (0, 260, 64, 230, 0, {"hier_enable": 1}, 0), (1, 260, 64, 230, 0, {"census_type": 0}, 0),
    (0, 201, 49, 128, 0, {}, 2), (1, 201, 49, 100, 0, {}, 2),
])
def test_sixteen_bit_sweeps_over_byte_volumes(apg, O, mode, w, h, dmax, dmin, over, cost8):
    """Penalties past a byte: the volume keeps one byte per voxel at 256 padded disparities (and on request at
    128), both forms of the last sweep widen it, and maps and path sums equal those over a two-byte volume."""
    L, R = synth(w, h, dmax, lo=max(0, dmin), hi=max(1, min(dmax, w) - 2), patch=0.2, seed=53)
    cfg = apg.config_from_mode(mode, dmax, dmin, P1=120, P2_base=700, **over)
    outs, sizes = [], []
    for form, split in ((cost8, 1), (cost8, 2), (1, 0)):
        e = apg.Engine(cfg, debug=apg.DEBUG_KEEP_SUM)
        e.set_tuning("cost8", form)
        e.set_tuning("sgm_split", split)
        o = e.process(L, R)
        o["sgm_sum"] = e.dump("sgm_sum")
        sizes.append(e.allocated_bytes)
        e.close()
        outs.append(o)
    Dp = 128 if cost8 else 256
    assert sizes[2] - sizes[0] >= w * h * Dp - 512  # two allocations, each rounded up to 256 bytes
    for o in outs[1:]:
        for k in o:
            assert same_bits(o[k], outs[0][k]), k
    if not over.get("hier_enable"):
        want = O.pipeline(to_oracle(O, cfg), L, R)
        for k in MAPS:
            assert same_bits(outs[0][k], want[k]), k
