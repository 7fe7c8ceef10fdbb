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


@pytest.mark.parametrize("mode,w,h,dmax,dmin,over", [
    (0, 200, 100, 48, 0, {}), (1, 333, 90, 128, 0, {}), (1, 150, 80, 200, 0, {}), (1, 120, 90, 40, 0, {"paths": 8}),
    (2, 160, 96, 64, 0, {}), (1, 97, 61, 24, -6, {}), (0, 64, 7, 16, 0, {}),
])
def test_last_sweep_on_one_and_two_warps(apg, mode, w, h, dmax, dmin, over):
    """Both forms of the 16-bit last sweep (tuning sgm_split) give the same maps and sums."""
    L, R = synth(w, h, dmax, lo=max(0, dmin), patch=0.2, seed=23)
    cfg = apg.config_from_mode(mode, dmax, dmin, P2_base=400, **over)
    outs = []
    for split in (1, 2):
        e = apg.Engine(cfg, debug=apg.DEBUG_KEEP_SUM)
        e.set_tuning("sgm_split", split)
        outs.append(e.process(L, R))
        outs[-1]["sgm_sum"] = e.dump("sgm_sum")
        e.close()
    for k in outs[0]:
        assert same_bits(outs[0][k], outs[1][k]), k


@pytest.mark.parametrize("mode,w,h,dmax,dmin,over", [
    (0, 384, 300, 128, 0, {}), (1, 352, 289, 192, 0, {}), (1, 300, 301, 256, 0, {}), (0, 333, 257, 250, 0, {}),
    (1, 320, 257, 100, -20, {}), (1, 340, 280, 128, 0, {"hier_enable": 1}),
])
def test_banded_last_sweep(apg, O, mode, w, h, dmax, dmin, over):
    """Host frames whose last 16-bit sweep runs in row bands equal those of one sweep and the oracle's."""
    L, R = synth(w, h, dmax, lo=max(0, dmin), hi=dmax - 8, seed=72)
    cfg = apg.config_from_mode(mode, dmax, dmin, P2_base=400, **over)
    want = None if over.get("hier_enable") else O.pipeline(to_oracle(O, cfg), L, R)
    for bands in (1, 2, 6, 16):
        e = apg.Engine(cfg)
        e.set_tuning("host_bands", bands)
        got = e.process(L, R)
        e.close()
        want = want or got
        for k in MAPS:
            assert same_bits(got[k], want[k]), (bands, k)


@pytest.mark.parametrize("opts", [{}, {"graphs": 0}, {"batched_sgm": 0}, {"unified_sgm": 0}, {"max_blocks_per_sm": 1, "autotune": 0},
                                  {"sgm_lanes": 16, "autotune": 0}])
@pytest.mark.parametrize("mode", [0, 1])
def test_batched_launch_over_all_ranges(apg, mode, opts):
    """Pairs of every padded range and several sizes in one persistent launch per phase (and in the forms the
    options choose): each pair's maps equal its own engine's; the second call replays the graph."""
    sizes = [(151, 81, 60), (151, 81, 60), (201, 99, 128), (259, 61, 190), (301, 49, 250)]
    b = apg.Batch(apg.config_from_mode(mode, 128, 0, P2_base=400), **opts)
    for seed in (600, 620):
        pairs = [(*synth(w, h, d, seed=seed + i), d) for i, (w, h, d) in enumerate(sizes)]
        for got, (L, R, d) in zip(b.process(pairs), pairs):
            e = apg.Engine(apg.config_from_mode(mode, d, 0, P2_base=400))
            want = e.process(L, R)
            e.close()
            for k in MAPS:
                assert same_bits(got[k], want[k]), (d, k)
    b.close()
