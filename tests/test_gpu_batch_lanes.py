"""Batches held to 16 lanes per chain: sizes that no other batch has tuned, and the option changed between
calls of one batch, against the single-pair engine, bit for bit (tolerance 0)."""
import pytest

from helpers import same_bits, synth

pytestmark = pytest.mark.gpu
KEYS = ("disparity", "confidence", "invalid_reason", "reliable_mask")


def _check(apg, b, mode, pairs):
    for got, (L, R, dmax) in zip(b.process(pairs), pairs):
        e = apg.Engine(apg.config_from_mode(mode, dmax))
        want = e.process(L, R)
        e.close()
        for k in KEYS:
            assert same_bits(got[k], want[k]), k


def _pairs(sizes, seed):
    return [(*synth(w, h, d, seed=seed + i), d) for i, (w, h, d) in enumerate(sizes)]


@pytest.mark.parametrize("mode,opts,sizes", [
    (1, {"sgm_lanes": 16}, [(167, 93, 64), (167, 93, 64), (203, 61, 128)]),
    (0, {"sgm_lanes": 16, "unified_sgm": 0}, [(169, 91, 64), (205, 63, 250)]),
    (1, {"sgm_lanes": 16, "autotune": 0}, [(171, 95, 64), (207, 65, 192)]),
])
def test_sixteen_lanes_on_sizes_of_their_own(apg, mode, opts, sizes):
    b = apg.Batch(apg.config_from_mode(mode, 128), **opts)
    for seed in (500, 510):
        _check(apg, b, mode, _pairs(sizes, seed))
    b.close()


def test_lanes_changed_between_calls(apg):
    b = apg.Batch(apg.config_from_mode(1, 128))
    for i, lanes in enumerate((0, 16, 32, 16, 0)):
        b.set_option("sgm_lanes", lanes)
        # a size of every call, and one that only this call has
        _check(apg, b, 1, _pairs([(173, 97, 64), (175 + 2 * i, 67, 128)], 520 + 10 * i))
    b.close()
