"""Batches of 16-bit sweeps whose buckets launch one after another: a bucket's table of pairs and scanlines is made
while earlier buckets' work fills the device, in memory that an earlier table may have had, and has to be there
before the sweeps read it.  Every call brings other pair counts, so other tables; graphs and plain launches; maps
equal the single-pair engine's, bit for bit (tolerance 0)."""
import random

import pytest

from helpers import same_bits, synth

pytestmark = pytest.mark.gpu
MAPS = ("disparity", "confidence", "invalid_reason", "reliable_mask")
SIZES = [(247, 38, 190), (163, 71, 64), (255, 17, 128), (211, 83, 240), (130, 8, 16)]


@pytest.mark.parametrize("mode,over,opts", [
    (0, {"hier_enable": 1}, {"unified_sgm": 0, "graphs": 0, "autotune": 0}),
    (1, {}, {"sgm_lanes": 16, "graphs": 0, "autotune": 0}),
    (2, {"hier_enable": 1}, {"unified_sgm": 0, "graphs": 0, "autotune": 0}),
    (1, {"agg_iterations": 2, "paths": 8}, {"unified_sgm": 0}),
])
def test_tables_are_there_before_the_sweeps(apg, mode, over, opts):
    rng = random.Random(5)
    cfg = lambda d: apg.config_from_mode(mode, d, 0, P2_base=300, **over)
    want = []
    for i, (w, h, d) in enumerate(SIZES):
        L, R = synth(w, h, d, seed=700 + i)
        e = apg.Engine(cfg(d))
        want.append(((L, R, d), e.process(L, R)))
        e.close()
    for _ in range(6):
        b = apg.Batch(cfg(128), **opts)
        for _ in range(4):
            call = [rng.choice(want) for _ in range(rng.randint(2, 14))]
            for got, (_, exp) in zip(b.process([p for p, _ in call]), call):
                for k in MAPS:
                    assert same_bits(got[k], exp[k]), k
        b.close()
