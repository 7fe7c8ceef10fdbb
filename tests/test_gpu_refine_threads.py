"""HighQuality engines of growing sizes first used from several threads at once: they share the host's draw tables,
which a longer frame lengthens, and copy them to their devices.  Radii no other test uses, so that the tables grow
here.  Maps equal those of engines used one after another, bit for bit (tolerance 0)."""
import threading

import pytest

from helpers import same_bits, synth

pytestmark = pytest.mark.gpu
MAPS = ("disparity", "confidence", "invalid_reason", "reliable_mask")


@pytest.mark.parametrize("radius", [23, 29])
def test_draw_tables_grow_under_threads(apg, radius):
    cfg = apg.config_from_mode(2, 32, 0, refine_random_radius=radius)
    pairs = [synth(40 + 24 * i, 33 + 9 * i, 32, patch=0.25, seed=80 + i) for i in range(12)]
    got = [None] * len(pairs)

    def run(first):
        for i in range(first, len(pairs), 4):
            e = apg.Engine(cfg)
            got[i] = e.process(*pairs[i])
            e.close()

    threads = [threading.Thread(target=run, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, p in enumerate(pairs):
        e = apg.Engine(cfg)
        want = e.process(*p)
        e.close()
        assert got[i] is not None, i
        for k in MAPS:
            assert same_bits(got[i][k], want[k]), (i, k)
