"""Device frames whose confidence stage works the right-image disparities out from the argmin keys and writes
the caller's maps itself: the maps equal those of a frame that keeps every stage (the right-image map of its
own launch), bit for bit, and so does the right-image map asked for afterwards.  Forms: 32- and 64-bit census,
ranges from the prior, a range below zero, sub-pixel off, the refiner with and without the check behind it,
and a float buffer off the 4-byte grid."""
import numpy as np
import pytest
import torch

from helpers import same_bits, synth

pytestmark = pytest.mark.gpu

CASES = [
    (0, 33, 9, 16, 0, {}), (0, 200, 64, 64, 0, {}), (1, 131, 70, 50, -7, {}), (1, 160, 48, 64, 0, {"subpixel": 0}),
    (1, 160, 48, 64, 0, {"census_type": 1}), (1, 160, 48, 64, 0, {"census_type": 0}), (1, 160, 48, 64, 0, {"lr_check": 0}),
    (2, 150, 64, 60, 0, {}), (2, 150, 64, 60, 0, {"refine_enable": 0}), (2, 150, 64, 60, 0, {"lr_check": 0}),
]
MAPS = (("disparity", torch.float32), ("confidence", torch.float32), ("invalid_reason", torch.uint8),
        ("reliable_mask", torch.uint8))


@pytest.mark.parametrize("skew", [0, 1])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"m{c[0]}_{c[1]}x{c[2]}_d{c[4]}..{c[3]}_{'_'.join(map(str, c[5].items())) or 'preset'}")
def test_direct_maps_equal_staged_ones(apg, case, skew):
    mode, w, h, dmax, dmin, over = case
    L, R = synth(w, h, dmax, lo=max(0, dmin), hi=max(1, min(dmax, w) - 2), patch=0.2, seed=29)
    cfg = apg.config_from_mode(mode, dmax, dmin, **over)
    staged = apg.Engine(cfg, debug=1)
    want = staged.process(L, R)
    e = apg.Engine(cfg)
    dl, dr = torch.from_numpy(L).cuda(), torch.from_numpy(R).cuda()
    raw = {k: torch.zeros(w * h * t.itemsize + 16, dtype=torch.uint8, device="cuda") for k, t in MAPS}
    off = {"disparity": 0, "confidence": skew, "invalid_reason": skew, "reliable_mask": skew}
    torch.cuda.synchronize()
    e.process_device(dl.data_ptr(), dr.data_ptr(), w, h, w, 1, *(raw[k].data_ptr() + off[k] for k, _ in MAPS))
    e.sync()
    for k, t in MAPS:
        got = raw[k][off[k]:off[k] + w * h * t.itemsize].cpu().numpy().copy()
        got = got.view(np.float32 if t == torch.float32 else np.uint8).reshape(h, w)
        assert same_bits(got, want[k]), k
        assert not raw[k][off[k] + w * h * t.itemsize:].any()
    for _ in range(2):
        assert same_bits(e.dump("disp_right"), staged.dump("disp_right"))
    e.close()
    staged.close()
