"""Aux planes (gray, gradients, census) of tiles staged by words or by bytes: device images at every byte offset
and stride remainder give the planes of the packed, aligned image, bit for bit.  Widths around a tile with its
halo (the words form starts at two tiles and four columns), heights around a tile."""
import pytest
import torch

from helpers import same_bits, synth

pytestmark = pytest.mark.gpu
PLANES = ("left_gray", "left_gx", "left_gy", "right_gray", "right_gx", "right_gy", "census_left", "census_right")


@pytest.mark.parametrize("w,h", [(33, 5), (67, 33), (68, 32), (69, 70), (100, 31), (131, 40), (264, 65)])
def test_word_staging_equals_byte_staging(apg, w, h):
    L, R = synth(w, h, 16, seed=3)
    e = apg.Engine(apg.config_from_mode(1, 16, 0))
    want = None
    for off in (0, 1, 2, 3):
        for pad in (0, 1, 2, 3, 4):
            stride = w + pad
            dev = []
            for im in (L, R):
                t = torch.zeros(off + stride * h + 8, dtype=torch.uint8, device="cuda")
                t[off:off + stride * h].view(h, stride)[:, :w] = torch.from_numpy(im).cuda()
                dev.append(t)
            torch.cuda.synchronize()
            e.process_device(dev[0].data_ptr() + off, dev[1].data_ptr() + off, w, h, stride, 1)
            e.sync()
            got = [e.dump(p) for p in PLANES]
            want = want or got
            for p, a, b in zip(PLANES, got, want):
                assert same_bits(a, b), (p, off, pad)
    e.close()
