"""Workspace sizes that admission and memory budgets rest on: what fits one form of a configuration is not
taken away by another (whole bytes, no tolerance but the stated one)."""
import pytest


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("w,h", [(1920, 1080), (301, 65)])
def test_penalties_past_a_byte_take_no_more(apg, mode, w, h):
    """At 256 padded disparities the volume takes one byte per voxel whatever the penalties are."""
    ws = [apg.workspace_bytes(apg.config_from_mode(mode, 256, 0, **over), w, h) for over in ({}, {"P2_base": 300})]
    assert ws[0] == ws[1]


def test_frames_of_four_gigavoxels_keep_the_byte_volume(apg):
    w, h = 8192, 2300  # 4.8e9 voxels at 256 disparities
    for mode, vols in ((0, 3.5), (1, 3.5), (2, 7.5)):
        vol = w * h * 256 * 2
        assert apg.workspace_bytes(apg.config_from_mode(mode, 256), w, h) < (vols + 0.3) * vol
