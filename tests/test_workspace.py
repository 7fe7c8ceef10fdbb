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


@pytest.mark.parametrize("w,h,dmax", [(64, 64, 16), (160, 120, 64), (1242, 375, 192), (1920, 1080, 256), (20, 2000, 16)])
@pytest.mark.parametrize("over", [{}, {"census_type": 0}, {"paths": 4}])
def test_refiner_workspace(apg, w, h, dmax, over):
    """The refiner's own buffers: a 4-byte draw index, two packed images and one 32-byte record per pixel at
    most, and scratch that does not grow with the frame's area (a kilobyte per 32 rows, 16 KB in all)."""
    pack = 32 if over.get("census_type") == 0 else 16
    ws = [apg.workspace_bytes(apg.config_from_mode(2, dmax, 0, refine_enable=r, **over), w, h) for r in (0, 1)]
    assert 0 < ws[1] - ws[0] <= w * h * (4 + pack + 32) + h * 32 + 16384
