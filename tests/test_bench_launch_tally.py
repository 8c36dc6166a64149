"""The ring kernels that bench.py counts for a pass: one per ring list, or one for both
common lists of a small pass."""

import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench  # noqa: E402


@pytest.mark.parametrize("nside,maps,kernels", [
    (32, 1, 1), (32, 16, 1), (32, 17, 2),  # 64 pairs
    (256, 8, 1), (256, 16, 1),             # 512 and 1024 CTAs
    (512, 8, 1), (512, 9, 2),              # 1024 and 2048 CTAs
    (600, 1, 3), (1024, 1, 3),             # with the 3072-point list
    (2, 4, 1),                             # powers of two only
])
def test_ring_launches(nside, maps, kernels):
    assert bench.ring_launches(nside, maps) == kernels


def test_kernels_of_a_batch_are_the_mean_over_its_passes():
    assert bench.kernels_in_stage("ring_fft_forward", "fp32", 256, 64) == 2
    assert bench.kernels_in_stage("ring_fft_forward", "fp32", 256, 8) == 1
    assert bench.kernels_in_stage("ring_fft_inverse", "fp32", 256, 72) == 1.5
    assert bench.kernels_in_stage("fold", "fp32", 256, 8) == 1
