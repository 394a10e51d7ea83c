"""The float32 flat step over eight-wide items (csrc/pic_wide.cuh) and the
tallies a segment's steps sum for one another, against the float64 step.

Tolerance as for the resident step: 1e-6 of the peak a step, steps added up."""

import importlib

import numpy as np
import pytest

from goldens import make_config, pkg
from test_resident import _case, _compare, _grid, _segment

# no_xy, no_z (four layers more in all): one interior column; a column of one
# vector, of exactly a warp, of a warp and one vector, of many; rows with one to
# eight padded layers; a grid of one block and of every block
SIZES = [(3, 1), (3, 600), (4, 3), (5, 20), (9, 252), (9, 255), (10, 260), (33, 57), (40, 28), (57, 203), (90, 124),
         (130, 300)]


@pytest.mark.gpu
@pytest.mark.parametrize("wall", [0, 1])
@pytest.mark.parametrize("n,no_z", SIZES)
def test_flat_segment_matches_the_float64_step(n, no_z, wall):
    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    for steps in (1, 2, 9):  # a step alone, a step and its last, both partial buffers in turn
        state, xs, ys, off = _case(n, no_z, steps, 100 * n + no_z + wall, 12)
        g = _grid(native, n, no_z, wall, native.PIC_F32, native.PIC_VARIANT_FLAT)
        g64 = _grid(native, n, no_z, wall, native.PIC_F64, native.PIC_VARIANT_FLAT)
        for variant in (native.PIC_DEPOSIT_AUTO, native.PIC_DEPOSIT_TRACKS):  # pairs kept and pairs cleared
            g.deposit_variant = g64.deposit_variant = variant
            got = _segment(native, g, torch, state, xs, ys, off, n & 1)
            ref = _segment(native, g64, torch, state, xs, ys, off, n & 1)
            _compare(native, got, ref, steps)
