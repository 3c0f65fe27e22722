"""The MIC(0) sweeps on grids whose edge words go through a ring: a word is
cleared, the chunk handed on and the word written again by another warp or the
edge warps, many times over.  Several laps of the ring, tiles along both axes,
the same system again and again: bit-identical to the CPU oracle's sequential
sweeps every time."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refsim
from test_sweep_tiles import box_factor


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(20, 36, 1100), (4, 3, 2500)])   # (K, J, I)
def test_ring_words_are_never_taken_twice(gpu, shape):
    import flipengine3d_gb300.fluidsimulation as fs
    fluid, fac, r = box_factor(shape, 9, 0.05)
    m = fluid > 0
    want = refsim.mic0_precondition_f32(fluid, fac, r, "orc")[m].view(np.uint32)
    for _ in range(10):
        for orientation in (0, 1):
            assert np.array_equal(fs.mic0_precondition(fluid, fac, r, orientation)[m].view(np.uint32), want)
