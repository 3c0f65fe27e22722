"""The MIC(0) sweeps at the sizes where their tiling can go wrong: fewer cells
than a warp, a tile exactly and one pencil more along each axis, a cluster of
tiles exactly, several clusters, and grids so long that the edge words go
through their ring.  Bit-identical to the CPU oracle's sequential sweeps, in
both tile orientations."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refsim

# (K, J, I); interior pencils are (K - 2) x (J - 2), tiles 16 x 8, clusters 32 x 32
SHAPES = [(3, 3, 3), (3, 5, 40), (10, 18, 12), (11, 19, 12), (18, 10, 9), (34, 34, 10), (35, 36, 9), (67, 41, 13),
          (5, 4, 700), (12, 20, 703), (36, 19, 760)]


def box_factor(shape, seed, holes):
    """A factor over the whole interior (with a fraction of holes): pivots'
    inverses and negative couplings towards flagged upper neighbours, with
    rows that sum to less than one, so the sweeps stay bounded."""
    rng = np.random.default_rng(seed)
    fluid = np.zeros(shape, bool)
    fluid[1:-1, 1:-1, 1:-1] = True
    fluid &= rng.random(shape) >= holes
    fac = np.zeros(shape + (4,), np.float32)
    fac[..., 0] = np.where(fluid, rng.uniform(0.3, 0.6, shape), 0)
    for q, (dk, dj, di) in enumerate(((0, 0, 1), (0, 1, 0), (1, 0, 0))):
        K, J, I = shape
        up = np.zeros(shape, bool)
        up[: K - dk, : J - dj, : I - di] = fluid[dk:, dj:, di:]
        fac[..., 1 + q] = np.where(fluid & up, -rng.uniform(0.1, 0.5, shape), 0)
    return fluid.astype(np.uint8), fac, np.where(fluid, rng.uniform(-1, 1, shape), 0).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("holes", [0.0, 0.1])
def test_sweeps_at_tile_edges(gpu, shape, holes):
    import flipengine3d_gb300.fluidsimulation as fs
    fluid, fac, r = box_factor(shape, 5, holes)
    m = fluid > 0
    z_ref = refsim.mic0_precondition_f32(fluid, fac, r, "orc")[m]
    for orientation in (0, 1):
        z = fs.mic0_precondition(fluid, fac, r, orientation)[m]
        assert np.array_equal(z.view(np.uint32), z_ref.view(np.uint32)), f"{int((z != z_ref).sum())} of {z.size} differ"
