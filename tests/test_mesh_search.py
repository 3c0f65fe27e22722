"""The surface mesher's searches over what decides how far they go: particle
scale (a fraction of a cell to several), subdivision level and so node spacing
and solid rule, lone particles and dense ones, grids that end within a word or
a block, and enough vertices for both group sizes.  Bit for bit the oracle's
mesh of the same particles."""
from __future__ import annotations

import numpy as np
import pytest

from flipengine3d_gb300 import fluidsimulation as fs
from oracle.mesher import mesh_particles


def drops(dims, dx, seed, lone, pool):
    """Lone particles all over the domain and a dense, ragged pool at its floor."""
    rng = np.random.default_rng(seed)
    size = np.array(dims) * dx
    a = rng.uniform(3.01 * dx, size - 3.01 * dx, (lone, 3))
    b = rng.uniform(3.01 * dx, size - 3.01 * dx, (pool, 3))
    b = b[b[:, 1] < (0.4 + 0.1 * np.sin(9 * b[:, 0] / size[0])) * size[1]]
    return np.concatenate([a, b]).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("dims,scale,level,lone,pool", [
    ((16, 11, 13), 3.0, 1, 40, 0), ((16, 11, 13), 0.4, 1, 60, 4000), ((31, 17, 12), 1.0, 2, 30, 6000),
    ((12, 12, 33), 8.0, 2, 6, 500), ((9, 10, 11), 3.0, 3, 20, 1500), ((20, 16, 18), 5.5, 1, 4, 9000),
    ((40, 44, 40), 3.0, 3, 50, 120000)])
def test_mesh_matches_oracle(gpu, dims, scale, level, lone, pool):
    dx = 1.0 / dims[0]
    pos = drops(dims, dx, 7, lone, pool)
    with fs.FluidSimulation(*dims, dx) as sim:
        sim.setSurfaceSubdivisionLevel(level)
        sim.setMarkerParticleScale(scale)
        sim.loadMarkerParticleData(pos, np.zeros_like(pos))
        sim.initialize()
        sim.buildIsomesh()
        v, t = sim.getIsomesh()
        p, solid = sim.getMarkerParticlePositionData(), sim.solid_sdf()
    ov, ot = mesh_particles(p, *dims, dx, solid, level, particle_scale=scale)
    assert np.array_equal(t, ot) and np.array_equal(v, ov)
