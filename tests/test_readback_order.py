"""Readback renumbers the ids it finds thinned out by removal.  What a program
reads, and what the frames after it make, must not depend on how often it read
before: with sources that emit and remove all the time, and after the removal
of the particles in the walls."""
from __future__ import annotations

import numpy as np
import pytest

from flipengine3d_gb300 import FluidSimulation, scenes


@pytest.mark.gpu
@pytest.mark.parametrize("scene", ["sources", "dam"])
def test_readbacks_do_not_change_the_order(gpu, scene):
    sc = scenes.fluid_sources(24, which="both", seed=2) if scene == "sources" else scenes.dam_break(20, seed=2, sphere=True)
    results = []
    for every in (1, 3):
        with FluidSimulation.from_scene(sc) as sim:
            for frame in range(6):
                sim.update(sc.frame_dt)
                if frame % every == every - 1:
                    pos, vel = sim.getMarkerParticlePositionData(), sim.getMarkerParticleVelocityData()
            binned, ids, _ = sim.binned_particles()
            assert np.array_equal(binned[np.argsort(ids, kind="stable")], pos)
            results.append((pos, vel))
    assert len(results[0][0]) > 0
    for a, b in zip(*results):
        assert np.array_equal(a, b)
