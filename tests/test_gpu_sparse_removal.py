"""A few particles in a large grid, some of which a frame removes: every cell is
then passed over, with the whole GPU and not with as many threads as there are
particles.  300 particles that drift into one cell, which keeps the first 250 of
them, against 250 that drift there: the binning takes as long but for the
crowded cell's sort, which is quadratic (a walk over all cells by 300 threads
takes more than two milliseconds longer)."""
from __future__ import annotations

import numpy as np
import pytest

from flipengine3d_gb300 import FluidSimulation

DIMS, DT = (256, 128, 128), 1 / 120


def frame(n):
    dx = 1.0 / 128
    rng = np.random.default_rng(6)
    pos = ((rng.uniform(0.05, 0.95, (300, 3)) + [60, 60, 60])[:n] * dx)
    pos[:, 0] -= 0.5 * dx   # about half of them in the cell before
    pos = pos.astype(np.float32)
    vel = np.zeros_like(pos)
    vel[:, 0] = 0.5 * dx / DT
    with FluidSimulation(*DIMS, dx) as sim:
        sim.loadMarkerParticleData(pos, vel)
        sim.initialize()
        sim.set_stage_timing(True)
        sim.update(DT)
        ms, substeps = sim.stage_times()
        return sim.getMarkerParticlePositionData(), sim.binned_particles()[2], ms["binning"] / substeps


@pytest.mark.gpu
def test_removal_among_few_particles(gpu):
    kept, _, _ = frame(250)
    assert len(kept) == 250
    plain = min(frame(250)[2] for _ in range(4))
    runs = [frame(300) for _ in range(4)]
    pos, start, _ = runs[0]
    counts = np.diff(start)
    assert len(pos) == 250 and counts.max() == 250 and np.count_nonzero(counts) == 1
    assert all(np.array_equal(pos, r[0]) for r in runs)
    assert min(r[2] for r in runs) <= 1.44 * plain + 0.5, (plain, [r[2] for r in runs])
