"""GPU: a wait of the viscous solver that runs out is reported as the other
device waits are (FLIP_E_DEVICE_TIMEOUT) and leaves the simulation usable: the
velocity field is not cleared, and the next update is, bit for bit, the one of a
simulation that was never disturbed.
The solver's CTAs are made to await an epoch that none writes, with a short
limit; nothing faults, traps or hangs."""
from __future__ import annotations

import time

import numpy as np
import pytest

from flipengine3d_gb300 import FlipDeviceTimeout, FluidSimulation
from flipengine3d_gb300.scenes import dam_break


@pytest.mark.gpu
@pytest.mark.parametrize("edge", [12, 40])   # a grid of a few CTAs, and of one per SM
def test_viscous_wait_times_out_and_the_next_update_recovers(gpu, edge):
    sc = dam_break(edge, seed=8)
    sc.viscosity = 0.05

    def frames(sim, n):
        for _ in range(n):
            sim.update(sc.frame_dt)
        return sim.getMarkerParticlePositionData(), sim.getMarkerParticleVelocityData(), sim.viscosity_solve()

    with FluidSimulation.from_scene(sc, tolerance=1e-9) as sim:
        want = frames(sim, 2)
    with FluidSimulation.from_scene(sc, tolerance=1e-9) as sim:
        sim.set_device_wait_limit(4096)
        sim.inject_sweep_stall(True)
        t0 = time.perf_counter()
        with pytest.raises(FlipDeviceTimeout, match="viscosity"):
            sim.update(sc.frame_dt)
        assert time.perf_counter() - t0 < 30.0, "the waits must end at their short limit"
        assert sim.getCurrentFrame() == 0, "a frame that timed out is not counted"
        assert np.abs(sim.mac_velocity()[1]).max() > 0, "the field that went into the solver is left as it was"
        sim.inject_sweep_stall(False)
        sim.set_device_wait_limit(0)
        got = frames(sim, 2)
    assert got[2] == want[2] and all(np.array_equal(a, b) for a, b in zip(got[:2], want[:2]))
