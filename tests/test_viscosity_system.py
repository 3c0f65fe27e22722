"""The viscosity solver on systems of all the sizes its launch distinguishes: few
rows, less than one pass of the grid's threads, several passes.  The expected
velocities come from an independent solver of the same systems (Jacobi CG as
five kernels an iteration, FP64, to the same 1e-9); bound: that of the
first-frame parity tests, 1e-5 of the largest velocity.  Two runs agree bit
for bit, since every sum has a fixed order."""
from __future__ import annotations

import numpy as np
import pytest

from flipengine3d_gb300 import FluidSimulation
from flipengine3d_gb300.scenes import dam_break

CASES = [
    ((10, 9, 11), (0.6, 0.5, 1.1), 1771, (497, 16),
     [[0.6580195, 0.48441866, 0.45472282], [-0.13658802, 0.21285453, -0.10620588], [1.1167685, -0.56401175, -0.0680266],
      [0.05123183, -0.10244446, -0.45530754], [-0.24356057, -0.60775393, -0.2536959]]),
    ((33, 20, 18), (0.5, 0.3, 0.4), 12888, (4645, 40),
     [[0.22760688, 0.6014983, 0.1444843], [0.5623645, -0.80720437, 0.3990535], [0.8123296, -0.39320597, 0.6696123],
      [0.87491876, 0.007680023, 0.8116514], [1.0244329, -0.76271015, 0.84031785]]),
    ((64, 48, 60), (0.9, 0.55, 0.9), 879826, (326530, 72),
     [[0.15213265, 0.77782273, 0.05799356], [0.23896928, -0.17591953, 0.2706975], [-0.106573895, 0.5609739, 0.15917659],
      [-0.26267135, 0.94572794, -0.6206203], [-0.5849184, -0.3259612, -0.8967141]]),
]


def frame(dims, fill):
    i, j, k = dims
    sc = dam_break(i, jsize=j, ksize=k, dx=1 / i, seed=3, fill=fill)
    pos = sc.positions
    vel = np.stack([np.sin(7 * pos[:, 1]), np.cos(5 * pos[:, 0]), np.sin(6 * pos[:, 2])], 1).astype(np.float32)
    with FluidSimulation(*dims, sc.dx) as sim:
        sim.addBodyForce(0, -9.81, 0)
        sim.setViscosity(0.05)
        sim.loadMarkerParticleData(pos, vel)
        sim.initialize()
        sim.update(sc.frame_dt)
        return sim.getMarkerParticleVelocityData(), sim.viscosity_solve()


@pytest.mark.gpu
@pytest.mark.parametrize("dims,fill,count,solve,expected", CASES)
def test_viscous_frame(gpu, dims, fill, count, solve, expected):
    v, (rows, iters, resid) = frame(dims, fill)
    assert len(v) == count and (rows, iters) == solve and resid <= 1e-9
    at = np.linspace(0, len(v) - 1, 5).astype(int)
    assert np.abs(v[at] - np.array(expected, np.float32)).max() <= 1e-5 * np.abs(v).max()
    again, _ = frame(dims, fill)
    assert np.array_equal(v, again)
