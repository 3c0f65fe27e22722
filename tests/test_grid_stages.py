"""Liquid level set, particle-to-grid, extrapolation and the particle update at
the sizes where their kernels change over: rows of faces that end at, before and after a
32-bit word, grids smaller than one block of ten cells, and grids on both
sides of the line between the two extrapolation variants.  Against the CPU
oracle: level set and known faces bit for bit, velocities to the bound of the
first-frame parity tests (1e-5 of the largest)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err
from flipengine3d_gb300 import FluidSimulation
from flipengine3d_gb300.scenes import dam_break
from oracle import refsim


@pytest.mark.gpu
@pytest.mark.parametrize("dims,fill", [
    ((8, 9, 7), (0.6, 0.5, 0.9)), ((30, 11, 12), (0.5, 0.5, 0.3)), ((31, 12, 21), (0.9, 0.2, 0.4)),
    ((32, 13, 10), (0.3, 0.3, 0.1)), ((33, 10, 20), (0.7, 0.1, 0.5)), ((62, 49, 66), (0.3, 0.2, 0.4)),
    ((64, 50, 63), (0.2, 0.5, 0.3))])
def test_level_set_and_face_velocities(gpu, dims, fill):
    i, j, k = dims
    sc = dam_break(i, jsize=j, ksize=k, dx=1 / i, seed=i, fill=fill, sphere=i > 60)
    ref = refsim.OracleSimulation(i, j, k, sc.dx).setup(sc, tolerance=1e-9).update_staged(sc.frame_dt)
    with FluidSimulation.from_scene(sc, tolerance=1e-9) as sim:
        st = sim.update_staged(sc.frame_dt)
    assert np.array_equal(st["phi"], ref["phi"])
    for f in "uvw":
        assert np.array_equal(st[f"v{f}_p2g"], ref[f"v{f}_p2g"])
        assert rel_err(st[f"{f}_p2g"], ref[f"{f}_p2g"]) <= 1e-5
        assert rel_err(st[f"{f}_final"], ref[f"{f}_final"]) <= 1e-5
    assert rel_err(st["vel_g2p"], ref["vel_g2p"]) <= 1e-5
    assert rel_err(st["pos_adv"], ref["pos_adv"]) <= 1e-5
