"""Particle to grid, bit for bit: faces recomputed in NumPy float32 with the
reference's expression trees, particles in (cell, id) order.  A sum contracted
with a product, or taken in another order, shows."""
from __future__ import annotations

import numpy as np
import pytest

from flipengine3d_gb300 import FluidSimulation
from flipengine3d_gb300.scenes import dam_break

f = np.float32


def face_value(d, ijk, pos, vel, dx):
    """The value of face ijk of direction d, None where no particle reaches it."""
    r = f(0.5 * dx * np.sqrt(3.0))
    h, rsq = f(0.5 * dx), f(r * r)
    c1 = f(f(4.0 / 9.0) * f(f(1) / f(f(f(f(f(r * r) * r) * r) * r) * r)))
    c2 = f(f(17.0 / 9.0) * f(f(1) / f(f(f(r * r) * r) * r)))
    c3 = f(f(22.0 / 9.0) * f(f(1) / f(r * r)))
    d2 = []
    for a in range(3):
        b = ijk[a] // 10
        off = f(float(f(b)) * (10 * dx))
        g = f(float(f(ijk[a] - 10 * b)) * dx)
        p = pos[:, a] if a == d else pos[:, a] - h
        q = g - (p - off)
        d2.append(q * q)
    d2 = (d2[0] + d2[1]) + d2[2]
    near = d2 < rsq
    if not near.any():
        return None
    s = w = f(0)
    for e, v in zip(d2[near], vel[near, d]):
        wgt = f(f(f(f(1) - f(f(f(c1 * e) * e) * e)) + f(f(c2 * e) * e)) - f(c3 * e))
        s, w = f(s + f(wgt * v)), f(w + wgt)
    return f(s / w) if w > f(1e-6) else None


@pytest.mark.gpu
@pytest.mark.parametrize("dims,ppc", [((14, 11, 13), 8), ((13, 12, 22), 5), ((21, 9, 10), 3)])
def test_face_velocities_bit_for_bit(gpu, dims, ppc):
    i, j, k = dims
    sc = dam_break(i, jsize=j, ksize=k, dx=1 / i, seed=4, fill=(0.7, 0.5, 0.8 * k / i), ppc=ppc)
    rng = np.random.default_rng(1)
    sc.velocities = rng.normal(0, 1, sc.positions.shape).astype(np.float32)
    with FluidSimulation.from_scene(sc, tolerance=1e-9) as sim:
        pos, ids, _ = sim.binned_particles()
        by_id = sim.getMarkerParticleVelocityData()
        rank = np.empty(len(ids), np.int64)
        rank[np.argsort(ids, kind="stable")] = np.arange(len(ids))
        vel = by_id[rank]
        st = sim.update_staged(sc.frame_dt)
    for d, name in enumerate("uvw"):
        known = np.argwhere(st[f"v{name}_p2g"].astype(bool))   # (k, j, i)
        pick = known[rng.choice(len(known), min(len(known), 150), replace=False)]
        for kk, jj, ii in pick:
            want = face_value(d, (int(ii), int(jj), int(kk)), pos, vel, sc.dx)
            got = st[f"{name}_p2g"][kk, jj, ii]
            assert want is not None and got.tobytes() == want.tobytes(), (name, ii, jj, kk, got, want)
