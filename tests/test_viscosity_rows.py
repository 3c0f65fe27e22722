"""The viscosity step alone, over every face of the system: |b - A x| with A and b
put together here in NumPy from the strain energy (Batty's method), apart from
the solver's own recurrence, and zeros off the system.  All CTAs of the solve
meet in a sum twice an iteration and read each other's directions after it, so
a value read too early shows as a residual.  Grids from less than one chunk of
rows to several chunks a warp, ragged ones and some with an obstacle.

Bound, per row: the solver's 1e-9 |b|inf, plus the rounding of the float
coefficients, right-hand side and result, at most eight roundings (8 x 2^-24)
of each term."""
from __future__ import annotations

import numpy as np
import pytest

f = np.float32
# control-volume grids: cells, faces, edges; extents beyond (I, J, K), offset of the centre in half cells
VOLUMES = {"c": ((0, 0, 0), (1, 1, 1)), "u": ((1, 0, 0), (0, 1, 1)), "v": ((0, 1, 0), (1, 0, 1)), "w": ((0, 0, 1), (1, 1, 0)),
           "yz": ((0, 1, 1), (1, 0, 0)), "xz": ((1, 0, 1), (0, 1, 0)), "xy": ((1, 1, 0), (0, 0, 1))}


def tet(p):
    p = np.sort(p, axis=0)
    with np.errstate(all="ignore"):
        def corner(a, b, c, d):
            return (a * a * a) / ((a - b) * (a - c) * (a - d))
        a, b = p[0] / (p[0] - p[2]), p[0] / (p[0] - p[3])
        c, d = p[1] / (p[1] - p[3]), p[1] / (p[1] - p[2])
        prism = (a * b * (f(1) - d) + b * (f(1) - c) * d) + c * d
        return np.select([p[3] <= 0, p[2] <= 0, p[1] <= 0, p[0] <= 0],
                         [np.ones_like(p[0]), f(1) - corner(p[3], p[2], p[1], p[0]), prism, corner(*p)], f(0)).astype(f)


def liquid_at(phi, dx, pos):
    """The level set read at p - dx/2 as a nodal grid; 0 outside it."""
    cell, frac = [], []
    for p in pos:
        q = p - f(0.5 * dx)
        i = np.floor(q.astype(np.float64) * (1.0 / dx)).astype(int)
        cell.append(i)
        frac.append((q - (i.astype(f).astype(np.float64) * dx).astype(f)).astype(np.float64) * (1.0 / dx))
    out = 0.0
    for o in ((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (0, 1, 1), (1, 1, 0), (1, 1, 1)):
        at = [c + s for c, s in zip(cell, o)]
        ok = np.all([(a >= 0) & (a < m) for a, m in zip(at, phi.shape[::-1])], axis=0)
        val = np.where(ok, phi[tuple(np.where(ok, a, 0) for a in at[::-1])], 0).astype(np.float64)
        for t, s in zip(frac, o):
            val = val * (t if s else 1 - t)
        out = out + val
    return out.astype(f)


def fractions(phi, valid, dx, grow, off):
    """Liquid fraction of each control volume of a grid, indexed [k, j, i]."""
    dims = [n + g for n, g in zip(phi.shape[::-1], grow)]
    a = np.meshgrid(*[np.arange(n + 1) for n in dims[::-1]], indexing="ij")[::-1]
    first = np.full(a[0].shape, -1)
    for q in range(7, -1, -1):   # the corner takes the first valid volume's sample
        c = [x - 1 + (q >> s & 1) for s, x in enumerate(a)]
        ok = np.all([(x >= 0) & (x < n) for x, n in zip(c, dims)], axis=0)
        first[ok & valid[tuple(np.where(ok, x, 0) for x in c[::-1])]] = q
    pos = []
    for s, x in enumerate(a):
        up = first >> s & 1
        centre = f(0.5 * dx * off[s]) + ((x - 1 + up).astype(np.float64) * dx + 0.5 * dx).astype(f)
        pos.append(centre + np.where(up, -f(1), f(1)) * (f(0.5) * f(dx)))
    node = np.where(first >= 0, liquid_at(phi, dx, pos), f(0))
    p = {(x, y, z): node[z:dims[2] + z, y:dims[1] + y, x:dims[0] + x] for x in (0, 1) for y in (0, 1) for z in (0, 1)}
    tets = [("000", "001", "101", "011"), ("000", "101", "100", "110"), ("000", "010", "011", "110"),
            ("101", "011", "111", "110"), ("000", "011", "101", "110"), ("100", "101", "001", "111"),
            ("100", "001", "000", "010"), ("100", "110", "111", "010"), ("001", "111", "011", "010"),
            ("100", "111", "001", "010")]
    total = np.zeros(node[1:, 1:, 1:].shape, f)
    for n, t in enumerate(tets):
        total += tet(np.stack([p[tuple(map(int, s))] for s in t])) * f(2 if n in (4, 9) else 1)
    every = np.stack(list(p.values()))
    vol = np.where((every < 0).all(0), f(1), np.where((every >= 0).all(0), f(0), total / f(12)))
    return np.where(valid[:dims[2], :dims[1], :dims[0]], vol, f(0)).astype(np.float64)


def scene(dims, seed, obstacle):
    I, J, K = dims
    rng = np.random.default_rng(seed)
    dx = 1.0 / max(dims)
    z, y, x = np.meshgrid(*[(np.arange(n) + 0.5) * dx for n in (K, J, I)], indexing="ij")
    ph = rng.uniform(0, 6, 3)
    phi = (y - (0.5 + 0.2 * np.sin(7 * x + ph[0]) * np.cos(5 * z + ph[1])) * J * dx).astype(f)
    n = [np.arange(m + 1) * dx for m in (K, J, I)]
    walls = [np.minimum(c, m * dx - c) - 1.5 * dx for c, m in zip(n, (K, J, I))]
    solid = np.minimum(np.minimum(walls[0][:, None, None], walls[1][None, :, None]), walls[2][None, None, :])
    if obstacle:
        r = np.sqrt(sum((c - 0.5 * m * dx) ** 2 for c, m in zip(np.meshgrid(*n, indexing="ij"), (K, J, I))))
        solid = np.minimum(solid, r - 0.2 * min(dims) * dx)
    field = [rng.normal(0, 1, s).astype(f) for s in ((K, J, I + 1), (K, J + 1, I), (K + 1, J, I))]
    return dx, phi, solid.astype(f), field


def system(phi, solid, dx):
    K, J, I = phi.shape
    sc = f(0.125) * sum(solid[z:K + z, y:J + y, x:I + x] for z in (0, 1) for y in (0, 1) for x in (0, 1))   # float, like its sums
    fluid = [np.zeros(s, bool) for s in ((K, J, I + 1), (K, J + 1, I), (K + 1, J, I))]
    fluid[0][:, :, 1:-1] = sc[:, :, 1:] + sc[:, :, :-1] > 0
    fluid[1][:, 1:-1] = sc[:, 1:] + sc[:, :-1] > 0
    fluid[2][1:-1] = sc[1:] + sc[:-1] > 0
    valid = np.zeros((K + 1, J + 1, I + 1), bool)
    valid[:-1, :-1, :-1] = phi < 0
    for _ in range(2):
        w = np.pad(valid, 1)
        valid = valid | w[:-2, 1:-1, 1:-1] | w[2:, 1:-1, 1:-1] | w[1:-1, :-2, 1:-1] | w[1:-1, 2:, 1:-1] | w[1:-1, 1:-1, :-2] | w[1:-1, 1:-1, 2:]
    return fluid, {name: fractions(phi, valid, dx, *g) for name, g in VOLUMES.items()}


def gradient(vols, k, nu, field, sign):
    """d/dx of the strain energy, 1/2 k nu sum(2 vol_c (du/dx)^2 + ...) + 1/2 k nu sum(vol_e (du/dy + dv/dx)^2 + ...), per
    face, and whether any of its volumes holds liquid; with sign +1 every term in absolute value."""
    u, v, w = field
    out, wet = [np.zeros(g.shape) for g in field], [np.zeros(g.shape, bool) for g in field]

    def add(d, at, val, vol):
        out[d][at] += val
        wet[d][at] |= vol > 0

    lo, hi, mid, full = slice(None, -1), slice(1, None), slice(1, -1), slice(None)
    for d, (g, axis) in enumerate(((u, 2), (v, 1), (w, 0))):
        a, b = [full] * 3, [full] * 3
        a[axis], b[axis] = lo, hi
        a, b = tuple(a), tuple(b)
        e = 2 * k * nu * vols["c"] * (g[b] + sign * g[a])
        add(d, b, e, vols["c"])
        add(d, a, sign * e, vols["c"])
    for name, (d1, ax1), (d2, ax2) in (("xy", (0, 1), (1, 2)), ("xz", (0, 0), (2, 2)), ("yz", (1, 0), (2, 1))):
        # face grid d1 differs along ax1 and d2 along ax2 across the edges inside both
        inner = [full] * 3
        inner[ax1] = inner[ax2] = mid
        vol = vols[name][tuple(inner)]
        g1, g2 = field[d1], field[d2]
        ends = []
        for ax, other in ((ax1, ax2), (ax2, ax1)):
            a, b = [full] * 3, [full] * 3
            a[ax], b[ax], a[other], b[other] = lo, hi, mid, mid
            ends.append((tuple(a), tuple(b)))
        (a1, b1), (a2, b2) = ends
        e = k * nu * vol * (g1[b1] + sign * g1[a1] + g2[b2] + sign * g2[a2])
        for d, a, b in ((d1, a1, b1), (d2, a2, b2)):
            add(d, b, e, vol)
            add(d, a, sign * e, vol)
    return out, wet


@pytest.mark.gpu
@pytest.mark.parametrize("dims,obstacle", [((5, 6, 5), False), ((8, 9, 7), False), ((17, 9, 23), True), ((33, 20, 18), False),
                                           ((40, 41, 39), True), ((64, 48, 61), False)])
def test_every_row_is_solved(gpu, dims, obstacle):
    from flipengine3d_gb300 import fluidsimulation as fs
    dx, phi, solid, field = scene(dims, 11, obstacle)
    nu, dt = 0.05, 1 / 60
    got, (rows, _, resid) = fs.viscosity_step(phi, solid, *field, dx, nu, dt)
    fluid, vols = system(phi, solid, dx)
    k = dt / dx ** 2
    face_vol = [vols[n] for n in "uvw"]
    _, wet = gradient(vols, k, nu, [g.astype(np.float64) for g in field], -1)
    inside = []
    for g, fl, wt, vf in zip(field, fluid, wet, face_vol):
        at = np.zeros(g.shape, bool)
        at[1:dims[2], 1:dims[1], 1:dims[0]] = True
        inside.append(at & fl & (wt | (vf > 0)))
    assert rows == sum(int(m.sum()) for m in inside) > 0 and resid <= 1e-9
    # the whole field: the solution in the system, known velocities in the solid, nothing elsewhere
    x = [np.where(m, g, np.where(fl, 0, g0)).astype(np.float64) for m, g, fl, g0 in zip(inside, got, fluid, field)]
    ax, _ = gradient(vols, k, nu, x, -1)
    size, _ = gradient(vols, k, nu, [np.abs(g) for g in x], +1)
    known = [np.where(fl, 0, g0).astype(np.float64) for fl, g0 in zip(fluid, field)]
    moved, _ = gradient(vols, k, nu, known, -1)
    bmax = max(np.abs((vf * g0 - mv)[m]).max() for vf, g0, mv, m in zip(face_vol, field, moved, inside) if m.any())
    for d in range(3):
        m = inside[d]
        assert not got[d][~m].any()
        r = np.abs(face_vol[d] * (field[d].astype(np.float64) - x[d]) - ax[d])[m]
        terms = (face_vol[d] * (np.abs(field[d]) + np.abs(x[d])) + size[d])[m]
        bound = 1e-9 * bmax + 8 * 2.0 ** -24 * terms
        assert (r <= bound).all(), f"{'uvw'[d]}: {int((r > bound).sum())} of {m.sum()} rows, worst {(r / bound).max()}"
