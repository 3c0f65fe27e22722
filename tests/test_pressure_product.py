"""The product of the pressure solve's loop alone: s = z + beta s, q = A s, s.q,
against FP64, in both orientations, with rows on tile edges, first and last
steps, ragged extents, holes, and (0 s, then 1 z) without and with a step in s.

Bounds.  s: the fused multiply-add, at most half an ulp of float from the exact
value, a whole one for FP64's own rounding here.  q: rows split into pairs of
floats (2^-48 of each coefficient), seven products whose second parts are
rounded to float (2^-47 of the product each) and their sums' errors added up in
float (seven times 2^-46 of the sum of magnitudes): below 2^-42 of the sum of
magnitudes |a s|.  A product contracted with the sum after it would cost 2^-24.
s.q: as many steps as a thread takes, below 2^-40 of the sum of |s q|."""
from __future__ import annotations

import numpy as np
import pytest

# (K, J, I); interior pencils are (K - 2) x (J - 2), tiles 16 x 8 in either orientation, chunks of 8 steps
SHAPES = [(3, 3, 3), (3, 5, 40), (10, 18, 12), (11, 19, 12), (18, 10, 9), (35, 36, 9), (67, 41, 13), (5, 4, 700), (36, 19, 150)]


def system(shape, seed, holes):
    """Rows with full FP64 mantissas over most of the interior: weights that span
    six orders, diagonals near the sum of the couplings."""
    rng = np.random.default_rng(seed)
    fluid = np.zeros(shape, bool)
    fluid[1:-1, 1:-1, 1:-1] = True
    fluid &= rng.random(shape) >= holes
    rows = np.zeros(shape + (4,))
    K, J, I = shape
    for q, (dk, dj, di) in enumerate(((0, 0, 1), (0, 1, 0), (1, 0, 0))):
        up = np.zeros(shape, bool)
        up[:K - dk, :J - dj, :I - di] = fluid[dk:, dj:, di:]
        rows[..., 1 + q] = np.where(fluid & up, -np.exp(rng.uniform(-7, 7, shape)), 0)
    rows[..., 0] = np.where(fluid, np.exp(rng.uniform(-7, 7, shape)) + rng.random(shape), 0)
    return fluid, rows, rng


def product(rows, s):
    """A s and the sum of the magnitudes of its terms, FP64."""
    a = [rows[..., 0] * s]
    for q, axis in ((1, 2), (2, 1), (3, 0)):
        lo = [slice(None)] * 3
        hi = [slice(None)] * 3
        lo[axis], hi[axis] = slice(None, -1), slice(1, None)
        lo, hi = tuple(lo), tuple(hi)
        plus, minus = np.zeros(s.shape), np.zeros(s.shape)
        plus[lo] = rows[..., q][lo] * s[hi]
        minus[hi] = rows[..., q][lo] * s[lo]
        a += [plus, minus]
    return sum(a), sum(np.abs(x) for x in a)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("holes,beta", [(0.0, 0.0), (0.1, 0.83)])
def test_product_holds_48_bits(gpu, shape, holes, beta):
    import flipengine3d_gb300.fluidsimulation as fs
    fluid, rows, rng = system(shape, 5, holes)
    z, s = (np.where(fluid, rng.normal(0, 1, shape), 0).astype(np.float32) for _ in range(2))
    for orientation in (0, 1):
        got, q, dot = fs.pressure_apply(fluid, rows, z, s, beta, orientation)
        want = z.astype(np.float64) + np.float64(np.float32(beta)) * s
        assert (np.abs(got - want) <= np.spacing(np.abs(want).astype(np.float32))).all() and not got[~fluid].any()
        s64 = got.astype(np.float64)
        exact, size = product(rows, s64)
        err = np.abs(q - exact)[fluid]
        assert (err <= 2.0 ** -42 * size[fluid]).all(), f"q: worst 2^{np.log2((err / size[fluid]).max())}"
        assert abs(dot - (s64 * q)[fluid].sum()) <= 2.0 ** -40 * np.abs(s64 * q)[fluid].sum()
