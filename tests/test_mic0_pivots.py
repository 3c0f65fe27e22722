"""What the MIC(0) factor takes for 1 / d and sqrt(d), against IEEE division and
square root over the whole exponent range: subnormal, huge, negative, zero,
infinite and NaN inputs, the ends of the range in which FP32 supplies the guess,
and guesses that are off by more and by less than the step can mend.  And a row
that is not a number: what depends on it is not one either, as in the
reference's elimination, and nothing else changes.

Bound: the remainder of either iteration is below 2^-56 of the result, so it is
within half a unit in the last place and a sixteenth of the exact value, and at
most one unit from the correctly rounded one.  Where CUDA's own operation is
taken, it is equal."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refsim


def inputs():
    rng = np.random.default_rng(3)
    e = np.concatenate([np.arange(-1074, 1024), np.repeat([-128, -127, -126, -121, -120, -119, 119, 120, 121, 126, 127, 128], 50)])
    d = np.ldexp(rng.uniform(1, 2, len(e)), e)
    d = np.concatenate([d, np.ldexp(1.0, e), np.ldexp(1 + rng.integers(-4, 5, len(e)) * 2.0 ** -20, e),
                        np.exp(rng.uniform(-20, 20, 200000)), [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, np.finfo(float).max]])
    return np.concatenate([d, -d])


def ulps(a, b):
    with np.errstate(all="ignore"):
        return np.where((a == b) | (np.isnan(a) & np.isnan(b)), 0, np.abs(a - b) / np.spacing(np.abs(b)))


@pytest.mark.gpu
@pytest.mark.parametrize("off", ["none", "little", "much", "odd"])
def test_pivot_functions(gpu, off):
    import flipengine3d_gb300.fluidsimulation as fs
    d = inputs()
    rng = np.random.default_rng(4)
    scale = {"none": np.ones(len(d)), "little": 1 + rng.uniform(-2e-6, 2e-6, len(d)), "much": 1 + rng.uniform(-1e-3, 1e-3, len(d)),
             "odd": rng.choice([0.0, -1.0, 3.0, np.inf, np.nan, 1e-30], len(d))}[off]
    recip, root = fs.mic0_pivot_functions(d, scale)
    with np.errstate(all="ignore"):
        want, want_root = 1.0 / d, np.sqrt(d)
    assert ulps(recip, want).max() <= 1, d[np.argmax(ulps(recip, want))]
    assert ulps(root, want_root).max() <= 1, d[np.argmax(ulps(root, want_root))]
    plain = ~np.isfinite(want) | (d == 0) | ~np.isfinite(d)
    assert np.array_equal(recip[plain], want[plain], equal_nan=True)
    assert np.array_equal(root[plain], want_root[plain], equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("what", [np.nan, -np.nan, np.inf])
@pytest.mark.parametrize("entry", [0, 1, 2, 3])   # diagonal, couplings to +x, +y, +z
def test_a_row_that_is_no_number(gpu, what, entry):
    import flipengine3d_gb300.fluidsimulation as fs
    fluid, rows = refsim.random_mic0_system((11, 13, 20), 3)
    at = tuple(np.argwhere((fluid > 0) & (rows[..., 1] != 0) & (rows[..., 2] != 0) & (rows[..., 3] != 0))[40])
    rows[at + (entry,)] = what
    got = fs.mic0_factor(fluid, rows)
    with np.errstate(all="ignore"):
        want, _ = refsim.mic0_factor(fluid, rows, "orc")
    m = (fluid > 0) & (rows[..., 0] != 0)   # a row of zeros has no pivot: 0 here, whatever is around it
    assert not got[~m].any()
    assert np.array_equal(np.isnan(got[m]), np.isnan(want[m])), (np.isnan(got[m]).sum(), np.isnan(want[m]).sum())
    ok = m & ~np.isnan(want)
    assert np.allclose(got[ok], want[ok], rtol=1e-12, atol=0)
