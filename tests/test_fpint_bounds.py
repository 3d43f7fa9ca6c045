"""Margins of the integer-pipe division and square root (csrc/fpint.h): their approximate
reciprocals may be off by twice the documented bounds (2^-23 for the reciprocal, 2^-22.9
for the reciprocal square root, of which the host build's unit, 2^-23, is 0.93) and every
result keeps its bits."""
import numpy as np
import pytest

from test_fpint import N, SPECIAL, fp, mantissas, same  # noqa: F401  (fp: fixture)


@pytest.mark.parametrize("ulp", [-2.2, -2.0, -1.08, 1.08, 2.0, 2.2])
def test_twice_the_documented_error_keeps_every_bit(fp, ulp):  # noqa: F811
    fp.set_ulp(ulp)
    rng = np.random.default_rng(17)
    a, b = mantissas(rng, 4 * N), mantissas(rng, 4 * N)
    near = (a.view(np.uint64) + rng.integers(0, 5, a.size, dtype=np.uint64)).view(np.float64)  # quotients near 1
    sa, sb = (v.ravel() for v in np.meshgrid(SPECIAL, SPECIAL))
    with np.errstate(all="ignore"):
        for x, y in ((a, b), (a, near), (a * b, b), (sa, sb)):
            assert same(fp(20, x, y), x / y)
        for x in (np.abs(a), np.abs(near) * np.abs(near), SPECIAL):
            assert same(fp(21, x), np.sqrt(x))
    fp.set_ulp(0.0)
