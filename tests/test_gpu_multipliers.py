"""Multipliers of the LU over the exponents of their pivots, one 2 x 2 system each: for [[u, 1], [a, 0]] x = (0, 1) the
second unknown is -u / a, the reciprocal of the multiplier a / u that the panel forms with the pivot's reciprocal (by
division where |u|^2 would leave the range).

Tolerance: |u|^2 and its reciprocal, the reciprocal's product with conj(u) and that with a take some 8 roundings, the
division of the back substitution as many.
"""
from fractions import Fraction

import numpy as np
import pytest

from refeff_gb300 import fms

pytestmark = pytest.mark.gpu


def _relative_error(x, u, a):
    def parts(z):
        return Fraction(float(z.real)), Fraction(float(z.imag))
    (xr, xi), (ur, ui), (ar, ai) = parts(x), parts(u), parts(a)
    dr, di = xr * ar - xi * ai + ur, xr * ai + xi * ar + ui  # x a + u
    return float((dr * dr + di * di) / (ur * ur + ui * ui)) ** 0.5


@pytest.mark.parametrize("form,exponents,unit", [(fms.FORM_FP64_LU, (-490, 491), 2.0 ** -53),
                                                 (fms.FORM_FP32_REFINED, (-40, 41), 2.0 ** -24)])
def test_multipliers_over_the_exponents_of_the_pivots(form, exponents, unit):
    rng = np.random.default_rng(4)
    n = 2000
    e = rng.integers(*exponents, size=n)
    u = (rng.uniform(0.5, 1, n) * rng.choice([-1, 1], n) + 1j * rng.uniform(-1, 1, n)) * 2.0 ** e
    a = (rng.uniform(0.1, 0.3, n) + 1j * rng.uniform(-0.2, 0.2, n)) * 2.0 ** (e - rng.integers(0, 3, n))
    A = np.zeros((n, 2, 2), complex)
    u, a = (z.astype(np.complex64).astype(complex) if form == fms.FORM_FP32_REFINED else z for z in (u, a))
    A[:, 0, 0], A[:, 1, 0], A[:, 0, 1] = u, a, 1
    b = np.zeros((n, 2, 1), complex)
    b[:, 1] = 1
    ctx = fms.Context(0)
    ctx.set_option(ctx.OPT_DENSE_REFINEMENT, 0)
    X, _, _ = fms.complex_lu_solve_batched(ctx, A, b, form)
    ctx.close()
    assert max(_relative_error(X[q, 1, 0], u[q], a[q]) for q in range(n)) <= 16 * unit
