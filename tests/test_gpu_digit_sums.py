"""One sum of 32 complex products of the FP64 block update, read off a solution and compared with exact rationals: the
bits that the join of the digit levels keeps, and level sums beyond 2^22.

Rows 0 .. 31 of the system are 4 I (larger than any |re| + |im| below it: the pivots) beside a column b, row 32 is (a, 0)
and row 33 (0.9 .. 0.9, -, 1): with the right-hand side e_32 the solution is x[32] = -4 / sum_k a_k b_k.  Row 33 keeps the
columns' balance at one and the largest entries of a and b lie in (1/2, 1), so that the grid of the sum is 2^0.

Tolerance: the join rounds to 2^-57; the dropped digit products have 7 pairs of digits, 64 real products each, of up to
2^14 at 2^-76, 2^-53.2 in all where every digit is near 127 and 6 standard deviations of 2^-59.2 where they are random;
x[32] itself takes eight roundings.
"""
from fractions import Fraction

import numpy as np
import pytest

from refeff_gb300 import fms

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _sum(a, b):
    re = im = Fraction(0)
    for x, y in zip(a, b):
        xr, xi, yr, yi = (Fraction(float(v)) for v in (x.real, x.imag, y.real, y.imag))
        re, im = re + xr * yr - xi * yi, im + xr * yi + xi * yr
    return re, im


def _errors(pairs):
    """|-4/x[32] - sum| and |sum| of every (a, b)."""
    A = np.zeros((len(pairs), 34, 34), complex)
    A[:] = np.diag([4.0] * 32 + [1, 1])
    for q, (a, b) in enumerate(pairs):
        A[q, :32, 32], A[q, 32, :32], A[q, 32, 32], A[q, 33, :32] = b, a, 0, 0.9
        A[q, 33, 32] = 0.9 * b.sum() / 4
    B = np.zeros((len(pairs), 34, 1), complex)
    B[:, 32] = 1
    ctx = fms.Context(0)
    X, st, _ = fms.complex_lu_solve_batched(ctx, A, B, fms.FORM_FP64_LU)
    ctx.close()
    assert (st == 0).all()
    err, size = [], []
    for q, (a, b) in enumerate(pairs):
        re, im = _sum(a, b)
        xr, xi = Fraction(X[q, 32, 0].real), Fraction(X[q, 32, 0].imag)
        n = xr * xr + xi * xi
        dr, di = -4 * xr / n - re, 4 * xi / n - im
        err.append(np.hypot(float(dr), float(di)))
        size.append(np.hypot(float(re), float(im)))
    return np.array(err), np.array(size)


def test_bits_kept_of_a_small_sum():
    rng = np.random.default_rng(1)
    pairs = []
    for _ in range(200):
        a, b = ((rng.uniform(0.5, 1, 32) + 1j * rng.uniform(0.5, 1, 32)) * rng.choice([-1, 1], 32) for _ in "ab")
        a[16:] *= 2.0 ** -7
        b[:16] *= 2.0 ** -7
        pairs.append((a, b))
    err, size = _errors(pairs)
    assert (size < 0.5).all()
    assert (err <= 2.0 ** -55 + 8 * U * size).all(), (err / (2.0 ** -55 + 8 * U * size)).max()


def test_level_sums_of_digits_near_127():
    tail = sum(127 * 2.0 ** -(6 + 8 * i) for i in range(1, 7)) + 124 * 2.0 ** -62
    a, b = np.full(32, tail * (1 + 1j)), np.full(32, tail * (1 + 1j))
    a[0] = b[1] = 0.99
    for sa in (1, -1):
        err, size = _errors([(sa * a, b), (a, 1j * sa * b)])
        assert (size > 2.0 ** -7).all() and (err <= 2.0 ** -53 + 2.0 ** -57 + 8 * U * size).all(), err
