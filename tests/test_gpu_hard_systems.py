"""LU solves of sparse and badly scaled systems: block triangular ones whose rows have other units, columns of L with one
entry, entries that are small in their row and column but decide a sum.  The digit products of the FP64 form and the
FP16 terms of the FP32 form lie on a grid set by a row's and a column's largest entries; what that grid cannot hold has
to be summed another way.

Tolerance: Gaussian elimination with partial pivoting in FP64 (any order of its sums) solves (A + E) x = b with
|E| <= g |L| |U| componentwise, g = 3 n u sqrt(8) < 10 n u for complex arithmetic; |L| |U| is LAPACK's (the same pivot
rule), row by row.
"""
import numpy as np
import pytest

from refeff_gb300 import fms

scipy_linalg = pytest.importorskip("scipy.linalg")
pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _normal(rng, *shape):
    return rng.normal(size=shape) + 1j * rng.normal(size=shape)


def _block_system(n, n1, q, rng, border):
    """[[s A11, s A12], [E, A22]], s = 2^q; E zero, or its row `border` of the size of the rows above."""
    A, b = _normal(rng, n, n), _normal(rng, n, 3)
    A[n1:, :n1] = 0
    if border is not None:
        A[n1 + border, :n1] = _normal(rng, n1) * 0.3
        A[n1 + border, :n1] *= 2.0 ** q
    A[:n1] *= 2.0 ** q
    b[:n1] *= 2.0 ** q
    return A, b


def _solve(A, b, form=fms.FORM_FP64_LU, tensor=1):
    c = fms.Context(0)
    c.set_option(c.OPT_TENSOR_CORES, tensor)
    X, st, _ = fms.complex_lu_solve_batched(c, A[None], b[None], form)
    c.close()
    return X[0], int(st[0])


def _worst(A, X, b):
    """The largest |A X - b| of a row over its |L| |U| |X| + |b|."""
    L, U = scipy_linalg.lu(A, permute_l=True)
    return float((np.abs(A @ X - b) / (np.abs(L) @ (np.abs(U) @ np.abs(X)) + np.abs(b))).max())


@pytest.mark.parametrize("q", [10, 40, 100])
@pytest.mark.parametrize("border", [None, 5])
@pytest.mark.parametrize("n", [48, 170, 700])
def test_blocks_of_other_units(n, border, q):
    A, b = _block_system(n, 16, q, np.random.default_rng(n + q), border)
    X, st = _solve(A, b)
    assert st == 0 and _worst(A, X, b) < 10 * n * EPS


def test_products_of_small_and_large_entries():
    """x[32] = 2^-70 / (3 2^-70 - (1 2^-70 + 2^-70 1)): neither product reaches 2^-69 of its row's largest entry times
    its column's."""
    n, t = 34, 2.0 ** -70
    A = np.eye(n, dtype=complex)
    A[32, 32], A[32, 0], A[32, 1], A[0, 32] = 3 * t, 1, t, t
    A[33, 1] = A[1, 32] = A[33, 32] = 1
    b = np.zeros((n, 1), complex)
    b[32] = t
    X, st = _solve(A, b)
    assert st == 0 and abs(X[32, 0] - 1) < 10 * n * EPS


@pytest.mark.parametrize("q", [40, 100])
@pytest.mark.parametrize("n1", [4, 20])
@pytest.mark.parametrize("n", [24, 48, 170, 700])
def test_units_that_change_inside_a_block_of_eight(n, n1, q):
    """Rows of other units inside the 8-row blocks of the panels and block solves, on half of the columns."""
    rng = np.random.default_rng(n + n1 + q)
    A, b = _block_system(n, n1, q, rng, None)
    b = np.concatenate([b, _normal(rng, n, 13)], 1)
    A[:n1, n1:] *= rng.choice([0, 1], n - n1)
    b[:n1] *= rng.choice([0, 1], 16)
    X, st = _solve(A, b)
    assert st == 0 and _worst(A, X, b) < 10 * n * EPS


@pytest.mark.parametrize("n", [24, 48, 170])
def test_entries_of_all_sizes(n):
    rng = np.random.default_rng(n)
    A = _normal(rng, n, n) * 2.0 ** rng.integers(-60, 61, (n, n)) * (rng.uniform(size=(n, n)) < 0.3) + np.diag(_normal(rng, n))
    b = _normal(rng, n, 16) * 2.0 ** rng.integers(-60, 61, (n, 16))
    X, st = _solve(A, b)
    assert st == 0 and _worst(A, X, b) < 10 * n * EPS


def _fp32_solution(A, b):
    """The FP32 LU's solution as it is, without corrections."""
    c = fms.Context(0)
    c.set_option(c.OPT_DENSE_REFINEMENT, 0)
    X, _, _ = fms.complex_lu_solve_batched(c, A[None], b[None], fms.FORM_FP32_REFINED)
    c.close()
    return X[0]


@pytest.mark.parametrize("q", [10, 30, 60])
@pytest.mark.parametrize("border", [None, 5])
@pytest.mark.parametrize("n", [48, 170, 700])
def test_fp32_blocks_of_other_units(n, border, q):
    """The same bound with the unit roundoff of FP32 (A rounded to it among the errors), and the refined solution's."""
    A, b = _block_system(n, 16, q, np.random.default_rng(n + q), border)
    assert _worst(A, _fp32_solution(A, b), b) < 10 * n * 2.0 ** -24
    X, st = _solve(A, b, fms.FORM_FP32_REFINED)
    assert st == 0 and np.isfinite(X).all()


@pytest.mark.parametrize("n", [48, 170, 700])
def test_fp32_entries_of_all_sizes(n):
    rng = np.random.default_rng(n)
    A = _normal(rng, n, n) * 2.0 ** rng.integers(-30, 31, (n, n)) * (rng.uniform(size=(n, n)) < 0.3) + np.diag(_normal(rng, n))
    b = _normal(rng, n, 16) * 2.0 ** rng.integers(-30, 31, (n, 16))
    assert _worst(A, _fp32_solution(A, b), b) < 10 * n * 2.0 ** -24


def test_fp32_right_hand_sides_near_the_end_of_the_range_keep_their_bits():
    """Scaling by a power of two changes no bit of an FP32 elimination but where a sum cancels into the denormals, 2^-149
    each: some 2^-31 of values of 2^-114 over a sum of 170."""
    n = 170
    rng = np.random.default_rng(3)
    A, b = (_normal(rng, n, n) + 3 * np.sqrt(n) * np.eye(n)) / 64, _normal(rng, n, 8)
    X, Y = _fp32_solution(A, b), _fp32_solution(A, b * 2.0 ** -114) * 2.0 ** 114
    assert np.abs(X - Y).max() <= 2.0 ** -29 * np.abs(X).max()


@pytest.mark.parametrize("n", [9, 32, 64, 170, 300])
def test_without_tensor_cores_no_digits_are_used(n):
    """Option 0 runs the panels, block solves and updates in FP64 multiply-adds: within the bound of the digit form's
    solution, and rounded differently (at n = 9 and 32 there is a panel and no block update)."""
    rng = np.random.default_rng(n)
    A, b = _normal(rng, n, n), _normal(rng, n, 16)
    X, X0 = _solve(A, b)[0], _solve(A, b, tensor=0)[0]
    L, U = scipy_linalg.lu(A, permute_l=True)
    bound = np.abs(np.linalg.inv(A)) @ (np.abs(L) @ (np.abs(U) @ np.abs(X)) + np.abs(b))
    assert (np.abs(X - X0) <= 20 * n * EPS * bound).all()
    assert not np.array_equal(X, X0)


@pytest.mark.parametrize("q", [40, 100])
@pytest.mark.parametrize("n1", [4, 16])
def test_blocks_of_other_units_without_tensor_cores(n1, q):
    A, b = _block_system(170, n1, q, np.random.default_rng(n1 + q), 5)
    X, st = _solve(A, b, tensor=0)
    assert st == 0 and _worst(A, X, b) < 10 * 170 * EPS
