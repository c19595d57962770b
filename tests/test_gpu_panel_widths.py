"""FP64 LU at the smallest sizes, and at those whose panels are 16 columns wide (n about 6200 to 12600) with one and with
two rows a thread: normwise backward error of partial pivoting (n u times a growth below 10), with a last panel narrower
than 8 columns at 6209 and 8437."""
import numpy as np
import pytest

from refeff_gb300 import fms

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _check(A, b):
    ctx = fms.Context(0)
    X, st, _ = fms.complex_lu_solve_batched(ctx, A, b, fms.FORM_FP64_LU)
    ctx.close()
    assert (st == 0).all()
    for q in range(A.shape[0]):
        n = A.shape[1]
        assert np.abs(A[q] @ X[q] - b[q]).max() < 10 * n * EPS * np.abs(A[q]).sum(-1).max() * np.abs(X[q]).max()


@pytest.mark.parametrize("n,m", [(1, 1), (1, 17), (2, 3), (7, 1), (8, 2), (9, 16), (15, 4), (31, 5), (32, 1)])
def test_smallest_systems(n, m):
    rng = np.random.default_rng(n)
    _check(rng.normal(size=(3, n, n)) + 1j * rng.normal(size=(3, n, n)), rng.normal(size=(3, n, m)) + 0j)


@pytest.mark.parametrize("n", [6209, 8437])
def test_sixteen_column_panels(n):
    rng = np.random.default_rng(n)
    A = np.empty((1, n, n), complex)
    A.real, A.imag = rng.random((1, n, n)) - 0.5, rng.random((1, n, n)) - 0.5
    _check(A, rng.normal(size=(1, n, 2)) + 0j)
