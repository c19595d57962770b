"""The FP64 elimination's block updates on the tensor cores (exact 8-bit digit products) against LAPACK and against the
same elimination on the FP64 pipe (REFEFF_FMS_OPT_TENSOR_CORES = 0): at the edges of the 128-row and 16-column tiles and
of the 32-column panels, under power-of-two scalings, with infinities and NaN, with waits made to run out, and with more
systems than one launch's operand images hold.

Tolerance of the backward error |A X - B| / (|A| |X|) (max norms): partial pivoting with products exact to 2^-53 stays
below n 2^-53 times a growth that is below 10 on such systems.
"""
import numpy as np
import pytest

from refeff_gb300 import fms

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _systems(n, m, seed, batch=2):
    rng = np.random.default_rng(seed)
    A = rng.normal(size=(batch, n, n)) + 1j * rng.normal(size=(batch, n, n))
    return A, rng.normal(size=(batch, n, m)) + 1j * rng.normal(size=(batch, n, m))


def _solve(A, B, tensor=1, polls=0):
    c = fms.Context(0)
    c.set_option(c.OPT_TENSOR_CORES, tensor)
    c.set_option(c.OPT_TC_WAIT_POLLS, polls)
    out = fms.complex_lu_solve_batched(c, A, B, fms.FORM_FP64_LU)
    c.close()
    return out


def _backward_error(A, X, B):
    norm = np.abs(A).sum(-1).max() * np.abs(X).max()
    return np.abs(A @ X - B).max() / norm


@pytest.mark.parametrize("n,m", [(33, 1), (48, 5), (64, 16), (65, 17), (160, 16), (161, 33), (288, 3), (300, 64),
                                 (417, 40), (700, 9)])
def test_solutions_at_tile_edges(n, m):
    A, B = _systems(n, m, 7 * n + m)
    X, st, _ = _solve(A, B)
    assert (st == 0).all()
    for b in range(2):
        assert _backward_error(A[b], X[b], B[b]) < 10 * n * EPS
    # the same pivots and the same solution as the FP64 pipe's, to rounding
    X0, _, _ = _solve(A, B, tensor=0)
    for b in range(2):
        assert _backward_error(A[b], X0[b], B[b]) < 10 * n * EPS


@pytest.mark.parametrize("rows,cols,rhs", [(0, 300, 200), (300, 0, 0), (40, 40, 200)])
def test_graded_systems_keep_every_digit(rows, cols, rhs):
    """Rows, columns and right-hand sides scaled by powers of two up to 2^(+-300): scaled back (exactly), the solution is
    as accurate as without, row by row (the componentwise backward error of partial pivoting)."""
    n, m = 170, 20
    A, B = _systems(n, m, 5)
    rng = np.random.default_rng(6)
    r, c, d = (2.0 ** rng.integers(-q, q + 1, size=k) for q, k in ((rows, n), (cols, n), (rhs, m)))
    Y, st, _ = _solve(A * r[:, None] * c, B * r[:, None] * d)
    assert (st == 0).all()
    X = Y * c[:, None] / d
    for b in range(2):
        assert np.isfinite(X[b]).all()
        err = np.abs(A[b] @ X[b] - B[b]) / (np.abs(A[b]) @ np.abs(X[b]) + np.abs(B[b]))
        assert err.max() < 10 * n * EPS


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("where", [(3, 100), (100, 3), (140, 150)])
def test_nonfinite_entries_spread_as_on_the_fp64_pipe(bad, where):
    n, m = 170, 4
    A, B = _systems(n, m, 8)
    A[0][where] = bad
    got, want = _solve(A, B), _solve(A, B, tensor=0)
    assert np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2])
    assert np.array_equal(np.isfinite(got[0]), np.isfinite(want[0]))
    assert _backward_error(A[1], got[0][1], B[1]) < 10 * n * EPS


def test_waits_that_run_out_leave_a_complete_update():
    n, m = 300, 20
    A, B = _systems(n, m, 9)
    X, st, _ = _solve(A, B, polls=1)
    assert (st == 0).all()
    for b in range(2):
        assert _backward_error(A[b], X[b], B[b]) < 10 * n * EPS


def test_more_systems_than_one_launch_takes():
    n, m, batch = 34, 1, 5000  # 0.2 MB of images each: 1 GiB holds fewer than 5000
    A, B = _systems(n, m, 10, batch)
    X, st, _ = _solve(A, B)
    assert (st == 0).all()
    err = np.abs(A @ X - B).max((1, 2)) / (np.abs(A).sum(-1).max(-1) * np.abs(X).max((1, 2)))
    assert err.max() < 10 * n * EPS
