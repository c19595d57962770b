"""The context's kept workspace and staging of the dense solves: calls of other shapes, forms and options in one context
give what a fresh context gives, bit for bit; batches beyond one staging buffer, systems beyond it, and a call after one
whose tensor-core waits ran out.
"""
import numpy as np
import pytest

from refeff_gb300 import fms

pytestmark = pytest.mark.gpu


def _systems(n, m, batch, seed):
    rng = np.random.default_rng(seed)
    A = rng.normal(size=(batch, n, n)) + 1j * rng.normal(size=(batch, n, n)) + 3 * np.sqrt(n) * np.eye(n)
    return A, rng.normal(size=(batch, n, m)) + 1j * rng.normal(size=(batch, n, m))


def _fresh(A, B, form, tensor=1):
    c = fms.Context(0)
    c.set_option(c.OPT_TENSOR_CORES, tensor)
    out = fms.complex_lu_solve_batched(c, A, B, form)
    c.close()
    return out


def test_calls_in_one_context_match_fresh_ones():
    ctx = fms.Context(0)
    F64, F32 = fms.FORM_FP64_LU, fms.FORM_FP32_REFINED
    calls = [(40, 3, 5, F64, 1), (40, 3, 2, F64, 1), (130, 16, 4, F32, 1), (130, 16, 4, F64, 1), (33, 1, 7, F64, 1),
             (130, 16, 6, F32, 0), (130, 16, 4, F64, 0), (40, 3, 5, F64, 1), (700, 9, 2, F32, 1), (130, 16, 4, F32, 1)]
    for q, (n, m, batch, form, tensor) in enumerate(calls):
        A, B = _systems(n, m, batch, q)
        ctx.set_option(ctx.OPT_TENSOR_CORES, tensor)
        got, want = fms.complex_lu_solve_batched(ctx, A, B, form), _fresh(A, B, form, tensor)
        for g, w in zip(got, want):
            assert np.array_equal(g, w), q
    ctx.close()


@pytest.mark.parametrize("n,m,batch", [(300, 5, 60), (2100, 2, 1)])  # 5.4 M entries in pieces; 4.4 M entries in one system
def test_batches_and_systems_beyond_the_staging_buffer(n, m, batch):
    A, B = _systems(n, m, batch, n)
    X, st, _ = _fresh(A, B, fms.FORM_FP64_LU)
    assert (st == 0).all()
    for b in range(batch):
        assert np.abs(A[b] @ X[b] - B[b]).max() < 10 * n * 2.0 ** -53 * np.abs(A[b]).sum(-1).max() * np.abs(X[b]).max()


def test_a_timed_out_call_leaves_the_next_one_whole():
    ctx = fms.Context(0)
    A, B = _systems(300, 8, 2, 3)
    want = fms.complex_lu_solve_batched(ctx, A, B, fms.FORM_FP32_REFINED)
    ctx.set_option(ctx.OPT_TC_WAIT_POLLS, 1)
    with pytest.raises(fms.FmsError):
        fms.complex_lu_solve_batched(ctx, A, B, fms.FORM_FP32_REFINED)
    ctx.set_option(ctx.OPT_TC_WAIT_POLLS, 0)
    got = fms.complex_lu_solve_batched(ctx, A, B, fms.FORM_FP32_REFINED)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
    ctx.close()


def test_reciprocal_calls_share_the_workspace():
    ctx = fms.Context(0)
    rng = np.random.default_rng(4)
    for n, K, form in ((16, 40, fms.FORM_FP32_REFINED), (50, 300, fms.FORM_FP64_LU), (16, 7, fms.FORM_FP64_LU)):
        G = (rng.normal(size=(K, n, n)) + 1j * rng.normal(size=(K, n, n))) * (0.6 / np.sqrt(n))
        w, T = rng.uniform(0.5, 2.0, size=K), np.diag(rng.normal(size=n) * 0.3 + 0.1j)
        got, st = fms.reciprocal_integrate(ctx, G, w, T, form)
        want = np.einsum("k,kij->ij", w / w.sum(), np.linalg.solve(np.eye(n) - G @ T, G))
        assert (st == 0).all() and np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)
    ctx.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_nonfinite_structure_factor_is_refused(bad):
    ctx = fms.Context(0)
    G = np.ones((30, 20, 20), complex) * 0.01
    G[29, 19, 19] = bad
    with pytest.raises(fms.FmsError) as e:
        fms.reciprocal_integrate(ctx, G, np.ones(30), np.eye(20, dtype=complex))
    assert e.value.name == "NonFiniteInput" and "structure factor" in str(e.value)
    ctx.close()
