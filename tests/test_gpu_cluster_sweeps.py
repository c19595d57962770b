"""The FP32 sweeps on clusters where their shapes change: one CTA, clusters of 2, 4 and 8, four right-hand sides a cluster
(few columns, and large systems), a last block of one row, odd orders, more CTAs than blocks left.  Random systems pivot
in almost every column, so the row moves cross the CTAs.  One solution without refinement against complex128 LAPACK (a
wrong row or block gives O(1) errors; FP32 elimination of such systems reaches 1e-4), and the refinement, whose steps are
sweeps, converges."""
import numpy as np
import pytest

from refeff_gb300 import fms

pytestmark = pytest.mark.gpu


# n, right-hand sides, batch: clusters of 1, 1, 2, 2, 4, 4, 8 CTAs; NB = 32 below 512
@pytest.mark.parametrize("n,m,batch", [(33, 3, 2), (511, 9, 2), (577, 8, 2), (1024, 1, 3), (1089, 16, 1), (2049, 4, 1),
                                       (2113, 9, 1), (4097, 17, 1)])
def test_sweeps(n, m, batch):
    rng = np.random.default_rng(n + m)
    A = rng.normal(size=(batch, n, n)) + 1j * rng.normal(size=(batch, n, n))
    B = rng.normal(size=(batch, n, m)) + 1j * rng.normal(size=(batch, n, m))
    ctx = fms.Context(0)
    try:
        ctx.set_option(ctx.OPT_DENSE_REFINEMENT, 0)
        raw, _, _ = fms.complex_lu_solve_batched(ctx, A, B, fms.FORM_FP32_REFINED)
        ctx.set_option(ctx.OPT_DENSE_REFINEMENT, 10)
        got, st, _ = fms.complex_lu_solve_batched(ctx, A, B, fms.FORM_FP32_REFINED)
    finally:
        ctx.close()
    assert (st == 0).all()
    for b in range(batch):
        ref = np.linalg.solve(A[b], B[b])
        assert np.linalg.norm(raw[b] - ref) <= 2e-2 * np.linalg.norm(ref)
