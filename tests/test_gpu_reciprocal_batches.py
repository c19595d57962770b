"""Reciprocal-space integration over more k-points than one batch holds (1024), and what it refuses."""
import numpy as np
import pytest

from refeff_gb300 import fms

pytestmark = pytest.mark.gpu


def _inputs(order, k_points, seed=1):
    rng = np.random.default_rng(seed)
    G = (rng.normal(size=(k_points, order, order)) + 1j * rng.normal(size=(k_points, order, order))) * (0.3 / order)
    return G, rng.uniform(0.5, 2.0, size=k_points), np.diag(rng.normal(size=order) * 0.3 + 0.1j)


def test_a_wait_that_runs_out_in_the_first_batch_is_reported():
    """1025 k-points at a poll budget that 1024 systems at a time exceed and one alone does not (16 .. 24 and 64 .. 96
    polls): the second batch's clean run must not hide the first one's."""
    ctx = fms.Context(0)
    ctx.set_option(ctx.OPT_TC_WAIT_POLLS, 40)
    _, st = fms.reciprocal_integrate(ctx, *_inputs(64, 1), fms.FORM_FP32_REFINED)
    assert (st == 0).all()
    with pytest.raises(fms.FmsError) as e:
        fms.reciprocal_integrate(ctx, *_inputs(64, 1025), fms.FORM_FP32_REFINED)
    assert "timed out" in str(e.value)
    ctx.close()
