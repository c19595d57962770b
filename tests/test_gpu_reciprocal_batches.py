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
    """1025 k-points at a poll budget that 1024 systems at a time exceed and one alone does not (between 24 and 64 polls
    where this was written): the second batch's clean run must not hide the first one's."""
    ctx = fms.Context(0)
    one, many, both = (_inputs(64, k) for k in (1, 1024, 1025))

    def times_out(inputs):
        try:
            fms.reciprocal_integrate(ctx, *inputs, fms.FORM_FP32_REFINED)
        except fms.FmsError as e:
            assert "timed out" in str(e)
            return True
        return False

    for polls in (40, 32, 48, 28, 56, 64, 80):
        ctx.set_option(ctx.OPT_TC_WAIT_POLLS, polls)
        if not any(times_out(one) for _ in range(4)) and all(times_out(many) for _ in range(4)):
            assert times_out(both)
            break
    else:
        pytest.skip("no poll budget tells the batches apart on this device")
    ctx.close()


def test_a_nonfinite_structure_factor_is_refused_first_and_before_anything_is_solved():
    ctx = fms.Context(0)
    G, w, T = _inputs(96, 30)
    fms.reciprocal_integrate(ctx, G, w, T)
    G[29, 95, 95] = np.nan
    launches = ctx._lib.refeff_fms_kernel_launches
    before = launches()
    with pytest.raises(fms.FmsError) as e:
        fms.reciprocal_integrate(ctx, G, w, T)
    assert e.value.name == "NonFiniteInput" and "structure factor" in str(e.value)
    assert launches() - before <= 2  # the packing of the batch
    T[3, 3] = np.inf
    with pytest.raises(fms.FmsError) as e:
        fms.reciprocal_integrate(ctx, G, w, T)
    assert "structure factor" in str(e.value)
    G[29, 95, 95] = 0
    with pytest.raises(fms.FmsError) as e:
        fms.reciprocal_integrate(ctx, G, w, T)
    assert "non-finite T" in str(e.value)
    ctx.close()
