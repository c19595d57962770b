"""The FP32 elimination with paired 64-column blocks where the right-hand sides no longer fit one CTA's shared memory and
the forward sweep runs block by block: it applies both blocks' row moves before the first block's solve.  An odd and an
even number of blocks, the last one narrow or nearly full, against the FP64 LU within the form's bound, in as many
refinement steps as without pairing (a wrong order of the moves would need more, or fall back)."""
import numpy as np
import pytest

from refeff_gb300 import fms, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms", [212, 215])  # n = 5300 (83 blocks, the last 52 wide), 5375 (84 blocks, the last 63)
def test_blocked_forward_sweep(atoms):
    cl, grid = wl.small_cluster(9.0, lmax=4, n_energies=8, seed=3)
    sel = np.arange(5, 7)
    k, ph = grid.wave_numbers[sel], grid.phase_shifts[sel]
    want, steps = None, {}
    for paired in (0, 1):
        ctx = fms.Context(0)
        try:
            ctx.set_option(ctx.OPT_PAIRED_BLOCKS, paired)
            plan = fms.fms_real_space_plan(ctx, cl.positions[:atoms], cl.potentials[:atoms], cl.lmaxph)
            assert plan.shape.n_states == 25 * atoms
            if want is None:
                want, _ = fms.fms_real_space_spectrum(plan, k, ph, fms.FORM_FP64_LU)
            got, st = fms.fms_real_space_spectrum(plan, k, ph, fms.FORM_FP32_REFINED)
            it, _, fallback = plan.refinement_stats(len(sel))
            assert (st == 0).all() and not fallback.any()
            assert np.linalg.norm(got - want) <= 1e-9 * np.linalg.norm(want)
            steps[paired] = int(it.sum())
        finally:
            ctx.close()
    assert abs(steps[1] - steps[0]) <= len(sel), steps
