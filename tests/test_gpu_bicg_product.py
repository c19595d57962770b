"""The BiCGSTAB form's tensor-core product (two FP16 terms a value) at the sizes where it can go wrong: fewer columns
than one slab, the ends of the 256-column accumulations, of the 512-column slices and of the 1024-row blocks that scale
its operand, 16 and 32 accumulator columns, both forms of the complex product; and the same systems with columns of
very different size (a phase shift scaled down by 1e6), against the FP64 LU within the form's 1e-6 gate."""
import numpy as np
import pytest

from refeff_gb300 import fms, workloads as wl

pytestmark = pytest.mark.gpu

# atoms, lmax: n = 5, 243, 256, 272, 496, 512, 513, 1024, 1025, 1040
SIZES = [(5, 0), (27, 2), (16, 3), (17, 3), (31, 3), (32, 3), (57, 2), (64, 3), (41, 4), (65, 3)]


@pytest.mark.parametrize("atoms,lmax", SIZES)
@pytest.mark.parametrize("mode,shrink", [(1, 1.0), (2, 1.0), (1, 1e-6)])
def test_product_sizes(atoms, lmax, mode, shrink):
    cl, grid = wl.small_cluster(7.0, lmax=lmax, n_energies=8, seed=5)
    sel = np.arange(4, 8)
    k, ph = grid.wave_numbers[sel], grid.phase_shifts[sel].copy()
    if lmax:
        ph[:, :, [0, -1]] *= shrink  # l = lmax
    ctx = fms.Context(0)
    try:
        ctx.set_option(ctx.OPT_BICG_TENSOR, mode)
        plan = fms.fms_real_space_plan(ctx, cl.positions[:atoms], cl.potentials[:atoms], cl.lmaxph)
        assert plan.shape.n_states == atoms * (lmax + 1) ** 2
        m = plan.shape.absorber_block
        want, _ = fms.fms_real_space_spectrum(plan, k, ph, fms.FORM_FP64_LU)
        got, st = fms.fms_real_space_spectrum(plan, k, ph, fms.FORM_BICGSTAB)
        flags = plan.bicgstab_lu_energies(len(sel))
        assert (st == 0).all()
        if plan.shape.n_states > 16:  # a few states: the iteration ends exactly, which may count as a breakdown
            assert (flags == 0).all(), flags
        for e in range(len(sel)):
            ref = want[e, :m, :m, 0]
            assert np.linalg.norm(got[e, :m, :m, 0] - ref) <= 1e-6 * np.linalg.norm(ref), e
    finally:
        ctx.close()
