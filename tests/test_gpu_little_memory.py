"""A batch of dense systems with room on the device for its matrices but not for the operand images of all of its FP64
updates: the updates run in smaller slices of the batch and give the same bits as with room."""
import numpy as np
import pytest

from refeff_gb300 import fms

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_operand_images_for_a_part_of_the_batch():
    n, m, batch = 300, 4, 600  # matrices 0.94 GB, images 0.7 GB, staging 0.1 GB
    rng = np.random.default_rng(2)
    A = rng.normal(size=(batch, n, n)) + 3 * np.sqrt(n) * np.eye(n) + 0j
    b = rng.normal(size=(batch, n, m)) + 0j
    ctx = fms.Context(0)
    want = fms.complex_lu_solve_batched(ctx, A, b)
    ctx.close()
    ctx = fms.Context(0)
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (1500 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = fms.complex_lu_solve_batched(ctx, A, b)
    finally:
        del hold
        torch.cuda.empty_cache()
        ctx.close()
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


def test_a_plan_takes_the_memory_that_a_dense_call_left_kept():
    """The context keeps up to 512 MB between dense calls; a plan that needs them gets them."""
    from refeff_gb300 import workloads as wl
    cl = wl.cu_fcc_cluster(4.5, lmax=3)  # n = 688: 0.32 GB of matrices for 40 energies
    grid = wl.energy_grid(cl, 40, -20.0, 60.0, 3)
    rng = np.random.default_rng(5)
    A, b = rng.normal(size=(100, 300, 300)) + 60 * np.eye(300) + 0j, rng.normal(size=(100, 300, 4)) + 0j

    def spectrum(ctx):
        plan = fms.fms_real_space_plan(ctx, cl.positions, cl.potentials, cl.lmaxph)
        plan.set_batch(40)
        return plan

    ctx = fms.Context(0)
    ctx.set_option(ctx.OPT_DUAL_STREAMS, 0)
    want, _ = fms.fms_real_space_spectrum(spectrum(ctx), grid.wave_numbers, grid.phase_shifts)
    ctx.close()
    ctx = fms.Context(0)
    ctx.set_option(ctx.OPT_DUAL_STREAMS, 0)
    plan = spectrum(ctx)
    fms.complex_lu_solve_batched(ctx, A, b)  # leaves 0.4 GB kept
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (260 << 20), dtype=torch.uint8, device="cuda")
    try:
        got, st = fms.fms_real_space_spectrum(plan, grid.wave_numbers, grid.phase_shifts)
    finally:
        del hold
        torch.cuda.empty_cache()
        ctx.close()
    assert (st == 0).all() and np.array_equal(got, want)


def test_a_call_without_room_leaves_the_next_one_alone():
    rng = np.random.default_rng(6)
    A, b = rng.normal(size=(40, 300, 300)) + 60 * np.eye(300) + 0j, rng.normal(size=(40, 300, 4)) + 0j
    ctx = fms.Context(0)
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (40 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(fms.FmsError) as e:
            fms.complex_lu_solve_batched(ctx, A, b)
        assert e.value.name == "OutOfMemory"
    finally:
        del hold
        torch.cuda.empty_cache()
    X, st, _ = fms.complex_lu_solve_batched(ctx, A, b)
    ctx.close()
    assert (st == 0).all() and np.isfinite(X).all()
