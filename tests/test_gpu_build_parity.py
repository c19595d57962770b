"""The system build's parity form (one spin channel, no spin selector: one mu sum serves the columns m2 and -m2) against the
FP64 oracle and the general form: every L it serves, clusters whose atoms carry different l cutoffs, atoms on the axes
(degenerate angles), damped pairs with an unsymmetric sigma^2 table, cut-off pairs, and the plain G0 of the iterative
forms.

Tolerances: the files' FP64 gate 1e-10 and chosen-form gate 1e-6, relative per energy.
"""
import numpy as np
import pytest

from oracle import pyoracle as po
from refeff_gb300 import fms, workloads as wl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = fms.Context(0)
    yield c
    c.close()


def _check(ctx, pos, pots, lmaxph, grid, **kw):
    ref = po.fms_spectrum(pos, pots, lmaxph, grid.wave_numbers, grid.phase_shifts, mode=po.F64, **kw)
    plan_kw = dict(kw)
    if "rdirec" in plan_kw:
        plan_kw["direct_cutoff"] = plan_kw.pop("rdirec")
    if "sigsqr" in plan_kw:
        plan_kw["mean_square_displacements"] = plan_kw.pop("sigsqr")
    plan = fms.fms_real_space_plan(ctx, pos, pots, lmaxph, **plan_kw)
    for form, tol in ((fms.FORM_FP64_LU, 1e-10), (fms.FORM_FP32_REFINED, 1e-6)):
        got, st = fms.fms_real_space_spectrum(plan, grid.wave_numbers, grid.phase_shifts, form)
        assert (st == 0).all()
        for e in range(len(st)):
            assert np.linalg.norm(got[e] - ref[e]) <= tol * np.linalg.norm(ref[e]), (form, e)
    plan.close()


@pytest.mark.parametrize("lmax", [0, 1, 2, 3, 4, 5])
def test_every_angular_limit(ctx, lmax):
    cl = wl.displaced_fcc_cluster(np.random.default_rng(lmax), 3.61, 2.7, 0.05, lmax)
    _check(ctx, cl.positions, cl.potentials, cl.lmaxph, wl.energy_grid(cl, 3, -5.0, 40.0, seed=lmax))


def test_mixed_cutoffs_and_axes(ctx):
    """Absorber lmax 2, hosts lmax 3 and 1, undisplaced rocksalt sites (pairs along every axis), 27 atoms: the row chunks
    of 16 atoms end inside the cluster."""
    pos, species = wl.rocksalt_sites(4.44, 4.5)
    pot = np.where(species == 0, 1, 2).astype(np.int32)
    order = np.argsort(np.linalg.norm(pos, axis=1), kind="stable")[:27]
    pos, pot = pos[order].astype(np.float32), pot[order]
    pot[0] = 0
    cl = wl.Cluster(pos, pot, np.array([2, 3, 1], np.int32))
    _check(ctx, cl.positions, cl.potentials, cl.lmaxph, wl.energy_grid(cl, 3, 0.0, 40.0, seed=3))


def test_unsymmetric_damping_and_cutoff(ctx):
    cl = wl.displaced_fcc_cluster(np.random.default_rng(9), 3.61, 3.7, 0.05, 2)
    n = cl.n_atoms
    sig = np.random.default_rng(10).uniform(0.0, 0.01, size=(n, n)).astype(np.float32)
    np.fill_diagonal(sig, 0.0)
    _check(ctx, cl.positions, cl.potentials, cl.lmaxph, wl.energy_grid(cl, 2, 0.0, 40.0, seed=4), rdirec=3.2,
           sigsqr=np.asfortranarray(sig))
