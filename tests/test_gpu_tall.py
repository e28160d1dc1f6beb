"""Lanczos runs of sectors, and of launches, whose columns and rows are of very
different lengths: every pair of widths that the plan takes for them (8 x 4,
4 x 8, 8 x 2, 2 x 8 by one sector; 4 x 2, 4 x 1 and 2 x 4 by scans of a long
row and a long column), with and without exchange terms.  As for the other
tile shapes: coefficients of 20 steps within 1e-9 of the oracle's, energies of
20 steps within 1e-10."""

import numpy as np
import pytest
from scipy.linalg import eigh_tridiagonal

from conftest import oracle_for, random_model

pytestmark = pytest.mark.gpu
STEPS = 20


def _model(pkg, norb, nsite):
    rng = np.random.default_rng(9000 * norb + nsite)
    return random_model(pkg, rng, norb, nsite - norb, J=0.5 if norb > 1 else 0.0, spin_dep=True)


@pytest.mark.parametrize("norb,nsite,nu,nd", [
    (1, 15, 7, 3), (1, 15, 3, 7), (2, 15, 7, 2), (2, 15, 2, 7), (1, 12, 6, 3), (1, 12, 3, 6), (2, 12, 6, 2), (1, 17, 2, 6),
])
def test_coefficients(pkg, solver, oracle_mod, norb, nsite, nu, nd):
    m = _model(pkg, norb, nsite)
    solver.set_model(m)
    o = oracle_for(oracle_mod, m)
    v0 = oracle_mod.start_vector(4, 0, o.dim(nu, nd)) + 0.1
    n_ref, a_ref, b_ref = o.lanczos_iteration(nu, nd, v0, STEPS)
    n, a, b = solver.lanczos_iteration(nu, nd, v0, STEPS)
    assert n == n_ref
    assert np.abs(a - a_ref).max() <= 1e-9 and np.abs(b - b_ref).max() <= 1e-9


@pytest.mark.parametrize("norb", [1, 2])
@pytest.mark.parametrize("nsite,sectors", [(16, [(8, 0), (0, 5)]), (17, [(8, 0), (0, 5)]), (17, [(5, 0), (0, 6)])])
def test_scans_of_long_rows_and_columns(pkg, solver, oracle_mod, norb, nsite, sectors):
    m = _model(pkg, norb, nsite)
    solver.set_model(m)
    o = oracle_for(oracle_mod, m)
    got = solver.ground_state(sectors, STEPS, seed=12)
    for i, (nu, nd) in enumerate(sectors):
        n, a, b = o.lanczos_iteration(nu, nd, oracle_mod.start_vector(12, i, o.dim(nu, nd)), STEPS)
        e = eigh_tridiagonal(a[:n], b[1:n], select="i", select_range=(0, 0))[0][0]
        assert abs(got["e_sector"][i] - e) <= 1e-10 * max(1.0, abs(e)), (nu, nd)
