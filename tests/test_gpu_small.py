"""Runs of up to 2,000 states in one CTA's shared memory: lines of one string,
sectors below and off the CTA's threads and its rows of four, the largest taken
and larger ones, exchange terms, a zero vector and every start vector.  First 20
coefficients against the oracle and against the persistent kernel (a pass cap
that is never reached selects it): a 1-ulp change grows to about 1e-11 by step
20, so 1e-9 is asked, as for the tile shapes."""

import numpy as np
import pytest

from conftest import oracle_for, random_model

pytestmark = pytest.mark.gpu
STEPS = 20


@pytest.mark.parametrize("norb,nsite,nu,nd", [
    (1, 2, 0, 1), (1, 2, 1, 1), (1, 3, 1, 2), (1, 6, 3, 3), (1, 7, 3, 2), (1, 7, 3, 4), (1, 8, 2, 4), (1, 8, 4, 4),
    (1, 13, 0, 6), (1, 13, 6, 0), (1, 9, 2, 4), (1, 16, 1, 3), (1, 13, 4, 1), (1, 11, 1, 5),
    (1, 9, 3, 3),
    (2, 4, 1, 2), (2, 7, 3, 4), (3, 8, 4, 2), (2, 8, 4, 4),
])
def test_small_run_coefficients(pkg, solver, oracle_mod, norb, nsite, nu, nd):
    rng = np.random.default_rng(77000 * norb + 100 * nsite + 10 * nu + nd)
    m = random_model(pkg, rng, norb, nsite - norb, J=0.5 if norb > 1 else 0.0, spin_dep=True)
    solver.set_model(m)
    o = oracle_for(oracle_mod, m)
    dim = o.dim(nu, nd)
    v0 = rng.random(dim) + 0.1
    n_ref, a_ref, b_ref = o.lanczos_iteration(nu, nd, v0, STEPS)
    n, a, b = solver.lanczos_iteration(nu, nd, v0, STEPS)
    solver.set_fault_test(pass_cap=10**6)
    try:
        n2, a2, b2 = solver.lanczos_iteration(nu, nd, v0, STEPS)
    finally:
        solver.set_fault_test()
    k = min(n_ref, dim - 1, STEPS)                       # a small sector's last norms are rounding
    assert min(n, k) == k and min(n2, k) == k
    for ar, br in ((a_ref, b_ref), (a2, b2)):
        assert np.abs(a[:k] - ar[:k]).max(initial=0.0) <= 1e-9
        assert np.abs(b[:k] - br[:k]).max(initial=0.0) <= 1e-9


def test_small_run_of_a_zero_vector(pkg, solver):
    solver.set_model(random_model(pkg, np.random.default_rng(3), 1, 5))
    n, a, b = solver.lanczos_iteration(3, 3, np.zeros(400), 10)
    assert n == 0 and not a.any() and not b.any()


@pytest.mark.parametrize("norb,nsite", [(1, 6), (2, 6), (1, 8)])
def test_solve_of_small_sectors(pkg, solver, norb, nsite):
    """A whole solve (scan with kept vectors, c and c^+ runs) both ways: the
    bounds of the batched form against single solves, E0 1e-10, G 1e-8."""
    rng = np.random.default_rng(40 + norb + nsite)
    solver.set_model(random_model(pkg, rng, norb, nsite - norb, J=0.5 if norb > 1 else 0.0))
    n = nsite // 2
    sectors = [(n, n), (n, n - 1), (n + 1, n)]
    omega = pkg.matsubara(64, 40.0)
    small = solver.solve(sectors, 30, omega, nspin=2, seed=8)
    solver.set_fault_test(pass_cap=10**6)
    try:
        ref = solver.solve(sectors, 30, omega, nspin=2, seed=8)
    finally:
        solver.set_fault_test()
    assert small["isector"] == ref["isector"]
    assert abs(small["e0"] - ref["e0"]) <= 1e-10 * max(1.0, abs(ref["e0"]))
    assert np.abs(np.asarray(small["G_cl"]) - np.asarray(ref["G_cl"])).max() <= 1e-8
