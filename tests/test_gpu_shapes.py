"""The persistent Lanczos kernel at the edges of its tile shapes: sectors with
one long and one short line, so that every shape (eight columns and rows with
two CTAs per SM or one, four, two) runs on remainders of its slabs, row groups
and planes, and the smallest sectors.  First 20 coefficients against the
oracle: a 1-ulp change grows to about 1e-11 by step 20, so 1e-9 is asked."""

import numpy as np
import pytest

from conftest import oracle_for, random_model

pytestmark = pytest.mark.gpu
STEPS = 20


@pytest.mark.parametrize("norb,nsite,nu,nd", [
    (1, 2, 1, 1), (1, 3, 2, 1), (1, 5, 2, 3), (1, 7, 3, 1), (1, 9, 4, 5),      # 4 to 15,876 states
    (1, 13, 1, 6), (1, 13, 7, 2), (1, 12, 4, 2),                               # two CTAs per SM
    (1, 14, 1, 7), (1, 14, 7, 2),                                              # 3,432 strings: one CTA, eight lines
    (1, 15, 1, 7), (1, 15, 8, 1),                                              # 6,435: four lines
    (1, 16, 1, 8), (1, 16, 8, 1),                                              # 12,870: two lines
    (2, 8, 3, 4), (2, 14, 7, 1), (2, 15, 1, 7), (3, 7, 3, 4),                  # exchange terms
])
def test_coefficients_of_every_tile_shape(pkg, solver, oracle_mod, norb, nsite, nu, nd):
    rng = np.random.default_rng(1000 * norb + 100 * nsite + 10 * nu + nd)
    m = random_model(pkg, rng, norb, nsite - norb, J=0.5 if norb > 1 else 0.0, spin_dep=True)
    solver.set_model(m)
    o = oracle_for(oracle_mod, m)
    v0 = rng.random(o.dim(nu, nd)) + 0.1
    n_ref, a_ref, b_ref = o.lanczos_iteration(nu, nd, v0, STEPS)
    n, a, b = solver.lanczos_iteration(nu, nd, v0, STEPS)
    k = min(n_ref, o.dim(nu, nd) - 1, STEPS)             # a small sector's last norms are rounding
    assert min(n, k) == k
    assert np.abs(a[:k] - a_ref[:k]).max() <= 1e-9 and np.abs(b[:k] - b_ref[:k]).max() <= 1e-9
