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
    (1, 17, 8, 1), (2, 17, 8, 0),                                              # 24,310: one row
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


@pytest.mark.parametrize("norb,nsite,nu,nd", [
    (1, 4, 2, 2), (1, 8, 4, 4), (1, 11, 5, 6), (1, 11, 6, 1), (1, 12, 7, 6),   # 1, 1, 3 -> 2, 1 and 4 rows a tile
    (1, 13, 6, 4), (1, 13, 7, 5), (2, 13, 6, 5),                               # 4 rows, 256 threads three times
    (1, 14, 7, 4), (1, 15, 7, 4), (1, 15, 7, 2),                               # 2 rows and 1 of 3,000 strings and more
    (1, 16, 8, 1), (1, 17, 8, 1), (2, 16, 8, 2),                               # one row of 8,000 and more
])
@pytest.mark.parametrize("add", [False, True])
def test_hx_of_every_tile_shape(pkg, solver, oracle_mod, norb, nsite, nu, nd, add):
    """y = H x, y += H x and y = H x over x itself against the oracle, to the
    rounding of a row's sum (HX_TOL of test_gpu_basis_hx)."""
    import torch
    rng = np.random.default_rng(7000 * norb + 100 * nsite + 10 * nu + nd)
    m = random_model(pkg, rng, norb, nsite - norb, J=0.5 if norb > 1 else 0.0, spin_dep=True, zero_frac=0.1)
    solver.set_model(m)
    o = oracle_for(oracle_mod, m)
    n = o.dim(nu, nd)
    x, y0 = rng.standard_normal(n), rng.standard_normal(n)
    ref = o.hx(nu, nd, x, y0, py=True) if add else o.hx(nu, nd, x)
    y = solver.hx(nu, nd, x, y0, py=add)
    assert np.abs(y - ref).max() <= 1e-13 * (np.abs(ref).max() + 1.0)
    if not add:
        t = torch.from_numpy(x).to("cuda:0")
        solver.hx(nu, nd, t, t)
        assert np.array_equal(t.cpu().numpy(), y)
