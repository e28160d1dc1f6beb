"""H.v of sectors with few up strings and many down strings: one column and more
(a warp a tile), 66 to 120 (128 threads), 220, with last tiles of two and three rows,
against the oracle to the rounding of a row's sum (HX_TOL of
test_gpu_basis_hx)."""

import numpy as np
import pytest

from conftest import oracle_for, random_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,nsite,nu,nd", [
    (1, 12, 0, 6), (1, 13, 13, 6), (1, 13, 1, 7), (1, 16, 15, 8), (2, 16, 1, 8), (4, 12, 1, 6),
    (1, 12, 2, 6), (1, 13, 11, 5), (1, 12, 9, 6), (1, 16, 2, 8), (2, 12, 2, 6), (4, 14, 2, 7),
])
@pytest.mark.parametrize("add", [False, True])
def test_hx_of_short_rows(pkg, solver, oracle_mod, norb, nsite, nu, nd, add):
    rng = np.random.default_rng(8000 * norb + 100 * nsite + 10 * nu + nd)
    m = random_model(pkg, rng, norb, nsite - norb, J=0.5 if norb > 1 else 0.0, spin_dep=True, zero_frac=0.1)
    solver.set_model(m)
    o = oracle_for(oracle_mod, m)
    n = o.dim(nu, nd)
    x, y0 = rng.standard_normal(n), rng.standard_normal(n)
    ref = o.hx(nu, nd, x, y0, py=True) if add else o.hx(nu, nd, x)
    y = solver.hx(nu, nd, x, y0, py=add)
    assert np.abs(y - ref).max() <= 1e-13 * (np.abs(ref).max() + 1.0)
