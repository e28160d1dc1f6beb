"""Many runs of very uneven sizes in one launch: every sector of a model, more
of them than CTAs and fewer.  Energies of 25 steps against the same sectors
alone, 1e-10 (the cut over the CTAs orders the sums of a(k) and b(k))."""

import numpy as np
import pytest

from conftest import random_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,nsite", [(1, 9), (1, 11), (1, 12), (2, 10)])
def test_every_sector_at_once(pkg, solver, norb, nsite):
    solver.set_model(random_model(pkg, np.random.default_rng(nsite), norb, nsite - norb, J=0.5 if norb > 1 else 0.0,
                                  spin_dep=True))
    sectors = [(u, d) for u in range(nsite + 1) for d in range(nsite + 1)]
    together = solver.ground_state(sectors, 25, seed=6, want_vec=False)["e_sector"]
    for i in list(range(0, len(sectors), 13)) + [sectors.index((nsite // 2, nsite // 2)), len(sectors) - 1]:
        alone = solver.diag_lanczos(*sectors[i], 25, seed=6, stream=i)["e0"]
        assert abs(together[i] - alone) <= 1e-10 * max(1.0, abs(alone)), sectors[i]
