"""What must not depend on the company or on memory: results of small models
alone and among others, and eigenvectors from kept vectors and from a second
run of the recurrence, which is the scan's arithmetic again."""

import numpy as np
import pytest

from conftest import random_model

pytestmark = pytest.mark.gpu


def _small(pkg, rng, norb, nsite, i):
    n = nsite // 2
    return dict(model=random_model(pkg, rng, norb, nsite - norb, J=0.5 if norb > 1 else 0.0, spin_dep=True),
                sectors=[(n, n), (n, n - 1), (n + 1, n)], nspin=1 + i % 2, seed=300 + i)


@pytest.mark.parametrize("others", [[(1, 7)], [(2, 6)], [(1, 7), (2, 7), (1, 9)]])
def test_small_models_do_not_see_their_company(pkg, solver, others):
    """Models of at most 512 states a run (6 sites) and of at most 2,000 (7),
    with and without exchange terms, and a larger one: E0 and G of the small
    ones are the same to the bit alone, in a batch and in a server."""
    rng = np.random.default_rng(61)
    omega = pkg.matsubara(32, 20.0)
    insts = [_small(pkg, rng, norb, ns, i) for i, (norb, ns) in enumerate([(1, 6), (1, 5), (2, 6)] + others)]
    steps = 40
    batch = solver.solve_batch(insts, steps, omega)
    sv = pkg.Server(solver, steps, omega)
    served, _, _ = pkg.serve(sv, insts, [0.0] * len(insts))
    sv.close()
    for i, inst in enumerate(insts):
        if inst["model"].nsite > 7:
            continue
        solver.set_model(inst["model"])
        one = solver.solve(inst["sectors"], steps, omega, nspin=inst["nspin"], seed=inst["seed"])
        assert batch["e0"][i] == one["e0"] and np.array_equal(batch["G_cl"][i], one["G_cl"]), i
        assert served[i]["e0"] == one["e0"] and np.array_equal(served[i]["G_cl"], one["G_cl"]), i
