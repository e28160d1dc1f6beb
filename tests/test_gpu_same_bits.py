"""What must not depend on the company or on memory: results of small models
alone and among others, and eigenvectors from kept vectors and from a second
run of the recurrence, which is the scan's arithmetic again."""

import numpy as np
import pytest

from conftest import random_model
from test_gpu_keep import _states

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


def _tolerance(steps):
    """Both ways sum coeff_k w_k of the same w_k in the same order: a term
    differs by at most two roundings and the sums add one a step, so an element
    by (steps + 4) 2^-53 sum_k |coeff_k| |w_k|, where the sum over k is at most
    2 (0.5 to 1.2 in a restatement of these runs).  The normalisation divides
    it by the sum's norm, which is 1 until copies of converged states come in
    and anything of order one then (0.02 to 1.4 there): 1e-4 is left for it,
    and a factor of two for the norms' own difference."""
    return (steps + 4) * 2.0**-53 * 2.0 * 2.0 / 1e-4


@pytest.mark.parametrize("nsite,sector", [(6, (3, 3)), (7, (3, 4))])
@pytest.mark.parametrize("steps", [80, 150, 300])
def test_small_scan_run_again(pkg, solver, nsite, sector, steps):
    """400 and 1,225 states far beyond convergence, where a second run in any
    other arithmetic loses the vectors' norm."""
    for seed in range(6):
        solver.set_model(random_model(pkg, np.random.default_rng(500 + seed), 1, nsite - 1))
        per_step = 8.0 * _states(pkg, nsite, [sector])
        got = []
        try:
            for keep, limit in ((1, 0.0), (0, 0.0), (1, per_step * (steps // 2 + 4))):
                solver.set_keep_vectors(keep)
                solver.set_keep_limit_test(limit)
                got.append(solver.ground_state([sector], steps, seed=seed))
        finally:
            solver.set_keep_vectors(1)
            solver.set_keep_limit_test(0)
        for r in got[1:]:
            assert r["e0"] == got[0]["e0"]
            assert np.abs(r["vec"] - got[0]["vec"]).max() <= _tolerance(steps), (seed, steps)


def test_small_winner_of_a_larger_scan_run_again(pkg, solver):
    """A scan with a sector for the persistent kernel takes all of the model's
    runs there: the small winner's second run goes there too."""
    for seed in range(3):
        m = random_model(pkg, np.random.default_rng(700 + seed), 1, 7)
        m.ek += 3.0                                      # few electrons: (1, 1) of 64 states or (2, 2) of 784
        m.mu = 0.0
        solver.set_model(m)
        steps, sectors = 150, [(1, 1), (2, 2), (4, 4)]
        got = []
        try:
            for keep in (1, 0):
                solver.set_keep_vectors(keep)
                got.append(solver.ground_state(sectors, steps, seed=seed))
        finally:
            solver.set_keep_vectors(1)
        assert got[0]["sector"] != (4, 4)
        assert got[0]["e0"] == got[1]["e0"]
        assert np.abs(got[0]["vec"] - got[1]["vec"]).max() <= _tolerance(steps)


def test_short_winner_of_a_scan_with_long_lines_run_again(pkg, solver):
    """Lines of 24,310 strings make the scan of every sector take rows one by
    one; the second run of (2, 1), 2,312 states, takes tiles of rows."""
    rng = np.random.default_rng(81)
    for seed in range(3):
        m = random_model(pkg, rng, 1, 16)
        m.ek += 3.0                                      # every electron costs: the emptier sector wins
        m.mu = 0.0
        solver.set_model(m)
        steps, got = 120, []
        try:
            for keep in (1, 0):
                solver.set_keep_vectors(keep)
                got.append(solver.ground_state([(8, 1), (2, 1)], steps, seed=seed))
        finally:
            solver.set_keep_vectors(1)
        assert got[0]["sector"] == (2, 1) and got[0]["e0"] == got[1]["e0"]
        assert np.abs(got[0]["vec"] - got[1]["vec"]).max() <= _tolerance(steps), seed
