"""Eigenvectors from kept Lanczos vectors: all steps kept, the first ones only
(the rest run again from the last kept one) and none give the same vector.

Both ways sum coeff_k w_k over m <= 60 steps in the same order; a term of one
is coeff_k rounded(v_k / b_k), of the other rounded(coeff_k / b_k) v_k, at most
two roundings apart, and the sums add m more: (m + 2) 2^-53 sum_k |coeff_k|
|w_k| <= 62 * 1.2e-16 * sqrt(60) < 1e-13 of a vector of norm one."""

import numpy as np
import pytest

from conftest import random_model
from test_gpu_batch import _check_against_alone

pytestmark = pytest.mark.gpu
TOL = 1e-13


def _pad(n):
    return (n + 3) // 4 * 4


def _states(pkg, nsite, sectors):
    from math import comb
    return sum(_pad(comb(nsite, u)) * _pad(comb(nsite, d)) for u, d in sectors)


@pytest.mark.parametrize("norb,nsite,sectors,steps", [
    (1, 6, [(3, 3), (2, 3)], 4), (1, 9, [(4, 5), (5, 4), (4, 4)], 41), (1, 10, [(5, 5)], 60),
    (1, 16, [(8, 1)], 20), (1, 17, [(8, 1)], 20), (2, 8, [(4, 4), (3, 4)], 40),
])
def test_partly_kept_vectors(pkg, solver, norb, nsite, sectors, steps):
    rng = np.random.default_rng(31 * norb + nsite)
    solver.set_model(random_model(pkg, rng, norb, nsite - norb, J=0.5 if norb > 1 else 0.0, spin_dep=True))
    per_step = 8.0 * _states(pkg, nsite, sectors)
    keeps = sorted({(steps + 1) // 2, steps // 2 + 2, steps - 3, steps - 1})
    try:
        solver.set_keep_vectors(0)
        ref = solver.ground_state(sectors, steps, seed=11)
        solver.set_keep_vectors(1)
        whole = solver.ground_state(sectors, steps, seed=11)
        part = []
        for k in (k for k in keeps if 2 <= k < steps):
            solver.set_keep_limit_test(per_step * (k + 2) if k + 2 < steps else per_step * (steps - 0.5))
            part.append(solver.ground_state(sectors, steps, seed=11))
    finally:
        solver.set_keep_vectors(1)
        solver.set_keep_limit_test(0)
    assert part
    for r in [whole] + part:
        assert r["isector"] == ref["isector"] and r["e0"] == ref["e0"]
        assert np.abs(r["vec"] - ref["vec"]).max() <= TOL


@pytest.mark.parametrize("share", [0.0, 0.4])
def test_batch_and_server_with_kept_vectors(pkg, solver, share):
    """Batches and a server with every instance's vectors kept, against none
    and (share) against some: the same sectors and E0, G to the rounding of the
    vectors (1e-10, as for one solve)."""
    rng = np.random.default_rng(99)
    omega = pkg.matsubara(64, 50.0)
    insts = []
    for i, ns in enumerate([6, 9, 8, 7]):
        n = ns // 2
        insts.append(dict(model=random_model(pkg, rng, 1, ns - 1), sectors=[(n, n), (n, n + 1), (n + 1, n)],
                          nspin=1 + i % 2, seed=50 + i))
    steps = 40
    total = 8.0 * steps * sum(_states(pkg, i["model"].nsite, i["sectors"]) for i in insts)

    def serve():
        sv = pkg.Server(solver, steps, omega)
        done, _, _ = pkg.serve(sv, insts, [0.0] * len(insts))
        return [(r["isector"], r["e0"], r["G_cl"]) for r in done]

    def batch():
        b = solver.solve_batch(insts, steps, omega)
        return list(zip(b["isector"], b["e0"], b["G_cl"]))

    kept = batch() + serve()
    try:
        if share:
            solver.set_keep_limit_test(share * total)
        else:
            solver.set_keep_vectors(0)
        other = batch() + serve()
    finally:
        solver.set_keep_vectors(1)
        solver.set_keep_limit_test(0)
    for (s1, e1, g1), (s2, e2, g2) in zip(kept, other):
        assert s1 == s2 and e1 == e2
        assert np.abs(np.asarray(g1) - np.asarray(g2)).max() <= 1e-10


def test_batch_of_more_instances_than_one_launch_takes(pkg, solver):
    """52 instances: the tables (40 per launch) and the vectors' sums (48) take
    several launches.  Against every instance alone, as the other batches are
    (the cut of a run over the CTAs, so the order of its sums, depends on what
    else is in the launch)."""
    rng = np.random.default_rng(5)
    omega = pkg.matsubara(16, 20.0)
    insts = [dict(model=random_model(pkg, rng, 1, 4 + i % 2), sectors=[(2, 2), (2, 3)], nspin=1, seed=900 + i)
             for i in range(52)]
    _check_against_alone(solver, insts, solver.solve_batch(insts, 8, omega), omega, 8)
