"""Running out of device memory, made on the host: a limit on what a context's
blocks hold (edzt_set_memory_limit_test) makes an allocation fail as one that
the device refuses.  Kept Lanczos vectors never make a call fail that succeeds
without them; a batch that does not fit at once runs in waves; a failed
admission or server step leaves the server as it was; a later call gets what
an earlier one left cached."""

import numpy as np
import pytest

from conftest import random_model
from test_gpu_keep import _states

pytestmark = pytest.mark.gpu
KB = 1024.0


def _run(pkg, f):
    """f() or None when it ran out of memory."""
    try:
        return f()
    except pkg.EDError as e:
        assert e.code == pkg.EDZT_ERR_OOM
        return None


def _limits(kept):
    """Limits around the kept vectors' size, 8 KB apart, and from little to plenty."""
    return sorted({kept + 8 * KB * k for k in range(130)} | {float(x) for x in np.geomspace(64 * KB, 2 * kept, 12)})


# The tolerance is that of the kept vectors' tests for m steps: (m + 4) 2^-53
# sqrt(m) < 1e-13 for m <= 60.
@pytest.mark.parametrize("sectors,steps,share", [([(4, 5), (5, 4), (4, 4)], 20, 1.0), ([(4, 4)], 40, 1.0),
                                                 ([(4, 4)], 40, 0.6)])
def test_kept_vectors_never_make_a_ground_state_fail(pkg, sectors, steps, share):
    m = random_model(pkg, np.random.default_rng(17), 1, 8, spin_dep=True)
    kept = 8.0 * _states(pkg, 9, sectors) * (steps if share == 1.0 else int(share * steps))

    def call(limit, keep):
        with pkg.Solver(0) as s:
            s.set_model(m)
            s.set_keep_vectors(keep)
            if share < 1.0:
                s.set_keep_limit_test(kept)
            s.set_memory_limit_test(limit)
            return _run(pkg, lambda: s.ground_state(sectors, steps, seed=3))

    ref = call(0, 0)
    outcomes = set()
    for limit in _limits(kept):
        without, with_ = call(limit, 0), call(limit, 1)
        outcomes.add((without is not None, with_ is not None))
        if with_ is not None:
            assert with_["isector"] == ref["isector"] and with_["e0"] == ref["e0"]
            assert np.abs(with_["vec"] - ref["vec"]).max() <= 1e-13
    assert (True, False) not in outcomes
    assert (True, True) in outcomes and (False, False) in outcomes


def _instances(pkg, sizes, one_sector=False):
    rng = np.random.default_rng(23)
    out = []
    for i, ns in enumerate(sizes):
        n = ns // 2
        out.append(dict(model=random_model(pkg, rng, 1, ns - 1, spin_dep=True),
                        sectors=[(n, n)] if one_sector else [(n, n), (n, n + 1), (n + 1, n)], nspin=1 + i % 2,
                        seed=70 + i))
    return out


def _same(got, ref):
    for (s1, e1, g1), (s2, e2, g2) in zip(got, ref, strict=True):
        assert s1 == s2 and abs(e1 - e2) <= 1e-10 * max(1.0, abs(e2))
        assert np.abs(np.asarray(g1) - np.asarray(g2)).max() <= 1e-8


def _batch(pkg, insts, steps, limit, keep, budget):
    with pkg.Solver(0) as s:
        s.set_keep_vectors(keep)
        s.set_memory_limit_test(limit)
        b = _run(pkg, lambda: s.solve_batch(insts, steps, pkg.matsubara(16, 20.0), hbm_budget=budget))
    return b and list(zip(b["isector"], b["e0"], b["G_cl"]))


def test_kept_vectors_never_make_a_batch_fail(pkg):
    insts, steps = _instances(pkg, [9, 9, 9], one_sector=True), 30
    kept = 8.0 * steps * _states(pkg, 9, [(4, 4)])
    ref = _batch(pkg, insts, steps, 0, 0, 1 << 30)
    outcomes = set()
    for limit in _limits(2 * kept):
        without, with_ = (_batch(pkg, insts, steps, limit, keep, 1 << 30) for keep in (0, 1))
        outcomes.add((without is not None, with_ is not None))
        if with_ is not None:
            _same(with_, ref)
    assert (True, False) not in outcomes and (True, True) in outcomes


@pytest.mark.parametrize("share", [0.3, 0.5, 0.9])
def test_batch_that_does_not_fit_at_once_runs_in_waves(pkg, share):
    """Without a budget of the caller's a batch takes what there is: instances
    that fit one by one are solved, whatever their sum."""
    insts = _instances(pkg, [9, 9, 10, 9, 10, 9])
    with pkg.Solver(0) as s:
        total = float(sum(s.footprint(i) for i in insts))
    ref = _batch(pkg, insts, 30, 0, 1, 0)
    got = _batch(pkg, insts, 30, share * total + 512 * KB, 1, 0)
    assert got is not None
    _same(got, ref)


def _serve(pkg, sv, insts, ids=None, steps=400):
    """Results of the requests, or None where a step ran out of memory."""
    ids = [sv.submit(i) for i in insts] if ids is None else ids
    res = [None] * len(ids)
    for _ in range(steps):
        if _run(pkg, sv.step) is None:
            return None, ids
        res = [r or sv.result(i) for r, i in zip(res, ids)]
        if all(res):
            return [(r["isector"], r["e0"], r["G_cl"]) for r in res], ids
    raise AssertionError("the server did not finish")


def test_failed_admission_leaves_the_request_queued(pkg):
    """Admissions that run out of memory, one step after the other, then memory:
    the requests are solved as if nothing had been, and both at a time, as the
    budget allows."""
    insts, omega = _instances(pkg, [9, 9]), pkg.matsubara(16, 20.0)
    with pkg.Solver(0) as s:
        ref = []
        for i in insts:
            s.set_model(i["model"])
            r = s.solve(i["sectors"], 20, omega, nspin=i["nspin"], seed=i["seed"])
            ref.append((r["isector"], r["e0"], r["G_cl"]))
    with pkg.Solver(0) as s:
        footprint = max(s.footprint(i) for i in insts)
        sv = pkg.Server(s, 20, omega, hbm_budget=int(2.5 * footprint))
        ids = [sv.submit(i) for i in insts]
        vectors = 24.0 * _states(pkg, 9, insts[0]["sectors"])     # of the scan's runs: more than any limit here
        for limit in np.linspace(8 * KB, 0.9 * vectors, 30):      # ever further into the admission
            s.set_memory_limit_test(limit)
            with pytest.raises(pkg.EDError) as e:
                sv.step()
            assert e.value.code == pkg.EDZT_ERR_OOM
        s.set_memory_limit_test(0)
        sv.set_step_ms(1e-3)
        assert sv.step() == (2, 0, 0)
        got, _ = _serve(pkg, sv, insts, ids, 4000)
        _same(got, ref)
        assert sv.step() == (0, 0, 0)
        sv.close()


def test_server_goes_on_after_a_step_without_memory(pkg):
    """Limits from the scan's vectors on, 16 KB apart: memory runs out between
    the phases of the requests.  With memory again the server finishes them."""
    insts, omega = _instances(pkg, [9, 6]), pkg.matsubara(16, 20.0)
    vectors = 24.0 * _states(pkg, 9, insts[0]["sectors"])

    def call(limit):
        with pkg.Solver(0) as s:
            s.set_keep_vectors(0)
            sv = pkg.Server(s, 20, omega)
            sv.set_step_ms(1000.0)                       # a step takes a request through
            ids, failed = [sv.submit(i) for i in insts], 0
            s.set_memory_limit_test(limit)
            for _ in range(4):
                failed += _run(pkg, sv.step) is None
            s.set_memory_limit_test(0)
            got, _ = _serve(pkg, sv, insts, ids)
            assert sv.step() == (0, 0, 0)
            sv.close()
            return failed, got

    _, ref = call(0)
    failures = []
    for k in range(60):
        failed, got = call(vectors + 16 * KB * k)
        failures.append(failed)
        _same(got, ref)
    assert max(failures) > 0 and min(failures) == 0


@pytest.mark.parametrize("second", [False, True])
def test_server_gives_kept_vectors_up(pkg, second):
    """Memory goes to others while a scan fills its kept vectors (and a second
    request waits): what is left serves the requests without them, so they are
    given up."""
    insts, omega = _instances(pkg, [9, 9][:1 + second]), pkg.matsubara(16, 20.0)

    def call(limited):
        with pkg.Solver(0) as s:
            sv = pkg.Server(s, 20, omega)
            sv.set_step_ms(1e-3)
            s.set_keep_vectors(int(limited))
            ids = [sv.submit(insts[0])]
            assert sv.step() == (1, 0, 0)                # the scan is on its way
            if limited:                                  # 2.7 MB a request; 8 MB are held, 7.8 MB of them kept
                s.set_memory_limit_test(1.5 * s.footprint(insts[0]))
            ids += [sv.submit(i) for i in insts[1:]]
            got, _ = _serve(pkg, sv, insts, ids, 4000)
            sv.close()
            return got

    ref, got = call(False), call(True)
    assert got is not None
    _same(got, ref)


def test_string_tables_get_what_earlier_calls_left_cached(pkg):
    """A scan leaves blocks cached; the string tables of a later model take
    their place when there is no other memory."""
    with pkg.Solver(0) as s:
        s.set_model(random_model(pkg, np.random.default_rng(2), 1, 9))
        s.ground_state([(5, 5)], 60, seed=1)             # 63,504 states, 60 steps: 30 MB kept
        s.set_model(random_model(pkg, np.random.default_rng(2), 1, 15))
        s.set_memory_limit_test(2048 * KB)               # the last ground state (500 KB) and the tables
        up, dn = s.generate_basis(8, 1)                  # rank tables of 2^16 strings, 256 KB each
        assert up.size == 12870 and dn.size == 16


def test_model_that_was_not_set_is_not_used(pkg):
    """Four orbitals' tables that do not fit: no model is set, not half of one."""
    m = random_model(pkg, np.random.default_rng(4), 1, 5)
    with pkg.Solver(0) as s:
        s.set_model(m)
        e0 = s.ground_state([(3, 3)], 20, seed=1)["e0"]
    with pkg.Solver(0) as s:
        s.set_model(m)
        s.set_memory_limit_test(1)
        with pytest.raises(pkg.EDError) as e:
            s.set_model(random_model(pkg, np.random.default_rng(4), 4, 2, J=0.5))
        assert e.value.code == pkg.EDZT_ERR_OOM
        s.set_memory_limit_test(0)
        with pytest.raises(pkg.EDError) as e:
            s.hx(3, 3, np.ones(400))
        assert e.value.code == pkg.EDZT_ERR_STATE
        s.set_model(m)
        assert s.ground_state([(3, 3)], 20, seed=1)["e0"] == e0
