"""Sectors that the kernels do not take are refused by every entry point."""

import numpy as np
import pytest

from conftest import random_model

pytestmark = pytest.mark.gpu


def test_sector_with_lines_too_long(pkg):
    """(10, 0) of 20 sites: within the no-allocation entry point's 262,144
    states, but one line of 184,756.  The tuner builds its tables before it
    refuses the sector, so that entry point finds them."""
    with pkg.Solver(0) as s:
        s.set_model(random_model(pkg, np.random.default_rng(6), 1, 19))
        v0 = np.ones(184756)
        for call in (lambda: s.tune_sector(10, 0, steps=4), lambda: s.lanczos_iteration_noalloc(10, 0, v0, 4),
                     lambda: s.lanczos_iteration(10, 0, v0, 4), lambda: s.hx(10, 0, v0)):
            with pytest.raises(pkg.EDError) as e:
                call()
            assert e.value.code == pkg.EDZT_ERR_ARG and "too large" in str(e.value)
        n, a, b = s.lanczos_iteration(1, 1, np.ones(400), 4)          # the context is still good
        assert n == 4 and np.isfinite(a).all() and np.isfinite(b).all()
