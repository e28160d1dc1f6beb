"""The launch count of the plain engine is the number of its launches."""

import numpy as np
import pytest

from conftest import random_model

pytestmark = pytest.mark.gpu


def test_launches_of_a_plain_step(pkg):
    """One Lanczos step more: the rescaling, H.v, the two of a(k), the axpy and
    the two of b(k)."""
    with pkg.Solver(0, engine=pkg.ENGINE_PLAIN) as s:
        s.set_model(random_model(pkg, np.random.default_rng(1), 1, 5))
        v0 = np.random.default_rng(2).random(400)
        n = []
        for steps in (3, 3, 4):                          # the first call also builds the tables
            before = s.launch_count()
            s.lanczos_iteration(3, 3, v0, steps)
            n.append(s.launch_count() - before)
        assert n[2] - n[1] == 7
