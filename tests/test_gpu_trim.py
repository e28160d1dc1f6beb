"""edzt_trim: what a scan left cached is free for others; the model and the
ground state stay."""

import numpy as np
import pytest
import torch

from conftest import random_model

pytestmark = pytest.mark.gpu


def test_trim_gives_cached_memory_back(pkg):
    with pkg.Solver(0) as s:
        s.set_model(random_model(pkg, np.random.default_rng(8), 1, 11))
        omega = pkg.matsubara(16, 20.0)
        s.ground_state([(6, 6)], 60, seed=2)             # 853,776 states, 60 steps kept: 410 MB
        ref = s.cluster_green_ftn(1, 40, omega)["G_cl"]
        before = torch.cuda.mem_get_info()[0]
        s.trim()
        assert torch.cuda.mem_get_info()[0] - before >= 8 * 853776 * 60
        s.trim()
        assert np.array_equal(s.cluster_green_ftn(1, 40, omega)["G_cl"], ref)
