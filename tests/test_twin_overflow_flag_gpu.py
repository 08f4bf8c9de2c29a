"""GPU test of the overflow flag of the shared lists (equation/ns_twin.cu): it is raised when a
particle has more neighbours than list slots, as with one particle per thread, not when only the
list that two particles share is full."""
from __future__ import annotations

import numpy as np
import pytest

from test_twin_gpu import run
from test_twin_seams_gpu import KEYS, with_fluid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,over", [(17, False), (18, True)])
def test_flag_of_two_full_lists(sphlib, cuda, size, over):
    """Two clusters of `size` particles, size - 1 neighbours each, 16 slots: at 17, odd, one thread
    holds a particle of either, whose shared list has 2 x 17 entries for 2 x 16 slots."""
    from tmp_sph_gb300 import api
    dx = 0.004
    g = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3)[:size]
    ball = 0.55 * dx * g  # diameter 1.91 dx, under the support radius 2.6 dx
    pos = np.concatenate([ball + [0.3, 0.2, 0.1], ball + [0.6, 0.3, 0.4]])
    st, p = with_fluid(pos, dx)
    assert len(st["rho"]) >= 400000
    o = {api.SPH_OPT_NEIGHBOR_CAP: 16, api.SPH_OPT_SKIN_PERMILLE: 0}
    two = run(st, p, o, steps=1)
    one = run(st, p, {**o, api.SPH_OPT_PARTICLES_PER_THREAD: 2}, steps=1)
    assert bool(one["flags"] & api.SPH_FLAG_NEIGHBOR_OVERFLOW) == over
    assert two["flags"] == one["flags"]
    for k in KEYS:
        assert np.array_equal(two[k], one[k]), k
