"""GPU tests of shared lists that fill up (equation/ns_twin.cu): clusters of many particles within one
support radius.  The overflow flag is raised when a particle has more neighbours than list slots, as
with one particle per thread, and the fields are the same bits, whether the list that two particles
share is whole, or full and they walk their cells."""
from __future__ import annotations

import numpy as np
import pytest

from test_twin_gpu import run
from test_twin_seams_gpu import KEYS, cluster, with_fluid

pytestmark = pytest.mark.gpu

SLOTS = 96  # a capacity that shared lists are used with (more than a lattice has within kh)


@pytest.mark.parametrize("size,over", [(97, False), (98, True), (250, True), (251, True)])
@pytest.mark.parametrize("precision", ["fp32", "mixed_abs"])
def test_flag_and_fields_of_full_lists(sphlib, cuda, precision, size, over):
    """Two clusters far apart, size - 1 neighbours a particle.  97: one thread holds a particle of
    either, whose shared list has 2 x 97 entries for 2 x 96 slots, though neither overflows.  98: both
    overflow, and the list of two of one cluster holds them.  250: no list holds them."""
    from tmp_sph_gb300 import api
    dx = 0.004
    pos = np.concatenate([cluster(size, dx) + [0.3, 0.2, 0.1], cluster(size, dx) + [0.6, 0.3, 0.4]])
    st, p = with_fluid(pos, dx)
    assert len(st["rho"]) >= 400000
    o = {api.SPH_OPT_NEIGHBOR_CAP: SLOTS, api.SPH_OPT_SKIN_PERMILLE: 0}
    two = run(st, p, o, precision, steps=1)
    one = run(st, p, {**o, api.SPH_OPT_PARTICLES_PER_THREAD: 2}, precision, steps=1)
    assert bool(one["flags"] & api.SPH_FLAG_NEIGHBOR_OVERFLOW) == over
    assert two["flags"] == one["flags"]
    for k in KEYS:
        assert np.isfinite(one[k]).all() and np.array_equal(two[k], one[k]), k


@pytest.mark.parametrize("slots", [16, 80, 96, 112])
def test_capacities_either_side_of_the_rule(sphlib, cuda, slots):
    """A disordered flow with lists most particles overflow (one particle per thread) and lists most
    fit (two): the fields and flags of one particle per thread."""
    from test_twin_gpu import state
    from tmp_sph_gb300 import api
    st, p = state(0.0061, True)
    o = {api.SPH_OPT_NEIGHBOR_CAP: slots}
    two = run(st, p, o)
    one = run(st, p, {**o, api.SPH_OPT_PARTICLES_PER_THREAD: 2})
    assert two["flags"] == one["flags"]
    for k in KEYS:
        assert np.array_equal(two[k], one[k]), k
