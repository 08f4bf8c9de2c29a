"""GPU tests of the two-particles-per-thread lists and passes (equation/ns_twin.cu): the resident
solver takes them in FP32 and in mixed precision on FP32 positions from 400,000 particles on.  They
sum every particle's pairs in cell-walk order like the one-particle passes, so both forms give the
same bits; SPH_OPT_PARTICLES_PER_THREAD above 1 selects the one-particle form."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def state(dx, disorder, seed=5, block=(0.4, 0.5, 0.3)):
    """A dam break in the 1.0 x 0.5 x 0.6 m tank; disordered: velocities, jitter and spray (a
    tenth of the fluid scattered through the empty part of the tank, rows of one particle)."""
    from tmp_sph_gb300 import cases
    st, p = cases.build("small", physics="config", dx=dx, jitter=0.01, block=block)
    st = {k: v.copy() if isinstance(v, np.ndarray) else v for k, v in st.items()}
    if disorder:
        rng = np.random.default_rng(seed)
        fl = np.nonzero(st["type"] == 1)[0]
        st["pos"][fl] += rng.uniform(-0.2, 0.2, (len(fl), 3)).astype(np.float32) * np.float32(dx)
        st["vel"][fl] = rng.uniform(-1.0, 1.0, (len(fl), 3)).astype(np.float32)
        spray = rng.choice(fl, len(fl) // 10, replace=False)
        st["pos"][spray] = rng.uniform([0.45, 0.02, 0.02], [0.98, 0.48, 0.55],
                                       (len(spray), 3)).astype(np.float32)
        st["p"][spray], st["rho"][spray] = 0.0, 1000.0
    return st, p


def run(st, p, opts, precision="fp32", steps=3, instances=0):
    import torch
    from tmp_sph_gb300 import solver as S
    s = torch.cuda.Stream()
    n = len(st["rho"]) * max(1, instances)
    with S.Solver(p, n, precision=precision) as sol:
        for k, v in opts.items():
            sol.set_option(k, v)
        if instances:
            sol.upload_instances([st] * instances, stream=s)
        else:
            sol.upload(st["pos"], st["vel"], st["rho"], st["p"], st["type"], stream=s)
        sol.step(steps, stream=s)
        out = sol.download(stream=s)
        out["flags"] = sol.error_flags(stream=s)
    return out


@pytest.mark.parametrize("precision,disorder,opts", [
    ("fp32", False, {}),
    ("fp32", True, {}),
    ("mixed_abs", True, {}),
    ("fp32", True, {"SPH_OPT_SKIN_PERMILLE": 0}),
    ("fp32", True, {"SPH_OPT_CELL_DIVISIONS": 2, "SPH_OPT_CONDITIONAL_GRAPH": 0}),
    ("fp32", True, {"SPH_OPT_CELL_DIVISIONS": 1, "SPH_OPT_PASS1_LANES": 1}),
    ("fp32", True, {"SPH_OPT_NEIGHBOR_CAP": 80}),  # some lists overflow and walk the cells
    ("fp32", True, {"SPH_OPT_NEIGHBOR_CAP": 80, "SPH_OPT_CELL_DIVISIONS": 1,  # both of a cell walk
                    "SPH_OPT_PASS1_LANES": 1}),
    ("mixed_abs", True, {"SPH_OPT_NEIGHBOR_CAP": 16, "SPH_OPT_CELL_DIVISIONS": 1}),
    ("fp32", True, {"SPH_OPT_BLOCK_THREADS": 256}),
])
def test_twin_gives_the_bits_of_one_particle_per_thread(sphlib, cuda, precision, disorder, opts):
    """Ordered rows, disorder, rows of single particles, odd counts, every cell size, overflowing
    lists and block sizes."""
    from tmp_sph_gb300 import api
    st, p = state(0.0061, disorder)
    assert len(st["rho"]) >= 400000
    o = {getattr(api, k): v for k, v in opts.items()}
    two = run(st, p, o, precision)
    one = run(st, p, {**o, api.SPH_OPT_PARTICLES_PER_THREAD: 2}, precision)
    assert two["flags"] == one["flags"]
    assert bool(one["flags"] & api.SPH_FLAG_NEIGHBOR_OVERFLOW) == ("SPH_OPT_NEIGHBOR_CAP" in opts)
    for k in ("pos", "vel", "rho", "p"):
        assert np.array_equal(two[k], one[k]), k


def test_twin_threshold_and_odd_counts(sphlib, cuda):
    """A particle count on either side of the threshold, odd and even: the first particles of the
    walls are left out until the count is right."""
    from tmp_sph_gb300 import api
    st, p = state(0.0061, False)
    n = len(st["rho"])
    for keep in (399999, 400000, 400001):
        cut = {k: np.ascontiguousarray(v[n - keep:]) for k, v in st.items()
               if isinstance(v, np.ndarray)}
        two = run(cut, p, {}, steps=2)
        one = run(cut, p, {api.SPH_OPT_PARTICLES_PER_THREAD: 2}, steps=2)
        for k in ("pos", "vel", "rho", "p"):
            assert np.array_equal(two[k], one[k]), (keep, k)


def test_twin_batch_equals_solo(sphlib, cuda):
    """Instances of a batch over the threshold, each below it alone: with lists rebuilt every half
    step each evolves bit for bit as it does alone."""
    from tmp_sph_gb300 import api
    st, p = state(0.0101, True, block=(0.39, 0.5, 0.29))
    n = len(st["rho"])
    assert n < 400000 <= 4 * n
    o = {api.SPH_OPT_SKIN_PERMILLE: 0}
    out = run(st, p, o, instances=4, steps=2)
    ref = run(st, p, o, steps=2)
    for b in range(4):
        for k in ("pos", "vel", "rho", "p"):
            assert np.array_equal(out[k][b * n:(b + 1) * n], ref[k]), (b, k)


def test_drop_in_ns_twin_gives_the_bits_of_one_particle_per_thread(sphlib, cuda):
    """sph_ns over the threshold: the shared lists give the rates, divergence and wall values of the
    one-particle path (which also returns the wall sums)."""
    import torch
    from gpu_util import dev, host
    from tmp_sph_gb300 import solver as S
    st, p = state(0.0061, True)
    n = len(st["rho"])
    h, idx = (torch.empty(n, dtype=torch.int32, device=cuda) for _ in range(2))
    S.calc_hash(p, dev(st["pos"], cuda), h, idx, n)
    S.sort_particles(h, idx, n)
    cs = torch.empty(p.num_cells, dtype=torch.int32, device=cuda)
    ce = torch.empty(p.num_cells, dtype=torch.int32, device=cuda)
    keys = ("pos", "vel", "rho", "p", "type")
    out = []
    with S.Solver(p, n) as sol:
        for sums in (False, True):
            q = {k: torch.empty_like(dev(st[k], cuda)) for k in keys}
            S.reorder(p, *(dev(st[k], cuda) for k in keys), None, *(q[k] for k in keys), None, h,
                      idx, cs, ce, n)
            r = {k: torch.empty(m, device=cuda) for k, m in (("rd", n), ("vd", 3 * n), ("dv", n),
                                                             ("rs", n), ("ws", n))}
            sol.ns(q["pos"], q["vel"], q["rho"], q["p"], q["type"], r["rd"], r["vd"], cs, ce, n, h,
                   r["dv"], r["rs"] if sums else None, r["ws"] if sums else None)
            out.append({k: host(v) for k, v in (("rd", r["rd"]), ("vd", r["vd"]), ("dv", r["dv"]),
                                                ("rho", q["rho"]), ("p", q["p"]))})
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
