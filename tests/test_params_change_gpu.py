"""GPU tests of sph_set_params with other physics on a loaded FP64 state: what the state keeps from
one half step to the next (the pair volume c_fr m / rho) follows the new parameters."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def case():
    """A perturbed dam break, and its parameters at h = 1.3 dx and at h = 1.5 dx with another mass."""
    from tmp_sph_gb300 import api, cases
    from gpu_util import perturbed
    st, p = cases.build("small", physics="config", dx=0.02, jitter=0.05)
    st = perturbed(st, vamp=0.5, ramp=0.01)
    c = cases.config(cases.geometry("small", dx=0.02), "config", len(st["rho"]))
    c.h_factor = 1.5
    q = api.params_derive(c)
    q.mass = 1.1 * p.mass
    q.dt = p.dt
    assert q.h > 1.1 * p.h
    return st, p, q


def put(sol, st, s):
    sol.upload(st["pos"], st["vel"], st["rho"], st["p"], st["type"], stream=s)


def test_fp64_params_changed_before_the_first_step(sphlib, cuda):
    """The bits of a solver created with the new parameters."""
    import torch
    from tmp_sph_gb300 import solver as S
    st, p, q = case()
    s = torch.cuda.Stream()
    out = []
    for first in (p, q):
        with S.Solver(first, len(st["rho"]), precision="fp64") as sol:
            put(sol, st, s)
            if first is p:
                torch.cuda.synchronize()
                sol.set_params(q)
            sol.step(2, stream=s)
            out.append(sol.download_f64(stream=s))
    for k in ("pos", "vel", "rho", "p"):
        assert np.array_equal(out[0][k], out[1][k]), k


def test_fp64_params_changed_between_steps(sphlib, cuda, report):
    """A step under the new parameters against a fresh upload of the same state (rounded to FP32:
    positions to 6e-8 m and pressures to 6e-8 of themselves, 3e-6 of a spacing; 1e-3 of the step's
    velocity increments leaves room for the sums that cancel)."""
    import torch
    from tmp_sph_gb300 import solver as S
    st, p, q = case()
    s = torch.cuda.Stream()
    with S.Solver(p, len(st["rho"]), precision="fp64") as sol:
        put(sol, st, s)
        sol.step(2, stream=s)
        mid = sol.download(stream=s)
        before = sol.download_f64(stream=s)
        torch.cuda.synchronize()
        sol.set_params(q)
        sol.step(1, stream=s)
        out = sol.download_f64(stream=s)
    with S.Solver(q, len(st["rho"]), precision="fp64") as sol:
        put(sol, mid, s)
        sol.step(1, stream=s)
        ref = sol.download_f64(stream=s)
    fl = st["type"] == 1
    d = out["vel"][fl] - before["vel"][fl]
    e = np.linalg.norm(d - (ref["vel"][fl] - mid["vel"][fl])) / np.linalg.norm(d)
    report("fp64 step after a change of h and mass, velocity increments", e, 1e-3)
    assert e < 1e-3
