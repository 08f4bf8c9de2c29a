"""CPU tests of what the autotuner compares its candidates with: the default as the solver runs it
(threads 0, the block size it picks itself), measured by a stand-in for the runs."""
from __future__ import annotations

import numpy as np
import pytest


class FakeSolver:
    def __init__(self, *a, **kw):
        self.options = []

    def __enter__(self):
        return self

    def __exit__(self, *a):
        return False

    def set_option(self, opt, value):
        self.options.append((opt, value))

    def upload(self, *a, **kw):
        pass


@pytest.fixture
def tuner(monkeypatch):
    """tune(ms): autotune.tune with every run timed by ms(choice)."""
    import torch
    from tmp_sph_gb300 import autotune as A

    class P:
        dt, kh, gravity = 1e-4, 0.01, -9.81

    st = {"type": np.array([1]), "pos": np.array([[0, 0, 0.3]]), "vel": None,
          "rho": np.ones(1), "p": None}
    monkeypatch.setattr(torch.cuda, "Stream", lambda *a, **kw: None)
    monkeypatch.setattr(A.S, "Solver", FakeSolver)

    def measure(sol, stream, threads, ppt, skin, lanes=1, divisions=1):
        return {"threads": threads, "ppt": ppt, "lanes": lanes, "skin_permille": skin,
                "divisions": divisions, "rebuild_ms": 1.0, "flags": 0,
                "pass_ms_per_half_step": 1.0 + 0.001 * (threads + ppt + lanes + divisions)}

    def tune(ms, precision):
        ran = []

        def timed_run(p, states, choice, prec, steps, stream):
            ran.append(dict(choice))
            return ms(choice)

        monkeypatch.setattr(A, "measure", measure)
        monkeypatch.setattr(A, "timed_run", timed_run)
        return A.tune(P, st, precision=precision), ran
    return tune


@pytest.mark.parametrize("precision", ["fp32", "mixed_abs", "mixed", "fp64"])
def test_default_runs_with_the_solvers_own_block_size(tuner, precision):
    best, ran = tuner(lambda c: 1.0 if c["threads"] == 0 else 2.0, precision)
    assert sum(c["default"] for c in best["confirm"]) == 1
    assert [c["threads"] for c in best["confirm"] if c["default"]] == [0]
    # the default is the faster: it is the choice, and applying it sets the option's default
    from tmp_sph_gb300 import api, autotune
    assert best["threads"] == 0 and best["ms_per_step"] == 1.0
    assert {c["threads"] for c in ran} > {0}
    sol = FakeSolver()
    autotune.apply(sol, best)
    assert (api.SPH_OPT_BLOCK_THREADS, 0) in sol.options


def test_candidates_hold_every_block_size_the_solver_picks(tuner):
    best, _ = tuner(lambda c: 2.0 if c["threads"] == 0 else 1.0, "fp64")
    assert {m["threads"] for m in best["table"]} >= {32, 64, 128, 256}
    assert best["threads"] == 32
