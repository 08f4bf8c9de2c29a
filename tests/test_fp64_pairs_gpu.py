"""GPU tests of the FP64 pair arithmetic (refined hardware approximations, the neighbour's volume
divided out once per particle): against the oracle in FP64, and where r^2 is 0 or tiny."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("physics", ["config", "reference"])
def test_fp64_step_matches_oracle(sphlib, oracle, cuda, report, physics):
    """Two steps against the oracle's FP64 restatement.  The oracle forms four constants in float
    (relative 6e-8 of the viscous, damping and diffusion terms, themselves below a tenth of the
    rates), so 1e-8 of the fields bounds it; pair arithmetic a bit short of FP64 would pass 1e-8
    only down to 1e-9 a pair."""
    import torch
    from tmp_sph_gb300 import cases, solver as S
    from gpu_util import perturbed
    st, p = cases.build("small", physics=physics, dx=0.02, jitter=0.05)
    st = perturbed(st, vamp=0.5, ramp=0.01)
    s = torch.cuda.Stream()
    with S.Solver(p, len(st["rho"]), precision="fp64") as sol:
        sol.upload(st["pos"], st["vel"], st["rho"], st["p"], st["type"], stream=s)
        sol.step(2, stream=s)
        out = sol.download_f64(stream=s)
    ref = oracle.run(oracle.params_like(p), st, 2, dtype=np.float64)
    fl = st["type"] == 1
    for k in ("vel", "rho"):
        base = 1000.0 if k == "rho" else 0.0
        e = (np.linalg.norm(out[k][fl] - ref[k][fl]) / np.linalg.norm(ref[k][fl] - base))
        report(f"fp64 2 steps vs oracle {physics} {k}", e, 1e-8)
        assert e < 1e-8


def test_fp64_coincident_and_close_particles(sphlib, cuda):
    """Particles at the same place (r^2 = 0) add nothing to each other and stay together; a pair
    1e-7 m apart stays finite."""
    import torch
    from tmp_sph_gb300 import cases, solver as S
    st, p = cases.build("small", physics="config", dx=0.02, jitter=0.01)
    fl = np.nonzero(st["type"] == 1)[0]
    a, b, c, d = fl[[1000, 1001, 3000, 3001]]
    for k in ("pos", "vel", "rho", "p"):
        st[k][b], st[k][d] = st[k][a], st[k][c]
    st["pos"][d, 0] += np.float32(1e-7)
    s = torch.cuda.Stream()
    with S.Solver(p, len(st["rho"]), precision="fp64") as sol:
        sol.upload(st["pos"], st["vel"], st["rho"], st["p"], st["type"], stream=s)
        sol.step(3, stream=s)
        out = sol.download_f64(stream=s)
    for k in ("pos", "vel", "rho", "p"):
        assert np.isfinite(out[k]).all(), k
    # the two sum the same pairs, each with the other as a zero term: equal to FP64 rounding
    np.testing.assert_allclose(out["vel"][a], out["vel"][b], rtol=1e-9, atol=1e-12)
