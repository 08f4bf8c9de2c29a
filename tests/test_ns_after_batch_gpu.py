"""GPU test of the drop-in sph_ns on a context whose resident batch rebuilds instance by instance: the
call builds a list of its own for every particle, whatever the instances last decided."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import dev, host

pytestmark = pytest.mark.gpu


def test_ns_after_instance_decisions(sphlib, cuda):
    import torch
    from gpu_util import perturbed
    from tmp_sph_gb300 import api, cases, solver as S
    states, p = cases.batch(2, dx=0.02, seed=11)
    st = perturbed(states[0])
    n = len(st["rho"])
    keys = ("pos", "vel", "rho", "p", "type")
    h, idx = (torch.empty(n, dtype=torch.int32, device=cuda) for _ in range(2))
    S.calc_hash(p, dev(st["pos"], cuda), h, idx, n)
    S.sort_particles(h, idx, n)
    cs, ce = (torch.empty(p.num_cells, dtype=torch.int32, device=cuda) for _ in range(2))
    out = []
    for batch in (True, False):
        with S.Solver(p, sum(len(q["rho"]) for q in states)) as sol:
            if batch:
                s = torch.cuda.Stream()
                sol.set_option(api.SPH_OPT_INSTANCE_DECISIONS, 1)
                sol.upload_instances(states, stream=s)
                sol.step(3, stream=s)
                torch.cuda.synchronize()
            q = {k: torch.empty_like(dev(st[k], cuda)) for k in keys}
            S.reorder(p, *(dev(st[k], cuda) for k in keys), None, *(q[k] for k in keys), None, h,
                      idx, cs, ce, n)
            r = {k: torch.empty(m, device=cuda) for k, m in (("rd", n), ("vd", 3 * n), ("dv", n))}
            sol.ns(q["pos"], q["vel"], q["rho"], q["p"], q["type"], r["rd"], r["vd"], cs, ce, n, h,
                   r["dv"], None, None)
            out.append({**{k: host(v) for k, v in r.items()}, "rho": host(q["rho"]),
                        "p": host(q["p"])})
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
