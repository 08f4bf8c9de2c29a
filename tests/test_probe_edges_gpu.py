"""GPU tests of the probes' FP32 pre-test: particles at, just inside and just outside a probe's
radius, at coordinates where FP32 rounding matters, give the values an FP64 scan of the downloaded
state gives, in every precision."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "mixed", "mixed_abs", "fp64"])
def test_probes_at_the_edges_of_their_radius(sphlib, cuda, precision):
    import torch
    from tmp_sph_gb300 import api, cases, solver as S
    st, p = cases.build("small", physics="config", dx=0.02, jitter=0.01)
    st["vel"][st["type"] == 1] = np.array([0.3, -0.2, 0.1], np.float32)
    fl = np.nonzero(st["type"] == 1)[0]
    # a ring of particles one float either side of the height gauge's radius and of kh
    x0, y0, r = np.float32(0.2), np.float32(0.25), np.float32(0.03)
    for k in range(8):
        edge = np.float32(x0 + r)
        for _ in range(abs(k - 4)):
            edge = np.nextafter(edge, np.float32(9 if k > 4 else -9), dtype=np.float32)
        st["pos"][fl[k]] = (edge, y0, np.float32(0.5 + 0.001 * k))
        st["pos"][fl[8 + k]] = (np.float32(0.7), np.float32(0.3),
                                np.float32(0.2 + float(p.kh)) + np.float32((k - 4) * 3e-8))
        st["p"][fl[8 + k]] = 100.0 + k
    probes = [(api.SPH_PROBE_HEIGHT, x0, y0, 0.0, r, 0.0),
              (api.SPH_PROBE_HEIGHT, x0, y0, 0.0, -1.0, 0.0),
              (api.SPH_PROBE_PRESSURE, 0.7, 0.3, 0.2, 0.0, 0.0),
              (api.SPH_PROBE_FRONT, 0, 0, 0, 0, 0)]
    s = torch.cuda.Stream()
    with S.Solver(p, len(st["rho"]), precision=precision) as sol:
        sol.upload(st["pos"], st["vel"], st["rho"], st["p"], st["type"], stream=s)
        vals, stats = sol.probe([api.SphProbe(*q) for q in probes], stream=s)
    x = st["pos"][st["type"] == 1].astype(np.float64)
    v = st["vel"][st["type"] == 1].astype(np.float64)
    pr = st["p"][st["type"] == 1].astype(np.float64)
    near = (np.abs(x[:, 0] - float(x0)) < float(r)) & (np.abs(x[:, 1] - float(y0)) < float(r))
    assert vals[0] == x[near, 2].max() and vals[1] == 0.0
    q = np.array([np.float32(0.7), np.float32(0.3), np.float32(0.2)], np.float64)
    h = float(p.h)
    sq = np.sqrt(((x - q) ** 2).sum(1)) / h
    w = np.where(((x - q) ** 2).sum(1) < float(p.kh) ** 2, (1 - 0.5 * sq) ** 4 * (2 * sq + 1), 0.0)
    assert w.sum() > 0.0
    # 1 - s/2 within 1e-7 of zero: its fourth power keeps few digits, so a loose comparison
    np.testing.assert_allclose(vals[2], (w * pr).sum() / w.sum(), rtol=1e-3)
    assert vals[3] == x[:, 0].max()
    assert stats["fluid"] == len(x) and stats["parked"] == 0
    np.testing.assert_allclose(stats["max_speed"], np.sqrt((v ** 2).sum(1)).max(), rtol=1e-12)
    np.testing.assert_allclose(stats["kinetic"], 0.5 * float(p.mass) * (v ** 2).sum(), rtol=1e-10)
