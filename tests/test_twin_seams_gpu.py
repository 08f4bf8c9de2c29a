"""GPU tests of the shared lists (equation/ns_twin.cu) where one list's two particles have nothing in
common: the last particle of one batched instance and the first of the next (positions are in each
instance's own frame, so distance alone does not tell them apart), and two clusters far apart."""
from __future__ import annotations

import numpy as np
import pytest

from test_twin_gpu import run

pytestmark = pytest.mark.gpu

KEYS = ("pos", "vel", "rho", "p")


def with_fluid(pos, dx, seed=0, tank=(1.0, 0.5, 0.6)):
    """The empty tank with fluid particles at `pos`, moving at random."""
    from tmp_sph_gb300 import cases
    st, p = cases.build("small", physics="config", dx=dx, tank=tank, block=(0.2, 0.2, 0.1))
    wall = st["type"] != 1
    m = len(pos)
    vel = np.random.default_rng(seed).uniform(-0.5, 0.5, (m, 3))
    out = {"pos": np.concatenate([pos, st["pos"][wall]]).astype(np.float32),
           "vel": np.concatenate([vel, st["vel"][wall]]).astype(np.float32),
           "rho": np.concatenate([np.full(m, 1001.0), st["rho"][wall]]).astype(np.float32),
           "p": np.concatenate([np.full(m, 500.0), st["p"][wall]]).astype(np.float32),
           "type": np.concatenate([np.ones(m), st["type"][wall]]).astype(st["type"].dtype)}
    return out, p


def cluster(size, dx):
    """`size` particles on a lattice 1.91 dx across: all within one support radius (2.6 dx)."""
    m = int(np.ceil(size ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:size]
    return 1.91 * dx * g / (np.sqrt(3) * (m - 1))


def heavy_drop(b, dx):
    """A drop at nearly the same place in every instance whose particles have 100 neighbours each."""
    return np.array([0.4, 0.2, 0.3]) + cluster(101 - b % 2, dx) + [0, 0, dx * (b % 3)]


def drop(b, dx):
    """A drop of 27 particles (28 or 26 in some instances, so that both parities of the seams occur)
    at nearly the same place in every instance."""
    rng = np.random.default_rng(b)
    g = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3)
    g = np.concatenate([g, [[1, 1, 3]]])[:(27, 28, 27, 26, 27)[b % 5]]
    return np.array([0.4, 0.2, 0.3]) + dx * (g + rng.uniform(-0.1, 0.1, g.shape) + [0, 0, b % 3])


def film(b, dx):
    """A film two layers deep and one particle above its corner nearest the origin: the last slot of
    an instance is then within reach of the first slots of the next."""
    rng = np.random.default_rng(b)
    g = np.stack(np.meshgrid(np.arange(49), np.arange(24), np.arange(2), indexing="ij"),
                 -1).reshape(-1, 3)[:-1 - b % 2]
    g = np.concatenate([g, [[0.2, 0.2, 2.3]]])
    return dx * (g + 0.6 + rng.uniform(-0.1, 0.1, g.shape))


def batch_of(kind, dx=0.02):
    made = [with_fluid(kind(b, dx), dx, seed=b) for b in range(22)]
    states = [m[0] for m in made]
    assert sum(len(s["rho"]) for s in states) >= 400000
    return states, made[0][1]


def run_batch(states, p, opts, precision, steps=2):
    import torch
    from tmp_sph_gb300 import solver as S
    s = torch.cuda.Stream()
    with S.Solver(p, sum(len(q["rho"]) for q in states), precision=precision) as sol:
        for k, v in opts.items():
            sol.set_option(k, v)
        off = sol.upload_instances(states, stream=s)
        sol.step(steps, stream=s)
        out = sol.download(stream=s)
        out["flags"] = sol.error_flags(stream=s)
    return out, off


@pytest.mark.parametrize("precision", ["fp32", "mixed_abs"])
@pytest.mark.parametrize("kind", [drop, film])
def test_instances_stay_apart(sphlib, cuda, kind, precision):
    """Instances that overlap in their own frames: with lists rebuilt every half step each evolves
    bit for bit as it does alone."""
    from tmp_sph_gb300 import api
    states, p = batch_of(kind)
    out, off = run_batch(states, p, {api.SPH_OPT_SKIN_PERMILLE: 0}, precision)
    for b, st in enumerate(states):
        ref = run(st, p, {api.SPH_OPT_SKIN_PERMILLE: 0}, precision, steps=2)
        for k in KEYS:
            assert np.array_equal(out[k][off[b]:off[b + 1]], ref[k]), (b, k)


def test_many_small_instances(sphlib, cuda):
    """700 tanks of 0.2 m: more than 1024 runs of one instance and kind in the work order."""
    from tmp_sph_gb300 import api
    made = [with_fluid(np.array([-0.33, -0.13, -0.2]) + drop(b, 0.04), 0.04, seed=b,
                       tank=(0.2, 0.2, 0.2)) for b in range(700)]
    states, p = [m[0] for m in made], made[0][1]
    assert sum(len(s["rho"]) for s in states) >= 400000
    out, off = run_batch(states, p, {api.SPH_OPT_SKIN_PERMILLE: 0}, "fp32")
    for b in [0, 1, 2, 3, 321, 322, 323, 324, 400, 510, 511, 512, 513, 697, 698, 699]:
        ref = run(states[b], p, {api.SPH_OPT_SKIN_PERMILLE: 0}, "fp32", steps=2)
        for k in KEYS:
            assert np.array_equal(out[k][off[b]:off[b + 1]], ref[k]), (b, k)


def test_particles_outside_the_search(sphlib, cuda):
    """Escaped particles outside the search (park_inactive) come after all instances: each instance
    as alone, whatever their number."""
    from tmp_sph_gb300 import api
    states, p = batch_of(film)
    for b, st in enumerate(states):  # an odd or even number of them above the tank's rim
        up = np.arange(5 + b % 3)
        st["pos"][up] = np.array([0.3, 0.2, 0.66]) + 0.005 * up[:, None].astype(np.float32)
    p.park_inactive = 1
    out, off = run_batch(states, p, {api.SPH_OPT_SKIN_PERMILLE: 0}, "fp32")
    parked = 0
    for b, st in enumerate(states):
        ref = run(st, p, {api.SPH_OPT_SKIN_PERMILLE: 0}, "fp32", steps=2)
        parked += int(np.all(ref["pos"][:8] == np.array(p.escape_park, np.float32), axis=1).sum())
        for k in KEYS:
            assert np.array_equal(out[k][off[b]:off[b + 1]], ref[k]), (b, k)
    assert parked == sum(5 + b % 3 for b in range(len(states)))


@pytest.mark.parametrize("kind,opts", [(drop, {}), (heavy_drop, {"SPH_OPT_NEIGHBOR_CAP": 96}),
                                       (drop, {"SPH_OPT_CELL_DIVISIONS": 1,
                                               "SPH_OPT_PASS1_LANES": 1})])
def test_seams_give_the_bits_of_one_particle_per_thread(sphlib, cuda, kind, opts):
    """The same batches at the default skin, with lists that overflow at the seams, and on cells of
    the cutoff: fields and flags of one particle per thread."""
    from tmp_sph_gb300 import api
    o = {getattr(api, k): v for k, v in opts.items()}
    states, p = batch_of(kind)
    two, _ = run_batch(states, p, o, "fp32", steps=4)
    one, _ = run_batch(states, p, {**o, api.SPH_OPT_PARTICLES_PER_THREAD: 2}, "fp32", steps=4)
    assert two["flags"] == one["flags"]
    assert bool(one["flags"] & api.SPH_FLAG_NEIGHBOR_OVERFLOW) == ("SPH_OPT_NEIGHBOR_CAP" in opts)
    for k in KEYS:
        assert np.array_equal(two[k], one[k]), k
