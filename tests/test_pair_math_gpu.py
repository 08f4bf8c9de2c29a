"""GPU test of the FP64 pair root and reciprocal themselves (equation/ns_pair.cuh): their errors over
the arguments a pair can have, against the exact values and against CUDA's square root and division.

Bounds, in units of the last place (2^-53 of the value at least): half a unit for the last rounding,
and what the one refinement step leaves of the relative error d of the hardware's approximation, d^4
for the reciprocal and 35/128 (2 d)^4 for the root (the first term its series leaves out); the other
roundings are below 2^-70 of the value.  The approximations read 20 bits of the argument and write 20
bits of the result, each off by at most 2^-20: d is at most 2^-19, and 3/4 of that for the root, which
halves the argument's part."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
RCP_START = 2.0 ** -19
SQRT_START = 0.75 * RCP_START
ROUNDINGS = 2.0 ** -17


def rcp_bound(d):
    return 0.5 + d ** 4 * 2.0 ** 53 + ROUNDINGS


def sqrt_bound(d):
    return 0.5 + 35 / 128 * (2 * d) ** 4 * 2.0 ** 53 + ROUNDINGS


@pytest.fixture(scope="module")
def pair_math(tmp_path_factory, cuda):
    from tmp_sph_gb300 import build as B
    lib = str(tmp_path_factory.mktemp("pair_math") / "pair_math.so")
    cmd = [B.nvcc(), *B.ARCH, *B.CFLAGS, "-I" + os.path.join(B.CSRC, "equation"), "-shared",
           "-cudart", "shared", "-o", lib, os.path.join(HERE, "pair_math.cu"),
           "-L" + B.cuda_libdir(), "-Xlinker", "-rpath," + B.cuda_libdir()]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    fn = ctypes.CDLL(lib).pair_math
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int]

    def call(x, values):
        import torch
        d = torch.from_numpy(np.ascontiguousarray(x)).to(cuda)
        out = torch.empty((len(x), 4), dtype=torch.float64, device=cuda)
        torch.cuda.synchronize()
        assert fn(d.data_ptr(), len(x), out.data_ptr(), int(values)) == 0
        return out.cpu().numpy()
    return call


def arguments():
    """r^2 and r^2 + eta^2 from 1e-14 m^2 to 1e3 m^2, densities and the padding record's 3e36: sweeps
    of the mantissa over two binades (a root's error depends on the parity of the exponent), random
    arguments, and the neighbours of powers of two."""
    rng = np.random.default_rng(1)
    sweep = 1.0 + np.arange(1 << 21) * 2.0 ** -21
    fine = sweep + rng.integers(0, 1 << 31, len(sweep)) * 2.0 ** -52
    spread = np.exp(rng.uniform(np.log(1e-14), np.log(1e3), 1 << 21))
    powers = 2.0 ** np.arange(-46, 122)
    edges = np.concatenate([powers * (1 + k * 2.0 ** -52) for k in range(-4, 5)])
    return np.concatenate([sweep, fine, 2 * fine, fine * 2.0 ** -40, spread, edges,
                           [3e36, 1e-14, 1000.0]])


def test_errors_of_pair_root_and_reciprocal(pair_math, report):
    x = arguments()
    e = np.abs(pair_math(x, False)).max(0)
    report("FP64 pair root, ulp", e[0], sqrt_bound(e[2]))
    report("FP64 pair reciprocal, ulp", e[1], rcp_bound(e[3]))
    report("FP64 root's start, relative", e[2], SQRT_START)
    report("FP64 reciprocal's start, relative", e[3], RCP_START)
    print(f"\nroot {e[0]:.7f} ulp, reciprocal {e[1]:.7f} ulp, starts 2^{np.log2(e[2]):.3f} "
          f"2^{np.log2(e[3]):.3f}")
    assert e[2] <= SQRT_START and e[3] <= RCP_START
    assert e[0] <= sqrt_bound(e[2])
    assert e[1] <= rcp_bound(e[3])


def test_pair_root_and_reciprocal_against_cuda(pair_math, report):
    """At most the neighbouring double of CUDA's correctly rounded results, and exact at 0 (root) and
    at even powers of two."""
    x = arguments()
    v = pair_math(x, True)
    for got, want, name in ((v[:, 0], v[:, 2], "root"), (v[:, 1], v[:, 3], "reciprocal")):
        d = np.abs(got.view(np.int64) - want.view(np.int64))
        report(f"FP64 pair {name}, differs from CUDA's, share", float((d > 0).mean()))
        assert d.max() <= 1, name
    zero = pair_math(np.array([0.0, 0.0]), True)
    assert (zero[:, 0] == 0.0).all()
    four = 4.0 ** np.arange(-20, 21)
    p = pair_math(four, True)
    assert np.array_equal(p[:, 0], np.sqrt(four)) and np.array_equal(p[:, 1], 1.0 / four)
