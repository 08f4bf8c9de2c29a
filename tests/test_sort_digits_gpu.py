"""GPU tests of the radix sort's passes that move nothing (every key has the same digit there): any
digit constant, tile remainders, one key that differs."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import dev, host

pytestmark = pytest.mark.gpu


def keys_of(kind, n, rng):
    k = rng.integers(0, 2 ** 31, n, dtype=np.int64)
    if kind == "top":            # cell keys below 2^24
        k &= 0x00ffffff
    elif kind == "middle":
        k = (k & ~0x0000ff00) | 0x00005a00
    elif kind == "low":
        k = (k & ~0xff) | 0x17
    elif kind == "two":
        k = (k & 0x0000ff00) | 0x12000034
    elif kind == "all":
        k[:] = 0x01020304
    elif kind == "one_differs":
        k = k & 0x00ffffff
        k[n // 2] |= 0x40000000
    elif kind == "negative":
        k = -1 - (k & 0x00ffffff)
    return k.astype(np.int32)


@pytest.mark.parametrize("kind", ["top", "middle", "low", "two", "all", "one_differs", "negative"])
@pytest.mark.parametrize("n", [2, 4095, 4096, 4097, 100003])
def test_constant_digits(sphlib, cuda, kind, n):
    from tmp_sph_gb300 import solver as S
    rng = np.random.default_rng(n)
    k = keys_of(kind, n, rng)
    v = rng.permutation(n).astype(np.int32)
    order = np.argsort(k, kind="stable")
    widths = [32] if kind == "negative" else [32, 31]
    for bits in widths:
        h, x = dev(k, cuda), dev(v, cuda)
        S.sort_particles(h, x, n, key_bits=bits)
        assert np.array_equal(host(h), k[order]), bits
        assert np.array_equal(host(x), v[order]), bits
