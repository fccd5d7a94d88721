"""The wall words that a sweep takes from the flags (compiled for the host) against a plain search: which links
bounce, and the kind bits, which must be set for the cells that have such a neighbour and for no others (a cell
marked for moving walls or per-link data is walked link by link, one dependent load after another)."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest

from lbmpy_b200.enums import Stencil
from lbmpy_b200.stencils import LBStencil

HERE = os.path.dirname(os.path.abspath(__file__))
SELF, FIXED_DENSITY, PER_LINK, UBB = 1, 1 << 29, 1 << 30, 1 << 31


@pytest.fixture(scope="module")
def host():
    out = os.path.join(tempfile.mkdtemp(), "walls_host.so")
    subprocess.run(["/usr/bin/g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-o", out,
                    os.path.join(HERE, "host", "walls_host.cpp")], check=True)
    return ctypes.CDLL(out).host_wall_words


def _finalize(types, dirs, periodic):
    """(flags with the near-wall bit, expected words) by search; arrays [x, y, z] with ghost layers."""
    n = [s - 2 for s in types.shape]
    flags, words = types.copy(), np.zeros(n, np.uint32)
    for c in np.ndindex(*n):
        if types[tuple(v + 1 for v in c)]:
            words[c] = SELF
            continue
        seen = set()
        for i, d in enumerate(dirs):
            if i == 0:
                continue
            s = [v - e for v, e in zip(c, d)]
            s = tuple((v % m if p else v) + 1 for v, m, p in zip(s, n, periodic))
            t = int(types[s])
            seen.add(t)
            if 1 <= t <= 5:
                words[c] |= 1 << i
        words[c] |= (FIXED_DENSITY if seen & {6, 7} else 0) | (PER_LINK if max(seen) >= 8 else 0) | \
                    (UBB if seen & {2, 3, 4, 5} else 0)
        if seen != {0}:
            flags[tuple(v + 1 for v in c)] |= 0x80
    return flags, words


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("size", [(1, 1, 1), (5, 4, 3), (7, 1, 6)])
@pytest.mark.parametrize("periodic", [(0, 0, 0), (1, 0, 1), (1, 1, 1)])
@pytest.mark.parametrize("kinds", [(1,), (1, 3), (2, 5), (1, 7), (8, 11), (1, 2, 3, 6, 7, 8, 9, 10, 11)])
def test_words_of_flags(host, q, size, periodic, kinds):
    rng = np.random.default_rng(q + sum(size))
    dirs = [tuple(int(v) for v in d) for d in LBStencil(Stencil.D3Q19 if q == 19 else Stencil.D3Q27)]
    shape = [s + 2 for s in size]
    for density in (0.0, 0.05, 0.4):
        types = np.where(rng.random(shape) < density, rng.choice(kinds, shape), 0).astype(np.uint8)
        flags, want = _finalize(types, dirs, periodic)
        got = np.zeros(size[::-1], np.uint32)
        field = np.ascontiguousarray(flags.transpose(2, 1, 0))
        host(q, *size, sum(b << k for k, b in enumerate(periodic)), field.ctypes.data_as(ctypes.c_void_p),
             got.ctypes.data_as(ctypes.c_void_p))
        assert (got.transpose(2, 1, 0) == want).all()
