"""lbm_walls_slab: the part of a domain's walls that a slab of its planes sweeps with."""
import ctypes

import pytest

from lbmpy_b200 import _native as N


def _whole(periodic=(1, 0, 0)):
    w = N.LbmWalls()
    w.flags, w.rows, w.words, w.stencil = 0x100000, 0x200000, 0x300000, 19
    w.dims[:] = (5, 33, 8)
    w.periodic[:] = periodic
    return w


def _slab(whole, z0, nz):
    out = N.LbmWalls()
    return N.lib().lbm_walls_slab(ctypes.byref(whole), z0, nz, ctypes.byref(out)), out


@pytest.mark.parametrize("z0,nz", [(0, 1), (7, 1), (1, 6), (0, 8)])
def test_offsets(z0, nz):
    rc, s = _slab(_whole(), z0, nz)
    assert rc == N.LBM_OK
    assert s.flags == 0x100000 + 7 * 35 * z0          # ghost-inclusive planes of bytes
    assert s.rows == 0x200000 + 4 * 2 * z0            # 33 rows take two words a plane
    assert s.words == 0x300000 + 4 * 5 * 33 * z0
    assert (s.stencil, list(s.dims), list(s.periodic)) == (19, [5, 33, nz], [1, 0, 0])


@pytest.mark.parametrize("z0,nz", [(-1, 2), (8, 1), (1, 8), (0, 0), (2, 2 ** 31 - 1)])
def test_planes_outside_are_refused(z0, nz):
    assert _slab(_whole(), z0, nz)[0] == N.LBM_E_INVALID


def test_a_domain_periodic_in_z_has_no_slabs():
    assert _slab(_whole((0, 0, 1)), 1, 2)[0] == N.LBM_E_INVALID
