"""The MRT collision specialised for rate-1 higher moments (lbm_collide_mrt1.cuh, compiled for the host)
against the general one (lbm_collide.cuh), cell by cell, over every form that takes it."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest

from tests.test_collision_host import FM, HERE, Physics


@pytest.fixture(scope="module")
def host():
    out = os.path.join(tempfile.mkdtemp(), "mrt1_host.so")
    subprocess.run(["/usr/bin/g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-o", out,
                    os.path.join(HERE, "host", "mrt1_host.cpp")], check=True)
    fn = ctypes.CDLL(out).host_mrt
    fn.restype = ctypes.c_double
    fn.argtypes = [ctypes.c_int] * 3 + [ctypes.POINTER(ctypes.c_double), ctypes.POINTER(Physics)]
    return fn


def _collide(host, q, special, fp32, f, p):
    g = np.array(f, np.float64)
    om = host(q, special, fp32, g.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), ctypes.byref(p))
    return g, om


def _physics(q, shear, bulk, fm, compressible, sgs):
    p = Physics()
    for k in range(q):
        p.rates[k] = 0.0 if k < 4 else shear if k < 9 else bulk if k == 9 else 1.0
    p.force_model = FM[fm]
    if fm:
        p.force[0], p.force[1], p.force[2] = 1e-3, -4e-4, 7e-4
    p.compressible, p.continuous_eq = int(compressible), 1
    if sgs:
        p.sgs, p.sgs_c18, p.tau0 = 1, 18 * 0.17 ** 2, 1 / shear
        p.sgs_mask = 0x1f0 | (0x200 if bulk == shear else 0)
    return p


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("fm", [None, "guo", "luo", "simple"])
@pytest.mark.parametrize("compressible", [True, False])
@pytest.mark.parametrize("shear,bulk,sgs", [(1.8, 1.6, False), (0.6, 1.0, False), (1.95, 1.95, False),
                                            (1.9, 1.0, True), (1.9, 1.9, True), (0.0, 2.0, False)])
def test_equals_the_general_collision(host, q, fm, compressible, shear, bulk, sgs):
    # FP64: both are exact up to rounding of populations of order 1e-1 through about a hundred terms
    # (1e-16 * 1e-1 * 100).  FP32: the special form may be no further from the FP64 result than the
    # general one, up to a factor for single cells.
    if shear == 0.0 and sgs:
        pytest.skip("a subgrid-scale model needs a positive shear rate")
    p = _physics(q, shear, bulk, fm, compressible, sgs)
    rng = np.random.default_rng(q + int(10 * shear))
    e32 = [0.0, 0.0]
    for amp in (1e-1, 1e-3, 1e-5):
        for _ in range(10):
            f = amp * rng.standard_normal(q) / q
            ref, om = _collide(host, q, 0, 0, f, p)
            got, om1 = _collide(host, q, 1, 0, f, p)
            assert np.abs(got - ref).max() < 1e-15 + 1e-13 * np.abs(ref).max()
            assert om1 == pytest.approx(om, rel=1e-12)
            for special in (0, 1):
                e32[special] += np.linalg.norm(_collide(host, q, special, 1, f, p)[0] - ref) / np.linalg.norm(ref)
    assert e32[1] <= 1.5 * e32[0], e32


@pytest.mark.parametrize("q", [19, 27])
def test_fp32_mass_and_momentum_do_not_drift(host, q):
    """Rebuilding the populations from moments must not scale the conserved ones: repeated collisions of
    one cell keep mass and momentum to rounding noise, where weights rounded by 3e-8 would add up."""
    p = _physics(q, 1.8, 1.6, None, True, False)
    from lbmpy_b200.stencils import LBStencil
    from lbmpy_b200.enums import Stencil
    c = np.array([tuple(d) for d in LBStencil(Stencil.D3Q19 if q == 19 else Stencil.D3Q27)], float)
    f = (1e-2 * np.random.default_rng(3).standard_normal(q) / q).astype(np.float32).astype(np.float64)
    m0, j0 = f.sum(), c.T @ f
    for _ in range(2000):
        f, _ = _collide(host, q, 1, 1, f, p)
    # 2000 steps of independent roundings of 1e-2 / 10 at 6e-8: 45 * 1e-3 * 6e-8 * a few; a drift of
    # 3e-8 per step would be 6e-5 of each
    scale = np.abs(f).sum()
    assert abs(f.sum() - m0) < 1e-5 * scale
    assert np.abs(c.T @ f - j0).max() < 1e-5 * scale
