"""Calls that the rules of the launch take to a special kernel or launch shape, against the general one:
row-shaped blocks against 32 x 8 blocks, the SRT/TRT sweeps without wall code against the same sweeps given
flags without a boundary, and the MRT sweep for rate-1 higher moments against the general MRT sweep."""
import ctypes

import numpy as np
import pytest
import torch

import lbmpy_b200 as L
from lbmpy_b200 import _native as N
from lbmpy_b200.fields import create_flag_array, create_pdf_array
from lbmpy_b200.kernel import BoundSweep, build_desc
from tests.test_gpu_parity import FP64_TOL, _interior, make_pair, pop_rel_linf, run_pair

pytestmark = pytest.mark.gpu


def _sweep(size, steps, stencil, method, dtype, pattern, rates, flags=False, force=None, e3m12=False, sgs=None):
    cfg = dict(stencil=L.Stencil[stencil], method=L.Method[method.upper()], streaming_pattern=pattern,
               compressible=True)
    cfg.update({"relaxation_rates": rates} if isinstance(rates, list) else {"relaxation_rate": rates})
    if pattern != "pull":
        cfg["timestep"] = L.Timestep.EVEN
    if force:
        cfg["force"] = force
    if sgs:
        cfg["subgrid_scale_model"] = (L.SubgridScaleModel.SMAGORINSKY, sgs)
    kernel = L.create_lb_function(lbm_config=L.LBMConfig(**cfg),
                                  lbm_optimisation=L.LBMOptimisation(storage_dtype=dtype),
                                  config=L.CreateKernelConfig(data_type="float64" if dtype == "float64" else "float32"))
    plan = N.Plan(build_desc(kernel.update_rule, size, (True, True, True), {}))
    q = kernel.method.stencil.Q
    a = create_pdf_array(size, q, dtype=dtype)
    b = a if pattern != "pull" else create_pdf_array(size, q, dtype=dtype)
    vel = np.random.default_rng(7).uniform(-0.05, 0.05, tuple(size) + (3,))
    L.macroscopic_values_setter(kernel.method, 1.0, torch.from_numpy(vel).cuda(), a, pattern,
                                L.Timestep.ODD if pattern != "pull" else L.Timestep.BOTH)
    f = create_flag_array(size) if flags else None
    stream = torch.cuda.current_stream().cuda_stream
    if flags:
        N.check(N.lib().lbm_flags_finalize(plan.handle, ctypes.c_void_p(f.data_ptr()), ctypes.c_void_p(stream)))
    sweep = BoundSweep(plan, a.stride(), f, stream)
    name = sweep.variant(a.data_ptr(), b.data_ptr(), 0)
    in_b = sweep.run(a.data_ptr(), b.data_ptr(), 0, steps)
    out = (b if in_b else a)[1:-1, 1:-1, 1:-1].clone()
    torch.cuda.synchronize()
    return out, name


@pytest.mark.parametrize("size", [(1, 3, 2), (5, 1, 4), (12, 46, 3), (16, 7, 5), (33, 9, 3), (100, 5, 3), (104, 13, 3),
                                  (127, 4, 2), (128, 5, 2), (129, 3, 2)])
@pytest.mark.parametrize("stencil,method,dtype,pattern", [("D3Q19", "trt", "float64", "pull"),
                                                          ("D3Q27", "cumulant", "float32", "aa"),
                                                          ("D3Q19", "trt", "float32", "esotwist")])
def test_row_shaped_blocks(cuda, size, stencil, method, dtype, pattern, monkeypatch):
    monkeypatch.setenv("LBM_B200_PAIR", "0")
    got, _ = _sweep(size, 4, stencil, method, dtype, pattern, 1.8)
    monkeypatch.setenv("LBM_B200_BX", "32")
    want, _ = _sweep(size, 4, stencil, method, dtype, pattern, 1.8)
    assert torch.equal(got, want)


@pytest.mark.parametrize("stencil", ["D3Q19", "D3Q27"])
@pytest.mark.parametrize("method", ["srt", "trt"])
@pytest.mark.parametrize("dtype,pattern", [("float32", "pull"), ("float16", "pull"), ("float16", "aa"),
                                           ("bfloat16", "aa"), ("e3m12", "pull")])
@pytest.mark.parametrize("size", [(4, 3, 2), (128, 5, 3), (132, 6, 3)])
def test_sweeps_without_wall_code(cuda, stencil, method, dtype, pattern, size):
    got, name = _sweep(size, 4, stencil, method, dtype, pattern, 1.8)
    want, same = _sweep(size, 4, stencil, method, dtype, pattern, 1.8, flags=True)
    assert name == same == ("cell" if dtype == "float32" else "quad")
    if dtype == "e3m12":        # codes: the same up to a last place in few of them
        d = (got.int() - want.int()).abs()
        assert d.max() <= 1 and (d != 0).float().mean() < 0.05
        return
    # the same FP32 operations up to contraction, rounded to storage four times
    eps = {"float32": 2e-7, "float16": 2 ** -10, "bfloat16": 2 ** -7}[dtype]
    scale = want.double().norm()
    assert (got.double() - want.double()).norm() <= 4 * eps * scale


@pytest.mark.parametrize("stencil,dtype,pattern", [("D3Q19", "float32", "pull"), ("D3Q19", "float16", "pull"),
                                                   ("D3Q19", "bfloat16", "aa"), ("D3Q27", "float32", "aa")])
@pytest.mark.parametrize("size", [(2, 3, 2), (34, 6, 3), (130, 5, 3)])
@pytest.mark.parametrize("force", [None, (1e-4, -2e-5, 3e-5)], ids=["plain", "force"])
def test_general_mrt_pairs_without_wall_code(cuda, stencil, dtype, pattern, size, force, monkeypatch):
    monkeypatch.setenv("LBM_B200_PAIR", "1")
    rates = [1.8, 1.6, 1.1, 1.2] + ([1.3, 1.1] if stencil == "D3Q27" else [])
    got, name = _sweep(size, 4, stencil, "mrt", dtype, pattern, rates, force=force)
    want, same = _sweep(size, 4, stencil, "mrt", dtype, pattern, rates, flags=True, force=force)
    assert name == same == "pair"
    # the same operations up to contraction, rounded to storage four times
    eps = {"float32": 2e-7, "float16": 2 ** -10, "bfloat16": 2 ** -7}[dtype]
    assert (got.double() - want.double()).norm() <= 4 * eps * want.double().norm()


@pytest.mark.parametrize("method,pattern,dtype", [("mrt", "pull", "float64"), ("mrt", "aa", "float64"),
                                                  ("cumulant", "pull", "float64"), ("cumulant", "aa", "float64"),
                                                  ("cumulant", "push", "float64"), ("cumulant", "esotwist", "float64")])
@pytest.mark.parametrize("size", [(2, 3, 2), (34, 6, 3), (130, 5, 3)])
def test_general_transforms_without_wall_code_match_oracle(cuda, method, pattern, dtype, size):
    rates = [1.8, 1.6, 1.1, 1.2, 1.3, 1.1] if method == "mrt" else [1.8, 1.0] + [1.1] * 8
    step, orc, f, flags, ubb, prev = make_pair("D3Q27", method, size, pattern, dtype, relaxation_rates=rates,
                                               compressible=True)
    res, _ = run_pair(step, orc, f, flags, ubb, prev, 20, pattern, (1, 1, 1))
    assert flags is None and step.sweep_variant() == "cell"
    err = pop_rel_linf(_interior(step.pdfs), res[1:-1, 1:-1, 1:-1], step.method.weights)
    assert err < FP64_TOL


@pytest.mark.parametrize("stencil,higher", [("D3Q19", 2), ("D3Q27", 4)])
@pytest.mark.parametrize("dtype,pattern,pair", [("float64", "pull", "0"), ("float64", "aa", "0"), ("float32", "pull", "0"),
                                                ("float32", "aa", "0"), ("float32", "pull", "1"),
                                                ("float16", "pull", "1"), ("bfloat16", "aa", "1")])
@pytest.mark.parametrize("options", [{}, {"force": (1e-4, -2e-5, 3e-5)}, {"sgs": 0.15}], ids=["plain", "force", "sgs"])
def test_mrt_with_rate_one_higher_moments(cuda, stencil, higher, dtype, pattern, pair, options, monkeypatch):
    if stencil == "D3Q27" and dtype.endswith("16"):
        pytest.skip("the D3Q27 MRT family is built for FP64 and FP32 storage")
    monkeypatch.setenv("LBM_B200_PAIR", pair)
    size, rates = (18, 9, 7), [1.8, 1.6] + [1.0] * higher
    got, _ = _sweep(size, 6, stencil, "mrt", dtype, pattern, rates, **options)
    # one higher rate off by a rounding: not the special case, the same result
    want, _ = _sweep(size, 6, stencil, "mrt", dtype, pattern, rates[:-1] + [float(np.nextafter(1.0, 2.0))], **options)
    eps = {"float64": 1e-13, "float32": 1e-6, "float16": 2 ** -10, "bfloat16": 2 ** -7}[dtype]
    assert (got.double() - want.double()).norm() <= 6 * eps * want.double().norm()
