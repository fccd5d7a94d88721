"""Wall words (lbm_walls_build) against the flags themselves, with the finalizing plan's row summary and
without: all must give the same populations, bit for bit.  The box mixes NoSlip, two UBB numbers meeting
in one cell, FixedDensity and per-link types
(bounced as NoSlip without link tables), on domain faces and around an obstacle, on sizes with
remainders in every kernel's tiles."""
import ctypes

import numpy as np
import pytest
import torch

import lbmpy_b200 as L
from lbmpy_b200 import _native as N
from lbmpy_b200.fields import create_pdf_array
from lbmpy_b200.kernel import BoundSweep, build_desc

pytestmark = pytest.mark.gpu


def _flags(size):
    f = np.zeros([s + 2 for s in size], np.uint8)
    f[0], f[-1] = 1, 8
    f[:, 0], f[:, -1] = 9, 2                # a UBB lid
    f[:, :, -1] = 3                         # a second UBB meeting it along an edge
    f[3:6, 2:4, 2:5] = 1                    # obstacle
    f[6:8, 3, 3] = 7                        # FixedDensity cells: left to the pre-pass
    f[2, 5, 1:3] = 11
    return f


@pytest.mark.parametrize("pattern", ["pull", "aa", "esotwist"])
@pytest.mark.parametrize("stencil,method,dtype,size", [
    ("D3Q19", "trt", "float64", (9, 7, 6)), ("D3Q19", "mrt", "float32", (33, 7, 6)),
    ("D3Q27", "cumulant", "float32", (34, 6, 7)), ("D3Q19", "trt", "float16", (36, 9, 6)),
    ("D3Q27", "cumulant", "bfloat16", (66, 6, 7)), ("D3Q19", "srt", "float32", (129, 6, 5))])
@pytest.mark.parametrize("periodic", [(False, False, False), (True, False, False)])
def test_words_equal_flags(cuda, stencil, method, dtype, size, pattern, periodic):
    cfg = dict(stencil=L.Stencil[stencil], method=L.Method[method.upper()], streaming_pattern=pattern,
               compressible=method != "mrt")
    cfg.update({"relaxation_rates": [1.8, 1.6, 1.1, 1.2]} if method == "mrt" else {"relaxation_rate": 1.7})
    if pattern != "pull":
        cfg["timestep"] = L.Timestep.EVEN
    kernel = L.create_lb_function(lbm_config=L.LBMConfig(**cfg),
                                  lbm_optimisation=L.LBMOptimisation(storage_dtype=dtype),
                                  config=L.CreateKernelConfig(data_type="float64" if dtype == "float64" else "float32"))
    desc = build_desc(kernel.update_rule, size, periodic, {}, [(0.03, 0, 0.01), (0, 0.02, 0)])
    flags = torch.from_numpy(_flags(size).transpose(2, 1, 0).copy()).cuda().permute(2, 1, 0)
    own, other = N.Plan(desc), N.Plan(desc)
    stream = torch.cuda.current_stream().cuda_stream
    N.check(N.lib().lbm_flags_finalize(own.handle, ctypes.c_void_p(flags.data_ptr()), ctypes.c_void_p(stream)))
    q = kernel.method.stencil.Q
    words = ctypes.c_int64(0)
    N.check(N.lib().lbm_walls_size(own.handle, ctypes.byref(words)))
    buffer, walls = torch.empty(words.value, dtype=torch.int32, device="cuda"), N.LbmWalls()
    N.check(N.lib().lbm_walls_build(own.handle, ctypes.c_void_p(flags.data_ptr()), ctypes.c_void_p(buffer.data_ptr()),
                                    ctypes.byref(walls), ctypes.c_void_p(stream)))
    gen = torch.Generator(device="cuda").manual_seed(5)
    results = []
    init = None
    for plan, w in ((own, N.Walls(walls, (flags, buffer), stream)), (own, None), (other, None)):
        a = create_pdf_array(size, q, dtype=dtype)
        b = a if pattern != "pull" else create_pdf_array(size, q, dtype=dtype)
        if init is None:
            init = (torch.rand(a.shape, generator=gen, device="cuda") - 0.5) * 1e-2
        a.copy_(init)
        sweep = BoundSweep(plan, a.stride(), flags, stream, w)
        in_b = sweep.run(a.data_ptr(), b.data_ptr(), 0, 5)
        results.append((b if in_b else a).clone())
    torch.cuda.synchronize()
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2])
    assert not torch.isnan(results[0].float()).any()
    assert (results[0].float() - init.to(results[0].dtype).float()).abs().max() > 1e-4
