"""A batch whose walls do not fit the device's memory any more takes them from the flags."""
import pytest
import torch

import lbmpy_b200 as L
from lbmpy_b200.batched import LatticeBoltzmannBatch

pytestmark = pytest.mark.gpu


def _batch(size):
    cfg = L.LBMConfig(stencil=L.Stencil.D3Q19, method=L.Method.TRT, relaxation_rate=1.8, compressible=False)
    b = LatticeBoltzmannBatch([size], lbm_config=cfg, lbm_optimisation=L.LBMOptimisation(storage_dtype="float32"),
                              config=L.CreateKernelConfig(data_type="float32"), use_cuda_graph=False)
    bh = b.boundary_handling(0)
    bh.set_boundary(L.UBB(velocity=(0.05, 0, 0)), L.slice_from_direction("N", 3))
    for d in ("W", "E", "S", "T", "B"):
        bh.set_boundary(L.NoSlip(), L.slice_from_direction(d, 3))
    return b


def test_walls_that_do_not_fit(cuda):
    size = (160, 160, 160)
    want = _batch(size)
    want.run_sweeps(3)
    b = _batch(size)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    for_flags = torch.empty(24 << 20, dtype=torch.uint8, device="cuda")
    rest = torch.empty((torch.cuda.mem_get_info()[0] - (12 << 20)) >> 21 << 21, dtype=torch.uint8, device="cuda")
    del for_flags
    try:
        assert torch.cuda.mem_get_info()[0] < 4 * 160 ** 3
        b.run_sweeps(3)
        torch.cuda.synchronize()
    finally:
        del rest
        torch.cuda.empty_cache()
    assert torch.equal(b.pdfs(0), want.pdfs(0))
