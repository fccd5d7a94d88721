"""Walls (lbm_walls_build) belong to a flag field: domains that share a plan keep their own, also in captured
graphs; a slab sweeps with its part of them; they are refused for another periodicity."""
import ctypes

import numpy as np
import pytest
import torch

import lbmpy_b200 as L
from lbmpy_b200 import _native as N
from lbmpy_b200.distributed import DistributedLatticeBoltzmannStep
from lbmpy_b200.kernel import build_desc

pytestmark = pytest.mark.gpu

SIZE = (34, 40, 9)


def _step(kernel=None, sides="NSTB", obstacle=None, periodicity=(True, False, False), dtype="float32", ubb=False):
    kw = dict(stencil=L.Stencil.D3Q19, method=L.Method.TRT, relaxation_rate=1.8, compressible=True)
    step = L.LatticeBoltzmannStep(domain_size=SIZE, periodicity=periodicity, lbm_kernel=kernel,
                                  config=L.CreateKernelConfig(data_type=dtype), **kw)
    bh = step.boundary_handling
    for d in sides:
        bh.set_boundary(L.NoSlip(), L.slice_from_direction(d, 3))
    if ubb:
        bh.set_boundary(L.UBB((0.03, 0, 0)), L.slice_from_direction("N", 3))
    if obstacle:
        bh.set_boundary(L.NoSlip(), obstacle)
    step.velocity_array[...] = np.random.default_rng(3).uniform(-0.05, 0.05, SIZE + (3,))
    step.set_pdf_fields_from_macroscopic_values()
    return step


BOX = tuple(slice(a, b) for a, b in ((6, 12), (5, 9), (2, 7)))


def test_domains_that_share_a_kernel_keep_their_walls(cuda):
    a = _step(obstacle=BOX)
    b = _step(kernel=a._kernels[0], sides="TB")
    init, tmp = a.pdfs.clone(), a.pdfs_tmp.clone()
    a.run_sweeps(4)
    want = a.pdfs.clone()
    a.pdfs.copy_(init)
    a.pdfs_tmp.copy_(tmp)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        a.run_sweeps(4)
    b.run_sweeps(4)                       # finalizes other flags with the plan that both steps use
    other = b.pdfs.clone()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(a.pdfs, want)
    a.pdfs.copy_(init)
    a.run_sweeps(4)
    assert torch.equal(a.pdfs, want)
    alone = _step(sides="TB")
    alone.run_sweeps(4)
    assert torch.equal(alone.pdfs, other)


@pytest.mark.parametrize("sides,periodicity", [("NSTB", (True, False, False)), ("WESTB", (False, False, False)),
                                               ("NS", (True, False, False))])
def test_a_slab_sweeps_with_its_part_of_the_walls(cuda, sides, periodicity):
    step = _step(sides=sides, obstacle=BOX, periodicity=periodicity, ubb=not periodicity[0])
    slab = object.__new__(DistributedLatticeBoltzmannStep)          # a slab with neighbours, without its ranks
    slab.local, slab.halo, slab.overlap, slab._aa, slab._split = step, object(), True, False, None
    parts = slab._overlap_sweeps()
    src, dst = step.pdfs, step.pdfs_tmp
    assert len(parts) == 3 and all(b._walls_ref is not None for _, b in parts)
    for off, b in parts:
        b.sweep(src.data_ptr() + off, dst.data_ptr() + off, 0)
    got = dst.clone()
    dst.zero_()
    step._bound().sweep(src.data_ptr(), dst.data_ptr(), 0)
    torch.cuda.synchronize()
    fluid = torch.from_numpy((step.boundary_handling.flag_array == 0)[1:-1, 1:-1, 1:-1]).cuda()
    assert torch.equal(got[1:-1, 1:-1, 1:-1][fluid], dst[1:-1, 1:-1, 1:-1][fluid])


def test_walls_of_another_periodicity_are_refused(cuda):
    step = _step()
    bound = step._bound()
    kernel = step._kernels[0]
    plan = N.Plan(build_desc(kernel.update_rule, SIZE, (True, True, False), {}))
    p, q = (ctypes.c_void_p(t.data_ptr()) for t in (step.pdfs, step.pdfs_tmp))
    walls = ctypes.byref(step.boundary_handling.walls.native)
    strides = N.i64_array(step.pdfs.stride())
    assert N.lib().lbm_sweep_walls(plan.handle, p, q, strides, walls, 0, None, None) == N.LBM_E_INVALID
    plan.update(build_desc(kernel.update_rule, SIZE, (True, False, False), {}))
    assert N.lib().lbm_sweep_walls(plan.handle, p, q, strides, walls, 0, None, None) == N.LBM_OK
    torch.cuda.synchronize()
    assert bound._walls_ref is step.boundary_handling.walls


def test_without_the_memory_the_sweeps_use_the_flags(cuda, monkeypatch):
    want = _step(obstacle=BOX)
    want.run_sweeps(3)
    step = _step(obstacle=BOX)
    real = torch.empty

    def no_memory(*a, **k):
        if k.get("dtype") is torch.int32:
            raise torch.cuda.OutOfMemoryError("no memory for the walls")
        return real(*a, **k)
    monkeypatch.setattr(torch, "empty", no_memory)
    step.run_sweeps(3)
    assert step.boundary_handling.walls is None
    torch.cuda.synchronize()
    assert torch.equal(step.pdfs, want.pdfs)


def test_walls_given_back_while_another_stream_still_sweeps(cuda):
    """New boundaries drop the walls of the old ones; their memory must not be handed out again while sweeps
    queued on another stream than the one they were built on still read them."""
    want = _step(obstacle=BOX)
    want.run_sweeps(40)
    step = _step(obstacle=BOX)
    step._bound()                                   # built on the current stream
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step.run_sweeps(40)
        got = step.pdfs
        step.boundary_handling.set_boundary(L.NoSlip(), L.slice_from_direction("N", 3))
        step._bound()                               # lets go of the first walls
    n = int(np.prod(SIZE)) + 2 * SIZE[2]
    junk = [torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    assert torch.equal(got, want.pdfs)
    del junk
