"""The training workspace kept with a closure: the same gradient as with a workspace of its own, on
several streams and threads at once, for sample counts around the kernel's chunk and block counts."""
import copy
import threading

import pytest
import torch

from lbmpy_b200 import closure as C

pytestmark = pytest.mark.gpu


def _samples(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(10, n, generator=g, device="cuda"), 1e-4 * torch.rand(n, generator=g, device="cuda"),
            torch.rand(n, generator=g, device="cuda") + 0.5)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 592 * 64, 592 * 64 + 1])
def test_kept_workspace_gives_the_same_bits(cuda, n):
    clo = C.MLPClosure(seed=1)
    data = _samples(n, n)
    loss0, grad0 = clo.loss_and_grad(*data, trainer=C._Trainer())
    for _ in range(2):
        loss, grad = clo.loss_and_grad(*data)
        assert torch.equal(loss, loss0) and torch.equal(grad, grad0)
    copied = copy.deepcopy(clo)
    assert torch.equal(copied.loss_and_grad(*data)[1], grad0)


def test_streams_and_threads_do_not_share_it(cuda):
    clo = C.MLPClosure(seed=2)
    sets = [_samples(20000 + 777 * k, k) for k in range(6)]
    want = [clo.loss_and_grad(*d, trainer=C._Trainer())[1] for d in sets]
    torch.cuda.synchronize()
    got = [None] * len(sets)

    def work(k):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(5):
                got[k] = clo.loss_and_grad(*sets[k])[1]
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sets))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert len(clo._workspaces) <= clo._MAX_WORKSPACES


def test_a_captured_graph_does_not_hold_the_kept_workspace(cuda):
    """The kept workspace may be given back while a graph that was captured with it lives on, so capture
    without a workspace of the caller's own is refused, also on a stream the call was warmed on."""
    clo = C.MLPClosure(seed=3)
    feats, target, _ = _samples(1000, 9)
    stream, own = torch.cuda.Stream(), C._Trainer()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        want = clo.loss_and_grad(feats, target)[1]
        clo.loss_and_grad(feats, target, trainer=own)
    torch.cuda.synchronize()
    refused, graph = False, torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        try:
            clo.loss_and_grad(feats, target)
        except RuntimeError:
            refused = True
        grad = clo.loss_and_grad(feats, target, trainer=own)[1]
    assert refused
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(grad, want)
    assert torch.equal(clo.loss_and_grad(feats, target)[1], want)
