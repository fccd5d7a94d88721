"""The training gradient's FP32 partial sums: no running sum may grow with the number of samples."""
import pytest
import torch

from lbmpy_b200 import closure as C

pytestmark = pytest.mark.gpu


def test_many_samples_per_block_keep_their_digits(cuda):
    """One sample repeated: its mean gradient is the same for every number of samples, so what differs is
    the rounding of the sums alone.  A block that adds groups of 128 samples on their own and then the groups
    is off by at most (128 + groups) half-ulps; one register that takes every sample loses its last digits to
    the size of the sum (3e-3 for the 2^19 samples of a block here)."""
    blocks, n = 2, 1 << 20
    g = torch.Generator().manual_seed(4)
    sample, target = torch.randn(10, 1, generator=g).cuda(), torch.tensor([3e-3]).cuda()
    clo = C.MLPClosure(seed=5)
    loss1, want = clo.loss_and_grad(sample.expand(10, 64).contiguous(), target.expand(64).contiguous())
    loss, got = clo.loss_and_grad(sample.expand(10, n).contiguous(), target.expand(n).contiguous(),
                                  trainer=C._Trainer(blocks))
    live = want != 0
    assert live.sum() > 1000
    off = ((got.double() - want.double()).abs()[live] / want.double().abs()[live]).max().item()
    groups = n // blocks // 128
    assert off <= (128 + 64 + groups) * 2.0 ** -24, off
    assert abs(loss.item() / loss1.item() - 1) < 1e-9
