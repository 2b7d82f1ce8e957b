"""Attention weights and score gradients of any number of heads: a group of lanes has up to four of them, or fewer where el cannot be
read four at a time, and other groups have the rest; rows of no edge, of as many as the lanes hold, of one more and of many.

Bounds, in the 2-norm against fp64: a lane adds up at most 500 / 4 terms one after another, sqrt(125 / 3) 2^-24 = 4e-7 of their sum, twice
(softmax, gradients), and exp is off by up to two units in the last place: 2e-6."""
import pytest
import torch

from apt_b200 import ops
from tests.test_gpu_stream import _layer

pytestmark = pytest.mark.gpu
LENGTHS = [0, 1, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 0, 500, 2, 0]


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("H", [1, 2, 3, 4, 5, 6, 8, 9, 12, 16])
@pytest.mark.parametrize("mean", [2, 9, 20, 60])
def test_heads_and_row_lengths(H, mean, shift):
    gen = torch.Generator(device="cuda").manual_seed(H * 100 + mean)
    # short or long rows behind them bring the mean, which decides on the lanes, to either side
    n = torch.cat([torch.tensor(LENGTHS, device="cuda"), torch.full((400,), mean, device="cuda")])
    col = torch.arange(n.numel(), device="cuda").repeat_interleave(n)
    n_dst, n_src, D = n.numel(), 197, 12
    row = torch.randint(0, n_src, (col.numel(),), device="cuda", generator=gen)
    make = lambda *shape: torch.randn(shape, device="cuda", generator=gen)
    ft, er, g = make(n_src, H, D), make(n_dst, H, 1), make(n_dst, H, D)
    el = make(n_src * H + shift)[shift:].view(n_src, H, 1)
    assert el.data_ptr() % 16 == 4 * shift
    want = _layer(row, col, ft, el, er, g, n_dst)
    got = (ops.gat_edge_softmax_sum(row, col, ft, el, er, n_dst),) + tuple(ops.gat_edge_softmax_sum_backward(row, col, ft, el, er, g))
    leaves = [t.detach().requires_grad_() for t in (ft, el, er)]
    out = ops.GATEdgeSoftmaxSum.apply(row, col, *leaves, n_dst, 0.2)
    for a, b in list(zip(got, want)) + list(zip((out,) + torch.autograd.grad(out, leaves, g), want)):
        assert float((a.double().view_as(b) - b).norm() / b.norm()) <= 2e-6
    ops.check_status()
