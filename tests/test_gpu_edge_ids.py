"""Destinations outside their table, on whose gaps the tables of edge ranges must not be written past their front: a flag and zeros
from the attention layer, and from sums told that the edges are grouped what the counting sort gives (such edges count for
nothing)."""
import ctypes

import pytest
import torch

from apt_b200 import ops
from apt_b200._lib import check, lib

pytestmark = pytest.mark.gpu


def _block(n_dst, fanout, first):
    gen = torch.Generator(device="cuda").manual_seed(n_dst)
    col = torch.arange(n_dst, device="cuda").repeat_interleave(fanout)
    col[:len(first)] = torch.tensor(first, device="cuda")
    row = torch.randint(0, 301, (col.numel(),), device="cuda", generator=gen)
    return row, col, gen


@pytest.mark.parametrize("first", [[-5], [-1], [-27, -26, -1], [0, -5]])
@pytest.mark.parametrize("n_dst,fanout,H,D", [(40, 5, 4, 8), (700, 3, 4, 64), (28_101, 14, 4, 64)])
def test_attention_of_a_negative_destination(first, n_dst, fanout, H, D):
    row, col, gen = _block(n_dst, fanout, first)
    make = lambda *shape: torch.randn(shape, device="cuda", generator=gen)
    ft, el, er, g = make(301, H, D), make(301, H, 1), make(n_dst, H, 1), make(n_dst, H, D)
    leaves = [t.clone().requires_grad_() for t in (ft, el, er)]
    out = ops.GATEdgeSoftmaxSum.apply(row, col, *leaves, n_dst, 0.2)
    got = (out, ops.gat_edge_softmax_sum(row, col, ft, el, er, n_dst)) + torch.autograd.grad(out, leaves, g)
    got += tuple(ops.gat_edge_softmax_sum_backward(row, col, ft, el, er, g))
    with pytest.raises(RuntimeError, match="grouped"):
        ops.check_status()
    assert not any(bool(t.any()) for t in got)


@pytest.mark.parametrize("first", [[-5], [-27, -26, -1]])
def test_sums_of_edges_called_grouped(first):
    n_dst, fanout, D = 700, 4, 20
    row, col, gen = _block(n_dst, fanout, first)
    x = torch.randint(-3, 4, (301, D), device="cuda", generator=gen).float()
    off = [torch.tensor([0, k], device="cuda") for k in (col.numel(), 301, n_dst)]
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    out = torch.empty((n_dst, D), device="cuda")
    nbytes = lib.apt_spmm_workspace_bytes(n_dst, col.numel())
    ws = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    check(lib.apt_spmm_sum_known(0, 0, p(row), p(col), col.numel(), p(x), None, D, D, *map(p, off), 1, n_dst, 1, 0, p(out), p(ws), nbytes, stream))
    there = col >= 0
    want = torch.zeros_like(out).index_add_(0, col[there], x[row[there]])
    assert torch.equal(out, want) and torch.equal(ops.spmm_copy_u_sum(row, col, x, *off), want)
