"""Wide rows of many edges, which are summed from shared memory behind bulk copies: a wait that runs out is reported and
leaves zeros, and the sums that look the block over on the device.

Bounds: a sum of n fp32 terms in any order is off by at most about n * 2^-24 of the sum of their magnitudes; 4e-6 of it
covers rows of 64 terms, and longer rows are sums of partial sums of about the root of their length."""
import ctypes

import pytest
import torch

from apt_b200 import _lib, ops
from apt_b200._lib import check, lib

pytestmark = pytest.mark.gpu
DST, SRC, DIM = 14_001, 20_003, 256


def _block(seed=0, fanout=15):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    col = torch.arange(DST, device="cuda").repeat_interleave(fanout)
    u = torch.rand(col.numel(), device="cuda", generator=gen, dtype=torch.float64)
    off = [torch.tensor([0, n], device="cuda") for n in (col.numel(), SRC, DST)]
    return (u ** 3 * SRC).long(), col, *off, gen


def _exact(out_index, in_index, x, rows):
    want = torch.zeros((rows, x.shape[1]), device="cuda", dtype=torch.float64).index_add_(0, out_index, x.double()[in_index])
    size = torch.zeros((rows, x.shape[1]), device="cuda", dtype=torch.float64).index_add_(0, out_index, x.double().abs()[in_index])
    return want, size


@pytest.fixture
def no_waiting():
    """Every wait for rows runs out at once."""
    check(lib.apt_set_tunable(b"bulk_wait_polls", 0))
    yield
    check(lib.apt_set_tunable(b"bulk_wait_polls", 1 << 20))
    torch.cuda.synchronize()
    lib.apt_pending_flags()
    ops.STATE.words().zero_()


def test_a_wait_that_ran_out_is_reported(no_waiting):
    row, col, eo, so, do, gen = _block()
    x, g = torch.randn((SRC, DIM), device="cuda", generator=gen), torch.randn((DST, DIM), device="cuda", generator=gen)
    torch.full((SRC, DIM), 5.0, device="cuda")                  # what the results' memory may hold
    for args, n in (((row, col, x, eo, so, do), DST), ((col, row, g, eo, do, so), SRC)):
        y = ops.spmm_copy_u_sum(*args)
        torch.cuda.synchronize()
        assert y.shape == (n, DIM) and not bool(y.any())
        small = row[:4], col[:4], x[:, :4].contiguous(), torch.tensor([0, 4], device="cuda"), so, do
        with pytest.raises(_lib.AptError, match="did not reach shared memory"):
            ops.spmm_copy_u_sum(*small)                         # a call of any size reports it, once
        ops.spmm_copy_u_sum(*small)
        ops.spmm_copy_u_sum(*args)
        with pytest.raises(RuntimeError, match="did not reach shared memory"):
            ops.check_status()
        ops.check_status()


def test_attention_reports_it_in_its_status(no_waiting):
    row, col, *_, gen = _block()
    make = lambda *shape: torch.randn(shape, device="cuda", generator=gen)
    args = row, col, make(SRC, 4, 64), make(SRC, 4, 1), make(DST, 4, 1)
    g_ft = ops.gat_edge_softmax_sum_backward(*args, make(DST, 4, 64))[0]
    with pytest.raises(RuntimeError, match="did not reach shared memory"):
        ops.check_status()
    assert not bool(g_ft.any()) and lib.apt_pending_flags() == 0


@pytest.mark.parametrize("reverse", [False, True], ids=["fixed", "order"])
def test_mode_left_on_the_device(reverse):
    row, col, eo, so, do, gen = _block(1)
    x = torch.randn((DST if reverse else SRC, DIM), device="cuda", generator=gen)
    args = (col, row, x, eo, do, so, SRC) if reverse else (row, col, x, eo, so, do, DST)
    src, dst, _, a, b, c, rows = args
    out = torch.full((rows, DIM), 9.0, device="cuda")
    nbytes = lib.apt_spmm_workspace_bytes(rows, src.numel())
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    check(lib.apt_spmm_sum(0, _lib.F32, p(src), p(dst), src.numel(), p(x), None, DIM, DIM, p(a), p(b), p(c), 1, rows, p(out),
                           p(ws), nbytes, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    want, size = _exact(dst, src, x, rows)
    assert bool(((out.double() - want).abs() <= 4e-6 * size + 1e-30).all())
    ops.check_status()
