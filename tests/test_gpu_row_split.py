"""Numbers of rows on either side of where they fill the chip by themselves and a row's edges are no longer taken side by side, for rows of two
lanes to a whole warp, rows of one length, of many and in no order, against the fp64 oracle. Bounds as in test_gpu_spmm_rows.py."""
import numpy as np
import pytest
import torch

from apt_b200 import ops
from oracle import oracle as orc
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu
LANES = 148 * 24 * 32


@pytest.mark.parametrize("dtype,dim", [(torch.float32, 1), (torch.bfloat16, 4), (torch.float32, 8), (torch.bfloat16, 30), (torch.float32, 36), (torch.bfloat16, 128)])
@pytest.mark.parametrize("side", [-1, 0, 1])
@pytest.mark.parametrize("lengths", ["fixed", "ragged", "no order"])
def test_rows_that_fill_the_chip(dtype, dim, side, lengths):
    rng = np.random.default_rng(dim + side)
    size = 4 if dtype == torch.float32 else 2
    slices = -(-dim * size // 16) if dim * size % 16 == 0 else dim if dim * size % 8 else dim * size // 8
    lanes = 1 << max(0, (min(slices, 32) - 1).bit_length())
    rows, n_in = max(50, LANES // lanes // 2 // (2 if lanes < 8 else 1) + side), 300
    n = np.full(rows, 6) if lengths == "fixed" else rng.integers(0, 13, rows)
    col = np.repeat(np.arange(rows), n).astype(np.int64)
    row = rng.integers(0, n_in, len(col)).astype(np.int64)
    if lengths == "no order":
        col = rng.permutation(col)
    x = torch.from_numpy(rng.standard_normal((n_in, dim)).astype(np.float32)).to(dtype)
    off = [np.array([0, k], dtype=np.int64) for k in (len(col), n_in, rows)]
    got = host(ops.spmm_copy_u_sum(dev(row), dev(col), x.cuda(), *(dev(o) for o in off))).astype(np.float64)
    xs = x.float().numpy()
    want, magnitude = (orc.spmm_sum("copy_u", row, col, v, None, *off) for v in (xs, np.abs(xs)))
    err = np.abs(got - want) / np.maximum(magnitude, 1e-30)
    assert err.max() <= (1e-5 if dtype == torch.float32 else 1e-2), err.max()


@pytest.mark.parametrize("dim", [16, 32, 64, 36])
@pytest.mark.parametrize("ordered", [False, True])
def test_sums_of_rows_an_edge_at_a_time_are_no_further_from_64_bits(dim, ordered):
    """24 edges a row of which every one is taken after the other: a rounding is off by 2.9e-8 of what it rounds (2^-24 / sqrt(3), over the mean mantissa).
    Added up by fours that is sqrt((12 x 2 + 6 x 4 + 8 + 12 + 16 + 20 + 24) / 24) of the sum, 6.7e-8, side by side about as much; one by one 1.03e-7."""
    rows, per, n_in = 60_000, 24, 30_000
    g = torch.Generator(device="cuda").manual_seed(dim)
    col, row = torch.arange(rows, device="cuda").repeat_interleave(per), torch.randint(0, n_in, (rows * per,), generator=g, device="cuda")
    if ordered:
        p = torch.randperm(rows * per, generator=g, device="cuda")
        row, col = row[p], col[p]
    x = torch.randn(n_in, dim, generator=g, device="cuda")
    off = [torch.tensor([0, n], device="cuda") for n in (rows * per, n_in, rows)]
    got = ops.spmm_copy_u_sum(row, col, x, *off).double()
    want = torch.zeros(rows, dim, dtype=torch.float64, device="cuda").index_add_(0, col, x.double()[row])
    assert float((got - want).norm() / want.norm()) <= 8e-8


@pytest.mark.parametrize("dim", [101, 128, 256])
def test_long_rows_are_no_further_from_64_bits(dim):
    """1000 edges a row, in no order, by k_spmm_stream. A warp's part of a row is 282 edges of a million here: added up by fours, 71 sums one after another, then
    the parts. A rounding is off by 2.9e-8 of what it rounds: sqrt(sum over 4, 8 ... 284 / 284 + what comes before and behind, a tenth of it) of a part's, 1.8e-7, and
    less where parts are cut short by row ends; one edge after another 3.5e-7."""
    rows, edges, n_in = 1000, 1_000_000, 60_000
    g = torch.Generator(device="cuda").manual_seed(dim)
    col, row = (torch.randint(0, n, (edges,), generator=g, device="cuda") for n in (rows, n_in))
    x = torch.randn(n_in, dim, generator=g, device="cuda")
    off = [torch.tensor([0, n], device="cuda") for n in (edges, n_in, rows)]
    got = ops.spmm_copy_u_sum(row, col, x, *off).double()
    want = torch.zeros(rows, dim, dtype=torch.float64, device="cuda").index_add_(0, col, x.double()[row])
    assert float((got - want).norm() / want.norm()) <= 2.0e-7
