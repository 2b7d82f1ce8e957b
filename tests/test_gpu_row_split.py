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
