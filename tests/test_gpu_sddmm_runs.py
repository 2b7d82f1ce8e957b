"""The per-edge operators make a chunk of edges as one run of slices: widths around one slice, a warp's lanes and the chunk's bytes, numbers of edges around
a warp's chunk and where chunks grow, several segments. Against the oracle; sums and products of two values, rounded once: 32-bit results to one
rounding (2^-23 relative), 16-bit ones to theirs (2^-8, 2^-10)."""
import numpy as np
import pytest
import torch

from apt_b200 import ops
from oracle import oracle as orc
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu
EPS = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("dim", [1, 2, 4, 8, 16, 24, 47, 64, 130, 256, 1023, 2050])
@pytest.mark.parametrize("edges,segments", [(1, 1), (31, 1), (33, 2), (127, 1), (2050, 3), (9473 * 2 + 1, 1)])
def test_widths_and_edges(dtype, dim, edges, segments):
    if edges * dim > 20_000_000:
        edges = 20_000_000 // dim
    rng = np.random.default_rng(dim + edges)
    cut = lambda n: np.concatenate([[0], np.sort(rng.integers(0, n + 1, segments - 1)), [n]]).astype(np.int64)      # noqa: E731
    eo, lo, ro = cut(edges), np.arange(segments + 1, dtype=np.int64) * 50, np.arange(segments + 1, dtype=np.int64) * 30
    row, col = rng.integers(0, 50, edges).astype(np.int64), rng.integers(0, 30, edges).astype(np.int64)
    lhs, rhs = (torch.from_numpy(rng.standard_normal((n * segments, dim)).astype(np.float32)).to(dtype) for n in (50, 30))
    for name, fn in (("u_add_v", ops.sddmm_u_add_v), ("u_mul_v", ops.sddmm_u_mul_v)):
        got = host(fn(dev(row), dev(col), lhs.cuda(), rhs.cuda(), dev(eo), dev(lo), dev(ro))).astype(np.float64)
        want = orc.sddmm(name, row, col, lhs.float().numpy(), rhs.float().numpy(), eo, lo, ro).astype(np.float64)
        assert got.shape == want.shape and np.all(np.abs(got - want) <= EPS[dtype] * np.abs(want) + 1e-7)
