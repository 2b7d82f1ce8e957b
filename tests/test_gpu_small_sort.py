"""Sums of few edges in no order, which one launch sorts: numbers of edges around a warp, a block's threads and what the warps' lists hold, of rows around
a block's share and the most that there can be, segments without edges, rows of very many edges, edges that belong to no row. Against the
fp64 oracle, bounds as in test_gpu_spmm_rows.py."""
import numpy as np
import pytest
import torch

from apt_b200 import ops
from oracle import oracle as orc
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu
I64 = np.int64


def _check(got, row, col, x, e, off, op):
    ab = [None if a is None else np.abs(a) for a in (x, e)]
    want, magnitude = orc.spmm_sum(op, row, col, x, e, *off), orc.spmm_sum(op, row, col, ab[0], ab[1], *off)
    err = np.abs(host(got).astype(np.float64) - want) / np.maximum(magnitude, 1e-30)
    assert err.max() <= 1e-5, err.max()


@pytest.mark.parametrize("edges", [2, 31, 33, 1023, 1025, 8193, 16383, 16384, 16385])
@pytest.mark.parametrize("rows", [1, 63, 65, 4097, 64 * 8192, 64 * 8192 + 1])
@pytest.mark.parametrize("skew", [1, 6])
def test_edges_and_rows(edges, rows, skew):
    rng = np.random.default_rng(edges + rows)
    n_in, dim = 70, 5
    col = np.minimum((rng.random(edges) ** skew * rows).astype(I64), rows - 1)      # skew: rows of thousands of edges in front
    col[:2] = [rows - 1, 0]
    row = rng.integers(0, n_in, edges).astype(I64)
    x = rng.standard_normal((n_in, dim)).astype(np.float32)
    off = [np.array([0, n], dtype=I64) for n in (edges, n_in, rows)]
    _check(ops.spmm_copy_u_sum(dev(row), dev(col), dev(x), *(dev(o) for o in off)), row, col, x, None, off, "copy_u")


@pytest.mark.parametrize("segments", [2, 3, 9, 64])
@pytest.mark.parametrize("op", ["copy_u", "copy_e", "u_mul_e"])
def test_segments(segments, op):
    rng = np.random.default_rng(segments)
    n_e, n_in, n_out = (rng.integers(0, k, segments) for k in (16384 // segments, 40, 90))
    n_e[0], n_in, n_out = 0, n_in + 1, n_out + 1
    row = np.concatenate([rng.integers(0, n_in[k], n_e[k]) for k in range(segments)]).astype(I64)
    col = np.concatenate([rng.integers(0, n_out[k], n_e[k]) for k in range(segments)]).astype(I64)
    off = [np.concatenate([[0], np.cumsum(n)]).astype(I64) for n in (n_e, n_in, n_out)]
    x = rng.standard_normal((int(n_in.sum()), 8)).astype(np.float32)
    e = rng.standard_normal((len(row), 8)).astype(np.float32)
    d = [dev(o) for o in off]
    if op == "copy_u":
        got, e = ops.spmm_copy_u_sum(dev(row), dev(col), dev(x), *d), None
    elif op == "copy_e":
        got, x = ops.spmm_copy_e_sum(dev(row), dev(col), dev(e), d[0], d[2]), None
    else:
        got = ops.spmm_u_mul_e_sum(dev(row), dev(col), dev(x), dev(e), *d)
    _check(got, row, col, x, e, off, op)


def test_edges_of_no_row():
    rng = np.random.default_rng(5)
    rows, n_in, edges = 300, 40, 5000
    col = rng.integers(0, rows, edges).astype(I64)
    row = rng.integers(0, n_in, edges).astype(I64)
    bad = rng.permutation(edges)[:400]
    col[bad] = rng.choice([-1, -7, rows, rows + 5, 1 << 40, -(1 << 40), (1 << 32) + 3], 400)
    x = rng.standard_normal((n_in, 12)).astype(np.float32)
    off = [np.array([0, n], dtype=I64) for n in (edges, n_in, rows)]
    got = ops.spmm_copy_u_sum(dev(row), dev(col), dev(x), *(dev(o) for o in off))
    good = np.setdiff1d(np.arange(edges), bad)
    _check(got, row[good], col[good], x, None, [np.array([0, len(good)], dtype=I64)] + off[1:], "copy_u")
