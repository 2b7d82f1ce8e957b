"""The row kernel of the SpMM at the edges of its lane splits, round lengths and row lengths, the probe in front of it
and the enqueue-only entry point, against the fp64 oracle. Bounds as in test_gpu_spmm.py: fp32 sums within 1e-5 and
16-bit results within 1e-2 of the summed magnitudes."""
import ctypes

import numpy as np
import pytest
import torch

from apt_b200 import _lib, ops
from apt_b200._lib import check, lib
from oracle import oracle as orc
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu
I64 = np.int64
TOL = {torch.float32: 1e-5, torch.bfloat16: 1e-2, torch.float16: 1e-2}


def _round(x, dtype):
    return torch.from_numpy(x).to(dtype).float().numpy() if dtype != torch.float32 else x


def _want(row, col, x, off):
    return orc.spmm_sum("copy_u", row, col, x, None, *off), orc.spmm_sum("copy_u", row, col, np.abs(x), None, *off)


def _close(got, want, magnitude, dtype):
    err = np.abs(host(got).astype(np.float64) - want) / np.maximum(magnitude, 1e-30)
    assert err.max() <= TOL[dtype], err.max()


# widths around one, two and four slices a lane, of 16, 8, 4 and 2 bytes, and beyond one column block
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [1, 2, 3, 8, 31, 33, 47, 66, 127, 128, 130, 256, 260, 516, 600])
@pytest.mark.parametrize("fanout", [1, 3, 33])
def test_row_widths_and_fanouts(dtype, D, fanout):
    rng = np.random.default_rng(D * 100 + fanout)
    S, n_src = 37, 90
    row = rng.integers(0, n_src, S * fanout).astype(I64)
    col = np.repeat(np.arange(S, dtype=I64), fanout)
    x = _round(rng.standard_normal((n_src, D)).astype(np.float32), dtype)
    g = _round(rng.standard_normal((S, D)).astype(np.float32), dtype)
    eo, io, oo = (np.array([0, n], dtype=I64) for n in (S * fanout, n_src, S))
    _close(ops.spmm_copy_u_sum(dev(row), dev(col), dev(x, dtype), dev(eo), dev(io), dev(oo)),
           *_want(row, col, x, (eo, io, oo)), dtype)
    _close(ops.spmm_copy_u_sum(dev(col), dev(row), dev(g, dtype), dev(eo), dev(oo), dev(io)),
           *_want(col, row, g, (eo, oo, io)), dtype)


# row lengths around what one group walks (32, 128), one item (64) and rows of several items; `wide` 2100-column rows
# find no room for the partial sums of their longest rows and are walked unsplit
@pytest.mark.parametrize("dtype,D", [(torch.float32, 8), (torch.float32, 128), (torch.bfloat16, 300), (torch.float32, 2100)])
@pytest.mark.parametrize("op", ["copy_u", "u_mul_e", "copy_e"])
def test_long_rows(dtype, D, op):
    rng = np.random.default_rng(D)
    lengths = np.array([0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 0, 500, 1500, 2, 0])
    n_in, n_out, E = 50, len(lengths), int(lengths.sum())
    col = rng.permutation(np.repeat(np.arange(n_out), lengths)).astype(I64)
    row = rng.integers(0, n_in, E).astype(I64)
    off = tuple(np.array([0, n], dtype=I64) for n in (E, n_in, n_out))
    eo, io, oo = (dev(o) for o in off)
    x = _round(rng.standard_normal((n_in, D)).astype(np.float32), dtype)
    if op == "copy_u":
        got, e = ops.spmm_copy_u_sum(dev(row), dev(col), dev(x, dtype), eo, io, oo), None
    elif op == "u_mul_e":
        e = _round(rng.standard_normal((E, 4 if D % 4 == 0 else 1)).astype(np.float32), dtype)
        got = ops.spmm_u_mul_e_sum(dev(row), dev(col), dev(x, dtype), dev(e, dtype), eo, io, oo)
    else:
        e = _round(rng.standard_normal((E, D)).astype(np.float32), dtype)
        x = None
        got = ops.spmm_copy_e_sum(dev(row), dev(col), dev(e, dtype), eo, oo)
    ab = [None if a is None else np.abs(a) for a in (x, e)]
    _close(got, orc.spmm_sum(op, row, col, x, e, *off), orc.spmm_sum(op, row, col, ab[0], ab[1], *off), dtype)


CASES = {
    "fixed": [2, 2, 2, 2], "fixed in segments": [3] * 6, "ragged": [1, 0, 4, 2], "empty first and last": [0, 3, 1, 0],
    "one row": [5], "long run": [2, 150, 1],
}


@pytest.mark.parametrize("name", sorted(CASES) + ["swapped pair", "drop behind a jump", "random"])
def test_probe_and_enqueue_only_form(name):
    """The mode the probe finds, and the same sums from the entry point that does not wait for it."""
    rng = np.random.default_rng(len(name))
    lengths = CASES.get(name, [2, 2, 2, 2])
    col = np.repeat(np.arange(len(lengths)), lengths).astype(I64)
    want_mode = {"fixed": 0, "fixed in segments": 0, "ragged": 1, "empty first and last": 1, "one row": 0}.get(name, 2)
    if name == "swapped pair":
        col[[3, 4]] = col[[4, 3]]
    elif name == "drop behind a jump":      # the edge after the drop fits the fanout again
        col[2] = 3
    elif name == "random":
        col = rng.permutation(col)
    E, n_out, n_in, D = len(col), len(lengths), 20, 24
    row = rng.integers(0, n_in, E).astype(I64)
    x = rng.standard_normal((n_in, D)).astype(np.float32)
    off = [np.array([0, n], dtype=I64) for n in (E, n_in, n_out)]
    if name == "fixed in segments":         # two blocks of three rows with ids of their own
        col, off = col % 3, [np.array(v, dtype=I64) for v in ([0, 9, 18], [0, 8, 20], [0, 3, 6])]
        row = np.concatenate([rng.integers(0, 8, 9), rng.integers(0, 12, 9)]).astype(I64)
    d_row, d_col, d_x = dev(row), dev(col), dev(x)
    eo, io, oo = (dev(o) for o in off)
    got = (ctypes.c_int64 * 3)()
    check(lib.apt_spmm_probe(d_col.data_ptr(), E, eo.data_ptr(), oo.data_ptr(), len(off[0]) - 1, got, None))
    assert got[0] == n_out and got[1] == want_mode and (want_mode != 0 or got[2] == lengths[0])
    want, magnitude = _want(row, col, x, off)
    _close(ops.spmm_copy_u_sum(d_row, d_col, d_x, eo, io, oo), want, magnitude, torch.float32)
    out = torch.full((n_out, D), 7.0, device="cuda")
    nbytes = lib.apt_spmm_workspace_bytes(n_out, E)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    check(lib.apt_spmm_sum(0, _lib.F32, d_row.data_ptr(), d_col.data_ptr(), E, d_x.data_ptr(), None, D, D, eo.data_ptr(),
                           io.data_ptr(), oo.data_ptr(), len(off[0]) - 1, n_out, out.data_ptr(), ws.data_ptr(), nbytes, None))
    torch.cuda.synchronize()
    _close(out, want, magnitude, torch.float32)


@pytest.mark.parametrize("dtype,D", [(torch.float32, 132), (torch.float32, 200), (torch.float32, 256),
                                     (torch.bfloat16, 264), (torch.bfloat16, 512), (torch.float16, 384)])
@pytest.mark.parametrize("shape", ["fixed", "ragged", "reverse", "segments"])
def test_wide_rows_of_many_edges(dtype, D, shape):
    # rows that travel through shared memory. Small whole numbers: exact in fp32, one rounding of the sum in 16 bits.
    gen = torch.Generator(device="cuda").manual_seed(D)
    fixed = shape in ("fixed", "segments")
    n_out, n_in, f = (20_002, 5001, 10) if fixed else (20_003, 5001, 21)
    lengths = torch.full((n_out,), f, device="cuda") if fixed else torch.randint(0, f, (n_out,), device="cuda", generator=gen)
    col = torch.repeat_interleave(torch.arange(n_out, device="cuda"), lengths)
    u = torch.rand(col.numel(), device="cuda", generator=gen, dtype=torch.float64)
    row = (u * u * n_in).long()
    if shape == "reverse":                      # hubs of thousands of edges, items of their own
        row, col, n_in, n_out = col, (u ** 4 * 50_000).long(), n_out, 50_000
    E = col.numel()
    assert E >= 196_608
    x = torch.randint(-4, 5, (n_in, D), device="cuda", generator=gen).to(dtype)
    T = lambda *v: torch.tensor(v, device="cuda")
    offsets = T(0, E), T(0, n_in), T(0, n_out)
    want = torch.zeros((n_out, D), device="cuda").index_add_(0, col, x.float()[row])
    if shape == "segments":                     # two blocks with ids of their own
        half, first = n_out // 2, col < n_out // 2
        row = torch.where(first, row % 2000, row % 3001)
        want = torch.zeros((n_out, D), device="cuda").index_add_(0, col, x.float()[torch.where(first, row, row + 2000)])
        col, offsets = col % half, (T(0, E // 2, E), T(0, 2000, n_in), T(0, half, n_out))
    assert torch.equal(ops.spmm_copy_u_sum(row, col, x, *offsets), want.to(dtype))


@pytest.mark.parametrize("E", [2, 5, 1023, 1024, 1025, 700_001])
def test_probe_finds_one_edge_out_of_order(E):
    # one thread block and several, the last of them ragged; more edges than one wave of blocks holds at a time
    gen = torch.Generator(device="cuda").manual_seed(E)
    n_out, n_in = E // 2 + 1, 50
    row = torch.randint(0, n_in, (E,), device="cuda", generator=gen)
    x = torch.arange(n_in, dtype=torch.float32, device="cuda")[:, None].contiguous()      # small integers: exact sums
    off = [torch.tensor([0, n], device="cuda") for n in (E, n_in, n_out)]
    for at in {1, E // 2, E - 1}:
        col = torch.arange(E, device="cuda") // 2
        col[at] = (col[at] + n_out // 2 + 1) % n_out
        want = torch.zeros(n_out, 1, device="cuda").index_add_(0, col, x[row])
        got = (ctypes.c_int64 * 3)()
        check(lib.apt_spmm_probe(col.data_ptr(), E, off[0].data_ptr(), off[2].data_ptr(), 1, got, None))
        rising = bool((col[1:] >= col[:-1]).all())
        assert got[0] == n_out and got[1] == (1 if rising else 2)
        assert torch.equal(ops.spmm_copy_u_sum(row, col, x, *off), want)


def test_probe_is_refused_inside_a_capture():
    one = torch.zeros(1, dtype=torch.int64, device="cuda")
    off = torch.tensor([0, 1], device="cuda")
    x = torch.ones((1, 4), device="cuda")
    ops.spmm_copy_u_sum(one, one, x, off, off, off)
    graph = torch.cuda.CUDAGraph()
    with pytest.raises(RuntimeError, match="stream capture"):
        with torch.cuda.graph(graph):
            ops.spmm_copy_u_sum(one, one, x, off, off, off)
    assert host(ops.spmm_copy_u_sum(one, one, x, off, off, off)).tolist() == [[1.0] * 4]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [1, 2, 6, 12, 33, 200])
def test_sddmm_widths(dtype, D):
    rng = np.random.default_rng(D)
    E, n_l, n_r = 1031, 77, 55
    row, col = rng.integers(0, n_l, E).astype(I64), rng.integers(0, n_r, E).astype(I64)
    lhs, rhs = (_round(rng.standard_normal((n, D)).astype(np.float32), dtype) for n in (n_l, n_r))
    off = [np.array([0, n], dtype=I64) for n in (E, n_l, n_r)]
    for name, fn in (("u_add_v", ops.sddmm_u_add_v), ("u_mul_v", ops.sddmm_u_mul_v)):
        want = orc.sddmm(name, row, col, lhs, rhs, *off)
        got = fn(dev(row), dev(col), dev(lhs, dtype), dev(rhs, dtype), *(dev(o) for o in off))
        # one rounding of an exact sum or product
        assert np.all(np.abs(host(got).astype(np.float64) - want) <= TOL[dtype] * np.abs(want) + 1e-38)


@pytest.mark.parametrize("num_rows", [4, 10, 11, 25, 50, 60])
@pytest.mark.parametrize("order", ["fixed", "ragged", "mixed"])
def test_more_or_fewer_rows_than_the_offsets_end_at(num_rows, order):
    # 50 edges over 10 rows, offsets that end at 10, a result of another length: rows behind are zero, edges of rows beyond it
    # are left out, also where the edges divide evenly among the rows there are
    rng = np.random.default_rng(num_rows)
    E, S, n_src, D = 50, 10, 17, 12
    col = np.repeat(np.arange(S), 5) if order == "fixed" else np.sort(rng.integers(0, S, E))
    if order == "mixed":
        rng.shuffle(col)
    row, col = rng.integers(0, n_src, E).astype(I64), col.astype(I64)
    x = rng.integers(-8, 9, (n_src, D)).astype(np.float32)          # whole numbers: sums are exact
    want = np.zeros((max(num_rows, S), D), np.float32)
    np.add.at(want, col, x[row])
    t = [dev(row), dev(col), dev(x)] + [dev(np.array([0, n], dtype=I64)) for n in (E, n_src, S)]
    out = torch.full((num_rows, D), 9.0, device="cuda")
    nbytes = lib.apt_spmm_workspace_bytes(num_rows, E)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    p = [ctypes.c_void_p(v.data_ptr()) for v in t]
    check(lib.apt_spmm_sum(0, _lib.F32, p[0], p[1], E, p[2], None, D, D, p[3], p[4], p[5], 1, num_rows, ctypes.c_void_p(out.data_ptr()),
                           ctypes.c_void_p(ws.data_ptr()), nbytes, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert np.array_equal(host(out), want[:num_rows])
    if num_rows >= S:
        longer = dev(np.array([0, S, num_rows], dtype=I64))         # the operator takes the number of rows from the last entry
        assert np.array_equal(host(ops.spmm_copy_u_sum(*t[:5], longer)), want)
    ops.check_status()
