"""Sums and dots of wide rows of many edges, which a warp takes from a stretch of the edges: row ends, rows without edges
and rows of many stretches, and the lanes that a row does not fill.

Bounds: sums of small whole numbers are exact in fp32, and a 16-bit result is one rounding of them. The attention layer is
held to the 2-norm of the fp64 results: about 15 fp32 terms a sum (2e-6), and 2^-9 or 2^-12 for a rounding to 16 bits. The
gradient of el is added up in fp32 one edge after another, in the order of arrival: n additions, each off by up to 2^-24 of the sum
so far (1 / sqrt(3) of that as a standard deviation), are off by sqrt(n / 3) 2^-24 of the largest sum on the way. The first source here
has 393 000 / 9001^(1/4) = 40 400 edges, which is 6.9e-6; three standard deviations are 2.1e-5 (seen: up to 7.2e-6 in 250 runs)."""
import ctypes

import pytest
import torch

from apt_b200 import ops
from apt_b200._lib import check, lib

pytestmark = pytest.mark.gpu
N_IN = 5003


def _lengths(shape, edges, gen):
    """Edges of every output row: a fanout; 0 to 32; one row of almost half of all edges (thousands of stretches) among short ones."""
    if shape == "fixed":
        return torch.full((edges // 13 + 1,), 13, device="cuda")
    # (16 edges a row, some more rows than that takes: none makes up for a small draw by a length of its own, and none of more than 32
    # edges makes the probe ask for the counting sort)
    n = torch.randint(0, 33 if shape == "ragged" else 9, (edges // (15 if shape == "ragged" else 8),), device="cuda", generator=gen)
    if shape == "hub":
        n[n.numel() // 3] = edges // 2
        n[-1] = n[0] = 0
    else:
        n[n.numel() // 2] = 0
    return n


def _mode(col, *off):
    """Where the probe says a row's edges are."""
    answer = (ctypes.c_int64 * 3)()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    check(lib.apt_spmm_probe(p(col), col.numel(), p(off[0]), p(off[2]), off[0].numel() - 1, answer,
                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return answer[1]


@pytest.mark.parametrize("dtype,D", [(torch.float32, 68), (torch.float32, 128), (torch.float32, 260 - 4), (torch.bfloat16, 136),
                                     (torch.bfloat16, 256), (torch.float16, 264)])
@pytest.mark.parametrize("shape,edges", [("fixed", 655_360), ("ragged", 655_360), ("hub", 98_304), ("hub", 400_000)])
def test_sums(dtype, D, shape, edges):
    gen = torch.Generator(device="cuda").manual_seed(D + edges)
    n = _lengths(shape, edges, gen)
    col = torch.arange(n.numel(), device="cuda").repeat_interleave(n)
    if shape == "hub":
        col = col[torch.randperm(col.numel(), device="cuda", generator=gen)]
        pad = edges - col.numel() + 3
        col = torch.cat([col, torch.full((max(0, pad),), n.numel() // 2, device="cuda")])
    row = torch.randint(0, N_IN, (col.numel(),), device="cuda", generator=gen)
    x = torch.randint(-3, 4, (N_IN, D), device="cuda", generator=gen).to(dtype)
    off = [torch.tensor([0, k], device="cuda") for k in (col.numel(), N_IN, n.numel())]
    assert col.numel() >= edges and _mode(col, *off) == {"fixed": 0, "ragged": 1, "hub": 2}[shape]
    want = torch.zeros((n.numel(), D), device="cuda", dtype=torch.float64).index_add_(0, col, x.double()[row]).to(dtype)
    assert torch.equal(ops.spmm_copy_u_sum(row, col, x, *off), want)


def _layer(row, col, ft, el, er, g, n_dst):
    """The attention layer and its gradients in fp64."""
    ft, el, er = (t.double().requires_grad_() for t in (ft, el, er))
    s = torch.nn.functional.leaky_relu(el[row] + er[col], 0.2)
    at = col[:, None, None].expand_as(s)
    most = torch.full((n_dst, *s.shape[1:]), -torch.inf, device="cuda", dtype=torch.float64).scatter_reduce(0, at, s.detach(), "amax")
    p = (s - most[col]).exp()
    a = p / torch.zeros_like(most).index_add(0, col, p)[col]
    out = torch.zeros((n_dst, *ft.shape[1:]), device="cuda", dtype=torch.float64).index_add(0, col, a * ft[row])
    return (out.detach(),) + torch.autograd.grad(out, (ft, el, er), g.double())


@pytest.mark.parametrize("dtype,H,D", [(torch.float32, 4, 32), (torch.float32, 1, 256), (torch.float32, 8, 32), (torch.float32, 4, 48),
                                       (torch.float32, 2, 44), (torch.float32, 16, 16), (torch.bfloat16, 4, 64), (torch.bfloat16, 8, 24), (torch.float16, 5, 40),
                                       (torch.float16, 2, 256)])
@pytest.mark.parametrize("ragged", [False, True])
def test_attention(dtype, H, D, ragged):
    gen = torch.Generator(device="cuda").manual_seed(H * D)
    n = torch.randint(0, 29, (30_001,), device="cuda", generator=gen) if ragged else torch.full((28_101,), 14, device="cuda")
    n[7] += 500
    col = torch.arange(n.numel(), device="cuda").repeat_interleave(n)
    n_dst, n_src, E = n.numel(), 9001, col.numel()
    assert E >= 393_216
    row = (torch.rand(E, device="cuda", generator=gen) ** 4 * n_src).long().clamp_(max=n_src - 1)
    make = lambda *shape: torch.randn(shape, device="cuda", generator=gen).to(dtype)
    ft, el, er, g = make(n_src, H, D), make(n_src, H, 1), make(n_dst, H, 1), make(n_dst, H, D)
    want = _layer(row, col, ft, el, er, g, n_dst)
    leaves = [t.clone().requires_grad_() for t in (ft, el, er)]
    out = ops.GATEdgeSoftmaxSum.apply(row, col, *leaves, n_dst, 0.2)
    bound = {torch.float32: 2e-6, torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -12}[dtype]
    for k, (got, ref) in enumerate(zip((out,) + torch.autograd.grad(out, leaves, g), want)):
        assert float((got.double() - ref).norm() / ref.norm()) <= (max(bound, 2.1e-5) if k == 2 else bound)


def test_dots_beside_infinite_features():
    # heads of 12 slices on 16 lanes: the lanes without a slice add nothing, and a head's infinities stay in it
    gen = torch.Generator(device="cuda").manual_seed(3)
    n_dst, n_src, H, D = 28_101, 9001, 4, 48
    col = torch.arange(n_dst, device="cuda").repeat_interleave(14)
    row = torch.randint(0, n_src, (col.numel(),), device="cuda", generator=gen)
    make = lambda *shape: torch.randn(shape, device="cuda", generator=gen)
    ft, el, er, g = make(n_src, H, D), make(n_src, H, 1), make(n_dst, H, 1), make(n_dst, H, D)
    plain = ops.gat_edge_softmax_sum_backward(row, col, ft, el, er, g)
    ft[:, 0] = torch.inf
    _, g_el, g_er = ops.gat_edge_softmax_sum_backward(row, col, ft, el, er, g)
    assert torch.equal(g_er[:, 1:], plain[2][:, 1:]) and not bool(g_er[:, 0].isfinite().any())
    assert float((g_el[:, 1:] - plain[1][:, 1:]).norm() / plain[1][:, 1:].norm()) <= 2e-6      # (44 edges a source, added up in the order of arrival)


@pytest.mark.parametrize("at", [1, 350_000, 699_999])
def test_edges_out_of_order_belong_to_nobody(at):
    # one edge out of its destination's turn, wherever it is: zeros everywhere, and the flag
    gen = torch.Generator(device="cuda").manual_seed(at)
    E, n_dst, n_src = 700_000, 50_000, 9001
    col = torch.arange(n_dst, device="cuda").repeat_interleave(14)
    col[at - 1], col[at] = n_dst - 1 if at < E // 2 else col[at - 1], 0
    row = torch.randint(0, n_src, (E,), device="cuda", generator=gen)
    make = lambda *shape: torch.randn(shape, device="cuda", generator=gen)
    ft, el, er, g = make(n_src, 4, 32), make(n_src, 4, 1), make(n_dst, 4, 1), make(n_dst, 4, 32)
    got = (ops.gat_edge_softmax_sum(row, col, ft, el, er, n_dst),) + tuple(ops.gat_edge_softmax_sum_backward(row, col, ft, el, er, g))
    with pytest.raises(RuntimeError, match="grouped"):
        ops.check_status()
    assert not any(bool(t.any()) for t in got)


@pytest.mark.parametrize("dtype,D", [(torch.float32, 128), (torch.bfloat16, 512)])
def test_rows_of_any_number_of_stretches(dtype, D):
    # one row among short ones, from one stretch of 32 to 88 edges to a hundred: parts are added up by 32s, a group of one among them
    gen = torch.Generator(device="cuda").manual_seed(D)
    E, n_out = 100_000, 9001
    x = torch.randint(-3, 4, (N_IN, D), device="cuda", generator=gen).to(dtype)
    row = torch.randint(0, N_IN, (E,), device="cuda", generator=gen)
    others = torch.randint(0, n_out, (E,), device="cuda", generator=gen)
    turn = torch.randperm(E, device="cuda", generator=gen)
    off = [torch.tensor([0, k], device="cuda") for k in (E, N_IN, n_out)]
    rest = torch.zeros((n_out, D), device="cuda", dtype=torch.float64)
    for n in range(40, 3400, 40):
        col = others.clone()
        col[turn[:n]] = 4000
        want = rest.zero_().index_add_(0, col, x.double()[row])
        assert torch.equal(ops.spmm_copy_u_sum(row, col, x, *off), want.to(dtype)), n


@pytest.mark.parametrize("dtype,D", [(torch.float32, 72), (torch.float32, 256), (torch.bfloat16, 256), (torch.float16, 512)])
@pytest.mark.parametrize("edges", [100_000, 210_000, 700_000])
@pytest.mark.parametrize("shape", ["fixed", "ragged", "none"])
@pytest.mark.parametrize("further", [0, 7])
def test_segments_in_any_order(dtype, D, edges, shape, further):
    """Three segments; edges of the same number each, of 0 to 32, or in no order. With further output rows behind the last segment's
    nothing about the edges is known to the host, and the kernels decide."""
    gen = torch.Generator(device="cuda").manual_seed(D + edges)
    fanout = 13
    parts, dst, src = [0], [0], [0]
    rows, cols = [], []
    for share in (0.5, 0.03, 0.47):
        n_dst, n_src = int(edges * share / fanout) + 1, int(3001 * share)
        n = torch.full((n_dst,), fanout, device="cuda") if shape == "fixed" else torch.randint(0, 33, (n_dst * fanout // 15 + 1,), device="cuda", generator=gen)
        col = torch.arange(n.numel(), device="cuda").repeat_interleave(n)
        if shape == "none":
            col = col[torch.randperm(col.numel(), device="cuda", generator=gen)]
        row = torch.randint(0, n_src, (col.numel(),), device="cuda", generator=gen)
        rows.append(row), cols.append(col)
        parts.append(parts[-1] + col.numel()), dst.append(dst[-1] + n.numel()), src.append(src[-1] + n_src)
    row, col = torch.cat(rows), torch.cat(cols)
    x = torch.randint(-3, 4, (src[-1], D), device="cuda", generator=gen).to(dtype)
    at = torch.cat([c + o for c, o in zip(cols, dst)])
    of = torch.cat([r + o for r, o in zip(rows, src)])
    total = dst[-1] + further
    mode = _mode(col, *(torch.tensor(v, device="cuda") for v in (parts, src, dst)))
    assert col.numel() >= edges and mode == {"fixed": 0, "ragged": 1, "none": 2}[shape]
    want = torch.zeros((total, D), device="cuda", dtype=torch.float64).index_add_(0, at, x.double()[of]).to(dtype)
    dev = lambda v: torch.tensor(v, device="cuda")
    got = ops.spmm_copy_u_sum(row, col, x, dev(parts), dev(src), dev(dst + [total] if further else dst))
    assert torch.equal(got, want)


@pytest.mark.parametrize("dtype,D", [(torch.float32, 72), (torch.bfloat16, 256), (torch.float32, 256)])
@pytest.mark.parametrize("shape,edges", [("fixed", 700_000), ("ragged", 700_000), ("hub", 100_000)])
def test_waits_that_run_out_leave_zeros(dtype, D, shape, edges):
    # 16-byte copies and bulk copies; in the counting sort's order a row of thousands of stretches, all of which have to be done
    gen = torch.Generator(device="cuda").manual_seed(D)
    n = _lengths(shape, edges, gen)
    if shape == "hub":
        n[1] += max(0, edges - int(n.sum()))
    col = torch.arange(n.numel(), device="cuda").repeat_interleave(n)
    if shape == "hub":
        col = col[torch.randperm(col.numel(), device="cuda", generator=gen)]
    row = torch.randint(0, N_IN, (col.numel(),), device="cuda", generator=gen)
    x = torch.ones((N_IN, D), device="cuda", dtype=dtype)
    off = [torch.tensor([0, k], device="cuda") for k in (col.numel(), N_IN, n.numel())]
    check(lib.apt_set_tunable(b"bulk_wait_polls", 0))
    try:
        y = ops.spmm_copy_u_sum(row, col, x, *off)
        torch.cuda.synchronize()
        assert not bool(y.any())
        with pytest.raises(RuntimeError, match="did not reach shared memory"):
            ops.check_status()
    finally:
        check(lib.apt_set_tunable(b"bulk_wait_polls", 1 << 20))
    y = ops.spmm_copy_u_sum(row, col, x, *off)
    assert torch.equal(y[:, 0], n.to(dtype))
    ops.check_status()
