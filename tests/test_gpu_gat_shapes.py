"""The attention block at the edges of its kernels (destinations of more edges than a thread keeps in registers or a
warp reads at once, more heads than lanes, head widths of every slice size and beyond one block of lanes, ragged and
empty destinations), the edge-part entry points of the C ABI and the backward that starts from what the forward saved,
against the fp64 oracle. Bounds as in test_gpu_gat.py: the sums of at most a few hundred fp32 terms within 1e-5 of the
largest value, 16-bit results within 1e-2."""
import ctypes

import numpy as np
import pytest
import torch

import apt_b200
from apt_b200 import _lib, ops
from apt_b200._lib import check, lib
from oracle import oracle as orc
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu
I64 = np.int64
TOL = {torch.float32: 1e-5, torch.bfloat16: 1e-2, torch.float16: 1e-2}
CODE = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16, torch.float16: _lib.F16}


def _round(x, dtype):
    return torch.from_numpy(x).to(dtype).float().numpy() if dtype != torch.float32 else x


def _inputs(lengths, H, Dh, dtype, seed):
    rng = np.random.default_rng(seed)
    S, E, n_src = len(lengths), int(sum(lengths)), 40
    col = np.repeat(np.arange(S), lengths).astype(I64)
    row = rng.integers(0, n_src, E).astype(I64)
    make = lambda *shape: _round(rng.standard_normal(shape).astype(np.float32), dtype)
    return row, col, make(n_src, H, Dh), make(n_src, H), make(S, H), make(S, H, Dh)


def _near(got, want, dtype, name):
    err = np.abs(host(got).astype(np.float64).reshape(want.shape) - want).max() / max(np.abs(want).max(), 1.0)
    assert err <= TOL[dtype], f"{name}: {err:.2e}"


RAGGED = [0, 1, 15, 16, 17, 0, 31, 32, 33, 64, 65, 130, 2, 0]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,Dh", [(1, 1), (4, 64), (3, 5), (8, 47), (9, 8), (33, 4), (1, 300), (2, 1030)])
@pytest.mark.parametrize("lengths", [[7] * 9, RAGGED], ids=["fixed", "ragged"])
def test_forward_and_backward(dtype, H, Dh, lengths):
    row, col, ft, el, er, go = _inputs(lengths, H, Dh, dtype, H * 100 + Dh)
    S = len(lengths)
    args = dev(row), dev(col), dev(ft, dtype), dev(el, dtype), dev(er, dtype)
    out, attn = ops.gat_edge_softmax_sum(*args, S, 0.2, return_attention=True)
    want, want_a = orc.gat_edge_softmax_sum(row, col, ft, el, er, S, 0.2)
    _near(out, want, dtype, "out")
    _near(attn, want_a, dtype, "attention")
    g_want = orc.gat_edge_softmax_sum_backward(row, col, ft, el, er, go, S, 0.2)[:3]
    for got, w, name in zip(ops.gat_edge_softmax_sum_backward(*args, dev(go, dtype), 0.2), g_want, ("ft", "el", "er")):
        _near(got, w, dtype, "grad_" + name)
    # through autograd the backward starts from the ranges and weights the forward left
    leaves = [t.requires_grad_() for t in args[2:]]
    y = apt_b200.GATEdgeSoftmaxSum.apply(args[0], args[1], *leaves, S, 0.2)
    for got, w, name in zip(torch.autograd.grad(y, leaves, dev(go, dtype)), g_want, ("ft", "el", "er")):
        _near(got, w, dtype, "autograd grad_" + name)
    ops.check_status()


def _pool_reserved():
    """Most bytes the device's stream-ordered memory pool has held so far."""
    rt = ctypes.CDLL("libcudart.so.12")            # the one PyTorch has loaded
    pool, most = ctypes.c_void_p(), ctypes.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 6, ctypes.byref(most)) == 0      # cudaMemPoolAttrReservedMemHigh
    return most.value


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,Dh", [(1, 1), (4, 16), (4, 64), (3, 5), (9, 8), (33, 4), (1, 300), (2, 1030)])
@pytest.mark.parametrize("captured", [False, True], ids=["direct", "captured"])
def test_edge_part_entry_points(dtype, H, Dh, captured):
    # they work in a few words a destination, allocate nothing and may be captured
    row, col, ft, el, er, go = _inputs(RAGGED, H, Dh, dtype, 1)
    S, E = len(RAGGED), len(row)
    t = [dev(row), dev(col)] + [dev(x, dtype) for x in (ft, el, er, go)]
    p = [x.data_ptr() for x in t]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, attn, attn_b, gs, ger = (torch.full(shape, 9.0, device="cuda", dtype=dtype)
                                  for shape in ((S, H, Dh), (E, H), (E, H), (E, H), (S, H)))
    nbytes = lib.apt_spmm_workspace_bytes(S, 0)
    room = torch.full((nbytes + 512,), 77, dtype=torch.uint8, device="cuda")
    ws = room[:nbytes]
    before = _pool_reserved()

    def call():
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        check(lib.apt_gat_edge_softmax_sum(CODE[dtype], p[0], p[1], E, p[2], p[3], p[4], H, Dh, 0.2, S, out.data_ptr(),
                                           attn.data_ptr(), ws.data_ptr(), nbytes, status.data_ptr(), stream))
        check(lib.apt_gat_edge_backward(CODE[dtype], p[0], p[1], E, p[2], p[3], p[4], p[5], H, Dh, 0.2, S, attn_b.data_ptr(),
                                        gs.data_ptr(), ger.data_ptr(), ws.data_ptr(), nbytes, status.data_ptr(), stream))

    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call()
        for _ in range(2):
            graph.replay()
    else:
        call()
    torch.cuda.synchronize()
    assert _pool_reserved() == before and bool((room[nbytes:] == 77).all())
    want, _ = orc.gat_edge_softmax_sum(row, col, ft, el, er, S, 0.2)
    _, _, w_er, w_attn, w_gs = orc.gat_edge_softmax_sum_backward(row, col, ft, el, er, go, S, 0.2)
    for got, w, name in ((out, want, "out"), (attn, w_attn, "attention"), (attn_b, w_attn, "attention of the backward"),
                         (gs, w_gs, "score gradient"), (ger, w_er, "grad_er")):
        _near(got, np.asarray(w).reshape(got.shape), dtype, name)
    assert int(status[0]) == 0
    st = lib.apt_gat_edge_softmax_sum(CODE[dtype], p[0], p[1], E, p[2], p[3], p[4], H, Dh, 0.2, S, out.data_ptr(), None, None, 0,
                                      status.data_ptr(), None)
    assert st == _lib.APT_ERR_BAD_ARG
    st = lib.apt_gat_edge_backward(CODE[dtype], p[0], p[1], E, p[2], p[3], p[4], p[5], H, Dh, 0.2, S, attn.data_ptr(), gs.data_ptr(),
                                   ger.data_ptr(), ws.data_ptr(), nbytes - 1, status.data_ptr(), None)
    assert st == _lib.APT_ERR_CAPACITY


def test_edge_part_of_ungrouped_edges():
    dtype, H, Dh = torch.float32, 2, 8
    row, col, ft, el, er, go = _inputs([3, 0, 4], H, Dh, dtype, 1)
    col = col[::-1].copy()
    t = [dev(x) for x in (row, col, ft, el, er, go)]
    p = [x.data_ptr() for x in t]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, attn, gs, ger = (torch.full(shape, 9.0, device="cuda") for shape in ((3, H, Dh), (7, H), (7, H), (3, H)))
    nbytes = lib.apt_spmm_workspace_bytes(3, 0)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    check(lib.apt_gat_edge_softmax_sum(_lib.F32, p[0], p[1], 7, p[2], p[3], p[4], H, Dh, 0.2, 3, out.data_ptr(), None, ws.data_ptr(),
                                       nbytes, status.data_ptr(), None))
    check(lib.apt_gat_edge_backward(_lib.F32, p[0], p[1], 7, p[2], p[3], p[4], p[5], H, Dh, 0.2, 3, attn.data_ptr(), gs.data_ptr(),
                                    ger.data_ptr(), ws.data_ptr(), nbytes, status.data_ptr(), None))
    torch.cuda.synchronize()
    assert not any(bool(x.any()) for x in (out, attn, gs, ger)) and int(status[0]) == _lib.FLAG_NOT_GROUPED


def test_ungrouped_backward_is_zero_and_flagged():
    col = np.array([1, 0, 1, 1], dtype=I64)
    row = np.array([0, 1, 2, 0], dtype=I64)
    ft, one = torch.ones((3, 2, 8), device="cuda"), torch.ones((3, 2), device="cuda")
    grads = ops.gat_edge_softmax_sum_backward(dev(row), dev(col), ft, one, one[:2], torch.ones((2, 2, 8), device="cuda"))
    torch.cuda.synchronize()
    assert not any(host(g).any() for g in grads)
    with pytest.raises(RuntimeError, match="not grouped"):
        ops.check_status()


@pytest.mark.parametrize("dtype,H,Dh", [(torch.float32, 4, 64), (torch.float32, 3, 44), (torch.float32, 16, 16),
                                        (torch.float32, 17, 12), (torch.bfloat16, 4, 128), (torch.float16, 1, 272)])
def test_source_rows_of_many_edges(dtype, H, Dh):
    # enough edges of rows above 512 bytes for the copies through shared memory: hubs, short rows and rows without edges
    gen = torch.Generator(device="cuda").manual_seed(H)
    S, n_src = 14_001, 20_003
    lengths = torch.randint(0, 31, (S,), device="cuda", generator=gen)
    col = torch.repeat_interleave(torch.arange(S, device="cuda"), lengths)
    u = torch.rand(col.numel(), device="cuda", generator=gen, dtype=torch.float64)
    row = (u ** 3 * n_src).long()
    rand = lambda *shape: torch.randn(shape, device="cuda", generator=gen).to(dtype)
    ft, el, er, go = rand(n_src, H, Dh), rand(n_src, H, 1), rand(S, H, 1), rand(S, H, Dh)
    assert col.numel() >= 200_000
    got = ops.gat_edge_softmax_sum_backward(row, col, ft, el, er, go, 0.2)
    # the formulas in fp64, from the rounded inputs, and for every sum the sum of its terms' magnitudes
    raw = el.double()[row] + er.double()[col]
    s = torch.where(raw > 0, raw, raw * 0.2)[:, :, 0]
    index = col[:, None].expand(-1, H)
    most = torch.full((S, H), -torch.inf, device="cuda", dtype=torch.float64).scatter_reduce_(0, index, s, "amax")
    p = (s - most[col]).exp()
    total = lambda at, rows, x: torch.zeros((rows, *x.shape[1:]), device="cuda", dtype=torch.float64).index_add_(0, at, x)
    attn = p / total(col, S, p)[col]
    g = go.double()[col]
    dot, dot_size = (g * ft.double()[row]).sum(-1), (g * ft.double()[row]).abs().sum(-1)
    factor = attn * torch.where(raw > 0, 1.0, 0.2)[:, :, 0]
    gs = factor * (dot - total(col, S, attn * dot)[col])
    gs_size = factor * (dot_size + total(col, S, attn * dot_size)[col])
    # fp32: rows of up to a few thousand terms, weights and dots of their own rounding: 1e-5 of the magnitudes, as for all sums
    # here. 16 bits: the result's own rounding (2^-9 and 2^-12 of the value) beside that.
    unit = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    for name, x, want, size in (("grad_ft", got[0], total(row, n_src, attn[:, :, None] * g), total(row, n_src, (attn[:, :, None] * g).abs())),
                                ("grad_el", got[1][:, :, 0], total(row, n_src, gs), total(row, n_src, gs_size)),
                                ("grad_er", got[2][:, :, 0], total(col, S, gs), total(col, S, gs_size))):
        over = (x.double() - want).abs() - (1e-5 * size + unit * want.abs() + 1e-7)
        assert float(over.max()) <= 0, f"{name}: {float(over.max()):.2e} beyond the bound"


def test_what_the_forward_saved_goes_with_the_backward():
    S, f, H, Dh = 20_000, 10, 8, 16
    row = torch.randint(0, S, (S * f,), device="cuda")
    col = torch.arange(S, device="cuda").repeat_interleave(f)
    leaves = [torch.randn(shape, device="cuda", requires_grad=True) for shape in ((S, H, Dh), (S, H, 1), (S, H, 1))]
    go = torch.randn((S, H, Dh), device="cuda")
    want = torch.autograd.grad(apt_b200.GATEdgeSoftmaxSum.apply(row, col, *leaves, S, 0.2), leaves, go)
    saved = S * f * H * 4
    out = apt_b200.GATEdgeSoftmaxSum.apply(row, col, *leaves, S, 0.2)
    before = torch.cuda.memory_allocated()
    grads = torch.autograd.grad(out, leaves, go)
    held = sum(g.numel() * 4 for g in grads)
    assert torch.cuda.memory_allocated() <= before + held - saved + (1 << 20)        # `out` and its graph are still there
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(out, leaves, go)
    # and to wherever a caller's hooks put what is saved
    with torch.autograd.graph.save_on_cpu():
        base = torch.cuda.memory_allocated()
        out = apt_b200.GATEdgeSoftmaxSum.apply(row, col, *leaves, S, 0.2)
        assert torch.cuda.memory_allocated() <= base + out.numel() * 4 + (1 << 20)
    for a, b in zip(torch.autograd.grad(out, leaves, go), want):
        assert (a - b).abs().max() <= 1e-5 * b.abs().max()


@pytest.mark.parametrize("H,Dh", [(1, 47), (3, 5), (2, 40), (1, 300)])
def test_infinite_rows_stay_where_they_belong(H, Dh):
    # one source's last column is infinite: its edge's gradient is not a number, the other edges' are infinite or, at other
    # destinations, what they are without it, in every head width (lanes beyond a head's last slice read that slice)
    row, col, ft, el, er, go = _inputs([4, 3, 5], H, Dh, torch.float32, 3)
    row[:] = np.arange(len(row))
    ft[1, :, -1] = np.inf
    go[:, :, -1] = 1.0
    args = [dev(x) for x in (row, col, ft, el, er)]
    g_ft, g_el, g_er = ops.gat_edge_softmax_sum_backward(*args, dev(go), 0.2)
    f, l, r, g = (torch.from_numpy(x).double() for x in (ft, el, er, go))
    rows, cols = torch.from_numpy(row), torch.from_numpy(col)
    raw = l[rows] + r[cols]
    s = torch.nn.functional.leaky_relu(raw, 0.2)
    a = torch.cat([torch.softmax(s[cols == d], 0) for d in range(3)])
    dot = (g[cols] * f[rows]).sum(-1)
    t = torch.stack([(a * dot)[cols == d].sum(0) for d in range(3)])
    gs = a * (dot - t[cols]) * torch.where(raw > 0, 1.0, 0.2)
    want = torch.zeros(l.shape, dtype=torch.float64).index_add_(0, rows, gs)
    got = g_el.cpu().double()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()) and int(want.isinf().sum()) == 3 * H
    assert torch.equal(got[got.isinf()], want[want.isinf()])
    fine = want.isfinite()
    assert bool(((got - want)[fine].abs() <= 1e-5 * want[fine].abs().max()).all()) and bool(g_ft.isfinite().all())


@pytest.mark.parametrize("dtype,H,Dh,zero", [(torch.bfloat16, 4, 64, True), (torch.float32, 8, 16, True), (torch.float32, 2, 64, True),
                                             (torch.float32, 1, 8, False), (torch.float32, 16, 16, False), (torch.bfloat16, 2, 64, False)])
@pytest.mark.parametrize("edges", [1, 15, 16, 17, 32, 33])
def test_masked_destinations(dtype, H, Dh, zero, edges):
    # every score of destination 1 is -inf: zeros up to 32 edges of wide rows, NaN elsewhere, and nothing for its neighbours
    row, col, ft, el, er, go = _inputs([5, edges, 4], H, Dh, dtype, 5)
    row[:] = np.arange(len(row)) % 9
    row[5:5 + edges] = 9 + np.arange(edges) % 31
    el[9:] = -np.inf
    leaves = [dev(x, dtype).requires_grad_() for x in (ft, el, er)]
    out = apt_b200.GATEdgeSoftmaxSum.apply(dev(row), dev(col), *leaves, 3, 0.2)
    grads = torch.autograd.grad(out, leaves, dev(go, dtype))
    zero = zero and edges <= 32
    masked = out[1].float()
    assert not bool(masked.any()) if zero else bool(masked.isnan().all())
    assert bool(out[0::2].isfinite().all()) and bool(out[0::2].any())
    assert bool(grads[0][:9].isfinite().all()) and bool(grads[1][:9].isfinite().all()) and bool(grads[2][0::2].isfinite().all())
    if zero:
        assert not bool(grads[0][9:].any()) and not bool(grads[2][1].any())
    # the entry points without a buffer agree
    t = [x.detach() for x in (dev(row), dev(col), *leaves)]
    alone = torch.full((3, H, Dh), 9.0, device="cuda", dtype=dtype)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    nbytes = lib.apt_spmm_workspace_bytes(3, 0)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    check(lib.apt_gat_edge_softmax_sum(CODE[dtype], *(x.data_ptr() for x in t[:2]), len(row), *(x.data_ptr() for x in t[2:]), H, Dh, 0.2, 3,
                                       alone.data_ptr(), None, ws.data_ptr(), nbytes, status.data_ptr(), None))
    torch.cuda.synchronize()
    assert bool((alone[1].isnan() == out[1].isnan()).all()) and bool(((alone - out).float().nan_to_num().abs() <= 2e-2).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,Dh", [(1, 8), (2, 8), (3, 16), (8, 8), (1, 64), (16, 4), (1, 128), (2, 40)])
@pytest.mark.parametrize("lengths", [[7] * 40, RAGGED], ids=["fixed", "ragged"])
def test_forward_without_a_backward(dtype, H, Dh, lengths):
    # rows of up to 256 bytes are summed by a kernel of their own, on both sides of that bound
    row, col, ft, el, er, _ = _inputs(lengths, H, Dh, dtype, H + Dh)
    S = len(lengths)
    args = dev(row), dev(col), dev(ft, dtype), dev(el, dtype), dev(er, dtype)
    want, want_a = orc.gat_edge_softmax_sum(row, col, ft, el, er, S, 0.2)
    out, attn = ops.gat_edge_softmax_sum(*args, S, 0.2, return_attention=True)
    _near(out, want, dtype, "out")
    _near(attn, want_a, dtype, "attention")
    plain = apt_b200.GATEdgeSoftmaxSum.apply(*args, S, 0.2)
    assert torch.equal(plain, out) and not plain.requires_grad
    leaf = args[2].clone().requires_grad_()
    with torch.no_grad():
        assert torch.equal(apt_b200.GATEdgeSoftmaxSum.apply(args[0], args[1], leaf, *args[3:], S, 0.2), out)
    kept = apt_b200.GATEdgeSoftmaxSum.apply(args[0], args[1], leaf, *args[3:], S, 0.2)
    assert kept.requires_grad
    _near(kept.detach(), want, dtype, "out of a training step")
    shifted = torch.empty(args[2].numel() + 1, device="cuda", dtype=dtype)[1:].view_as(args[2])        # no 16-byte alignment
    shifted.copy_(args[2])
    _near(ops.gat_edge_softmax_sum(args[0], args[1], shifted, *args[3:], S, 0.2), want, dtype, "out of unaligned rows")
    ops.check_status()


def test_forward_mode_is_refused():
    row, col, ft, el, er, _ = _inputs([3, 4], 2, 8, torch.float32, 1)
    args = [dev(x) for x in (row, col, ft, el, er)]
    with torch.autograd.forward_ad.dual_level():
        args[2] = torch.autograd.forward_ad.make_dual(args[2], torch.ones_like(args[2]))
        with pytest.raises(Exception, match="jvp|forward"):
            apt_b200.GATEdgeSoftmaxSum.apply(*args, 2, 0.2)


@pytest.mark.parametrize("dtype,unit", [(torch.bfloat16, 2.0 ** -9), (torch.float16, 2.0 ** -12)])
@pytest.mark.parametrize("S,f,n_src,H,Dh", [(358, 24, 1541, 1, 64), (1881, 10, 9408, 4, 8), (3000, 15, 7000, 4, 64)])
def test_results_of_16_bits_are_rounded_once(dtype, unit, S, f, n_src, H, Dh):
    # weights and score gradients stay in fp32 between the kernels: outputs miss the fp64 ones by the rounding of the result
    # (at most `unit` of each value, 0.58 of that in the mean square) and not by that of anything on the way (1.4 times it and more)
    rng = np.random.default_rng(S)
    row, col = rng.integers(0, n_src, S * f).astype(I64), np.repeat(np.arange(S), f).astype(I64)
    make = lambda *shape: _round(rng.standard_normal(shape).astype(np.float32), dtype)
    ft, el, er, go = make(n_src, H, Dh), make(n_src, H), make(S, H), make(S, H, Dh)
    args = dev(row), dev(col), dev(ft, dtype), dev(el, dtype), dev(er, dtype)
    want = (orc.gat_edge_softmax_sum(row, col, ft, el, er, S, 0.2)[0],
            *orc.gat_edge_softmax_sum_backward(row, col, ft, el, er, go, S, 0.2)[:3])
    got = (ops.gat_edge_softmax_sum(*args, S, 0.2), *ops.gat_edge_softmax_sum_backward(*args, dev(go, dtype), 0.2))
    for x, w, name in zip(got, want, ("out", "grad_ft", "grad_el", "grad_er")):
        err = np.linalg.norm(host(x.float()).astype(np.float64).reshape(w.shape) - w) / np.linalg.norm(w)
        assert err <= unit, f"{name}: {err:.2e}"
