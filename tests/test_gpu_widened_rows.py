"""Sums over rows that are no whole number of 16-byte slices, whose input is laid out anew first (csrc/widen.cuh): the lines of
the rule, the ends of rows and of tiles, and an input that starts and ends anywhere."""
import pytest
import torch

from apt_b200 import ops
from apt_b200._lib import check, lib

pytestmark = pytest.mark.gpu
_EPS = {torch.float32: 2.0 ** -24, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _block(dst, src, per, ordered, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    row = torch.randint(0, src, (dst * per,), generator=g, device="cuda")
    col = torch.arange(dst, device="cuda").repeat_interleave(per)
    if not ordered:
        p = torch.randperm(dst * per, generator=g, device="cuda")
        row, col = row[p], col[p]
        col[0], col[-1] = dst - 1, 0      # (in no order, whatever the permutation)
    return row, col, g


def _expect(got, row, col, x, dst, most):
    want = torch.zeros(dst, x.shape[1], dtype=torch.float64, device="cuda").index_add_(0, col, x[row].double())
    size = torch.zeros(dst, x.shape[1], dtype=torch.float64, device="cuda").index_add_(0, col, x[row].double().abs())
    # fp32 sums of up to `most` terms in some order, and one rounding to the result's type
    bound = size * most * 2.0 ** -24 + want.abs() * _EPS[x.dtype] * 1.01 + 1e-7
    assert ((got.double() - want).abs() <= bound).all()


def _whole(shape, dtype, g, most):
    """Whole numbers, whose sums are exact in fp32: one edge more or less shows."""
    return torch.randint(-most, most + 1, shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("dim", [9, 17, 18, 31, 61, 101, 119, 137, 197, 198, 251, 255, 301, 511, 1001])
@pytest.mark.parametrize("segments", [1, 3])
def test_sums_in_no_order(dtype, dim, segments):
    # (rows of about as many edges: most widths are read as they are; with some rows of very many below)
    dst, src, per = 19_997, 9_001, 11
    parts = [_block(dst, src, per, False, 7 * dim + k) for k in range(segments)]
    x = torch.randn(segments * src, dim, generator=parts[0][2], device="cuda").to(dtype)
    off = lambda n: torch.arange(segments + 1, device="cuda") * n
    row, col = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
    got = ops.spmm_copy_u_sum(row, col, x, off(dst * per), off(src), off(dst))
    for k, (r, c, _) in enumerate(parts):
        most = int(torch.bincount(c).max()) + 40
        _expect(got[k * dst:(k + 1) * dst], r, c, x[k * src:(k + 1) * src], dst, most)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("dim", [9, 17, 18, 31, 61, 101, 119, 137, 197, 198, 251, 255, 301, 511, 1001])
@pytest.mark.parametrize("segments", [1, 3])
def test_sums_in_no_order_with_rows_of_many_edges(dtype, dim, segments):
    """Whole numbers, exactly: 220 000 edges and more drawn at u^2 of the rows go the widened way where the width does."""
    dst, src, edges = 19_997, 9_001, 219_967
    g = torch.Generator(device="cuda").manual_seed(7 * dim)
    off = lambda n: torch.arange(segments + 1, device="cuda") * n      # noqa: E731
    row = torch.randint(0, src, (segments * edges,), generator=g, device="cuda")
    u = torch.rand(segments * edges, generator=g, device="cuda", dtype=torch.float64)
    col = (u * u * dst).long().clamp_(max=dst - 1)
    x = _whole((segments * src, dim), dtype, g, 9)
    got = ops.spmm_copy_u_sum(row, col, x, off(edges), off(src), off(dst))
    part = torch.arange(segments, device="cuda").repeat_interleave(edges)
    want = torch.zeros(segments * dst, dim, dtype=torch.float64, device="cuda").index_add_(0, col + part * dst, x.double()[row + part * src])
    assert torch.equal(got, want.float().to(dtype))


@pytest.mark.parametrize("dtype,dim", [(torch.float32, 31), (torch.float32, 101), (torch.bfloat16, 17), (torch.bfloat16, 61), (torch.bfloat16, 119),
                                       (torch.float16, 251), (torch.float32, 251), (torch.float16, 601)])
def test_rows_that_many_edges_share(dtype, dim):
    """Rows cut into items, or into stretches of several warps: their parts meet in scratch."""
    dst, src, per = 30_011, 9_001, 8
    row, col, g = _block(dst, src, per, False, dim)
    hub = torch.rand(dst * per, generator=g, device="cuda")
    col[hub < 0.2], col[(hub > 0.2) & (hub < 0.21)] = 5, 29_000
    x = torch.randn(src, dim, generator=g, device="cuda").to(dtype)
    off = lambda n: torch.tensor([0, n], device="cuda")
    got = ops.spmm_copy_u_sum(row, col, x, off(dst * per), off(src), off(dst))
    _expect(got, row, col, x, dst, 4096)      # sums of sums: no term goes through more additions than that


@pytest.mark.parametrize("heads,head_dim", [(4, 47), (1, 33), (8, 17)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_attention_gradients_of_sources_that_many_edges_share(dtype, heads, head_dim):
    dst, src, per = 30_011, 20_001, 15
    row, col, g = _block(dst, src, per, True, head_dim)
    hub = torch.rand(dst * per, generator=g, device="cuda")
    row[hub < 0.2], row[(hub > 0.2) & (hub < 0.21)] = 7, 19_000
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(dtype)
    ft, el, er, grad = normal(src, heads, head_dim), normal(src, heads, 1), normal(dst, heads, 1), normal(dst, heads, head_dim)
    leaves = [t.requires_grad_() for t in (ft, el, er)]
    out = ops.GATEdgeSoftmaxSum.apply(row, col, *leaves, dst, 0.2)
    got = torch.autograd.grad(out, leaves, grad)[0].double()
    score = torch.nn.functional.leaky_relu(el.detach().double()[row, :, 0] + er.detach().double()[col, :, 0], 0.2).view(dst, per, heads)
    weight = torch.softmax(score, 1).view(-1, heads, 1)
    zeros = torch.zeros(src, heads, head_dim, dtype=torch.float64, device="cuda")
    want = zeros.index_add(0, row, weight * grad.double()[col])
    size = zeros.index_add(0, row, weight * grad.double()[col].abs())
    # weights within a few 2^-24 of themselves (an exponential, a sum of 15 and a quotient, from fp32 scores of up to 8), fp32 sums of up to 4096
    # additions a term, one rounding
    assert ((got - want).abs() <= size * (4096 + 64) * 2.0 ** -24 + want.abs() * _EPS[dtype] * 1.01 + 1e-7).all()


@pytest.mark.parametrize("dim", [17, 31, 61, 119, 251, 257])
@pytest.mark.parametrize("ragged", [False, True])
def test_sums_of_grouped_edges(dim, ragged):
    dst, src, per = 40_001, 90_000, 10
    row, col, g = _block(dst, src, per, True, dim)
    if ragged:
        keep = torch.rand(dst * per, generator=g, device="cuda") < 0.99
        row, col = row[keep], col[keep]
    x = torch.randn(src, dim, generator=g, device="cuda").to(torch.bfloat16)
    off = lambda n: torch.tensor([0, n], device="cuda")
    got = ops.spmm_copy_u_sum(row, col, x, off(row.numel()), off(src), off(dst))
    _expect(got, row, col, x, dst, 2 * per)


@pytest.mark.parametrize("dtype,dim", [(torch.float32, 101), (torch.bfloat16, 61), (torch.float16, 251), (torch.bfloat16, 255)])
@pytest.mark.parametrize("first", [0, 1, 2, 3, 5, 7])
def test_input_anywhere_is_read_within_its_ends(dtype, dim, first):
    """What lies around the input (NaN) is not part of any sum, and the result ends where it ends."""
    dst, src, per = 10_007, 1_003, 10
    row, col, g = _block(dst, src, per, False, first)
    room = torch.full((first + src * dim + 64,), float("nan"), dtype=dtype, device="cuda")
    x = room[first:first + src * dim].view(src, dim)
    x.copy_(torch.randn(src, dim, generator=g, device="cuda"))
    off = lambda n: torch.tensor([0, n], device="cuda")
    e, d, s = off(dst * per), off(dst), off(src)
    code = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}[dtype]
    wide = lib.apt_spmm_widened_bytes(code, dst * per, src, dim, 2)
    assert wide >= src * dim * x.element_size()
    ws_bytes = lib.apt_spmm_workspace_bytes(dst, dst * per)
    buf, ws = torch.empty(wide, dtype=torch.uint8, device="cuda"), torch.empty(ws_bytes, dtype=torch.uint8, device="cuda")
    out = torch.full((first + dst * dim + 64,), 7.0, dtype=dtype, device="cuda")
    at = out.data_ptr() + first * x.element_size()
    run = lambda size: lib.apt_spmm_copy_u_widened(code, row.data_ptr(), col.data_ptr(), dst * per, x.data_ptr(), src, dim, e.data_ptr(), s.data_ptr(),
                                                   d.data_ptr(), 1, dst, 2, 0, at, buf.data_ptr(), size, ws.data_ptr(), ws_bytes,
                                                   torch.cuda.current_stream().cuda_stream)
    check(run(wide))
    got = out[first:first + dst * dim].view(dst, dim)
    _expect(got, row, col, x, dst, int(torch.bincount(col).max()) + 40)
    assert (out[:first] == 7.0).all() and (out[first + dst * dim:] == 7.0).all()
    assert run(wide - 1) != 0      # a buffer that is too small is refused


def test_rows_that_stay_as_they_are():
    bytes_of = lib.apt_spmm_widened_bytes
    assert bytes_of(1, 1_000_000, 67_000, 256, 2) == 0          # whole slices
    assert bytes_of(1, 90_000, 8_000, 101, 2) == 0              # few edges
    assert bytes_of(1, 1_000_000, 400_000, 101, 2) == 0         # input rows that few edges read
    assert bytes_of(1, 1_000_000, 150_000, 102, 1) == 0         # grouped, read four bytes a lane
    assert bytes_of(1, 1_000_000, 67_000, 101, -1) == 0         # unknown block
    assert bytes_of(1, 1_000_000, 67_000, 101, 2) == 67_000 * 208


def test_rows_that_all_have_as_many_edges_stay_as_they_are():
    """Mode 3: in no order, and no row with very many of the edges."""
    bytes_of = lib.apt_spmm_widened_bytes
    assert bytes_of(1, 390_000, 20_000, 251, 3) == 0 and bytes_of(0, 900_000, 20_000, 137, 3) == 0 and bytes_of(0, 400_000, 20_000, 101, 3) == 0
    assert bytes_of(1, 1_000_000, 67_000, 101, 3) == 0 and bytes_of(1, 1_000_000, 67_000, 198, 3) == 0
    assert bytes_of(1, 1_000_000, 200_000, 251, 3) == 0 and bytes_of(0, 1_000_000, 67_000, 602, 3) == 0
    assert bytes_of(1, 400_000, 40_000, 251, 3) == 40_000 * 512 and bytes_of(0, 1_000_000, 67_000, 137, 3) == 67_000 * 560
    # with such rows, but a copy that takes longer than it gives
    assert bytes_of(0, 1_000_000, 300_000, 602, 2) == 0 and bytes_of(0, 150_000, 9_000, 31, 2) == 0 and bytes_of(1, 100_000, 9_000, 17, 2) == 0


def test_copies_are_of_bounded_size():
    edges = 200_000_000
    assert lib.apt_spmm_widened_bytes(1, edges, 8_388_608, 251, 2) == 4 << 30 and lib.apt_spmm_widened_bytes(1, edges, 8_388_609, 251, 2) == 0
    assert lib.apt_gat_widened_bytes(1, edges, 11_184_810, 0, 4, 47) > 0 and lib.apt_gat_widened_bytes(1, edges, 11_184_811, 0, 4, 47) == 0


def test_attention_over_sources_that_few_edges_read_stays_as_it_is():
    bytes_of = lib.apt_gat_widened_bytes
    assert bytes_of(1, 200_000, 180_000, 0, 2, 127) == 0 and bytes_of(1, 200_000, 100_000, 0, 2, 127) > 0      # forward
    assert bytes_of(1, 200_000, 180_000, 20_000, 2, 127) > 0                                                     # backward
    assert bytes_of(0, 240_000, 72_000, 60_000, 1, 47) == 0 and bytes_of(0, 240_000, 60_000, 60_000, 1, 47) > 0
    assert bytes_of(0, 900_000, 270_000, 60_000, 1, 47) > 0


@pytest.mark.parametrize("edges", [98_304, 100_003, 606_208, 606_241, 1_500_001])
@pytest.mark.parametrize("rows", [40, 5_003, 20_000])
@pytest.mark.parametrize("segments", [1, 4])
@pytest.mark.parametrize("drawn", ["alike", "u^2", "u^3", "one row", "grouped"])
def test_rows_with_very_many_of_the_edges_are_seen(edges, rows, segments, drawn):
    import ctypes

    g = torch.Generator(device="cuda").manual_seed(edges + rows)
    u = torch.rand(edges, generator=g, device="cuda", dtype=torch.float64)
    col = (u.pow({"u^2": 2, "u^3": 3}.get(drawn, 1)) * rows).long().clamp_(max=rows - 1)
    if drawn == "one row":
        col[torch.rand(edges, generator=g, device="cuda") < 0.1] = rows // 2
    cut = [edges * k // segments for k in range(segments + 1)]
    if drawn == "grouped":
        for a, b in zip(cut, cut[1:]):
            col[a:b] = col[a:b].sort()[0]
    off, out = torch.tensor(cut, device="cuda"), torch.arange(segments + 1, device="cuda") * rows
    got, old = (ctypes.c_int64 * 4)(), (ctypes.c_int64 * 3)()
    for want_hubs in (1, 0):
        check(lib.apt_spmm_probe_rows(col.data_ptr(), edges, off.data_ptr(), out.data_ptr(), segments, want_hubs, got, None))
        check(lib.apt_spmm_probe(col.data_ptr(), edges, off.data_ptr(), out.data_ptr(), segments, old, None))
        assert list(got)[:3] == list(old)
        many = drawn != "grouped" and (edges // 128 >= rows * segments or drawn in ("u^2", "u^3") or (drawn == "one row" and rows > 200))
        if drawn == "grouped":
            assert got[1] in (1, 2)
        else:
            # (what 40 rows' drawn differences come to is left open)
            assert got[1] == 2 and (rows == 40 and drawn != "alike" or got[3] == (many and want_hubs))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,head_dim", [(4, 47), (1, 47), (8, 10), (4, 10), (3, 33), (2, 255), (1, 601), (9, 18), (17, 9)])
def test_attention_of_heads_that_are_no_whole_slices(dtype, heads, head_dim):
    """Against the same heads with columns of zeros behind them, which are read as they are."""
    dst, src, per = 20_003, 60_001, 14
    row, col, g = _block(dst, src, per, True, head_dim)
    keep = torch.rand(dst * per, generator=g, device="cuda") < 0.95
    row, col = row[keep], col[keep]
    code = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}[dtype]
    size = heads * head_dim * dtype.itemsize
    if head_dim % 2:
        assert (lib.apt_gat_widened_bytes(code, row.numel(), src, dst, heads, head_dim) > 0) == (row.numel() * size >= 32 << 20 and size <= 4096)
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(dtype)
    ft, el, er, grad = normal(src, heads, head_dim), normal(src, heads, 1), normal(dst, heads, 1), normal(dst, heads, head_dim)
    per_slice = 16 // dtype.itemsize
    more = -head_dim % per_slice
    pad = lambda x: torch.nn.functional.pad(x, (0, more)).contiguous()

    def layer(ft, grad):
        leaves = [ft.detach().requires_grad_(), el.detach().requires_grad_(), er.detach().requires_grad_()]
        out = ops.GATEdgeSoftmaxSum.apply(row, col, *leaves, dst, 0.2)
        return (out.detach(),) + torch.autograd.grad(out, leaves, grad)

    got, want = layer(ft, grad), layer(pad(ft), pad(grad))
    want = (want[0][..., :head_dim], want[1][..., :head_dim], want[2], want[3])
    for a, b in zip(got, want):
        assert a.shape == b.shape and torch.isfinite(a).all()
        # the same terms in another order: fp32 sums a few 2^-24 of their terms apart, and then at most one rounding further
        a, b = a.double(), b.double()
        assert ((a - b).abs() <= 2 * _EPS[dtype] * b.abs() + 2e-5 * b.abs().max()).all()


# ---- every edge once
@pytest.mark.parametrize("dtype,dim", [(torch.float32, 31), (torch.float32, 101), (torch.bfloat16, 17), (torch.bfloat16, 61), (torch.float16, 251), (torch.float32, 251),
                                       (torch.float16, 601)])
@pytest.mark.parametrize("edges", [240_088, 1_000_003])
def test_every_edge_of_a_shared_row_counts_once(dtype, dim, edges):
    dst, src = 30_011, 9_001
    g = torch.Generator(device="cuda").manual_seed(dim)
    row, col = torch.randint(0, src, (edges,), generator=g, device="cuda"), torch.randint(0, dst, (edges,), generator=g, device="cuda")
    hub = torch.rand(edges, generator=g, device="cuda")
    col[hub < 0.2], col[(hub > 0.2) & (hub < 0.21)] = 5, 29_000
    x = _whole((src, dim), dtype, g, 9)
    off = lambda n: torch.tensor([0, n], device="cuda")      # noqa: E731
    got = ops.spmm_copy_u_sum(row, col, x, off(edges), off(src), off(dst))
    want = torch.zeros(dst, dim, dtype=torch.float64, device="cuda").index_add_(0, col, x[row].double())
    assert want.abs().max() < 2 ** 24 and torch.equal(got, want.float().to(dtype))      # (one rounding to the result's type)


@pytest.mark.parametrize("heads,head_dim", [(4, 47), (1, 33), (8, 17), (1, 31), (4, 63), (2, 127)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_every_edge_of_a_shared_source_counts_once(dtype, heads, head_dim):
    """Equal scores and 16 edges to a destination: weights of 1/16, which whole numbers keep exact."""
    dst, src, per = 30_011, 20_001, 16
    row, col, g = _block(dst, src, per, True, head_dim)
    hub = torch.rand(dst * per, generator=g, device="cuda")
    row[hub < 0.2], row[(hub > 0.2) & (hub < 0.21)] = 7, 19_000
    ft, grad = _whole((src, heads, head_dim), dtype, g, 9), _whole((dst, heads, head_dim), dtype, g, 9)
    el, er = torch.ones(src, heads, 1, dtype=dtype, device="cuda"), torch.ones(dst, heads, 1, dtype=dtype, device="cuda")
    leaves = [t.requires_grad_() for t in (ft, el, er)]
    out = ops.GATEdgeSoftmaxSum.apply(row, col, *leaves, dst, 0.2)
    got = torch.autograd.grad(out, leaves, grad)[0]
    zeros = lambda n: torch.zeros(n, heads, head_dim, dtype=torch.float64, device="cuda")      # noqa: E731
    want = zeros(src).index_add(0, row, grad.double()[col] / 16)
    assert want.abs().max() < 2 ** 20 and torch.equal(got, want.float().to(dtype))
    assert torch.equal(out.detach(), (zeros(dst).index_add(0, col, ft.detach().double()[row]) / 16).float().to(dtype))


@pytest.mark.parametrize("heads,head_dim", [(1, 31), (4, 31), (2, 63), (4, 63), (2, 127)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_widened_heads_that_the_tensor_cores_take(dtype, heads, head_dim):
    """Heads whose widened rows are those of k_gat_dots_mma, against the same with a column of zeros."""
    per, src = 15, 30_001
    dst = max((32 << 20) // (per * heads * head_dim * 2), 98_304 // per) + 101      # the bytes and the edges from which on rows are widened
    row, col, g = _block(dst, src, per, True, head_dim)
    code = {torch.bfloat16: 1, torch.float16: 2}[dtype]
    assert lib.apt_gat_widened_bytes(code, dst * per, src, dst, heads, head_dim) > 0
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(dtype)      # noqa: E731
    ft, el, er, grad = normal(src, heads, head_dim), normal(src, heads, 1), normal(dst, heads, 1), normal(dst, heads, head_dim)
    pad = lambda x: torch.nn.functional.pad(x, (0, 1)).contiguous()      # noqa: E731

    def gradients(ft, grad):
        leaves = [t.detach().requires_grad_() for t in (ft, el, er)]
        return torch.autograd.grad(ops.GATEdgeSoftmaxSum.apply(row, col, *leaves, dst, 0.2), leaves, grad)

    for k, (a, b) in enumerate(zip(gradients(ft, grad), gradients(pad(ft), pad(grad)))):
        a, b = a.double(), b[..., :head_dim].double() if k == 0 else b.double()
        # the same products; sums in no order (sources) a few 2^-24 of their terms apart, and a rounding further
        assert ((a - b).abs() <= 2 * _EPS[dtype] * b.abs() + 2e-5 * b.abs().max()).all(), k


def test_widened_attention_in_a_captured_graph():
    dst, src, per, heads, head_dim = 20_003, 30_001, 15, 4, 47
    row, col, g = _block(dst, src, per, True, 3)
    ft, grad = (_whole((n, heads, head_dim), torch.bfloat16, g, 3) for n in (src, dst))
    el, er = (torch.randn(n, heads, 1, generator=g, device="cuda").bfloat16() for n in (src, dst))
    assert lib.apt_gat_widened_bytes(1, dst * per, src, 0, heads, head_dim) > 0

    def layer():
        out = ops.gat_edge_softmax_sum(row, col, ft, el, er, dst)
        return (out,) + tuple(ops.gat_edge_softmax_sum_backward(row, col, ft, el, er, grad, 0.2))

    want = [t.double() for t in layer()]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        layer()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = layer()
    for fill in (0.0, float("nan")):      # what the results held before is not part of them
        for t in got:
            t.fill_(fill)
        graph.replay()
        for a, b in zip(got, want):
            assert ((a.double() - b).abs() <= 2 * _EPS[torch.bfloat16] * b.abs() + 2e-5 * b.abs().max()).all()


def test_sums_without_room_for_the_copy():
    dst, src, edges, dim = 10_007, 500_003, 1_700_003, 251
    g = torch.Generator(device="cuda").manual_seed(2)
    row, col = torch.randint(0, src, (edges,), generator=g, device="cuda"), torch.randint(0, dst, (edges,), generator=g, device="cuda")
    x = _whole((src, dim), torch.bfloat16, g, 3)
    off = [torch.tensor([0, n], device="cuda") for n in (edges, src, dst)]
    need = lib.apt_spmm_widened_bytes(1, edges, src, dim, 2)
    assert need >= src * 512
    want = ops.spmm_copy_u_sum(row, col, x, *off)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total, before = torch.cuda.get_device_properties(0).total_memory, torch.cuda.memory_stats().get("num_ooms", 0)
    kept = torch.cuda.memory_reserved()
    torch.cuda.set_per_process_memory_fraction((kept + need * 3 // 4) / total)
    try:
        got = ops.spmm_copy_u_sum(row, col, x, *off)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.cuda.memory_stats().get("num_ooms", 0) > before and torch.equal(got, want)      # (whole numbers: exact in any order)
