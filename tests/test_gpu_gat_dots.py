"""The attention backward's dots by tensor-core products of 16 edges with 8 destinations: every split of a row into heads that they take, groups of
edges whose destinations fill one tile of them, several, or lie far apart, stretches that end inside a group, and infinite rows, which are
nobody else's business. Against the fp64 oracle, bounds as in test_gpu_gat.py."""
import numpy as np
import pytest
import torch

from apt_b200 import ops
from oracle import oracle as orc
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu
SPLITS = [(1, 32), (2, 32), (4, 32), (8, 32), (1, 64), (2, 64), (4, 64), (1, 128), (2, 128), (1, 256)]
LENGTHS = {
    "one each": [1] * 75, "three each": [3] * 331, "fifteen each": [15] * 70, "long": [500, 1, 700, 0, 90],
    "gaps": [2, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 5, 1, 0, 0, 0, 0, 0, 0, 0, 0, 30, 0, 7] * 3, "one": [1], "sixteen": [16], "seventeen": [17],
    "a warp's": [31, 1], "and one more": [31, 2],
}


def _round(x, dtype):
    return torch.from_numpy(x).to(dtype).float().numpy()


def _inputs(lengths, H, D, dtype, n_src=90):
    rng = np.random.default_rng(H * 1000 + D + len(lengths))
    col = np.repeat(np.arange(len(lengths)), lengths).astype(np.int64)
    row = rng.integers(0, n_src, len(col)).astype(np.int64)
    make = lambda *shape: _round(rng.standard_normal(shape).astype(np.float32), dtype)      # noqa: E731
    return row, col, make(n_src, H, D), make(n_src, H), make(len(lengths), H), make(len(lengths), H, D)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,D", SPLITS)
@pytest.mark.parametrize("lengths", sorted(LENGTHS))
def test_gradients(dtype, H, D, lengths):
    n = LENGTHS[lengths]
    row, col, ft, el, er, go = _inputs(n, H, D, dtype)
    want = orc.gat_edge_softmax_sum_backward(row, col, ft, el, er, go, len(n), 0.2)[:3]
    got = ops.gat_edge_softmax_sum_backward(dev(row), dev(col), *(dev(x, dtype) for x in (ft, el, er, go)), 0.2)
    for a, b, name in zip(got, want, ("ft", "el", "er")):
        err = np.abs(host(a).astype(np.float64).reshape(b.shape) - b).max() / max(np.abs(b).max(), 1.0)
        assert err <= 1e-2, f"grad_{name}: {err:.2e}"
    ops.check_status()


def test_infinite_rows_stay_with_their_edges():
    H, D, n = 4, 64, [3] * 40
    row, col, ft, el, er, go = _inputs(n, H, D, torch.bfloat16)
    row[:] = np.arange(len(row)) % 80
    clean = [host(x) for x in ops.gat_edge_softmax_sum_backward(dev(row), dev(col), *(dev(x, torch.bfloat16) for x in (ft, el, er, go)), 0.2)]
    ft[85] = np.inf      # of no edge
    ft[7, 1] = np.inf
    got = [host(x) for x in ops.gat_edge_softmax_sum_backward(dev(row), dev(col), *(dev(x, torch.bfloat16) for x in (ft, el, er, go)), 0.2)]
    hit = np.unique(col[row == 7])
    others = np.setdiff1d(np.arange(len(n)), hit)
    er_got, er_clean = (x.reshape(len(n), H) for x in (got[2], clean[2]))
    assert np.array_equal(er_got[others], er_clean[others]) and np.array_equal(er_got[:, [0, 2, 3]], er_clean[:, [0, 2, 3]])
    assert not np.isfinite(er_got[hit, 1]).any()


def test_ids_that_have_changed_since_the_forward():
    """The ranges are the forward's; what the destinations' ids have become since is read within its ends, and the pass comes to its end."""
    H, D, n = 2, 64, [15] * 40
    row, col, ft, el, er, go = _inputs(n, H, D, torch.bfloat16)
    row, ids = dev(row), dev(col)
    leaves = [dev(x, torch.bfloat16).view(-1, H, x.size // H // len(x)).requires_grad_() for x in (ft, el, er)]
    layer = lambda: ops.GATEdgeSoftmaxSum.apply(row, ids, *leaves, len(n), 0.2)      # noqa: E731
    out, grad = layer(), dev(go, torch.bfloat16)
    want = torch.autograd.grad(out, leaves, grad, retain_graph=True)
    kept = ids.clone()
    for bad in (-1, -9, 2 ** 31 - 1, 2 ** 31, 2 ** 32 - 4, 2 ** 40 + 3, 39):
        ids.data[5::16] = bad
        torch.autograd.grad(out, leaves, grad, retain_graph=True)
        torch.cuda.synchronize()
        ids.data.copy_(kept)
    # (sums over a source's edges are in no order: two roundings to 16 bits apart, and a few 2^-24 of their terms)
    for a, b in zip(torch.autograd.grad(layer(), leaves, grad), want):
        a, b = a.double(), b.double()
        assert ((a - b).abs() <= 2.0 ** -7 * b.abs() + 2e-5 * b.abs().max()).all()
    ops.check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,D", [(2, 128), (1, 256)])
def test_dots_are_rounded_sums(dtype, H, D):
    """Two sources of a destination whose rows have the same dot with its gradient, the same products in another order, and the same score: half of each
    weight, and gradients of the scores that are a quarter of what the two computed dots differ by."""
    dst = 3000
    g = torch.Generator(device="cuda").manual_seed(D)
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(dtype)      # noqa: E731
    pairs = torch.randperm(D, generator=g, device="cuda").view(2, D // 2)
    swap = torch.empty(D, dtype=torch.int64, device="cuda")
    swap[pairs[0]], swap[pairs[1]] = pairs[1], pairs[0]
    grad = normal(dst, H, D)
    grad[..., pairs[1]] = grad[..., pairs[0]]
    ft = torch.empty(2 * dst, H, D, dtype=dtype, device="cuda")
    ft[::2] = normal(dst, H, D)
    ft[1::2] = ft[::2][..., swap]
    col = torch.arange(dst, device="cuda").repeat_interleave(2)
    el, er = torch.ones(2 * dst, H, 1, dtype=dtype, device="cuda"), torch.ones(dst, H, 1, dtype=dtype, device="cuda")
    got = ops.gat_edge_softmax_sum_backward(torch.arange(2 * dst, device="cuda"), col, ft, el, er, grad, 0.2)[1].double()
    dots = (ft[::2].double() * grad.double()).sum(-1)
    # An fp32 value is off by 2^-24 / sqrt(3) of the largest it may be, at 0.7 of that in the mean, wherever it is rounded: eight times from product to
    # sum, down a tree, by less every time, less than three such steps together, and once more for the mean of the two.
    error = 4 * got.norm() / 2 ** 0.5 / 2 ** 0.5 / dots.norm()
    assert error <= 2.0 ** -23, float(error)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,D", [(4, 32), (2, 64), (1, 256)])
@pytest.mark.parametrize("what", ["infinity", "a sum beyond fp32"])
def test_infinite_dots_are_infinite(dtype, H, D, what):
    """Four sources of a destination with the same score; the dot of one is infinite, for an infinite value or from finite ones. Its own gradient is none,
    the other three's are minus what infinity it is. All other destinations' are what they are without it."""
    dst, at = 40, 3 * D // 4 + 1
    if what != "infinity" and dtype == torch.float16:
        pytest.skip("products of 16-bit floats of this range have no such sum")
    g = torch.Generator(device="cuda").manual_seed(D)
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(dtype)      # noqa: E731
    row, col = torch.arange(4 * dst, device="cuda"), torch.arange(dst, device="cuda").repeat_interleave(4)
    ft, grad = normal(4 * dst, H, D), normal(dst, H, D)
    el, er = torch.ones(4 * dst, H, 1, dtype=dtype, device="cuda"), torch.ones(dst, H, 1, dtype=dtype, device="cuda")
    clean = ops.gat_edge_softmax_sum_backward(row, col, ft, el, er, grad, 0.2)[1].view(dst, 4, H)
    for d, sign in ((5, 1), (22, -1)):
        if what == "infinity":
            grad[d, 0, at] = 2.0
            ft[4 * d + 1, 0, at] = sign * float("inf")
        else:
            grad[d, 0, at - 1:at + 1] = 2.0 ** 100
            ft[4 * d + 1, 0, at - 1:at + 1] = sign * 2.0 ** 30
            ft[[4 * d, 4 * d + 2, 4 * d + 3], 0, at - 1:at + 1] = 0
    got = ops.gat_edge_softmax_sum_backward(row, col, ft, el, er, grad, 0.2)[1].view(dst, 4, H)
    for d, sign in ((5, 1), (22, -1)):
        assert got[d, 1, 0].isnan() and (got[d, [0, 2, 3], 0] == -sign * float("inf")).all(), got[d, :, 0]
        got[d, :, 0] = clean[d, :, 0]
    assert torch.equal(got, clean)
    ops.check_status()
