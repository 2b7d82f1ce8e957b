"""The gather's widths around a warp's lanes, its eight elements in flight and the bytes of a chunk, with rows of the host table and rows of neither among
them, in requests so small that every row has a warp to itself (rows that share a chunk: test_gpu_gather_host_rows.py). Copied bytes: exact."""
import numpy as np
import pytest
import torch

from apt_b200 import ops
from apt_b200 import _lib
from tests.gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _own_tables():
    """The tables installed before come back."""
    saved, ops.STATE.feat = ops.STATE.feat, ops.FeatStorage()
    yield
    ops.STATE.feat = saved
    ops.STATE.generation += 1

TYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}


@pytest.mark.parametrize("dtype,dim", [("bf16", 1), ("f32", 1), ("f16", 3), ("bf16", 8), ("f32", 9), ("f16", 31), ("bf16", 33), ("f32", 64), ("bf16", 255),
                                       ("f16", 257), ("bf16", 441), ("f32", 300), ("f32", 999), ("f16", 1024), ("bf16", 8191), ("f16", 8193), ("f32", 8196)])
@pytest.mark.parametrize("rows", [1, 31, 33, 1000])
def test_widths_and_rows(dtype, dim, rows):
    rng = np.random.default_rng(dim + rows)
    n, n_dev, n_host = 90, 50, 36      # the last 4 nodes are in neither table
    table = torch.from_numpy(rng.integers(-9, 10, (n, dim)).astype(np.float32)).to(TYPES[dtype])
    ops.cache_feats_shared(n, table[n_dev:n_dev + n_host].contiguous().pin_memory(), table[:n_dev].cuda(), torch.arange(n_dev),
                           torch.arange(n_dev, n_dev + n_host), 0)
    ids = rng.integers(0, n_dev + n_host, rows).astype(np.int64)
    ids[[0, -1]] = [n_dev - 1, n_dev + n_host - 1][:len(ids[[0, -1]])]
    assert torch.equal(ops.load_subtensor(dev(ids)).cpu(), table[torch.from_numpy(ids)])
    ops.check_status()
    ids[rows // 2] = n - 1
    got = ops.load_subtensor(dev(ids)).cpu()
    want = table[torch.from_numpy(ids)]
    want[torch.from_numpy(ids) >= n_dev + n_host] = 0
    assert torch.equal(got, want)
    with pytest.raises(RuntimeError, match=_lib_text()):
        ops.check_status()


def _lib_text():
    from apt_b200.ops import _flag_text

    return _flag_text(_lib.FLAG_FEAT_NOT_EXIST)


@pytest.mark.parametrize("first", [0, 1, 7, 500])
def test_rows_behind_the_first_ones(first):
    """Rows [first, n) of a request, which start at no multiple of anything in the result; the others stay as they are."""
    rng = np.random.default_rng(first)
    n, dim = 400, 77
    table = torch.from_numpy(rng.standard_normal((n, dim)).astype(np.float32)).to(torch.bfloat16)
    ops.cache_feats_shared(n, table[:2].contiguous().pin_memory(), table.cuda(), torch.arange(n), torch.arange(2), 0)
    ids = dev(rng.integers(0, n, 700).astype(np.int64))
    out = torch.full((700, dim), 3.0, dtype=torch.bfloat16, device="cuda")
    word = torch.tensor([first, 650], device="cuda")
    ops._gather_enqueue(ids, word[1:2], out=out, first_dev=word[0:1])
    want = torch.full((700, dim), 3.0, dtype=torch.bfloat16)
    want[first:650] = table[ids.cpu()][first:650]
    assert torch.equal(out.cpu(), want)
