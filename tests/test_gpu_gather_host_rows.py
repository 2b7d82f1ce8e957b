"""Gathers whose rows share a chunk, with rows of the host table and rows of no table among them: numbers of rows on both sides of every doubling of the
rows a warp takes (148 x 64 warps each), narrow, odd and whole rows, windows of wider host rows, host tables that begin at any element. The first and last
rows of the host table are always asked for: the vectors that cover them reach beyond it. Copied bytes: exact."""
import numpy as np
import pytest
import torch

from apt_b200 import ops
from tests.gpu_util import dev

pytestmark = pytest.mark.gpu

TYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}


@pytest.fixture(autouse=True)
def _own_tables():
    """The tables installed before come back."""
    saved, ops.STATE.feat = ops.STATE.feat, ops.FeatStorage()
    yield
    ops.STATE.feat = saved
    ops.STATE.generation += 1


def _bits(t):
    return t.view(torch.int16 if t.element_size() == 2 else torch.int32)


@pytest.mark.parametrize("dtype,dim", [("f16", 1), ("f16", 3), ("bf16", 31), ("bf16", 33), ("f32", 1), ("f32", 9), ("f32", 17), ("f16", 12), ("f32", 20),
                                       ("f32", 100), ("f32", 128), ("bf16", 201), ("bf16", 255), ("f16", 999), ("f32", 1025)])
@pytest.mark.parametrize("rows", [1, 40, 9472, 9473, 18_945, 37_890, 75_777, 151_558])
@pytest.mark.parametrize("hosted,more,skip", [(0.1, 0, 0), (1.0, 0, 1), (0.5, 5, 1)])
def test_chunks_with_host_rows(dtype, dim, rows, hosted, more, skip):
    if rows * dim > 20_000_000:
        rows = 20_000_000 // dim
    rng = np.random.default_rng(dim + rows)
    n_dev, n_host, offset = 300, 200, min(more, 3)
    full = torch.from_numpy(rng.integers(-99, 100, (n_dev + n_host + 1, dim)).astype(np.float32)).to(TYPES[dtype])
    wide = torch.full((n_host + skip, dim + more), 7.0).to(TYPES[dtype])
    wide[skip:, offset:offset + dim] = full[n_dev:-1]
    full[-1] = 0
    # (a table that begins `skip` rows into its storage)
    ops.cache_feats_shared(n_dev + n_host + 1, wide.pin_memory()[skip:], full[:n_dev].cuda(), torch.arange(n_dev), torch.arange(n_dev, n_dev + n_host),
                           offset)
    ids = np.where(rng.random(rows) < hosted, rng.integers(n_dev, n_dev + n_host, rows), rng.integers(0, n_dev, rows))
    ids[0], ids[-1] = n_dev, n_dev + n_host - 1
    ids[rows // 2:rows // 2 + 1] = [n_dev + n_host] if rows > 2 else ids[rows // 2:rows // 2 + 1]
    want = full.cuda()[dev(ids)]
    assert torch.equal(_bits(ops.load_subtensor(dev(ids))), _bits(want))
    if rows > 2:
        with pytest.raises(RuntimeError, match="neither cached nor in host memory"):
            ops.check_status()
        # rows behind the first ones, up to a count of the device's
        out = torch.full((rows, dim), 3.0, dtype=TYPES[dtype], device="cuda")
        keep = out.clone()
        word = torch.tensor([rows // 3, rows - 1], device="cuda")
        ops._gather_enqueue(dev(ids), word[1:2], out=out, first_dev=word[0:1])
        keep[rows // 3:rows - 1] = want[rows // 3:rows - 1]
        assert torch.equal(_bits(out), _bits(keep))
        with pytest.raises(RuntimeError, match="neither cached nor in host memory"):
            ops.check_status()
    ops.check_status()
