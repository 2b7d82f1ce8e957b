"""Mini-batches whose counts reach the host before the feature rows are there: errors of the rows are still raised by
sample(), rows are ordered behind their gather on any stream, the data-parallel sampler's single read gives what hop by
hop gives, and the polled word block of the C ABI."""
import ctypes

import numpy as np
import pytest
import torch

import apt_b200
from apt_b200 import _lib, ops
from apt_b200._lib import check, lib
from tests.gpu_util import dev, install_graph, reset_world
from tests.helpers import small_graph

pytestmark = pytest.mark.gpu
I64 = np.int64
MAKE = {
    "np": lambda f: apt_b200.MixedNeighborSampler(0, f),
    "np_eager": lambda f: apt_b200.MixedNeighborSampler(0, f, use_graph=False),
    "snp_gat": lambda f: apt_b200.SPGATSampler(0, f),
    "sage": lambda f: apt_b200.SPVirtualSampler(0, f),
    "gcn": lambda f: apt_b200.SPVirtualSampler(0, f, model="GCN"),
    "sage_dst": lambda f: apt_b200.SPVirtualSampler(0, f, shuffle_with_dst=True),
    "dp": lambda f: apt_b200.DPNeighborSampler(0, f),
}


def _install(missing=0, dim=24):
    n, indptr, indices = small_graph(scale=12, edge_factor=8)
    install_graph(indptr, indices)
    reset_world(1, 0)
    ops.register_min_vids(torch.tensor([0, n]))
    table = torch.arange(n, dtype=torch.float32, device="cuda")[:, None] + torch.zeros(dim, device="cuda")
    held = torch.arange(n - missing)
    cached, hosted = held[::2], held[1::2]
    ops.cache_feats_shared(n, table[hosted.cuda()].cpu().pin_memory(), table[cached.cuda()], cached, hosted, 0)
    return n, table


@pytest.mark.parametrize("kind", sorted(MAKE))
def test_rows_follow_on_any_stream(kind):
    # rows of 4 KiB, all of them in host memory: a gather of two thousand takes 200 us and is still running when sample() has
    # returned. The buffers rows may land in hold -1 before.
    n, _ = _install()
    table = (torch.arange(n, dtype=torch.float32)[:, None] + torch.zeros(1024)).pin_memory()
    ops.cache_feats_shared(n, table, table[:1].cuda(), torch.arange(1), torch.arange(n), 0)
    rng = np.random.default_rng(2)
    smp = MAKE[kind]([6, 4])
    other = torch.cuda.Stream()
    for k in range(6):
        seeds = dev(rng.permutation(n)[:1000].astype(I64))
        if k:
            rows.fill_(-1)                  # a replay's buffer: of the batch after the next one
        torch.empty(4096 * 1024, device="cuda").fill_(-1)
        torch.cuda.synchronize()
        got = smp.sample(None, seeds)
        with torch.cuda.stream(other if k % 2 else torch.cuda.current_stream()):
            rows = ops.load_subtensor(got[0])
            seen = rows[:, ::512].clone()
        torch.cuda.synchronize()
        ids = got[0].cpu()
        assert len(ids) > 1500 and torch.equal(seen.cpu(), table[ids][:, ::512])
    ops.check_status()


@pytest.mark.parametrize("kind", sorted(MAKE))
def test_missing_rows_are_raised_by_sample(kind):
    n, _ = _install(missing=500)
    smp = MAKE[kind]([6, 4])
    seeds = dev(np.arange(n - 400, n, dtype=I64))       # nodes without a feature row
    for _ in range(2):                                  # the first pass of a shape, and a replay
        with pytest.raises(RuntimeError, match="neither cached"):
            got = smp.sample(None, seeds)
            if kind in ("snp_gat", "gcn", "sage_dst"):  # destinations need no rows of their own here
                ops.load_subtensor(got[0])
                ops.check_status()
        torch.cuda.synchronize()
        ops.STATE.words().zero_()
    _, table = _install()
    got = smp.sample(None, seeds)
    assert torch.equal(ops.load_subtensor(got[0]), table[got[0]])
    ops.check_status()


@pytest.mark.parametrize("fanouts", [[5], [10, 5], [15, 10, 5]])
@pytest.mark.parametrize("replace", [True, False])
def test_dp_one_read_equals_hop_by_hop(fanouts, replace):
    n, table = _install()
    rng = np.random.default_rng(4)
    batches = [dev(rng.permutation(n)[:k].astype(I64)) for k in (200, 200, 1, 333)]
    runs = []
    try:
        for chained in (True, False):
            ops.set_sampling(key=9, call_id=0, replace=replace)
            smp = apt_b200.DPNeighborSampler(0, fanouts, chained=chained)
            runs.append([smp.sample(None, s) for s in batches])     # all kept: every batch has tensors of its own
    finally:
        ops.set_sampling(replace=True)
    for (ia, oa, ba), (ib, ob, bb), seeds in zip(*runs, batches):
        assert torch.equal(ia, ib) and oa is seeds and ob is seeds and len(ba) == len(bb) == len(fanouts)
        for x, y in zip(ba, bb):
            assert (x.num_src, x.num_dst, x.fanout) == (y.num_src, y.num_dst, y.fanout)
            assert all(torch.equal(p, q) for p, q in ((x.coo_row, y.coo_row), (x.coo_col, y.coo_col), (x.src_ids, y.src_ids)))
        assert torch.equal(ops.load_subtensor(ia), table[ia])
    empty = apt_b200.DPNeighborSampler(0, fanouts).sample(None, dev(np.empty(0, dtype=I64)))
    assert empty[0].numel() == 0
    ops.check_status()


def test_call_id_alone_keeps_captured_batches():
    n, _ = _install()
    smp = MAKE["np"]([4, 3])
    seeds = dev(np.arange(50, dtype=I64))
    ops.set_sampling(key=3, call_id=7)
    first = [smp.sample(None, seeds)[0].clone() for _ in range(2)]
    before = ops.STATE.generation
    ops.set_sampling(key=3, call_id=7)
    again = [smp.sample(None, seeds)[0].clone() for _ in range(2)]
    assert ops.STATE.generation == before and all(torch.equal(a, b) for a, b in zip(first, again))
    ops.set_sampling(key=4, call_id=7)
    assert ops.STATE.generation == before + 1
    assert not torch.equal(smp.sample(None, seeds)[0], first[0])


def test_published_words():
    words = torch.arange(300, device="cuda")
    host = torch.zeros(301, dtype=torch.int64).pin_memory()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for seq in (1, 2):
        words += 1
        check(lib.apt_publish_words(ptr(words), 300, None, seq, ptr(host), stream))
        check(lib.apt_wait_published(ptr(host), 300, seq, stream))
        assert host[:300].tolist() == list(range(seq, 300 + seq))
    seq_dev = torch.tensor([77], device="cuda")
    check(lib.apt_publish_words(ptr(words), 300, ptr(seq_dev), 0, ptr(host), stream))
    check(lib.apt_wait_published(ptr(host), 300, 77, stream))
    # nothing published and the stream idle: a status, no wait without end
    assert lib.apt_wait_published(ptr(host), 300, 78, stream) == _lib.APT_ERR_TIMEOUT
