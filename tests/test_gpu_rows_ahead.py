"""Rows that a sampler gathered ahead: load_subtensor hands them out only while the tables and the ids they were gathered
for are what they were. Rows are copied bytes: compared bit for bit."""
import numpy as np
import pytest
import torch

import apt_b200
from apt_b200 import ops
from tests.gpu_util import dev, install_graph, reset_world
from tests.helpers import small_graph
from tests.test_gpu_counts_first import MAKE

pytestmark = pytest.mark.gpu
I64 = np.int64


def _table(n, scale, dim=24):
    """A feature table of its own, half of it cached: (table, what is to be kept alive)."""
    table = (torch.arange(n, dtype=torch.float32, device="cuda")[:, None] + torch.zeros(dim, device="cuda")) * scale
    cached, hosted = torch.arange(n)[::2], torch.arange(n)[1::2]
    parts = table[hosted.cuda()].cpu().pin_memory(), table[cached.cuda()]
    ops.cache_feats_shared(n, parts[0], parts[1], cached, hosted, 0)
    return table, parts


def _install():
    n, indptr, indices = small_graph(scale=12, edge_factor=8)
    install_graph(indptr, indices)
    reset_world(1, 0)
    ops.register_min_vids(torch.tensor([0, n]))
    return n


def _seeds(n, seed=2, count=300):
    return dev(np.random.default_rng(seed).permutation(n)[:count].astype(I64))


@pytest.mark.parametrize("kind", sorted(MAKE))
def test_another_table_is_read(kind):
    n = _install()
    old = _table(n, 1.0)
    smp = MAKE[kind]([6, 4])
    for _ in range(2):                      # the first pass of a shape, and a replay
        got = smp.sample(None, _seeds(n))
        new = _table(n, -3.0)
        assert torch.equal(ops.load_subtensor(got[0]), new[0][got[0]])
        old = _table(n, 1.0)
    ops.check_status()
    del old


@pytest.mark.parametrize("kind", sorted(MAKE))
def test_changes_in_place_are_read(kind):
    n = _install()
    table, (host, cached) = _table(n, 1.0)
    smp = MAKE[kind]([6, 4])
    for _ in range(2):
        got = smp.sample(None, _seeds(n))
        cached.mul_(2)
        table[::2] *= 2
        assert torch.equal(ops.load_subtensor(got[0]), table[got[0]])
        got = smp.sample(None, _seeds(n))
        torch.cuda.synchronize()
        host.add_(1)
        table[1::2] += 1
        assert torch.equal(ops.load_subtensor(got[0]), table[got[0]])
        got = smp.sample(None, _seeds(n))
        torch.cuda.synchronize()
        got[0].copy_(got[0].flip(0))
        assert torch.equal(ops.load_subtensor(got[0]), table[got[0]])
    ops.check_status()


@pytest.mark.parametrize("kind", ["np", "snp_gat", "sage"])
def test_batches_in_flight_meet_another_table(kind):
    n = _install()
    old = _table(n, 1.0)
    it = MAKE[kind]([6, 4]).sample_iter(None, [_seeds(n, k) for k in range(6)])
    got = next(it)
    assert torch.equal(ops.load_subtensor(got[0]), old[0][got[0]])
    new = _table(n, 5.0)                    # the batches launched by now were gathered from the old one
    for got in it:
        assert torch.equal(ops.load_subtensor(got[0]), new[0][got[0]])
    ops.check_status()


def test_rows_ahead_are_used_when_nothing_changed():
    n = _install()
    table, _ = _table(n, 1.0)
    for kind in ("np", "dp", "sage"):
        got = MAKE[kind]([6, 4]).sample(None, _seeds(n))
        rows = ops.STATE.prefetched.rows
        assert ops.load_subtensor(got[0]).data_ptr() == rows.data_ptr()
        got = MAKE[kind]([6, 4]).sample(None, _seeds(n))
        assert torch.equal(ops.load_subtensor(got[0].view(-1)), table[got[0]])
    ops.check_status()


def _wide_host_table(n, dim):
    """Rows of several KiB in host memory: a gather of some thousands of them is still running when sample() returns."""
    host = (torch.arange(n, dtype=torch.float32)[:, None] + torch.zeros(dim)).pin_memory()
    ops.cache_feats_shared(n, host, host[:1].cuda(), torch.arange(1), torch.arange(n), 0)
    return host


@pytest.mark.parametrize("fanouts", [[10], [6, 4]])
def test_data_parallel_rows_on_another_stream(fanouts):
    # the rows are ordered behind their gather, and operators on other streams do not change how many there are
    n = _install()
    host = _wide_host_table(n, 1024)
    smp = apt_b200.DPNeighborSampler(0, fanouts)
    other = torch.cuda.Stream()
    few = torch.arange(3, device="cuda")
    for k in range(6):
        seeds = _seeds(n, k, 2000)
        torch.empty(4096 * 1024, device="cuda").fill_(-1.0)         # rows not written yet show
        torch.cuda.synchronize()
        got = smp.sample(None, seeds)
        with torch.cuda.stream(other):
            if k % 2:
                ops.relabel_csc(few, few)                           # leaves its own count in the shared words
            rows = ops.load_subtensor(got[0])
            seen = rows[:, ::512].clone()
        other.synchronize()
        ids = got[0].cpu()
        assert len(ids) > 2000 and torch.equal(seen.cpu(), host[ids][:, ::512])
    ops.check_status()


def test_data_parallel_batches_hold_what_they_consist_of():
    n = _install()                          # 4096 nodes: three hops meet the same ones again and again
    _table(n, 1.0, dim=256)
    got = apt_b200.DPNeighborSampler(0, [15, 15, 15]).sample(None, _seeds(n, 0, 256))
    rows = ops.load_subtensor(got[0])
    assert got[0] is got[2][0].src_ids
    held = [(rows.untyped_storage().nbytes(), rows.numel() * 4 + 512)]
    for b in got[2]:
        held += [(t.untyped_storage().nbytes(), 2 * t.numel() * 8 + (1 << 20)) for t in (b.coo_row, b.coo_col, b.src_ids)]
        assert torch.equal(b.coo_col, torch.arange(b.num_dst, device="cuda").repeat_interleave(15))
    assert all(size <= most for size, most in held), held
    ops.check_status()


@pytest.mark.parametrize("kind", ["np", "snp_gat", "sage", "gcn", "sage_dst"])
def test_a_batch_keeps_its_counts_to_itself(kind):
    # the gather behind a replay reads its counts when other operators, on other streams, may be writing theirs
    n = _install()
    table, _ = _table(n, 1.0)
    smp = MAKE[kind]([6, 4])
    smp.sample(None, _seeds(n))
    ops.check_status()
    words = ops.STATE.words()
    words[:-1].fill_(-7)
    got = smp.sample(None, _seeds(n, 3))
    assert bool((words[:-1] == -7).all()) and int(words[-1]) & ~4 == 0
    assert torch.equal(ops.load_subtensor(got[0]), table[got[0]])
    # flags of operators outside the replay are still raised by it
    ops.STATE.lane_words()[-1] = 32
    with pytest.raises(RuntimeError, match="not grouped"):
        smp.sample(None, _seeds(n, 3))
    ops.check_status()


def test_an_iterator_given_up_leaves_nothing_behind():
    # its batches may not have begun when the next iterator launches on the same buffer sets; their seeds' memory is not
    # handed out before they have
    n = _install()
    table, _ = _table(n, 1.0)
    smp = apt_b200.MixedNeighborSampler(0, [4, 3], lanes=2)
    batches = [_seeds(n, k, 200) for k in range(8)]
    for got in smp.sample_iter(None, batches):
        ops.load_subtensor(got[0])
    torch.cuda.synchronize()

    junk = []

    def broken():
        for k in range(2):
            yield batches[k].clone()
        raise KeyError("no more")

    def fresh():
        for b in batches:
            yield b.clone()
            junk.append(torch.full((200,), -5, device="cuda"))         # takes whatever memory has been given back

    for lane in (1, 2):
        with torch.cuda.stream(ops.STATE.lane_stream(lane)):
            torch.cuda._sleep(400_000_000)
    with pytest.raises(KeyError):
        list(smp.sample_iter(None, broken()))
    for got in smp.sample_iter(None, fresh()):
        assert torch.equal(ops.load_subtensor(got[0]), table[got[0]])
    ops.check_status()
