"""The id kernels and the gather at the edges of their splits: rows around a chunk and a warp and of every access width
(gather), dense and sparse id ranges around what a lane walks alone (sorted unique), layers around a tile, the one-block
limit and the number of tiles a block adds up (relabelling). Bytes and whole numbers: exact."""
import numpy as np
import pytest
import torch

from apt_b200 import DPNeighborSampler, ops
from apt_b200._lib import check, lib
from oracle import oracle as orc
from tests.gpu_util import dev, host, install_graph
from tests.helpers import small_graph

pytestmark = pytest.mark.gpu
I64 = np.int64


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("dim", [1, 3, 8, 17, 47, 100, 128, 130, 195, 600, 1024])
def test_gather_rows_and_widths(dtype, dim):
    table, n_host, n = 300, 90, 420                     # ids 390.. are in neither table
    gen = torch.Generator(device="cuda").manual_seed(dim)
    cached = torch.randn((table, dim), device="cuda", generator=gen).to(dtype)
    hosted = torch.randn((n_host, dim), device="cuda", generator=gen).to(dtype)
    ops.cache_feats_shared(n, hosted.cpu().pin_memory(), cached, torch.arange(table), torch.arange(table, table + n_host), 0)
    whole = torch.cat([cached, hosted, torch.zeros((n - table - n_host, dim), dtype=dtype, device="cuda")])
    for rows in (1, 2, 7, 31, 32, 33, 257, 5000):
        ids = torch.randint(0, table + n_host, (rows,), device="cuda", generator=gen)
        assert torch.equal(ops.load_subtensor(ids), whole[ids])
        ops.check_status()
    ids = torch.randint(0, n, (333,), device="cuda", generator=gen)
    assert torch.equal(ops.load_subtensor(ids), whole[ids])
    with pytest.raises(RuntimeError, match="neither cached"):
        ops.check_status()



@pytest.mark.parametrize("rows", [1, 1184, 37_889, 200_001])
def test_gather_on_few_blocks(rows):
    # fewer rows than its warps, one chunk more than they take at once, many
    table, n_host, dim = 5000, 700, 36
    gen = torch.Generator(device="cuda").manual_seed(rows)
    cached = torch.randn((table, dim), device="cuda", generator=gen)
    hosted = torch.randn((n_host, dim), device="cuda", generator=gen)
    ops.cache_feats_shared(table + n_host, hosted.cpu().pin_memory(), cached, torch.arange(table),
                           torch.arange(table, table + n_host), 0)
    ids = torch.randint(0, table + n_host, (rows,), device="cuda", generator=gen)
    got = ops._gather_enqueue(ids, torch.tensor([rows], device="cuda"), beside=True)
    assert torch.equal(got, torch.cat([cached, hosted])[ids])
    ops.check_status()


def _patterns():
    rng = np.random.default_rng(8)
    for words in (7, 8, 9, 32):                        # level-0 words below one level-1 word
        for per in (1, 4, 5, 32):                      # ids to a word: 32 and 33 ids, and full words
            yield f"{words} words of {per}", 5000, np.concatenate([2048 + 32 * w + np.arange(per) for w in range(words)])
    yield "dense", 70_000, np.arange(70_000)
    yield "runs", 9_000, np.repeat(np.arange(900) * 9, 25)
    yield "dense among sparse", 40_000_000, np.concatenate([np.arange(5000) + 1_000_000, rng.integers(0, 40_000_000, 3000)])
    yield "one id", 1, np.zeros(3, dtype=I64)
    yield "sparse", 1 << 27, rng.integers(0, 1 << 27, 20_000)


@pytest.mark.parametrize("name,rng_hi,ids", list(_patterns()), ids=[p[0] for p in _patterns()])
def test_unique_sorted_patterns(name, rng_hi, ids):
    ids = np.random.default_rng(1).permutation(ids.astype(I64)) if "runs" not in name else ids.astype(I64)
    for _ in range(2):                                 # the second call finds what the first one left: nothing
        uniq, inv = ops.unique_sorted(dev(ids), 0, rng_hi)
        want, want_inv = np.unique(ids, return_inverse=True)
        assert np.array_equal(host(uniq), want) and np.array_equal(host(inv), want_inv)


@pytest.mark.parametrize("small", [0, 1])
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 4097, 8191, 8192, 8193, 70_001])
def test_relabel_sizes(n, small):
    rng = np.random.default_rng(n)
    seeds = rng.permutation(n * 2)[: max(1, n // 9)].astype(I64)
    nbr = np.minimum(rng.zipf(1.2, n - len(seeds)), 2 * n).astype(I64) if n > len(seeds) else np.empty(0, dtype=I64)
    check(lib.apt_set_tunable(b"relabel_small", small))
    try:
        for _ in range(2):
            uniq, rel = ops.relabel_csc(dev(seeds), dev(nbr))
            want_u, want_r = orc.relabel_csc(seeds, nbr)
            assert np.array_equal(host(uniq), want_u) and np.array_equal(host(rel), want_r)
    finally:
        check(lib.apt_set_tunable(b"relabel_small", 1))


def test_relabel_beyond_the_tiles_of_one_size():
    # 4.5 M items: more than 4096 tiles of 1024, so that tiles are twice as large
    gen = torch.Generator(device="cuda").manual_seed(5)
    n = 4_500_001
    items = torch.randint(0, 3_000_000, (n,), device="cuda", generator=gen)
    S = 1000
    uniq, rel = ops.relabel_csc(items[:S], items[S:])
    assert torch.equal(uniq[rel], items[S:])
    first = torch.full((3_000_000,), n, device="cuda").scatter_reduce_(0, items, torch.arange(n, device="cuda"), "amin")
    order = first[uniq]                                # positions of first occurrence: rising, and all of them
    assert bool((order[1:] > order[:-1]).all()) and uniq.numel() == int((first < n).sum())


@pytest.mark.parametrize("id_range", [1 << 18, (1 << 18) + 1, 1 << 28, (1 << 28) + 1, (1 << 31) + 1])
def test_unique_around_the_numbers_of_tiles(id_range):
    # one tile and two; the most whose counts a block adds up first and one more; enough for sums over groups of tiles
    gen = torch.Generator(device="cuda").manual_seed(3)
    edge = torch.tensor([0, id_range - 1, id_range - 1, id_range // 2], device="cuda")
    ids = torch.cat([torch.randint(0, id_range, (20_000,), device="cuda", generator=gen), edge])
    for _ in range(2):
        uniq, inv = ops.unique_sorted(ids, 0, id_range)
        want, want_inv = torch.unique(ids, return_inverse=True)
        assert torch.equal(uniq, want) and torch.equal(inv, want_inv)
    for key in [k for k in ops.STATE._ws if k[0].startswith("unique")]:
        del ops.STATE._ws[key]                         # the widest bitmap is 0.8 GB


@pytest.mark.parametrize("fanout", [1, 7, 8, 9, 15, 16, 31, 32, 33])
def test_sample_and_relabel_around_the_group_widths(fanout):
    # with a lane left over the seed enters the table beside its draws, without one behind them
    n, indptr, indices = small_graph(scale=12, edge_factor=8)
    install_graph(indptr, indices)
    seeds = dev(np.random.default_rng(fanout).permutation(n)[:1003].astype(I64))
    ops.set_sampling(key=5, call_id=9)
    _, neighbours = ops.local_sample_one_layer(seeds, fanout)
    uniq, rel = ops.relabel_csc(seeds, neighbours)
    got = DPNeighborSampler(0, [fanout], prefetch_features=False)
    ops.set_sampling(key=5, call_id=9)
    input_nodes, _, blocks = got.sample(None, seeds)[:3]
    assert torch.equal(input_nodes, uniq) and torch.equal(blocks[0].coo_row, rel)
