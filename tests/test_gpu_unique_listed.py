"""Distinct ids with the list that begins with other ids, and their inverse in a call of its own (apt_unique_ids, apt_unique_inverse), against numpy:
numbers of ids around a thread block and a wave, narrow and wide ranges, counts on the device, ids outside the range, no ids at all. Whole numbers:
exact."""
import numpy as np
import pytest
import torch

from apt_b200 import ops
from tests.gpu_util import dev, host, reset_world

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _own_tables():
    """The tables installed before come back."""
    saved, ops.STATE.feat = ops.STATE.feat, ops.FeatStorage()
    yield
    ops.STATE.feat = saved
    ops.STATE.generation += 1



@pytest.mark.parametrize("lo,hi", [(0, 1), (0, 40), (5, 3000), (7, 300_000), (0, 40_000_000)])
@pytest.mark.parametrize("groups,per", [(1, 1), (85, 3), (257, 1), (3000, 10), (40_000, 5)])
@pytest.mark.parametrize("listed", ["head", "no head", "no list"])
def test_against_numpy(lo, hi, groups, per, listed):
    rng = np.random.default_rng(groups + hi)
    reset_world()
    used = max(1, groups * 2 // 3)
    ids = rng.integers(lo, hi, groups * per).astype(np.int64)
    head = rng.integers(0, 50, 700).astype(np.int64) if listed == "head" else np.zeros(0, np.int64)
    heads = 600 if listed == "head" else 0
    counts = torch.tensor([used, heads, -1, -1, -1, -1, -1], device="cuda")
    word = lambda k: counts[k:k + 1]      # noqa: E731
    ops.register_min_vids(torch.tensor([0, 1 << 30]))
    for turn in range(2):      # the bitmap is left empty
        uniq = ops._unique_ids(dev(ids), word(0), per, lo, hi, word(2), "unique_test")
        inv, perm, all_ids = ops._unique_inverse(dev(ids), word(0), per, lo, hi, "unique_test", uniq, word(2), counts[4:6], counts[6:7],
                                                 3 if turn else None, None if listed == "no list" else dev(head), word(1) if heads else None,
                                                 None if listed == "no list" else word(3))
        ops.STATE.join(3)
        want, want_inv = np.unique(ids[:used * per], return_inverse=True)
        n = len(want)
        assert counts.tolist()[2:] == [n, -1 if listed == "no list" else heads + n, n, n, n]
        assert np.array_equal(host(uniq)[:n], want) and np.array_equal(host(inv)[:used * per], want_inv)
        assert np.array_equal(host(perm)[:n], np.arange(n))
        if listed != "no list":
            assert np.array_equal(host(all_ids)[:heads + n], np.concatenate([head[:heads], want]))
    ops._unique_ids(dev(ids), word(0), per, lo, hi, word(2), "unique_test")
    inv, perm, _ = ops._unique_inverse(dev(ids), word(0), per, lo, hi, "unique_test", sizes=counts[4:6], offsets=counts[6:7])
    assert counts.tolist()[4:] == [used * per] * 3 and np.array_equal(host(perm)[:used * per], np.arange(used * per))
    ops.check_status()


def test_ids_outside_and_rows_that_do_not_exist():
    reset_world()
    table = torch.zeros((8, 4))
    ops.cache_feats_shared(12, table.pin_memory(), table.cuda(), torch.arange(8), torch.arange(8), 0)
    word = torch.zeros(2, dtype=torch.int64, device="cuda")
    ids, head = np.array([3, 11, 3, 5], np.int64), np.array([1, 2], np.int64)

    def both(ids, hi, look_up):
        uniq = ops._unique_ids(ids, None, 1, 0, hi, word[0:1], "unique_t2")
        return ops._unique_inverse(ids, None, 1, 0, hi, "unique_t2", uniq, word[0:1], head=dev(head), all_out=word[1:2], look_up=look_up)

    inv, _, all_ids = both(dev(ids), 12, True)
    assert word.tolist() == [3, 5] and host(all_ids)[:5].tolist() == [1, 2, 3, 5, 11] and host(inv).tolist() == [0, 2, 0, 1]
    with pytest.raises(RuntimeError, match="neither cached nor in host memory"):
        ops.check_status()
    inv, _, all_ids = both(dev(ids), 6, False)
    assert word.tolist() == [2, 4] and host(inv).tolist() == [0, -1, 0, 1] and host(all_ids)[:4].tolist() == [1, 2, 3, 5]
    with pytest.raises(RuntimeError, match="id outside"):
        ops.check_status()
    _, _, all_ids = both(torch.empty(0, dtype=torch.int64, device="cuda"), 6, False)
    assert word.tolist() == [0, 2] and host(all_ids).tolist() == [1, 2]


def test_a_second_half_that_fails():
    """The distinct ids by themselves: what they leave in the bitmap is gone before anybody else's, a captured graph's too."""
    reset_world()
    lo, hi = 7, 300_000
    ids = np.random.default_rng(3).integers(lo, hi, 20_000).astype(np.int64)
    ids_dev, word = dev(ids), torch.zeros(4, dtype=torch.int64, device="cuda")
    want, want_inv = np.unique(ids, return_inverse=True)

    def both():
        uniq = ops._unique_ids(ids_dev, None, 1, lo, hi, word[0:1], "unique_half")
        return uniq, ops._unique_inverse(ids_dev, None, 1, lo, hi, "unique_half")[0]

    def right(uniq, inv):
        torch.cuda.synchronize()
        return int(word[0]) == len(want) and np.array_equal(host(uniq)[:len(want)], want) and np.array_equal(host(inv), want_inv)

    assert right(*both())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        of_graph = both()
    saved, ops.STATE.shuffle_min_vids = ops.STATE.shuffle_min_vids, None
    try:
        for then in ("call", "graph"):
            ops._unique_ids(ids_dev, None, 1, lo, hi, word[0:1], "unique_half")
            with pytest.raises(RuntimeError, match="register_min_vids"):
                ops._unique_inverse(ids_dev, None, 1, lo, hi, "unique_half", sizes=word[1:3], offsets=word[3:4])
            # (the bitmap is looked at before it is used: counts left in it would send the next call beyond its buffers)
            torch.cuda.synchronize()
            assert int(ops._unique_bitmap(hi - lo, "unique_half").count_nonzero()) == 0
            if then == "graph":
                graph.replay()
                assert right(*of_graph)
            else:
                assert right(*both())
        # a first half whose second never came: the next call starts from an empty bitmap
        ops._unique_ids(ids_dev, None, 1, lo, hi, word[0:1], "unique_half")
        assert right(*both())
    finally:
        ops.STATE.shuffle_min_vids = saved
    ops.check_status()
