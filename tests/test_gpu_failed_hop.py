"""A mini-batch whose outermost hop cannot be enqueued (no memory) while side streams are at work on its inverse and its frontier's rows: the stream that
the next one begins on waits for them."""
import numpy as np
import pytest
import torch

import apt_b200
from apt_b200 import ops
from tests.gpu_util import dev, host, install_graph, reset_world
from tests.helpers import feature_setup, small_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [2, 3])
def test_side_streams_are_joined(monkeypatch, side):
    n, indptr, indices = small_graph(scale=12, edge_factor=8)
    install_graph(indptr, indices)
    reset_world(1, 0)
    ops.register_min_vids(torch.tensor([0, n]))
    rng = np.random.default_rng(4)
    feats, uva, devf, cached_idx, local_idx, pos_map, cpu_map = feature_setup(n, 32, 0.5, rng)
    ops.cache_feats_shared(n, torch.from_numpy(uva).pin_memory(), dev(devf), torch.from_numpy(cached_idx), torch.from_numpy(local_idx), 0)
    seeds = dev(rng.permutation(n)[:200].astype(np.int64))
    smp = apt_b200.MixedNeighborSampler(0, [10, 5], chained=True, use_graph=False)
    smp.gather_split = 1

    def batch():
        ops.set_sampling(key=4242, call_id=5)
        nodes, seen_seeds = smp.sample(None, seeds)[:2]
        return [host(x) for x in (nodes, seen_seeds, ops.load_subtensor(nodes))]

    want, enqueue, seen = batch(), ops._sample_relabel_enqueue, []

    def fails(*args, **kw):
        seen.append(torch.cuda.current_stream())
        if len(seen) < 2:
            return enqueue(*args, **kw)
        with torch.cuda.stream(ops.STATE.side_stream(side)):
            torch.cuda._sleep(200_000_000)      # 0.1 s
            seen.append(torch.cuda.Event())
            seen[-1].record()
        raise torch.OutOfMemoryError("no room")

    monkeypatch.setattr(ops, "_sample_relabel_enqueue", fails)
    with pytest.raises(torch.OutOfMemoryError):
        batch()
    monkeypatch.undo()
    after = torch.cuda.Event()
    after.record(seen[1])
    after.synchronize()
    assert seen[2].query()
    assert all(np.array_equal(a, b) for a, b in zip(batch(), want))
    ops.check_status()
