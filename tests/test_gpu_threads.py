"""Operators that read counts or flags on the host, called by several threads at once."""
import threading

import numpy as np
import pytest
import torch

import apt_b200
from apt_b200 import ops
from tests.gpu_util import dev, install_graph, reset_world
from tests.helpers import small_graph

pytestmark = pytest.mark.gpu


def test_threads_read_the_word_block_at_once():
    # their copies to the host all start at the same moment, behind one event
    ops.STATE.words()
    ops.check_status()
    threads, rounds, failures = 16, 8, []
    ready = threading.Barrier(threads + 1)
    gates = [torch.cuda.Event() for _ in range(rounds)]
    streams = [torch.cuda.Stream() for _ in range(threads + 1)]

    def work(k):
        try:
            torch.cuda.set_device(0)
            with torch.cuda.stream(streams[k]):
                ops.check_status()
                for gate in gates:
                    ready.wait(60)
                    streams[k].wait_event(gate)
                    ops.check_status()
                    ready.wait(60)
        except Exception as exc:
            failures.append(exc)
            ready.abort()

    pool = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for t in pool:
        t.start()
    try:
        for gate in gates:
            with torch.cuda.stream(streams[-1]):
                torch.cuda._sleep(40_000_000)
                gate.record()
            ready.wait(60)
            ready.wait(60)
    except threading.BrokenBarrierError:
        pass
    for t in pool:
        t.join()
    failures = [f for f in failures if not isinstance(f, threading.BrokenBarrierError)]
    assert not failures, failures


def test_one_thread_samples_while_others_check():
    n, indptr, indices = small_graph(scale=12, edge_factor=8)
    install_graph(indptr, indices)
    reset_world(1, 0)
    seeds = [dev(np.random.default_rng(k).permutation(n)[:200].astype(np.int64)) for k in range(40)]
    ops.set_sampling(key=5, call_id=0)
    smp = apt_b200.DPNeighborSampler(0, [5, 4], prefetch_features=False)
    want = [smp.sample(None, s)[0].clone() for s in seeds]
    stop, failures = threading.Event(), []

    def check():
        try:
            torch.cuda.set_device(0)
            with torch.cuda.stream(torch.cuda.Stream()):
                while not stop.is_set():
                    ops.check_status()
        except Exception as exc:
            failures.append(exc)

    pool = [threading.Thread(target=check) for _ in range(2)]
    for t in pool:
        t.start()
    try:
        ops.set_sampling(key=5, call_id=0)
        got = [smp.sample(None, s)[0].clone() for s in seeds]
    finally:
        stop.set()
        for t in pool:
            t.join()
    assert not failures and all(torch.equal(a, b) for a, b in zip(got, want)), failures
