"""Word blocks that reach the host with a sequence number in every word, by themselves and beside the rows of a gather, and
arrays of words copied together."""
import ctypes

import pytest
import torch

from apt_b200 import _lib
from apt_b200._lib import check, lib

pytestmark = pytest.mark.gpu


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _blocks(count):
    words = torch.arange(count, dtype=torch.int64, device="cuda") * 7
    words[0], words[count // 2] = -1, 2 ** 31 - 1
    last = torch.tensor([0x11], device="cuda")
    want = words.tolist()
    want[-1] = 0x11
    return words, last, want, torch.zeros(count, dtype=torch.int64).pin_memory()


@pytest.mark.parametrize("count", [1, 31, 256, 300])
def test_words_arrive_with_their_sequence(count):
    words, last, want, host = _blocks(count)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for seq in (1, 2, 2 ** 32 + 3):      # the lower half counts
        check(lib.apt_publish_tagged(_ptr(words), count, _ptr(last), None, seq, _ptr(host), stream))
        check(lib.apt_wait_tagged(_ptr(host), count, seq, stream))
        assert host.tolist() == want
    seq_dev = torch.tensor([9], device="cuda")
    check(lib.apt_publish_tagged(_ptr(words), count, _ptr(last), _ptr(seq_dev), 0, _ptr(host), stream))
    check(lib.apt_wait_tagged(_ptr(host), count, 9, stream))
    assert host.tolist() == want
    # an idle stream without an answer ends the wait
    assert lib.apt_wait_tagged(_ptr(host), count, 10, stream) == _lib.APT_ERR_TIMEOUT


@pytest.mark.parametrize("rows,first", [(0, 0), (1, 0), (1203, 0), (1203, 1000), (40_000, 7)])
def test_words_beside_the_rows_of_a_gather(rows, first):
    count = 256
    words, last, want, host = _blocks(count)
    nodes, dim = 50_000, 36
    feats = torch.arange(nodes * dim, dtype=torch.float32, device="cuda").view(nodes, dim)
    pos = torch.arange(nodes, device="cuda")
    ids = torch.randperm(nodes, device="cuda")[:max(rows, 1)]
    out = torch.full((max(rows, 1), dim), -5.0, device="cuda")
    first_dev, status = torch.tensor([first], device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    check(lib.apt_gather_rows_publish(_ptr(ids), rows, None, _ptr(first_dev), _ptr(pos), nodes, _ptr(feats), nodes, dim * 4, None, 0, dim * 4, 0,
                                      _ptr(out), _ptr(status), _ptr(words), count, _ptr(last), None, 5, _ptr(host), stream))
    check(lib.apt_wait_tagged(_ptr(host), count, 5, stream))
    assert host.tolist() == want and int(status) == 0
    assert torch.equal(out[first:rows], feats[ids[first:rows]]) and bool((out[:min(first, rows)] == -5).all())


@pytest.mark.parametrize("counts", [[0], [1], [0, 5, 1023, 1024, 1025], [70_001] * 3, list(range(30))])
def test_arrays_copied_in_one_call(counts):
    src = [torch.arange(n + 1, dtype=torch.int64, device="cuda") * 3 + k for k, n in enumerate(counts)]
    dst = [torch.full((n + 1,), -9, dtype=torch.int64, device="cuda") for n in counts]
    pointers = ctypes.c_void_p * len(counts)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    check(lib.apt_copy_words(pointers(*(t.data_ptr() for t in src)), pointers(*(t.data_ptr() for t in dst)),
                             (ctypes.c_int64 * len(counts))(*counts), len(counts), stream))
    for n, a, b in zip(counts, src, dst):
        assert torch.equal(a[:n], b[:n]) and int(b[n]) == -9


@pytest.mark.parametrize("seq", [0, 2 ** 32 - 1, 2 ** 32, -1])
def test_words_that_were_read_answer_no_later_wait(seq):
    # a plain value's upper half is 0 or all ones, and so is that of a sequence number now and then
    words, last, want, host = _blocks(40)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    check(lib.apt_publish_tagged(_ptr(words), 40, _ptr(last), None, 7, _ptr(host), stream))
    check(lib.apt_wait_tagged(_ptr(host), 40, 7, stream))
    torch.cuda.synchronize()
    host[:] = 5 if seq in (0, 2 ** 32) else -5
    assert lib.apt_wait_tagged(_ptr(host), 40, seq, stream) == _lib.APT_ERR_TIMEOUT
    check(lib.apt_publish_tagged(_ptr(words), 40, _ptr(last), None, seq, _ptr(host), stream))
    check(lib.apt_wait_tagged(_ptr(host), 40, seq, stream))
    assert host.tolist() == want


def test_a_wait_in_vain_names_itself():
    host = torch.zeros(3, dtype=torch.int64).pin_memory()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for wait in ("apt_wait_tagged", "apt_wait_published"):
        assert getattr(lib, wait)(_ptr(host), 2, 4, stream) == _lib.APT_ERR_TIMEOUT
        with pytest.raises(RuntimeError, match=wait + ": the stream is idle"):
            check(_lib.APT_ERR_TIMEOUT)
