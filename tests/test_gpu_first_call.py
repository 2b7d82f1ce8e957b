"""The first call that needs something of the library's own (page-locked words) may come inside a stream capture, or while
another thread captures: it works and the capture stays valid. In processes of their own, so that it is the first."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BLOCK = """
import ctypes, sys, threading
import torch
from apt_b200 import _lib, ops
from apt_b200._lib import check, lib
p = lambda t: ctypes.c_void_p(t.data_ptr())
def block(dst, src, fanout, dim):
    gen = torch.Generator(device="cuda").manual_seed(1)
    col = torch.arange(dst, device="cuda").repeat_interleave(fanout)
    row = torch.randint(0, src, (col.numel(),), device="cuda", generator=gen)
    off = [torch.tensor([0, n], device="cuda") for n in (col.numel(), src, dst)]
    x = torch.randint(-8, 9, (src, dim), device="cuda", generator=gen).float()      # whole numbers: sums are exact
    return row, col, x, off
def want(b, dst):
    return torch.zeros((dst, b[2].shape[1]), device="cuda").index_add_(0, b[1], b[2][b[0]])
def sum_into(b, out, ws):
    row, col, x, off = b
    check(lib.apt_spmm_sum(0, _lib.F32, p(row), p(col), row.numel(), p(x), None, x.shape[1], x.shape[1], p(off[0]), p(off[1]),
                           p(off[2]), 1, out.shape[0], p(out), p(ws), ws.numel(),
                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
def room(b, dst):
    return torch.empty(lib.apt_spmm_workspace_bytes(dst, b[0].numel()), dtype=torch.uint8, device="cuda")
"""

CAPTURED = BLOCK + """
b = block(14_001, 20_003, 15, 256)
out, ws = torch.zeros((14_001, 256), device="cuda"), room(b, 14_001)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    sum_into(b, out, ws)
graph.replay()
assert torch.equal(out, want(b, 14_001))
print("fine")
"""

BESIDE = BLOCK + """
b = block(300, 500, 7, 32)
out, ws = torch.zeros((300, 32), device="cuda"), room(b, 300)
sum_into(b, out, ws)                          # the kernels are loaded; nothing of the library's own has been needed yet
expect, got, errors = want(b, 300), [], []
captured = torch.zeros(8, device="cuda")
stream = torch.cuda.Stream()
with torch.cuda.stream(stream):
    torch.cuda._sleep(1000)
    ops.check_status()
torch.cuda.synchronize()
def other():
    try:
        torch.cuda.set_device(0)
        with torch.cuda.stream(stream):
            torch.cuda._sleep(200_000_000)    # the host asks the stream how it stands meanwhile
            got.append(ops.spmm_copy_u_sum(b[0], b[1], b[2], *b[3]))
            torch.cuda._sleep(200_000_000)
            ops.check_status()
    except Exception as exc:
        errors.append(exc)
graph = torch.cuda.CUDAGraph()
try:
    with torch.cuda.graph(graph):
        captured += 1
        thread = threading.Thread(target=other)
        thread.start()
        thread.join()
        captured += 1
finally:
    print(*errors, file=sys.stderr)
graph.replay()
torch.cuda.synchronize()
assert not errors, errors
assert torch.equal(got[0], expect) and captured.tolist() == [2.0] * 8
print("fine")
"""


@pytest.mark.parametrize("program", [CAPTURED, BESIDE], ids=["captured", "beside_a_capture"])
def test_first_call(program):
    done = subprocess.run([sys.executable, "-c", program], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and done.stdout.strip() == "fine", done.stderr[-2000:]
