"""Which sums and dots go to the kernel that walks the edges as a stream: the rule itself, compiled for the host."""
import os
import shutil
import subprocess

import pytest

from apt_b200._lib import lib

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "apt_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
PROGRAM = r"""
#include <cstdio>
#include "spmm_rows.cuh"
int main() {
  int op, slice, dim, esz, heads, what;
  long long edges;
  while (scanf("%d %d %d %d %d %lld %d", &op, &slice, &dim, &esz, &heads, &edges, &what) == 7)
    printf("%d\n", what == 20 ? apt::stream_blocks(dim, edges, apt::part_room(edges), apt::stream_plan(op, dim, esz, heads).warps, false)
                              : (int)apt::stream_fits(op, slice, dim, esz, heads, edges, what != 0));
}
"""
COPY_U, MUL_W, DOTS = 0, 4, 5
SORTED, GROUPED, BLOCKS = 0, 1, 20


@pytest.fixture(scope="module")
def fits(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("needs nvcc")
    folder = tmp_path_factory.mktemp("rule")
    (folder / "rule.cu").write_text(PROGRAM)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC, str(folder / "rule.cu"), "-o",
                    str(folder / "rule")], check=True)

    def ask(*questions):
        text = "\n".join(" ".join(str(int(v)) for v in q) for q in questions)
        return [int(v) for v in subprocess.run([str(folder / "rule")], input=text, capture_output=True, text=True, check=True).stdout.split()]
    return ask


@pytest.mark.parametrize("op,heads", [(COPY_U, 1), (MUL_W, 4), (DOTS, 4)])
def test_slots_stay_within_31_bits(fits, op, heads):
    # a warp looks at slots behind the last one: the number of the last of these has to fit an int
    ahead = 159
    got = fits(*[(op, 16, 128, 4, heads, e, g) for e in (1 << 30, 2 ** 31 - 2 - ahead, 2 ** 31 - 2) for g in (SORTED, GROUPED)])
    assert got[:2] == [1, 1] and got[4:] == [0, 0]
    # not further up than that, where it still fits
    assert fits((op, 16, 128, 4, heads, 2 ** 31 - 8192, SORTED)) == [1]


@pytest.mark.parametrize("esz,dim,warps", [(4, 128, 12), (4, 256, 10), (2, 256, 12), (2, 512, 10)])
def test_partial_sums_find_room(fits, esz, dim, warps):
    # stretches of 32 edges, on up to two blocks an SM, whatever the width
    for edges in (98_304, 135_000, 196_608, 1_013_760):
        assert fits((COPY_U, 16, dim, esz, 1, edges, BLOCKS)) == [min(296, edges // (32 * warps))]


@pytest.mark.parametrize("edges,heads", [(1, 1), (50_000, 4), (98_303, 16), (98_304, 16), (98_304, 17), (1_013_760, 4)])
def test_the_attention_backward_holds_one_order(edges, heads):
    # beside what the sums behind a sort take: fp32 sums of the score gradients, the dots, and 16 bytes a slot where the stream may
    # take the walk instead of 8
    sources = 20_000
    sums, dots = -(-sources // 1024) * 1024 * heads * 4, edges * heads * 4
    more = 8 * edges if edges >= 98_304 and heads <= 16 else 0
    extra = lib.apt_gat_backward_workspace_bytes(sources, edges, heads) - lib.apt_spmm_workspace_bytes(sources, edges)
    assert sums + dots + more <= extra <= sums + dots + more + 3 * 256
