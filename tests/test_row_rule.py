"""How sums divide their rows among lanes: the rule itself, compiled for the host."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "apt_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
PROGRAM = r"""
#include <cstdio>
#include "spmm_rows.cuh"
int main() {
  long long dim, edges, rows;
  int ve, ordered;
  while (scanf("%lld %d %lld %lld %d", &dim, &ve, &edges, &rows, &ordered) == 5) {
    const apt::RowSplit r = apt::row_split(dim, ve, edges, rows, ordered != 0);
    printf("%d %d\n", r.lpe, r.ep);
  }
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("needs nvcc")
    folder = tmp_path_factory.mktemp("rule")
    (folder / "rule.cu").write_text(PROGRAM)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC, str(folder / "rule.cu"), "-o",
                    str(folder / "rule")], check=True)

    def ask(*questions):
        text = "\n".join(" ".join(str(int(v)) for v in q) for q in questions)
        out = subprocess.run([str(folder / "rule")], input=text, capture_output=True, text=True, check=True).stdout.split()
        return list(zip(map(int, out[::2]), map(int, out[1::2])))
    return ask


@pytest.mark.parametrize("dim,ve", [(16, 4), (32, 4), (64, 8), (64, 4), (128, 8), (10, 2), (256, 8)])
def test_long_rows_keep_their_edges_side_by_side(split, dim, ve):
    """Rows that fill the chip take one edge at a time up to a length of row, beyond it as many as go; the length is that of rows in a list, of
    many of them, or of rows whose edges are one after another."""
    for rows, ordered, longest in ((7_000, 1, 16), (24_575, 1, 16), (24_576, 1, 24), (300_000, 1, 24), (7_000, 0, 40), (300_000, 0, 40)):
        at, above = split((dim, ve, rows * longest, rows, ordered), (dim, ve, rows * longest + 1, rows, ordered))
        lanes = at[0]
        most = 1
        while 2 * most <= min(32 // lanes, longest // 2):
            most *= 2
        assert above == (lanes, most)
        filled = rows * max(lanes, 4) * 2 > 148 * 24 * 32
        assert at[1] == (1 if filled and lanes >= 4 else at[1]) <= most
    assert split((dim, ve, 15 * 60_000, 60_000, 1))[0][1] == 1


def test_few_rows_take_as_many_edges_as_go(split):
    assert split((16, 4, 500 * 15, 500, 1), (16, 4, 500 * 15, 500, 0), (16, 4, 500 * 100, 500, 1)) == [(4, 4), (4, 4), (4, 8)]


DOTS = r"""
#include <cstdio>
#include "gat_dots.cuh"
int main() {
  int bf16, heads, dim, slice;
  long long edges, dst;
  while (scanf("%d %d %d %d %lld %lld", &bf16, &heads, &dim, &slice, &edges, &dst) == 6)
    printf("%d\n", (int)(bf16 ? apt::dots_mma_fits<__nv_bfloat16>(heads, dim, slice, edges, dst) : apt::dots_mma_fits<__half>(heads, dim, slice, edges, dst)));
}
"""


def test_dots_of_blocks_whose_destinations_are_sparse(tmp_path):
    """Wide rows of many edges with few edges to a destination go to the kernel that fetches the gradient's rows in use alone."""
    if not os.path.exists(NVCC):
        pytest.skip("needs nvcc")
    (tmp_path / "dots.cu").write_text(DOTS)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr", "-I", CSRC, str(tmp_path / "dots.cu"),
                    "-o", str(tmp_path / "dots"), "-cudart", "shared", "-Xlinker", "--unresolved-symbols=ignore-all"], check=True)
    ask = lambda *q: [int(v) for v in subprocess.run([str(tmp_path / "dots")], input="\n".join(" ".join(map(str, x)) for x in q), capture_output=True,      # noqa: E731
                                                     text=True, check=True).stdout.split()]
    wide = [(b, h, d, 16, e, n) for b, h, d in ((1, 4, 64), (1, 1, 256), (0, 8, 32)) for e, n in
            ((1_000_000, 66_666), (1_000_000, 200_000), (1_000_000, 200_001), (1_000_000, 500_000), (1_000_000, 500_001), (393_215, 400_000))]
    assert ask(*wide) == [1, 1, 0, 0, 0, 1] * 2 + [1, 1, 1, 1, 0, 1]
    # narrow rows, heads that are no power of two, rows that are no whole slices
    assert ask((1, 4, 32, 16, 1_000_000, 900_000), (1, 3, 64, 16, 1_000_000, 60_000), (1, 4, 48, 16, 1_000_000, 60_000), (1, 4, 64, 8, 1_000_000, 60_000)) == [1, 0, 0, 0]
    # bf16 heads of 32 columns, whose products are made twice: wide rows of many edges are the stream's
    assert ask((1, 8, 32, 16, 1_000_000, 60_000), (1, 8, 32, 16, 393_215, 60_000), (1, 4, 64, 16, 1_000_000, 60_000)) == [0, 1, 1]
