"""Which sums and dots go to the kernel that walks the edges as a stream: the rule itself, compiled for the host."""
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
  int op, slice, dim, esz, heads, grouped;
  long long edges;
  while (scanf("%d %d %d %d %d %lld %d", &op, &slice, &dim, &esz, &heads, &edges, &grouped) == 7)
    printf("%d\n", (int)apt::stream_fits(op, slice, dim, esz, heads, edges, grouped != 0));
}
"""
COPY_U, MUL_W, DOTS = 0, 4, 5


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
    got = fits(*[(op, 16, 128, 4, heads, e, g) for e in (1 << 30, 2 ** 31 - 2 - ahead, 2 ** 31 - 2) for g in (0, 1)])
    assert got[:2] == [1, 1] and got[4:] == [0, 0]
    # not further up than that, where it still fits
    assert fits((op, 16, 128, 4, heads, 2 ** 31 - 8192, 0)) == [1]
