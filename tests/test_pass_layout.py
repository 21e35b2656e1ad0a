"""How the quadrature passes fill an SM: the host side of pffrg_flow.cuh, run on the CPU.

A small host program built from the header prints what the passes would use.
"""
import os
import shutil
import subprocess

import pytest

PROGRAM = r"""
#include <cstdio>
#include "pffrg_flow.cuh"
using namespace pffrg;
template <typename R, int T, int C, int SPL>
void shape(int Ns, int nm, long long rows) {
    std::printf("shape %d %d %d %d %d %d %zu %d\n", (int)sizeof(R), T, C, SPL, Ns, eval_min_blocks<R, T, SPL, C>(),
                SmemLayout<R, T, C, SPL>(Ns, nm, rows, false).total, (int)stage_rows<R, T, C, SPL>(Ns, nm, rows, 0));
}
int main() {
    const int nm = 51 + 2 * 16 + 2 * 11;
    shape<float, 8, 2, 1>(6, nm, 55);
    shape<float, 16, 2, 1>(9, nm, 136);
    shape<float, 16, 2, 1>(12, nm, 426);
    shape<float, 16, 2, 1>(15, nm, 605);
    shape<float, 32, 2, 1>(31, nm, 3007);
}
"""


@pytest.fixture(scope="module")
def printed(pkg, tmp_path_factory):
    import pffrg_gb300.build as b

    nvcc = b.NVCC if os.path.exists(b.NVCC) else shutil.which("nvcc")
    if not nvcc:
        pytest.skip("nvcc is not installed")
    d = tmp_path_factory.mktemp("layout")
    (d / "layout.cu").write_text(PROGRAM)
    subprocess.run([nvcc, *b.ARCH, "-std=c++17", "-I", str(b.CSRC), "-o", str(d / "layout"), str(d / "layout.cu")], check=True)
    out = subprocess.run([str(d / "layout")], check=True, capture_output=True, text=True).stdout.splitlines()
    return [line.split() for line in out]


def test_blocks_asked_of_the_compiler_fit_on_an_sm(printed):
    """Registers are held down for a number of blocks that shared memory allows, and rows are staged where
    that costs none of these blocks (15 sites: 57.2 KB a block, four fit, with 2.5 KB of rows three)."""
    shapes = [list(map(int, x[1:])) for x in printed if x[0] == "shape"]
    assert len(shapes) == 5
    for size, T, C, SPL, Ns, blocks, smem, staged in shapes:
        assert blocks * (smem + 1024) <= 228 * 1024, (T, Ns)
        assert staged == (Ns < 15), (T, Ns)
