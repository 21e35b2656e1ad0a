"""How the quadrature passes cut a level and fill an SM: the host side of pffrg_flow.cuh, run on the CPU.

A small host program built from the header prints what the passes would use; the expectations are restated
here.  A level of n new nodes on nact subdomains is cut into chunks of at most 32 nodes (at most 256 chunks
per subdomain); the chunks are halved while fewer than `teams` of them exist, within half the capacity, and
the partial sums' upper half is then free for the sums of |node values|.
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
    for (int batch : {1, 2, 4})
        for (int least : {1, batch})
            for (int teams : {4864, 19456})
                for (int qcap : {64, 100, 1024, 65536, 1 << 20})
                    for (int nact : {0, 1, 3, 17, 150, 4000, 70000})
                        for (int wave = 1; wave <= 21; ++wave) {
                            const LevelCut k = cut_level(nact, 2ll << wave, qcap, batch, least, teams);
                            std::printf("cut %d %d %d %d %d %d %d %d %d %d %d\n", batch, least, teams, qcap, nact, wave,
                                        k.nact, k.coarse, k.chunks, k.per, (int)k.overflow);
                        }
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


def test_cut_of_a_level(printed):
    cuts = [list(map(int, x[1:])) for x in printed if x[0] == "cut"]
    assert len(cuts) == 3 * 2 * 2 * 5 * 7 * 21
    finer = 0
    for batch, least, teams, qcap, nact, wave, act, coarse, chunks, per, overflow in cuts:
        n = 2 << wave
        assert coarse == min(256, max(1, n // 32))
        assert chunks * per == n and chunks % coarse == 0  # every node once, coarse chunks cut evenly
        assert overflow == (nact * coarse > qcap)
        assert act == (qcap // coarse if overflow else nact)
        assert act * chunks <= qcap
        assert per >= min(least, 32)
        if chunks != coarse and act:
            finer += 1
            assert 2 * act * chunks <= qcap  # the other half holds the fine chunks' sums of |node values|
            assert act * chunks <= teams
        if per > batch:  # no finer cut of whole batches was left
            assert 2 * act * chunks > min(teams, qcap // 2)
    assert finer > 1000


def test_capacity_just_above_the_coarse_chunks_forbids_the_fine_cut(printed):
    """A capacity of less than twice the coarse chunks is the way to compare both cuts of a level."""
    cuts = {tuple(map(int, x[1:7])): tuple(map(int, x[7:])) for x in printed if x[0] == "cut"}
    for batch in (1, 2, 4):
        coarse = cuts[batch, batch, 19456, 1024, 17, 9]  # 1024 new nodes, 32 coarse chunks on each of 17 subdomains
        fine = cuts[batch, batch, 19456, 1 << 20, 17, 9]
        assert coarse[1:4] == (32, 32, 32)
        assert fine[1:4] == (32, 1024 // batch, batch)


def test_blocks_asked_of_the_compiler_fit_on_an_sm(printed):
    """Registers are held down for a number of blocks that shared memory allows, and rows are staged where
    that costs none of these blocks (15 sites: 57.2 KB a block, four fit, with 2.5 KB of rows three)."""
    shapes = [list(map(int, x[1:])) for x in printed if x[0] == "shape"]
    assert len(shapes) == 5
    for size, T, C, SPL, Ns, blocks, smem, staged in shapes:
        assert blocks * (smem + 1024) <= 228 * 1024, (T, Ns)
        assert staged == (Ns < 15), (T, Ns)
