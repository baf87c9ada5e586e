"""Ranks of a crowded SRD cell's members, computed on the host by the function
that the collision uses: a permutation also where indices repeat, so that
every place of the ordered members is written."""
import subprocess

import pytest

from conftest import REPO
from nwgb import build

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "nw_device.cuh"
int main(int argc, char** argv)
{
    uint32_t ids[384], n = (uint32_t)argc - 1u;
    for (uint32_t k = 0; k < n; ++k) ids[k] = (uint32_t)std::strtoul(argv[k + 1], nullptr, 10);
    for (uint32_t k = 0; k < n; ++k) std::printf("%u\n", nw::rank_of(ids, n, k));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("rank")
    (d / "p.cu").write_text(PROGRAM)
    subprocess.run([str(build._cuda_home() / "bin" / "nvcc"), *build.ARCH, "-std=c++17", f"-I{build.CSRC}", "-o", str(d / "p"),
                    str(d / "p.cu")], check=True)
    return str(d / "p")


@pytest.mark.parametrize("ids", [[3], [5, 5], [9, 2, 7, 4], [8, 0, 8, 0, 8, 1], [4] * 20, [0, 4294967295, 4294967295, 1],
                                 [(k * 37) % 50 // 3 for k in range(60)]])
def test_ranks_are_a_permutation(program, ids):
    out = subprocess.run([program, *map(str, ids)], check=True, capture_output=True, text=True).stdout.split()
    ranks = [int(x) for x in out]
    assert sorted(ranks) == list(range(len(ids)))
    assert [ids[k] for k in sorted(range(len(ids)), key=lambda k: ranks[k])] == sorted(ids)


def test_the_collision_of_crowded_cells_ranks_by_it():
    src = (REPO / "nematic-worms_gb300" / "csrc" / "nw_srd.cu").read_text()
    kernel = src[src.index("srd_collide_big_kernel(const DevParams"):]
    assert "rank_of(" in kernel and "s_in[w][j] < x" not in kernel
