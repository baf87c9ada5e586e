"""The address of a cell list's slot in the largest grids that a system takes
(just below 2^30 cells of 8 or 16 slots), computed on the host by the function
that the list build uses."""
import subprocess

import pytest

from conftest import REPO
from nwgb import build

PROGRAM = r"""
#include <cstdio>
#include "nw_device.cuh"
int main()
{
    const uint32_t cells[] = {0u, 1u, (1u << 28) - 1u, 1u << 28, (1u << 29) + 5u, (1u << 30) - 1u};
    for (uint32_t cap : {8u, 16u})
        for (uint32_t c : cells) std::printf("%u %u %llu\n", cap, c, (unsigned long long)nw::list_slot(c, cap - 1u, cap));
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    d = tmp_path_factory.mktemp("address")
    (d / "p.cu").write_text(PROGRAM)
    subprocess.run([str(build._cuda_home() / "bin" / "nvcc"), *build.ARCH, "-std=c++17", f"-I{build.CSRC}", "-o", str(d / "p"),
                    str(d / "p.cu")], check=True)
    return subprocess.run([str(d / "p")], check=True, capture_output=True, text=True).stdout.splitlines()


def test_slots_of_large_grids(lines):
    assert len(lines) == 12
    for line in lines:
        cap, cell, at = map(int, line.split())
        assert at == cell * cap + cap - 1


def test_the_list_builds_take_their_slots_from_it():
    src = (REPO / "nematic-worms_gb300" / "csrc" / "nw_fused_impl.cuh").read_text()
    build_3d = src[src.index("uint32_t verlet_build("):src.index("uint32_t verlet_build(") + 4000]
    assert "list_slot(" in build_3d and "* CAP" not in build_3d
