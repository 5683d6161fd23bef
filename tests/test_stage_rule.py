"""Which launches stage their neighbourhood windows (csrc/runtime/internal.h): those whose blocks are all resident,
by their shared memory and by the registers of the variant that stages. Compiled for the host; no GPU is used."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "runtime/internal.h"
int main(int, char** argv) {
    fg_spatial_grid g{};
    g.dims = 2;
    g.gridDim[0] = g.gridDim[1] = 8;
    g.gridDim[2] = 1;
    g.binCount = 64;
    std::printf("%d\n", flamegpu::detail::stage_window_fits(g, 0.5, 4, 128, std::atoi(argv[1]) * 1024, std::atoi(argv[2]), 152));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from flamegpu2_gb300.build import ARCH, NVCC
    d = tmp_path_factory.mktemp("stage_rule")
    (d / "main.cu").write_text(MAIN)
    subprocess.run([NVCC] + ARCH + ["-std=c++20", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"),
                                    "-I", os.path.join(ROOT, "flamegpu2_gb300", "csrc"), str(d / "main.cu"), "-o", str(d / "main")],
                   check=True)
    return str(d / "main")


@pytest.mark.parametrize("kb,per_sm", [(8, 4), (24, 4), (40, 4), (48, 3), (96, 2), (200, 1)])
def test_staged_launches_are_resident(program, kb, per_sm):
    for blocks, want in ((1, 1), (152 * per_sm, 1), (152 * per_sm + 1, 0)):
        out = subprocess.run([program, str(kb), str(blocks)], capture_output=True, text=True, check=True)
        assert out.stdout.strip() == str(want), (kb, blocks)
