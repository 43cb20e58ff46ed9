"""Index arithmetic of the kernels at the ends of its range, compiled for the host."""
import os
import subprocess

import pytest

from conftest import ROOT

PROGRAM = """
#include "grws_common.cuh"
#include <stdlib.h>
int main(int argc, char **argv) {
    for (int lane = 0; lane < 32; ++lane) printf("%d", (int)grws::lane_has_entry(atoi(argv[1]), lane, atoi(argv[2])));
}
"""


@pytest.fixture(scope="module")
def lanes(tmp_path_factory):
    d = tmp_path_factory.mktemp("index")
    (d / "main.cu").write_text(PROGRAM)
    subprocess.check_call(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-ccbin", "/usr/bin/g++",
                           "-I", os.path.join(ROOT, "graph_rws_b200", "csrc"), str(d / "main.cu"), "-o", str(d / "main")])
    return lambda p, end: subprocess.check_output([str(d / "main"), str(p), str(end)], text=True)


@pytest.mark.parametrize("p,end", [(0, 0), (0, 1), (5, 36), (5, 37), (5, 38), (2 ** 31 - 34, 2 ** 31 - 2), (2 ** 31 - 10, 2 ** 31 - 2),
                                   (2 ** 31 - 2, 2 ** 31 - 2)])
def test_lanes_of_a_run_of_entries(lanes, p, end):
    assert lanes(p, end) == "".join(str(int(p + lane < end)) for lane in range(32))
