"""The fused tile kernel numbers its work items in 32 bits: the steps one launch may
run (tile_plan.cuh) keep every item number, and one more per CTA, in range."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = r"""
#define __host__
#define __device__
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include "tile_plan.cuh"
int main(int, char **v) {
  std::printf("%d\n", alp::tile::max_steps_per_launch(std::atoi(v[1]), std::atoi(v[2]),
                                                      std::atoi(v[3]), std::atoi(v[4])));
}
"""


@pytest.fixture(scope="module")
def steps(tmp_path_factory):
    d = tmp_path_factory.mktemp("steps")
    (d / "steps.cpp").write_text(SOURCE)
    exe = str(d / "steps")
    subprocess.run(["g++", "-std=c++17", "-Wno-unknown-pragmas", "-o", exe, str(d / "steps.cpp"),
                    "-I", os.path.join(HERE, "..", "alpaca_b200", "csrc")], check=True)
    return lambda *a: int(subprocess.run([exe] + [str(x) for x in a], check=True,
                                         capture_output=True, text=True).stdout)


@pytest.mark.parametrize("nwork,parts", [(1, 4), (37, 4), (38, 2), (147, 2), (148, 1),
                                         (2048, 1), (100000, 1)])
@pytest.mark.parametrize("nstages", [2, 3])
def test_items_stay_in_32_bits(steps, nwork, parts, nstages):
    ctas = 148
    n = steps(nwork, parts, nstages, ctas)
    assert n * nstages * nwork * parts + ctas < 2 ** 31 <= (n + 1) * nstages * nwork * parts + ctas
