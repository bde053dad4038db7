"""CPU replay of the fused tile kernel's plan for items of eight or four of a
block's sixteen x-planes (inner x neighbours the block itself), as
test_tile_plan.py replays whole blocks: every face once, no buffer reused
early, every wait satisfied in stream order."""
import itertools
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    out = {}
    for n in (8, 4):
        out[n] = str(tmp_path_factory.mktemp("tile") / f"tile_plan_part_emu_{n}")
        subprocess.run(["g++", "-O1", "-std=c++17", "-Wno-unknown-pragmas", f"-DNX_PLANES={n}",
                        "-o", out[n], os.path.join(HERE, "tile_plan_emu.cpp")], check=True)
    return out


@pytest.mark.parametrize("planes,x0", [(8, 0), (8, 8), (4, 0), (4, 4), (4, 8), (4, 12)])
@pytest.mark.parametrize("x", list(itertools.product((0, 1, 2), repeat=2)))
@pytest.mark.parametrize("yz", [(0, 0, 0, 0), (1, 2, 2, 1), (2, 0, 1, 1), (0, 2, 0, 1)])
def test_part_plan_replay(emu, x, yz, planes, x0):
    r = subprocess.run([emu[planes]] + [str(k) for k in x + yz + (x0,)], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    # x faces of planes + 1 face planes, 17 x 16 y and z faces of each plane
    assert r.stdout.split() == ["ok", str(256 * (planes + 1) + 2 * 272 * planes), str(256 * planes)]
