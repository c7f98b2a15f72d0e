"""The two roles of the slot sum through shared memory, run lane by lane on host threads (warp_emulation.cpp): the sums, and
what an aborting launch does to lanes that see it at different polls."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "unimonomoe_b200", "csrc")


@pytest.fixture(scope="module")
def emulation(tmp_path_factory):
    d = tmp_path_factory.mktemp("warps")
    for name in ("bounded_wait.cuh", "slot_copies.cuh"):
        text = open(os.path.join(CSRC, name)).read()
        (d / name).write_text(text.replace('#include "ptx_sm100.cuh"\n', ""))
    exe = str(d / "warps")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-w", f'-DSOURCE="{d}/bounded_wait.cuh"', "-I", str(d),
                    os.path.join(HERE, "warp_emulation.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("case", ["sum", "lanes", "drain", "settle"])
def test_every_lane_comes_to_the_end(emulation, case):
    r = subprocess.run([emulation, case], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
