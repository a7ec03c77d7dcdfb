"""A cell's mass and centre from integer sums (csrc/moments.cuh, compiled for the
host) are those of the reference's double sums, bit for bit: ordinary cells,
masses over eleven binades, centres halfway between floats, coordinates of both
signs, sums that cancel, more children than the integer path takes."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = "/usr/local/cuda/include"
KINDS = ["ordinary", "wide masses", "ties", "both signs", "cancelling", "many children"]


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if not shutil.which("g++") or not os.path.isdir(CUDA):
        pytest.skip("no host compiler or CUDA headers")
    exe = str(tmp_path_factory.mktemp("moments") / "driver")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", CUDA,
                    os.path.join(HERE, "cell_moments_driver.cpp"), "-o", exe], check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("kind", KINDS)
def test_cells_match_the_double_sums(driver, kind):
    out = subprocess.run([driver, str(KINDS.index(kind)), "300000", "7"], check=True, capture_output=True, text=True)
    assert int(out.stdout) == 0, out.stdout
