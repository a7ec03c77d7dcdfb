"""A handle's creation that fails at any of its runtime calls leaves no stream,
event or buffer behind (csrc/resources.cuh against a counting runtime)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if not shutil.which("g++") or not os.path.isdir(CUDA):
        pytest.skip("no host compiler or CUDA headers")
    exe = str(tmp_path_factory.mktemp("resources") / "driver")
    subprocess.run(["g++", "-std=c++17", "-x", "c++", "-I", CUDA, os.path.join(HERE, "resources_driver.cpp"), "-o", exe],
                   check=True, capture_output=True)

    def call(*args):
        return subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True).stdout.split("\n")[:-1]
    return call


def test_every_failure_is_cleaned_up(run):
    whole = run()
    assert len(whole) == 1 and whole[0].startswith("rc 0 ") and whole[0].endswith("live 0"), whole
    calls = int(whole[0].split()[3])
    assert calls > 10
    for k in range(calls):
        out = run(k)
        assert len(out) == 1 and not out[0].startswith("rc 0 ") and out[0].endswith("live 0"), (k, out)


def test_nothing_is_pending_when_the_handle_is_returned(run):
    """The ticket is zero before any stream, the caller's own included, can reach a kernel that takes it."""
    assert " pending 0 " in run()[0]
