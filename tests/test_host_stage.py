"""Host copies through the page-locked stage (csrc/host_stage.cpp) against a
CUDA runtime made of host memory (tests/emu/stage_fake.cpp): what a copy does
when the stage cannot be had or another engine holds it up."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "artisynth_core_b200", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("stage") / "stage_fake")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-pthread", "-I", CSRC, "-I", CUDA_INC,
                        os.path.join(ROOT, "tests", "emu", "stage_fake.cpp"), os.path.join(CSRC, "host_stage.cpp"),
                        "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return out


@pytest.mark.parametrize("scenario", ["no_host_memory", "no_stream", "stage_in_use", "stream_busy"])
def test_copies_without_a_stage(scenario, exe):
    r = subprocess.run([exe, scenario], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
