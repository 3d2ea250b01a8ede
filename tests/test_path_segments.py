"""Which paths a whole-path launch takes when a lane that an earlier launch has finished is still
among its segments (the job engine's waves in flight), on the CPU: the kernel's own segment
functions (luxion_b200/csrc/path_segs.h) in a model of its blocks and its work assignment
(path_segs_model.cpp)."""
import os
import subprocess

import pytest

from luxion_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def cases(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("path_segs") / "model")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + build.CSRC, "-I" + os.path.join(build.CUDA_HOME, "include"),
                    os.path.join(HERE, "path_segs_model.cpp"), "-o", exe], check=True)
    lines = [ln.split() for ln in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert len(lines) == 128
    return lines


def test_blocks_agree_whenever_they_start(cases):
    assert [c for c in cases if c[3] != "agree"] == []


def test_every_path_not_yet_finished_is_taken_once(cases):
    assert [c for c in cases if c[4] != "cover"] == []
