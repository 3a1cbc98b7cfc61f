"""Builds and runs tests/cpp/segment_sum_test.cpp: the rules by which the whole-vocabulary sampler rows are summed in segments
(segment_sum.cuh, the header the CUDA kernel is compiled from), with lanes, guessed binades and a walk restated on the CPU."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = tmp_path_factory.mktemp("segment_sum") / "segment_sum_test"
    cmd = ["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "openvino.genai_b200" / "csrc"),
           str(ROOT / "tests" / "cpp" / "segment_sum_test.cpp"), "-o", str(out)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return out


def run(exe, *args):
    res = subprocess.run([str(exe), *args], capture_output=True, text=True)
    sys.stdout.write(res.stdout)
    assert res.returncode == 0, res.stdout + res.stderr


def test_sums_and_crossings_are_those_of_the_plain_loop(exe):
    run(exe, "sums", "3")


def test_rows_whose_sum_begins_late_are_walked_by_their_amounts(exe):
    """Grammar masks, low temperatures, a late peak: a segment that adds nothing, or to a sum that is zero or tiny, is no wrong guess."""
    run(exe, "late", "3")
