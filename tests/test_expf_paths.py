"""The exponentials of whole-vocabulary rows have the host libm's bits in every form that the kernel uses: the form for
non-positive arguments is compared with libm here, and what sampler_b200_selftest_expf runs on the device covers them all."""
import re
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
SOURCE = re.sub(r"//[^\n]*", "", (ROOT / "openvino.genai_b200" / "csrc" / "sampler_exact.cu").read_text())


def test_nonpositive_form_has_the_bits_of_libm(tmp_path):
    exe = tmp_path / "expf_nonpositive_test"
    cmd = ["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "openvino.genai_b200" / "csrc"),
           str(ROOT / "tests" / "cpp" / "expf_nonpositive_test.cpp"), "-o", str(exe)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    run = subprocess.run([str(exe), "61"], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout + run.stderr


def test_the_selftest_runs_every_form_that_the_rows_use():
    forms = set(re.findall(r"\bfloat (expf_\w+)\(", SOURCE))
    assert forms, "no exponential found"
    at = re.search(r"void expf_selftest_kernel\([^)]*\)\s*\{", SOURCE)
    body = SOURCE[at.end():SOURCE.index("\n}", at.end())]
    rows = SOURCE[:at.start()] + SOURCE[at.end() + len(body):]
    used = {f for f in forms if len(re.findall(r"\b%s\(" % f, rows)) > 1}
    assert used and all(re.search(r"\b%s\(" % f, body) for f in used), (used, body)
