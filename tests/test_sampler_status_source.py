"""The sampler's status bits, read from the source: what the public header describes as an error is set by a kernel, and the hosts
look at no other bit."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "openvino.genai_b200" / "csrc"


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def test_status_bits_that_are_described_and_looked_at_are_set():
    kernels = "".join(_code(p) for p in [*CSRC.glob("sampler*.cu"), *CSRC.glob("sampler*.cuh")])
    set_bits = {int(v).bit_length() - 1 for v in re.findall(r"atomicOr\([^;]*?,\s*(\d+)u\)", kernels)}
    assert set_bits, "no status bit is set"
    header = (ROOT / "include" / "sampler_b200.h").read_text()
    text = header[header.index("Reads (and clears) the device status word"):]
    text = re.sub(r"\s+\*?\s*", " ", text[:text.index("*/")])
    described = {int(b) for b, what in re.findall(r"bit (\d) = ([^,(]*)", text) if "not used" not in what}
    assert described == set_bits
    hosts = _code(CSRC / "sampler_api.cu") + _code(CSRC / "host" / "sampler_host.cpp")
    looked_at = {int(v).bit_length() - 1 for expr in re.findall(r"\bbits & (\d+u|\([^)]*\))", hosts) for v in re.findall(r"(\d+)u", expr)}
    assert looked_at <= set_bits
