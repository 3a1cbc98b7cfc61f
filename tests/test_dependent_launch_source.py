"""The kernels of an attention step are programmatic dependents of one another, read from the source: each that is launched as one waits
for the kernel before it, on every path, and each that waits is launched as one."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "openvino.genai_b200" / "csrc"
SOURCES = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("pa_*.cu"))}


def _kernels(text):
    """name -> body of every __global__ function."""
    out = {}
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\([^{;]*?\)\s+)?(\w+)\([^)]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out[m.group(1)] = text[m.end():i]
    return out


def test_dependents_wait_and_waiting_kernels_are_dependents():
    checked = 0
    for name, text in SOURCES.items():
        dependents = "".join(re.findall(r"\bkern(?:el)?\s*=[^;]*;|launch_dependent\([^;]*;|launch\([^;]*;", text))
        for kernel, body in _kernels(text).items():
            waits = "grid_wait()" in body
            assert waits == bool(re.search(r"\b%s\b" % kernel, dependents)), f"{name}: {kernel}"
            assert not (waits and re.search(r"\b%s\s*(<[^;]*>)?\s*<<<" % kernel, text)), f"{name}: {kernel} waits but is launched as any other"
            if waits:
                assert "return" not in body[:body.index("grid_wait()")], f"{name}: {kernel} may leave before it has waited"
                checked += 1
    assert checked >= 7


def test_the_cache_write_releases_early_only_in_front_of_one_cta_per_sm():
    """Two or three waiting CTAs per SM do not all fit beside the cache write's blocks, and those that come late end late."""
    write = _kernels(SOURCES["pa_cache_ops.cu"])["write_kv_kernel"]
    assert re.search(r"if \(a\.release_early\)\s*grid_release\(\)", write) and write.count("grid_release()") == 1
    assert re.search(r"release_early = shared_decode\b", SOURCES["pa_api.cu"])
    shared, sliced = (SOURCES[n] for n in ("pa_decode_shared.cu", "pa_decode.cu"))
    assert re.search(r"__launch_bounds__\(kShMaxWarps \* 32, 1\) decode_shared_kernel", shared)
    assert not re.search(r"__launch_bounds__\([^;{]*?, 1\) decode_kernel", sliced)
