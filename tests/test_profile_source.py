"""The cycle trace of the tensor-core prefill kernel (-DPA_PREFILL_PROF), read from the source: what it prints has been
written, by every role that the kernel has."""
import re
from pathlib import Path

SOURCE = (Path(__file__).resolve().parent.parent / "openvino.genai_b200" / "csrc" / "pa_prefill_tc.cu").read_text()


def test_every_printed_role_of_the_prefill_trace_is_recorded():
    roles = int(re.search(r"trace\[(?:kTraceRoles|(\d+))\]\[\d+\]\[\d+\];", SOURCE).group(1) or re.search(r"kTraceRoles = (\d+)", SOURCE).group(1))
    recorded = set()
    for role in re.findall(r"PA_TRACE\(([^,]+),", SOURCE):
        recorded |= {eval(role, {"X": x}) for x in (0, 1)} if role != "role" else set()
    assert recorded == set(range(roles))
    base = re.search(r"base = trace\[(\d+)\]\[(\d+)\]\[0\]", SOURCE)
    assert re.search(r"PA_TRACE\(%s(?: \+ 2 \* X)?, %s," % base.groups(), SOURCE), "nothing records the trace's origin"


def test_the_prefill_trace_takes_no_shared_memory():
    """The 16-bit variants use every byte of shared memory that a CTA can have: with a record of their own there the build with
    the trace could not be launched."""
    assert not re.search(r"__shared__[^;]*\btrace\b", SOURCE)
