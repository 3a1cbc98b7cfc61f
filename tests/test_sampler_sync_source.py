"""How the warps of the sampler's top-k path hand over to one another, read from the source (comments apart): what the PTX documentation asks
of the instructions used holds by what is written, not by how the compiler happens to schedule a branch.  (A missing wait
or an unconverged barrier is a race that a run on the GPU may or may not show.)"""
import re
from pathlib import Path

SOURCE = re.sub(r"//[^\n]*", "", (Path(__file__).resolve().parent.parent / "openvino.genai_b200" / "csrc" / "sampler.cu").read_text())


def _function(name):
    """Body of the first function called `name`."""
    at = re.search(r"\b%s\([^;{]*\)\s*\{" % name, SOURCE)
    assert at, name
    depth, i = 1, at.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(SOURCE[i], 0)
        i += 1
    return SOURCE[at.end():i - 1]


def test_aligned_barriers_are_reached_by_converged_warps():
    """bar.* and barrier.*.aligned ask for all threads of a warp to execute the same instruction together."""
    helpers = [n for n in ("named_sync", "named_count") if re.search(r"\b(bar|barrier)\.", _function(n))]
    assert helpers == ["named_sync", "named_count"]
    for name in helpers:
        body = _function(name)
        assert "__syncwarp()" in body[:body.index("asm")], f"{name}: nothing converges the warp in front of the barrier"
    rest = SOURCE
    for name in helpers:
        rest = rest.replace(_function(name), "")
    assert not re.search(r'"[^"\n]*\b(bar|barrier)\.[a-z]', rest), "a barrier instruction outside the two helpers"


def test_ring_entries_are_read_and_overwritten_behind_an_acquired_count():
    """The consumer's lane 0 acquires the counts and the warp synchronises before any lane reads an entry; the producers
    acquire the consumer's count before they write to a place again; counts are stored with release."""
    consume, produce = _function("consume_candidates"), _function("produce_candidates")
    acquire, read = consume.index("load_acquire(&sh.head)"), consume.index("sh.ring[")
    assert acquire < read and "__syncwarp()" in consume[acquire:read]
    taken, freed = read, consume.index("store_release(&sh.tail")
    assert taken < freed and "__syncwarp()" in consume[taken:freed]
    assert produce.index("load_acquire(&sh.tail)") < produce.index("sh.ring[")
    for body in (consume, produce):
        assert not re.search(r"volatile[^;]*&sh\.(head|tail|done)\b", body), "a count of the ring without its ordering"
