"""Rules of the persistent attention kernel that a run cannot show without a wait that runs out: they are read off its
source.  A timed-out CTA must come to its end, so no warp may wait, without a bound, for a warp that may have gone home."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "chitudiffusion_b200", "csrc")


@pytest.fixture(scope="module")
def code():
    text = open(os.path.join(CSRC, "attn_persist.cuh")).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def test_no_barrier_between_start_and_end_of_a_cta(code):
    """Warps decide on their own whether to take up another unit once a role has given up; a barrier among some of
    them (bar.sync has no bound) would hold those that go on for ever."""
    assert not re.search(r"\bbar\.sync|\bbarrier\.|__barrier_sync|\bbar\.red", code)
    body = code[code.index("attn_persist_kernel("):]
    assert body.count("__syncthreads()") == 2  # after the set-up, before tensor memory is freed


def test_a_warp_decides_as_one(code):
    """Lanes poll separately, so a decision that a branch or a loop depends on is voted on."""
    uses = [m.start() for m in re.finditer(r"\*abort_flag", code[code.index("attn_persist_kernel("):])]
    assert uses
    body = code[code.index("attn_persist_kernel("):]
    assert len(re.findall(r"__any_sync\(0xffffffffu, \*abort_flag", body)) + len(re.findall(r"\*abort_flag = 0", body)) == len(uses)
    for m in re.finditer(r"(if|while)\s*\(\s*!?\s*mbar_wait", body):
        pytest.fail("control flow on one lane's wait: " + body[m.start():m.start() + 80])


def test_lanes_meet_after_a_wait_that_only_some_take(code):
    """Tensor-memory loads and stores are instructions of the whole warp (.sync.aligned): a wait behind a condition that a
    lane evaluated for itself is followed by __syncwarp before the next of them."""
    conditional = re.findall(r"if \(!pv_done\) mbar_wait\([^;]*;\s*(\S+)", code)
    assert conditional and all(nxt.startswith("__syncwarp()") for nxt in conditional)
