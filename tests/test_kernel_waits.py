"""Bounded waits of the kernels, by reading their sources: a wait that gives up must answer for the whole warp.  The lanes of a warp poll a
barrier at different times; one that leaves its role alone leaves the others at the warp's next collective (a vote, __syncwarp,
tcgen05.ld.sync.aligned) for good, which cannot be tried on a device."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kronos-2t_b200", "csrc")
PER_THREAD = r"\bmbar_wait_(?:thread|bounded)\("
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and f != "k2t_device.cuh" and re.search(PER_THREAD, open(os.path.join(CSRC, f)).read()))


def lone_waits(text):
    """Per-thread waits whose answer a warp's lanes take apart: neither inside a block (or behind a condition) of one thread, nor voted on
    in their statement or in the one behind it."""
    text = re.sub(r"//[^\n]*", "", text)
    bad = []
    for m in re.finditer(PER_THREAD, text):
        headers, depth, start = [], 0, m.start()
        for i in range(m.start() - 1, -1, -1):          # headers of the enclosing blocks
            if text[i] == "}":
                depth += 1
            elif text[i] == "{":
                depth -= 1
                if depth < 0:
                    depth = 0
                    j = max(text.rfind(c, 0, i) for c in ";{}")
                    headers.append(text[j + 1:i])
        start = max(text.rfind(c, 0, m.start()) for c in ";{}") + 1
        end = text.index(";", m.end())
        following = text[end:].split(";", 2)
        here, behind = text[start:end], following[1] if len(following) > 1 else ""
        if "__device__" in here + "".join(headers[:1]) and "bool mbar_wait" in here + "".join(headers[:1]):
            continue          # its own definition
        voted = re.search(r"__(all_sync|any_sync|syncthreads_or)\(", here + behind)
        if not voted and not any(re.search(r"\b(lane|tid) == 0\b", h) for h in headers):
            bad.append(text[start:end].strip())
    return bad


@pytest.mark.parametrize("source", SOURCES)
def test_a_wait_that_gives_up_answers_for_the_warp(source):
    assert lone_waits(open(os.path.join(CSRC, source)).read()) == []


def test_the_reading_sees_a_lane_that_leaves_alone():
    role = "if (warp < 4) { for (;;) { ok = %s; if (!ok) break; __syncwarp(); } }"
    assert lone_waits(role % "mbar_wait_thread(bar, 0, 9, s_abort)")
    assert lone_waits(role % "mbar_wait_warp(bar, 0, 9, s_abort)") == []
    assert lone_waits(role.replace("warp < 4", "lane == 0") % "mbar_wait_thread(bar, 0, 9, s_abort)") == []
