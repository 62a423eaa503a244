"""Bounded waits of the kernels, by reading their sources: a wait that gives up must not split a warp.  The lanes of a warp poll a barrier at
different times; one that leaves its role alone leaves the others at the warp's next collective (a vote, __syncwarp,
tcgen05.ld.sync.aligned) for good, which cannot be tried on a device."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kronos-2t_b200", "csrc")
WAIT = re.compile(r"\bmbar_wait_(?:thread|bounded)\(")
VOTE = re.compile(r"__all_sync\(|__any_sync\(|__syncthreads_or\(|mbar_wait_warp\(")
LEAVE = re.compile(r"if \([^;{}]*!(ok)\b[^;{}]*\)\s*(?:\{[^{}]*)?\b(?:break|return)\b|if \([^;{}]*\b(failed)\b[^;{}]*\)\s*(?:\{[^{}]*)?\b(?:break|return)\b"
                   r"|for \([^;]*;[^;]*&& (ok)\b[^;]*;|for \([^;]*;[^;]*&& !(failed)\b[^;]*;")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and f != "k2t_device.cuh" and WAIT.search(open(os.path.join(CSRC, f)).read()))


def headers(text, at):
    """What stands in front of the blocks around a place, from the inside out."""
    out, depth = [], 0
    for i in range(at - 1, -1, -1):
        if text[i] == "}":
            depth += 1
        elif text[i] == "{" and depth:
            depth -= 1
        elif text[i] == "{":
            out.append(text[max(text.rfind(c, 0, i) for c in ";{}") + 1:i])
    return out


def of_one_thread(text, at):
    return any(re.search(r"\b(?:lane|tid) == 0\b", h) for h in headers(text, at)) or re.search(r"\b(?:lane|tid) == 0\)\s*$", text[:at])


def drained(text, at):
    """The loop around a place is followed by the __syncwarps that it had left (its only collectives), or the place runs its own."""
    if re.match(r"[^;{}]*\)\s*\{ __syncwarp\(\); return false; \}", text[at:]):
        return True
    depth = 0
    for i in range(at - 1, -1, -1):
        depth += {"}": 1, "{": -1}.get(text[i], 0)
        if depth < 0:
            depth = 0
            if re.search(r"\bfor \([^{}]*$", text[max(text.rfind(c, 0, i) for c in "{}") + 1:i]):
                break
    else:
        return False
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            body = text[i:j]
            return not re.search(r"__(all|any)_sync|shfl|tcgen05|hf_ld16|tc_ld", body) and bool(re.match(r"\}\s*for \(; [^)]*\) (?:\{\s*)?(?:if \([^)]*\) )?__syncwarp\(\);", text[j:]))
    return False


def splits(text):
    """Places of a role of several lanes where a lane takes its own answer and leaves, or takes one that it may leave by."""
    text = re.sub(r"//[^\n]*", "", text)
    bad = []
    for m in WAIT.finditer(text):
        start, end = max(text.rfind(c, 0, m.start()) for c in ";{}") + 1, text.index(";", m.end())
        statement, behind = text[start:end], text[end + 1:].split(";", 1)[0]
        if re.search(r"bool mbar_wait\w+\($|__device__", statement) or "bool mbar_wait" in "".join(headers(text, m.start())[:1]) or of_one_thread(text, m.start()):
            continue
        stays = re.search(r"\bok = ok && |\bfailed = failed \|\| ", statement)
        if not stays and not VOTE.search(statement + ";" + behind) and not drained(text, m.start()):
            bad.append(statement.strip())
    for m in LEAVE.finditer(text):
        name = next(g for g in m.groups() if g)
        before = re.findall(rf"\b{name} = ([^;]*);", text[:m.start()])
        loop = m.start() if m.group(0).startswith("if") else text.index("{" if ") {" in text[m.start():m.start() + 200] else ";", m.end()) + 1
        if of_one_thread(text, m.start()) or (before and VOTE.search(before[-1])) or drained(text, loop):
            continue
        if m.group(0).startswith("for") and re.match(r"[^;{}]*\) [^;{}]*;\s*for \(; [^)]*\) __syncwarp\(\);", text[m.end():]):
            continue          # a loop of one statement
        bad.append(m.group(0))
    return bad


@pytest.mark.parametrize("source", SOURCES)
def test_a_wait_that_gives_up_does_not_split_its_warp(source):
    assert splits(open(os.path.join(CSRC, source)).read()) == []


@pytest.mark.parametrize("role,found", [
    ("ok = mbar_wait_thread(bar, 0, 9, s_abort); if (!ok) break; __syncwarp();", True),
    ("if (!mbar_wait_bounded(bar, 0)) return false; __syncwarp();", True),
    ("ok = ok && mbar_wait_thread(bar, 0, 9, s_abort); if (!ok) { failed = true; break; } __syncwarp();", True),
    ("ok = mbar_wait_warp(bar, 0, 9, s_abort); if (!ok) break; __syncwarp();", False),
    ("ok = ok && mbar_wait_thread(bar, 0, 9, s_abort); __syncwarp();", False),
    ("ok = mbar_wait_thread(bar, 0, 9, s_abort); if (!ok) break; __syncwarp(); } for (; i < n; ++i) { __syncwarp();", False),
    ("ok = mbar_wait_thread(bar, 0, 9, s_abort); if (!ok) break; tc_ld8(t, v); } for (; i < n; ++i) { __syncwarp();", True),
])
def test_the_reading_itself(role, found):
    assert bool(splits("void kernel() { if (warp < 4) { for (;;) { " + role + " } } }")) is found
    assert splits("void kernel() { if (lane == 0) { for (;;) { " + role + " } } }") == []


@pytest.mark.parametrize("source", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_a_wait_is_not_cut_short_by_an_earlier_one(source):
    """A role that asks for its next copy whatever the last wait said polls for each of them up to the limit: a loop that an earlier answer ends
    would let the CTA leave while copies into its shared memory are in flight."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, source)).read())
    assert re.findall(r"for \([^;]*\bspin\b[^;]*;[^;]*(?<![!\w])ok\b[^;]*;[^)]*\)", text) == []


def test_prompt_gemm_waits_for_what_it_issued():
    """The threads that ask for activations and issue products wait for the last of them on every way out: a role that gives up elsewhere would otherwise
    let the CTA leave, and its tensor memory go back, while these are in flight."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "k2t_gemm_prompt.cu")).read())
    drains = list(re.finditer(r"spin < \w*WAIT_LIMIT && !mbar_try_wait\((bar_last|bar_bfull)", text))
    assert [m.group(1) for m in drains] == ["bar_last", "bar_bfull"]
    for m in drains:
        assert not any("!ok" in h for h in headers(text, m.start()))
