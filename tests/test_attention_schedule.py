"""The order of a softmax group's steps in ns_attention_prompt.cu: every interleaving of the warp that issues the MMAs, of the tensor pipe and of softmax warps
that run apart, for a few key blocks.  A wait names the parity of a phase: a warp two phases behind its barrier passes too early, one that is a phase too late never
does, and on a quiet GPU no result shows either.  The waits for P.V are read out of the source."""
import os
import re

import pytest

from nn_b200 import build

WARPS = 2        # of the group's four: two suffice to run apart


def _waits():
    """[(condition, d)] of the waits for P.V number k - d: where O is rescaled, before the second half of P is handed over, and where O is read out."""
    text = open(os.path.join(build.CSRC, "ns_attention_prompt.cu")).read()
    text = text[text.index("softmax and output"):]
    cuts = [text.index("hand_over(0, pk)"), text.index("hand_over(1, pk)"), text.index("const float inv")]
    found = [[], [], []]
    for m in re.finditer(r"(?:if \(([^()]*)\) (?:\{\s*)?)?ok = (?:ok && )?wait\(PB_O_DONE \+ g, k - (\d), \d+\)", text):
        found[sum(m.start() > c for c in cuts)].append((m.group(1) or "True", int(m.group(2))))
    return found


def _explore(solo, n, waits):
    """Runs every order of steps.  Fails where O is rescaled before the P.V in front of it or read before the last one, and where a warp waits for good."""
    # the warp that issues the MMAs: S scores, V a half of P.V, ? waits for that half of P
    program = ["S0"]
    for j in range(n):
        scores = [f"S{j + 1}"] if j + 1 < n else []
        halves = [f"?{2 * j}", f"V{2 * j}", f"?{2 * j + 1}", f"V{2 * j + 1}"]
        program += scores + halves if solo else halves + scores
    passes = lambda done, phase: (done & 1) != (phase & 1)           # an mbarrier with `done` completed phases, asked for the parity of `phase`
    asked = lambda at, j: [d for c, d in waits[at] if eval(c.replace("&&", "and"), {"SOLO": solo, "n": n, "j": j})]
    # (steps issued, MMAs completed, the step of each warp): four steps a block (scores, rescale or not, first half, second half), then the read-out's waits
    reads = asked(2, n)
    end = 4 * n + len(reads)
    start = (0, 0, (0,) * WARPS)
    seen, todo = {start}, [start]
    while todo:
        issued, completed, warps = state = todo.pop()
        mmas = [s for s in program[:issued] if s[0] != "?"]
        done = mmas[:completed]
        pv = sum(s[0] == "V" and int(s[1:]) % 2 for s in done)
        after = []
        if completed < len(mmas):
            after.append((issued, completed + 1, warps))
        if issued < len(program):
            half = int(program[issued][1:])
            if program[issued][0] != "?" or all(w > 4 * (half // 2) + 2 + half % 2 for w in warps):
                after.append((issued + 1, completed, warps))
        for i, w in enumerate(warps):
            block, step = min(w // 4, n), w % 4
            ready = True
            if block == n:
                ready = w < end and passes(pv, n - reads[w - 4 * n])
                if ready and w + 1 == end:
                    assert pv == n, f"O of {n} blocks is read after {pv}: {state}"
            elif step == 0:
                scores = sum(s[0] == "S" and (not solo or int(s[1:]) % 2 == block % 2) for s in done)
                ready = passes(scores, block // 2 if solo else block)
            elif step == 1:
                # the maximum may have stayed; else:
                if block > 0 and all(passes(pv, block - d) for d in asked(0, block)):
                    assert pv == block, f"O of block {block} is rescaled after {pv}: {state}"
            elif step == 3:
                ready = all(passes(pv, block - d) for d in asked(1, block))
            if ready:
                after.append((issued, completed, warps[:i] + (w + 1,) + warps[i + 1:]))
        assert after or (issued == len(program) and all(w == end for w in warps)), f"stuck: {state}"
        for x in after:
            if x not in seen:
                seen.add(x)
                todo.append(x)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("solo", [True, False])
def test_o_is_complete_where_it_is_rescaled_and_read(solo, n):
    waits = _waits()
    assert waits[0] and waits[2]
    _explore(solo, n, waits)
