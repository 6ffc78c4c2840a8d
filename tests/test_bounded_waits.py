"""Every wait on an mbarrier ends: it gives up after a number of polls, and the kernel returns an error. That holds only if threads that
meet again give up together. A lane that leaves its warp's loop alone is waited for, for ever, at the warp's next election, vote,
shuffle or tensor-memory access, and a warp that leaves a role alone at the role's next named barrier. Read from the sources: where a
role has such instructions, its waits are a warp's (mbar_wait_warp) or are agreed on by the role before anybody acts on them."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cwick_b200", "csrc")
SOURCES = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu")) if "mbar_wait" in open(f).read())
WARP_WIDE = re.compile(r"elect_one\(|_sync\(|__syncwarp\(|\.sync\.aligned|TMEM_(?:LD|ST)\d+\(|mbar_wait_warp\(|\barrive\(")
ONE_LANE = re.compile(r"\blane == 0\b|\btid == \d+\b")


def strip(text):
    text = re.sub(r"/\*.*?\*/", lambda m: re.sub(r"[^\n]", " ", m[0]), text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def blocks(text):
    """(header, begin, end, parent) of every pair of braces; the header is what stands before it since the last statement."""
    out, stack, last = [], [], 0
    depth = 0
    for i, c in enumerate(text):
        depth += (c == "(") - (c == ")")
        if c == "{":
            out.append([text[last:i].strip(), i, None, stack[-1] if stack else None])
            stack.append(len(out) - 1)
            last = i + 1
        elif c == "}":
            out[stack.pop()][2] = i
            last = i + 1
        elif c == ";" and depth == 0:
            last = i + 1
    return out


def waits(text):
    """Bare waits whose result decides something: (position, enclosing blocks from the inside out)."""
    bl = blocks(text)
    for m in re.finditer(r"\bmbar_wait\(", text):
        inside = [b for b in bl if b[1] < m.start() < b[2]]
        inside.sort(key=lambda b: b[1] - b[2], reverse=True)
        statement = re.split(r"[;{}]", text[:m.start()])[-1].strip()
        statement = re.sub(r"^(for|if|else)\b.*\)\s*(?=$)", "", statement, flags=re.S)
        if statement:                                        # (otherwise: the result is not used, the thread carries on)
            yield m.start(), statement, inside


@pytest.mark.parametrize("name", SOURCES)
def test_a_warp_gives_up_as_a_whole(name):
    text = strip(open(os.path.join(CSRC, name)).read())
    bad = []
    for at, statement, inside in waits(text):
        if any(ONE_LANE.search(b[0]) for b in inside) or "__all_sync(0xffffffffu," in statement:
            continue
        lambda_ = any("->" in b[0] for b in inside)          # (several roles call it)
        role = next((b for b in inside if re.search(r"\bif \(.*\bwarp\b", b[0])), inside[-1])
        # voted on further down, with no way out in between; or told to the whole role, which looks at it together
        vote = text.find("__all_sync(0xffffffffu, here)", at)
        agreed = ("bool here =" in statement and 0 < vote < role[2] and not re.search(r"\b(break|continue|return)\b", text[at:vote])
                  or re.match(r"[^;]*\)\) s_\w+\[[^\]]+\] = 1;", text[at:]))
        if not agreed and (lambda_ or WARP_WIDE.search(text[role[1]:role[2]])):
            bad.append("line %d: %s" % (text.count("\n", 0, at) + 1, text[at:text.index(";", at)]))
    assert not bad, "\n".join(bad)


@pytest.mark.parametrize("name", [n for n in SOURCES if "mbar_wait_on(" in open(os.path.join(CSRC, n)).read()])
def test_a_loop_that_carries_on_only_issues_and_commits(name):
    """mbar_wait_on carries on when it gives up. Its loop must have no way out that a lane could take alone, do nothing that counts bytes at a
    barrier, and let what was issued end before the block does."""
    text = strip(open(os.path.join(CSRC, name)).read())
    for m in re.finditer(r"\bmbar_wait_on\(", text):
        inside = sorted((b for b in blocks(text) if b[1] < m.start() < b[2]), key=lambda b: b[1] - b[2], reverse=True)
        loop = next(b for b in inside if re.search(r"\bfor \(", b[0]))
        role = next(b for b in inside if re.search(r"\bif \(.*\bwarp\b", b[0]))
        body, after = text[loop[1]:loop[2]], text[loop[2]:role[2]]
        assert not re.search(r"\b(break|continue|return|mbar_expect_tx|copy_to_peer|tma_load\w*)\b", body), body
        assert "&& ok" not in loop[0] and "settle(patience != WAIT_LIMIT);" in after, loop[0]


@pytest.mark.parametrize("name", [n for n in SOURCES if re.search(r"softmax_bar\(|\bbar\.sync", open(os.path.join(CSRC, n)).read())])
def test_a_role_gives_up_as_a_whole_where_its_warps_meet(name):
    """Where a role has named barriers, a wait that gives up is told to all of it (a word in shared memory) before the next barrier in the text."""
    text = strip(open(os.path.join(CSRC, name)).read())
    meet = re.compile(r"softmax_bar\(\);|\"bar\.(?:sync|red)[^\"]* 1, \d+")
    for m in re.finditer(r"\bmbar_wait(?:_warp)?\(", text):
        inside = sorted((b for b in blocks(text) if b[1] < m.start() < b[2]), key=lambda b: b[1] - b[2], reverse=True)
        if any(ONE_LANE.search(b[0]) for b in inside):
            continue
        role = next((b for b in inside if re.search(r"\bif \(.*\bwarp\b", b[0]) or b[0].endswith("else")), inside[-1])
        if not meet.search(text[role[1]:role[2]]):
            continue
        nxt = meet.search(text, m.end())
        assert re.search(r"\bs_\w+\[[^\]]+\] = 1;", text[m.end():nxt.start() if nxt and nxt.start() < role[2] else role[2]]), text[m.start():text.index(";", m.start())]
