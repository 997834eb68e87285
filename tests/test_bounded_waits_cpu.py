"""Every wait of the tensor-core kernels gives up after a while, and a warp that gave up leaves its loop.  A hardware barrier
(``bar.sync``) waits for all of its threads without a limit, so none may stand in a loop that a warp can leave on its own: those
have counted barriers with bounded waits.  Read from the sources; the failure itself cannot be provoked on a GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastmax_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def closing(s, i, pair):
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == pair[0]) - (s[j] == pair[1])
        if depth == 0:
            return j
    raise ValueError("unbalanced")


def statement_end(s, i):
    """End of the statement that begins at i: a block, a nested loop or condition, or up to a semicolon."""
    while s[i].isspace():
        i += 1
    if s[i] == "{":
        return closing(s, i, "{}") + 1
    m = re.compile(r"(for|while|if( constexpr)?)\s*\(").match(s, i)
    if m:
        end = statement_end(s, closing(s, m.end() - 1, "()") + 1)
        other = re.compile(r"\s*else\b").match(s, end)
        return statement_end(s, other.end()) if m.group(1).startswith("if") and other else end
    while s[i] != ";":
        i = closing(s, i, "{}" if s[i] == "{" else "()") + 1 if s[i] in "{(" else i + 1
    return i + 1


def loops(s):
    """(condition, start and end of the body) of every loop."""
    for m in re.finditer(r"\b(for|while)\s*\(", s):
        end = closing(s, m.end() - 1, "()")
        yield s[m.end():end], end + 1, statement_end(s, end + 1)


def barriers_in_loops_that_warps_leave(text):
    s = re.sub(r"//[^\n]*|^\s*#[^\n]*", "", text, flags=re.M)
    bodies = {m.group(1): s[m.end() - 1:closing(s, m.end() - 1, "{}")]
              for m in re.finditer(r"auto (\w+) = \[[^\]]*\]\s*(?:\([^()]*\))?\s*(?:->\s*\w+\s*)?\{", s)}
    meeting = set()
    while True:
        more = {n for n, b in bodies.items() if "bar.sync" in b or any(re.search(r"\b%s\(" % x, b) for x in meeting)}
        if more == meeting:
            break
        meeting = more
    meets = re.compile("|".join(["bar\\.sync"] + [r"\b%s\(" % n for n in sorted(meeting)]))
    every = list(loops(s))
    found = []
    for cond, lo, hi in every:
        body = s[lo:hi]
        # what a lambda defined inside does happens where it is called
        for b in bodies.values():
            body = body.replace(b, " " * len(b))
        if not meets.search(body):
            continue
        inner = [(a - lo, b - lo) for _, a, b in every if lo < a and b <= hi]
        own = [m.start() for m in re.finditer(r"\bbreak;|\breturn\b", body)
               if not any(a <= m.start() < b for a, b in inner)]
        if own or re.search(r"\bok\b", cond):
            found.append((cond.strip(), s[:lo].count("\n")))
    return found


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_unbounded_barrier_where_a_warp_may_leave(path):
    with open(path) as f:
        text = f.read()
    if "mbar_wait" in text:
        assert barriers_in_loops_that_warps_leave(text) == []


def test_the_reading_finds_what_it_looks_for():
    leave = "void f() { auto meet = []() { asm volatile(\"bar.sync 1, 256;\"); }; bool ok = true;\n"
    assert barriers_in_loops_that_warps_leave(leave + "for (; ok && more(); next()) { meet(); } }")
    assert barriers_in_loops_that_warps_leave(leave + "while (more()) { if (!mbar_wait(b, 0)) { ok = false; break; } meet(); } }")
    assert not barriers_in_loops_that_warps_leave(leave + "while (more()) { if (ok && !mbar_wait(b, 0)) ok = false; meet(); } }")
    assert not barriers_in_loops_that_warps_leave(leave + "while (more()) { meet(); for (;;) { if (!ok) break; } } }")
    assert not barriers_in_loops_that_warps_leave(leave + "for (; ok && more(); next()) { } meet(); }")


# Warpgroups that take registers wait for them until the block has them, so the block must have been launched with enough: the
# compiler decides, and where it gave fewer another kernel serves the call.  A call that other kernels can serve is not refused.
@pytest.mark.parametrize("name", ["fm_dense_tc_walk.cu", "fm_dense_split_rows.cu"])
def test_missing_registers_choose_another_kernel(name):
    with open(os.path.join(CSRC, name)) as f:
        s = re.sub(r"//[^\n]*", "", f.read())
    assert "regs_up<" in s
    assert re.search(r"launch_registers\([^;]*>=", s)
    assert not [c for c in re.findall(r"\bfail\([^;]*;", s) if re.search(r"\bregs|registers", c, re.I)]
