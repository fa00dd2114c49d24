"""Warps that meet at a named barrier must all reach it, also after one of them has given up on a
bounded wait: in the kernels' sources no loop that holds such a barrier is left early, unless a loop
of the remaining barriers, walked to its end, follows it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "modiff_b200", "csrc")
BARRIER = re.compile(r'bar(?:rier\.cta)?\.sync\s+[1-9]')


def early_exits(text):
    """(line, what) of every way out of a loop whose body holds a named barrier, other than its
    count: a `break` of that loop, a `return` inside it, a condition on `ok`."""
    text = re.sub(r'//[^\n]*', lambda m: ' ' * len(m.group()), text)
    # bodies as (start, end, header) of every `for` / `while` with braces
    loops = []
    for m in re.finditer(r'\b(?:for|while)\s*\(', text):
        depth, i = 1, m.end()
        while depth:
            depth += {'(': 1, ')': -1}.get(text[i], 0)
            i += 1
        header, j = text[m.end():i - 1], i
        while text[j].isspace():
            j += 1
        if text[j] != '{':
            continue
        depth, k = 1, j + 1
        while depth:
            depth += {'{': 1, '}': -1}.get(text[k], 0)
            k += 1
        loops.append((j, k, header))
    found = []

    def same_scope(a, b):                 # text from a to b closes no scope that is open at a
        depth = 0
        for ch in text[a:b]:
            depth += {'{': 1, '}': -1}.get(ch, 0)
            if depth < 0:
                return False
        return True

    def followed(beg, end):               # by a loop with barriers, behind this loop or one around it
        around = [e for b, e, _ in loops if b <= beg and end <= e]
        return any(same_scope(a, b) and BARRIER.search(text[b:e]) and not re.search(r'\b(break|return)\b', text[b:e])
                   for a in around for b, e, _ in loops if b > a)

    line = lambda pos: text.count('\n', 0, pos) + 1
    for beg, end, header in loops:
        body = text[beg:end]
        if not BARRIER.search(body):
            continue
        if re.search(r'\bok\b', header):
            found.append((line(beg), 'condition'))
        for m in re.finditer(r'\b(break|return)\b', body):
            pos = beg + m.start()
            inner = [(b, e) for b, e, _ in loops if beg < b < pos < e]
            # a break of an inner loop without a barrier leaves only that loop (loop bodies without
            # braces hold one statement, in which no kernel breaks)
            if m.group(1) == 'break' and (inner or followed(beg, end)):
                continue
            found.append((line(pos), m.group(1)))
    return found


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_loops_with_named_barriers_are_walked_to_their_end(path):
    with open(path) as f:
        assert early_exits(f.read()) == []


def test_the_search_finds_early_exits():
    loop = 'for (int t = 0; t < n%s; ++t) {\n %s\n asm volatile("bar.sync 1, 256;" ::: "memory");\n}'
    assert early_exits(loop % ('', 'if (!ok) continue;')) == []
    assert early_exits(loop % ('', 'for (;;) { break; }')) == []
    assert early_exits(loop % ('', 'if (!ok) break;')) == [(2, 'break')]
    assert early_exits(loop % (' && ok', '')) == [(1, 'condition')]
    rest = '\nfor (t += 1; t < n; ++t) { asm volatile("bar.sync 1, 256;" ::: "memory"); }'
    assert early_exits(loop % ('', 'if (!ok) break;') + rest) == []
    assert early_exits(loop % ('', 'if (!ok) break;') + '\n}\nvoid f() {' + rest) == [(2, 'break')]
