"""The hand-over protocol of the diagonal tile factorisation's warps
(csrc/cholesky_df.cu: factor_chain, factor_lead, factor_help, factor_finish),
on the host: the barriers and the panel counts as they stand in the source,
run in every order that the barriers allow.

The last warp follows the published count of panels at its own pace, so the
count must never fall back, must end at 8, and a count n must stand for a
stored panel n - 1 and for everything of panel n - 2."""
import os
import re

from conftest import ROOT

HELPERS = 4


def _source():
    with open(os.path.join(ROOT, "pybrown_b200", "csrc", "cholesky_df.cu")) as f:
        return f.read()


def _body(src, name):
    start = src.index(f"void {name}(")
    return src[start:src.index("\n}\n", start)]


EVENT = re.compile(r"(bar_wait|bar_arrive|panels_done)\(([^)]*)\)")


def _events(body, panels):
    """[(event, argument, threads), ...] of a warp whose loop runs over `panels`:
    barrier calls and published counts, with the conditions on p in front of
    them (on their own line or on the line that opens their block)."""
    out = []
    for p in range(panels):
        guard = True  # the condition of the innermost `if (p ...) {` / `} else {` block
        for line in body.split("\n"):
            line = line.split("//")[0]
            block = re.match(r"\s*if \((?:j == 4 && )?p (<|>) (\d+)\) \{\s*$", line)
            if block:
                guard = p < int(block[2]) if block[1] == "<" else p > int(block[2])
                continue
            if re.match(r"\s*\} else \{", line):
                guard = not guard
                continue
            if re.match(r"    \}\s*$", line):
                guard = True
                continue
            if re.match(r"\s*if \(p == 5\) break;", line) and p == 5:
                return out
            m = EVENT.search(line)
            if not m or not guard:
                continue
            cond = re.search(r"if \(p (<|>) (\d+)\)", line[:m.start()])
            if cond and not (p < int(cond[2]) if cond[1] == "<" else p > int(cond[2])):
                continue
            if m[1] == "panels_done":
                assert m[2] == "f, p + 1"
                out.append(("count", p + 1, 0))
            else:
                bar, threads = (int(v) for v in m[2].split(","))
                out.append((m[1], bar, threads))
    return out


def _programs(src):
    chain = _events(_body(src, "factor_chain"), 8)
    lead = _events(_body(src, "factor_lead"), 6)
    helper = _events(_body(src, "factor_help"), 6)
    # the parser read what it is meant to read
    assert [e for e in chain if e[0] == "bar_arrive"] == [("bar_arrive", 1, 192)] * 6
    assert [e for e in chain if e[0] == "bar_wait"] == [("bar_wait", 3, 64)] * 6
    assert [e[1] for e in lead if e[0] == "count"] == [1, 2, 3, 4, 5, 6]
    assert [e[:2] for e in helper] == [("bar_wait", 1), ("bar_wait", 4)] * 5 + [("bar_wait", 1)]
    return [chain, lead] + [helper] * HELPERS


def _monotone(src):
    """Whether a count is published as a maximum (else as a plain store)."""
    body = _body(src, "panels_done")
    return re.search(r"(red|atom)\.release\.cta\.shared(::cta)?\.max\.", body) is not None


def test_panel_count_never_falls_back():
    src = _source()
    programs = _programs(src)
    keep_max = _monotone(src)
    names = ["chain", "lead"] + ["helper"] * HELPERS
    # state: pc of each warp, arrived[barrier] (threads and waiting warps), count
    start = (tuple(0 for _ in programs), (), 0)
    seen, todo, finals = {start}, [start], set()
    while todo:
        pcs, bars, count = todo.pop()
        arrived = {b: (n, set(w)) for b, n, w in bars}
        waiting = {w for _, ws in arrived.values() for w in ws}
        moves = [w for w in range(len(programs)) if pcs[w] < len(programs[w]) and w not in waiting]
        if not moves:
            assert all(pc == len(p) for pc, p in zip(pcs, programs)), "the warps wait for one another"
            finals.add(count)
            continue
        for w in moves:
            kind, arg, threads = programs[w][pcs[w]]
            pc2, arr2, c2 = list(pcs), {b: (n, set(ws)) for b, (n, ws) in arrived.items()}, count
            if kind == "count":
                # panel arg - 1 is stored: the chain is past its hand-over of it (its own
                # counts follow its stores directly)
                if w != 0:
                    before = programs[0][:pcs[0]]
                    assert sum(e[0] == "bar_arrive" for e in before) >= arg
                    # and every helper has left panel arg - 2
                    for h in range(2, 2 + HELPERS):
                        assert sum(e[1] == 1 for e in programs[h][:pcs[h]]) + (h in waiting) >= arg - 1
                c2 = max(count, arg) if keep_max else arg
                assert c2 >= count, f"the {names[w]} lowers the count from {count} to {arg}"
                pc2[w] += 1
            else:
                n, ws = arr2.get(arg, (0, set()))
                n += 32
                if kind == "bar_wait":
                    ws = ws | {w}
                else:
                    pc2[w] += 1
                if n == threads:  # complete: the waiting warps go on
                    for v in ws:
                        pc2[v] += 1
                    arr2.pop(arg, None)
                else:
                    assert n < threads, f"barrier {arg} entered twice"
                    arr2[arg] = (n, ws)
            state = (tuple(pc2), tuple(sorted((b, n, tuple(sorted(ws))) for b, (n, ws) in arr2.items())), c2)
            if state not in seen:
                seen.add(state)
                todo.append(state)
    assert finals == {8}
