"""The order of k_delta_chunk's shared memory, on the CPU: its waits, arrivals, copies, reads and writes are taken from the source as they stand, and every read of a
place has to be ordered before the next write to it by barriers, whatever the warps' speeds."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent.parent / "dnet_b200" / "csrc" / "dn_seq_delta_chunk.cuh"
CHUNKS = 6
# what a line of the loop does: kind, then the barrier or the place
EVENTS = [(r"mbar_wait\(&?(\w+_(?:full|free))\b", "wait"), (r"mbar_arrive\((\w+_free)\)", "arrive"), (r"\bpart\(sK\b", "copy K"), (r"\bpart\(sQ\b", "copy Q"), (r"\brest\(c \+ 1\)", "copy T"),
          (r"\bmine\[.*\] =", "write xch"), (r"\bother\[", "read xch"), (r"bar\.sync", "meet"), (r"\b(?:load\(Ks\)|ldsm_x4_t\(w, Ks)", "read K"), (r"\bload\(Qs\)", "read Q"),
          (r"\b(?:tile16\((?:Ts|As)|Vs\[|gm \+|gm\[)", "read T")]
FULL = {"K": "k_full", "Q": "q_full", "T": "t_full"}


def loop_events():
    """[(kind, name, warp or None)] of one chunk, in the order of the source; a statement under `if (warp == n ...)` is warp n's alone"""
    body = SRC.read_text().split("for (int c = 0; c < chunks; c++) {")[1]
    out, depth, guard = [], 1, None
    for line in body.splitlines():
        line = re.sub(r"//.*", "", line)
        m = re.search(r"if \(warp == (\d) && c \+ 1 < chunks\) \{", line)
        if m:
            guard = (int(m.group(1)), depth)
        for pos, kind, name in sorted((x.start(), kind, x.group(1) if x.groups() else None) for pattern, kind in EVENTS for x in re.finditer(pattern, line)):
            out.append((kind, name, guard[0] if guard else None))
        depth += line.count("{") - line.count("}")
        if guard and depth <= guard[1]:
            guard = None
        if depth <= 0:
            return out
    raise AssertionError("the loop over the chunks does not end")


def accesses(events, cg):
    """the graph of what is ordered before what, and the accesses of each place: (place, is_write, chunk of what it holds, warp, node)"""
    edges, seen, nodes, waits, done = {}, [], 0, [], {}      # done: (barrier, number of its phase) -> nodes that complete it
    for warp in range(2 * cg):
        prev = None
        for c in range(-1, CHUNKS):
            todo = events if c >= 0 else [("copy K", None, 0), ("copy Q", None, 0), ("copy T", None, 0)]      # (the first chunk's copies, ahead of the loop)
            for kind, name, only in todo:
                if only is not None and (warp != only or c + 1 >= CHUNKS):
                    continue
                if kind == "wait" and only == 0 and name == "k_free" and c == 0:
                    continue      # (`if (c > 0)`)
                node, nodes = nodes, nodes + 1
                edges[node] = []
                if prev is not None:
                    edges[prev].append(node)
                prev = node
                what, _, place = kind.partition(" ")
                if what == "wait":
                    waits.append((name, c - 1 if name == "k_free" else c, node))
                elif what == "arrive":
                    done.setdefault((name, c), []).append(node)
                elif what == "meet":      # the two warps of a column group
                    done.setdefault(("meet", warp % cg, c), []).append(node)
                    after, nodes = nodes, nodes + 1
                    edges[after] = []
                    edges[prev].append(after)
                    prev = after
                    waits.append((("meet", warp % cg), c, after))
                elif what == "copy":
                    done.setdefault((FULL[place], c + 1), []).append(node)
                    seen.append(((place, (c + 1) & 1 if place == "K" else 0), True, c + 1, None, node))
                elif place == "xch":
                    seen.append((("xch", warp if what == "write" else (warp + cg) % (2 * cg)), what == "write", c, warp, node))
                else:
                    seen.append(((place, c & 1 if place == "K" else 0), False, c, warp, node))
    for name, c, node in waits:
        for x in done[(*name, c) if isinstance(name, tuple) else (name, c)]:
            edges[x].append(node)
    return edges, seen


@pytest.mark.parametrize("cg", [2, 4])
def test_every_read_is_ordered_before_the_next_write_and_behind_its_own(cg):
    events = loop_events()
    kinds = [k for k, _, _ in events]
    assert kinds.count("meet") == 1 and all(kinds.count(k) >= 1 for _, k in EVENTS)
    assert {n for k, n, _ in events if k == "wait"} == {"k_full", "q_full", "t_full", "k_free", "q_free", "t_free"}
    edges, seen = accesses(events, cg)
    reach = {}

    def after(node):      # every node that is ordered behind this one
        if node not in reach:
            todo, got = [node], set()
            while todo:
                for x in edges[todo.pop()]:
                    if x not in got:
                        got.add(x)
                        todo.append(x)
            reach[node] = got
        return reach[node]

    unordered = set()
    for place, is_write, c, warp, node in seen:
        for place2, is_write2, c2, warp2, node2 in seen:
            if place2 == place and not is_write and is_write2:
                if c2 > c and node2 not in after(node):
                    unordered.add(f"{place[0]}: warp {warp} may still read chunk {c}'s when chunk {c2}'s are written")
                if c2 == c and node not in after(node2):
                    unordered.add(f"{place[0]}: warp {warp} may read chunk {c}'s before they are written")
    assert not unordered, sorted(unordered)[:6]
