"""Rows of a split program dealt to the warps that share a node.

The explicit kernels can give a node to the four warps of a block, each of
which evaluates some rows (``group_kernel`` in ``csrc/goss_kernels.cuh``).  What
a warp's rows do not need falls out of its copy of the program, so the groups
are balanced by the cost of the statements that their rows need.
"""
from __future__ import annotations

import re
from typing import Dict, List, Sequence

# FP64 instructions of the models::F64 functions and of a multiply or add
_COST = ((r"gexp2?\(", 24), (r"glog\(", 40), (r"gsqrt\(", 20), (r"gpow\(", 64), (r"/", 14), (r"[*+-]", 1))
_DEFINITION = re.compile(r"const (?:T|double|bool) (\w+) = (.*);$")
_OUTPUT = re.compile(r"\w+\[(\d+)\] = (.*);$")
PARTS = 4
# states of a model worth dealing out, and those the exchange buffers hold
MIN_ROWS, MAX_ROWS = 9, 64


def row_groups(lines: Sequence[str], rows: int, update: int) -> List[int]:
    """The group of each row of a program given as its C statements.

    A group costs the statements that its rows need (what two groups need
    counts in both) and ``update`` per row.  Rows go, dearest first, to the
    group that leaves the dearest group cheapest, then move singly while that
    lowers the sorted costs.
    """
    def price(e):
        return sum(c * len(re.findall(p, e)) for p, c in _COST)

    cost: Dict[str, int] = {}
    needs: Dict[str, frozenset] = {}
    need, own = [frozenset()] * rows, [update] * rows

    def operands(e):
        return frozenset().union(*[needs[n] for n in re.findall(r"[A-Za-z_]\w*", e) if n in needs])

    for line in lines:
        line = line.strip()
        m = _DEFINITION.match(line)
        if m:
            cost[m[1]] = price(m[2])
            needs[m[1]] = operands(m[2]) | {m[1]}
            continue
        m = _OUTPUT.match(line)
        if not m:
            continue
        i = int(m[1])
        need[i] = need[i] | operands(m[2])
        own[i] += price(m[2])

    def total(g):
        return sum(cost[n] for n in frozenset().union(*[need[i] for i in g])) + sum(own[i] for i in g)

    groups: List[List[int]] = [[] for _ in range(PARTS)]
    for i in sorted(range(rows), key=lambda i: (-total([i]), i)):
        now, grown = [total(g) for g in groups], [total(g + [i]) for g in groups]
        k = min(range(PARTS), key=lambda k: (max(now + [grown[k]]), grown[k], k))
        groups[k].append(i)
    best, moved = sorted(map(total, groups), reverse=True), True
    while moved:
        moved = False
        for i in range(rows):
            for k in range(PARTS):
                at = next(q for q in range(PARTS) if i in groups[q])
                if k == at:
                    continue
                groups[at].remove(i)
                groups[k].append(i)
                now = sorted(map(total, groups), reverse=True)
                if now < best:
                    best, moved = now, True
                else:
                    groups[k].remove(i)
                    groups[at].append(i)
    return [next(k for k in range(PARTS) if i in groups[k]) for i in range(rows)]


def declarations(linearized: Sequence[str], rhs: Sequence[str], rows: int) -> List[str]:
    """The model's row groups as C++ (28: a GRL update; 4: an RK4 stage's sums)."""
    out = ["  // the rows of linearized_split and of rhs_split dealt to the four warps of a block"]
    for name, lines, update in (("linear_group", linearized, 28), ("rhs_group", rhs, 4)):
        digits = "".join(map(str, row_groups(lines, rows, update)))
        out.append(f"  __host__ __device__ static constexpr int {name}(int i) {{ return \"{digits}\"[i] - '0'; }}")
    return out
