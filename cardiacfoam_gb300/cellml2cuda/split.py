"""Partition of a model's states over the warps that share a cell.

GB300 issues one FP64 instruction per SM partition every 64 clocks, whatever
the number of active lanes, so a mesh with fewer cells than the chip has lanes
is bound by the FP64 instruction count of one warp.  There the plain form runs
four warps per 32 cells, each integrating a part of the states (and evaluating
only the statements those states' rates need) and exchanging the stage inputs
through shared memory.

:func:`partition` assigns the states so that the most expensive part is as
cheap as a deterministic descent makes it.  A part's cost counts every
statement that at least one of its rates needs once, in FP64 instructions of
the CUDA form: the intermediate values two parts need are evaluated by both.
"""
from __future__ import annotations

from typing import Dict, FrozenSet, List

from .cexpr import Bin, Call, Cond, Node, Num, Ref, Unary, refs, walk
from .gates import linear_gates
from .hoist import analyse
from .model import If, Model, iter_assigns

PARTS = 4
# FP64 instructions of the functions and of a division (measured order)
_CALLS = {"exp": 17, "log": 22, "pow": 65, "sqrt": 10, "tanh": 30}
_DIVIDE, _DIVIDE_BY_CONSTANT = 9, 3
_STAGE, _GATE = 9, 6          # stage sums and error of a state, per evaluation
_EVALS = 6                    # stages of a substep; invariants once
_CONTROL = 80                 # the step control of a substep


def _constant(e: Node) -> bool:
    return all(not isinstance(n, Ref) or n.array == "CONSTANTS" for n in walk(e))


def expr_cost(e: Node) -> float:
    c = 0.0
    for n in walk(e):
        if _constant(n):
            continue
        if isinstance(n, Call):
            if n.fn == "pow" and isinstance(n.args[1], Num):
                k = n.args[1].value
                c += 4 if k == int(k) else (10 if k == 0.5 else _CALLS["pow"])
            else:
                c += _CALLS.get(n.fn, 1)
        elif isinstance(n, Bin):
            c += ((_DIVIDE_BY_CONSTANT if _constant(n.r) else _DIVIDE) if n.op == "/"
                  else 0.75)
        elif isinstance(n, (Unary, Cond)):
            c += 0.25
    return c


def _statements(m: Model):
    """Per top-level statement: what it assigns, what it reads, its cost."""
    out = []
    for st in m.rates:
        assigns = list(iter_assigns([st]))
        reads, cost = set(), 0.0
        for a in assigns:
            reads |= {r.name for r in refs(a.expr, "ALGEBRAIC")}
            cost += expr_cost(a.expr)
        if isinstance(st, If):
            reads |= {r.name for r in refs(st.cond, "ALGEBRAIC")}
        out.append((assigns, reads, cost))
    return out


def closures(m: Model) -> Dict[str, FrozenSet[int]]:
    """state -> the statements its rate needs."""
    stmts = _statements(m)
    rates: Dict[str, set] = {}
    for k, (assigns, _, _) in enumerate(stmts):
        for a in assigns:
            if a.target.array == "RATES":
                rates.setdefault(a.target.name, set()).add(k)
    return {s: frozenset().union(*({k} | _needs(stmts, k) for k in rates[s]))
            if s in rates else frozenset() for s in m.states}


def _needs(stmts, k: int) -> FrozenSet[int]:
    """The statements before k whose values k reads, directly or not (a name
    read before its assignment is zero)."""
    out: set = set()
    todo = [k]
    while todo:
        i = todo.pop()
        for j in range(i):
            if j not in out and any(a.target.array == "ALGEBRAIC" and
                                    a.target.name in stmts[i][1] for a in stmts[j][0]):
                out.add(j)
                todo.append(j)
    return frozenset(out)


def partition(m: Model, solve_vm: bool) -> List[int]:
    stmts = _statements(m)
    need = closures(m)
    h = analyse(m, m.rates)
    gates = {} if solve_vm else linear_gates(m, h.invariant)
    invariant = set() if solve_vm else {
        k for k, (assigns, _, _) in enumerate(stmts)
        if assigns and all(a.target.array == "ALGEBRAIC" and a.target.name in h.invariant
                           for a in assigns)}
    weight = [c * (1.0 if k in invariant else _EVALS) for k, (_, _, c) in enumerate(stmts)]
    for k, (assigns, _, _) in enumerate(stmts):
        if len(assigns) == 1 and assigns[0].target.array == "RATES" and \
                assigns[0].target.name in gates:
            weight[k] = expr_cost(assigns[0].expr)
    states = list(m.states) if solve_vm else list(m.states[1:])
    own = {s: (_GATE if s in gates else _STAGE) * _EVALS for s in states}

    # the current at the end of the step, which part 0 evaluates once
    current = frozenset().union(*(
        frozenset({k}) | _needs(stmts, k) for k, (assigns, _, _) in enumerate(stmts)
        if any(a.target.array == "ALGEBRAIC" and a.target.name == m.iion_name for a in assigns)))

    def cost(group, part=1):
        used = set().union(*(need[s] for s in group)) if group else set()
        c = sum(weight[k] for k in used) + sum(own[s] for s in group)
        if part == 0:
            c += _CONTROL + sum(stmts[k][2] for k in current
                                if k not in invariant or k not in used)
        return c

    parts: List[List[str]] = [[] for _ in range(PARTS)]
    for s in sorted(states, key=lambda s: (-cost([s]), states.index(s))):
        best = min(range(PARTS), key=lambda p: (max(cost(parts[q] + ([s] if q == p else []), q)
                                                    for q in range(PARTS)),
                                                cost(parts[p] + [s], p), p))
        parts[best].append(s)

    def total(ps):
        c = sorted((cost(p, q) for q, p in enumerate(ps)), reverse=True)
        return (c[0], sum(x * x for x in c))
    improved = True
    while improved:
        improved = False
        now = total(parts)
        for a in range(PARTS):
            for s in list(parts[a]):
                for b in range(PARTS):
                    if a == b:
                        continue
                    trial = [list(p) for p in parts]
                    trial[a].remove(s)
                    trial[b].append(s)
                    t = total(trial)
                    if t < now:
                        parts, now, improved = trial, t, True
                        break
    where = {s: k for k, p in enumerate(parts) for s in p}
    return [where.get(s, 0) for s in m.states]
