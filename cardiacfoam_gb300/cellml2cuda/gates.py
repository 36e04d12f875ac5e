"""States that are linear gates in tissue mode.

While the PDE owns Vm (see :mod:`hoist`), the rate of a Hodgkin-Huxley gate,
(g_inf(Vm) - g) / tau_g(Vm) or a(Vm) (1 - g) - b(Vm) g, is linear in the gate
with coefficients that do not change over a PDE step, and no other state
enters it.  A Runge-Kutta step of such an equation is a polynomial in
z = -h * decay times the rate at the step's start, so a solver needs the rate
once per step and the decay coefficient once per cell; the stage loop does not
have to evaluate the gate at all.

:func:`linear_gates` finds these states: exactly one assignment of the rate,
outside any conditional, linear in the state, every other operand a constant,
the tissue flag, the membrane potential or an invariant algebraic.
:func:`decay` is the coefficient, -d(rate)/d(state), as an expression.
"""
from __future__ import annotations

from typing import Dict, Optional

from .cexpr import Bin, Call, Node, Num, Ref, Unary, Var, refs, walk
from .model import Assign, Model, iter_assigns

_ALLOWED_VARS = {"tissueFlag", "dimension"}
_ONE = Num("1.0")


def _depends(e: Node, state: str) -> bool:
    return any(r.name == state for r in refs(e, "STATES"))


def slope(e: Node, state: str) -> Optional[Node]:
    """d(e)/d(state) of an expression linear in the state with a slope that is
    not zero; raises ValueError where it is not linear."""
    if isinstance(e, Ref):
        return _ONE
    if isinstance(e, Unary) and e.op == "-":
        return Unary("-", slope(e.e, state))
    if isinstance(e, Bin) and e.op in "+-":
        l = slope(e.l, state) if _depends(e.l, state) else None
        r = slope(e.r, state) if _depends(e.r, state) else None
        if l is not None and r is not None:
            return Bin(e.op, l, r)
        return l if l is not None else (r if e.op == "+" else Unary("-", r))
    if isinstance(e, Bin) and e.op == "*":
        dl, dr = _depends(e.l, state), _depends(e.r, state)
        if dl and dr:
            raise ValueError("product of two terms in the state")
        inner, other = (slope(e.l, state), e.r) if dl else (slope(e.r, state), e.l)
        return other if inner == _ONE else Bin("*", inner, other)
    if isinstance(e, Bin) and e.op == "/" and not _depends(e.r, state):
        return Bin("/", slope(e.l, state), e.r)
    raise ValueError("not linear in the state")


def _negated(e: Node) -> Node:
    """-e, with the sign moved to where one is written already."""
    if isinstance(e, Unary) and e.op == "-":
        return e.e
    if isinstance(e, Bin) and e.op in "*/" and isinstance(e.l, Unary) and e.l.op == "-":
        return Bin(e.op, e.l.e, e.r)
    if isinstance(e, Bin) and e.op == "-" and isinstance(e.l, Bin) and \
            isinstance(e.l.l, Unary) and e.l.l.op == "-":
        return Bin("+", _negated(e.l), e.r)
    return Unary("-", e)


def linear_gates(m: Model, invariant) -> Dict[str, Node]:
    """state -> its decay coefficient, in the order of the states."""
    vm = m.states[0]
    sites: Dict[str, list] = {}
    for st in iter_assigns(m.rates):
        if st.target.array == "RATES":
            sites.setdefault(st.target.name, []).append(st)
    out: Dict[str, Node] = {}
    for s in m.states[1:]:
        if len(sites.get(s, ())) != 1 or sites[s][0] not in [x for x in m.rates
                                                             if isinstance(x, Assign)]:
            continue
        e = sites[s][0].expr
        if not _depends(e, s):
            continue
        ok = all(r.array == "CONSTANTS" or (r.array == "STATES" and r.name in (vm, s)) or
                 (r.array == "ALGEBRAIC" and r.name in invariant) for r in refs(e))
        ok = ok and all(n.name in _ALLOWED_VARS for n in walk(e) if isinstance(n, Var))
        ok = ok and not any(isinstance(n, Call) and n.fn == "computeIstim" for n in walk(e))
        if not ok:
            continue
        try:
            out[s] = _negated(slope(e, s))
        except ValueError:
            continue
    return out
