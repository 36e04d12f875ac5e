"""Reverse-mode derivative (vector-Jacobian product) of a model's right-hand
side in tissue mode, emitted as a CUDA device function.

The body the tissue step evaluates (``rates``: RATES of every state but V, and
``Iion_cm``) is turned into three-address code: every operator node of every
expression gets a named temporary, conditionals (``c ? a : b`` and
``tissueSelect``) become if/else blocks so that only the taken branch is
evaluated and differentiated.  The emitted function first runs that code
forward (the same operations as the forward RHS, in the header's order), then
walks the statements backwards, pushing the adjoint of each statement's target
down its expression tree with the derivative rule of each operator:

    a + b, a - b      (g, g), (g, -g)
    a * b, a / b      (g b, g a), (g / b, -g v / b)      v = the node's value
    -a, exp a, log a  -g, g v, g / a
    sqrt a, tanh a    g / (2 v), g (1 - v^2)
    pow(a, n)         g n a^(n-1) (and g v log a for a non-constant exponent)
    fabs a            g sign(a);  floor, heaviside, comparisons: 0
    exp(x) - 1        evaluated as cfg_expm1(x), adjoint g (v + 1)

Algebraics read before their assignment are the zeroed scratch of
``derivatives()`` (constant 0).  The single-cell stimulus does not exist in
tissue mode (the reference refuses it) and differentiates to 0.

    rhs_vjp<R, KS>(t, y, K, tissue, dbar, ibar, ybar, pbar)

adds to ybar[NS] the product of the transposed Jacobian of (dydt, Iion_cm) with
respect to the states with (dbar, ibar), and to pbar[NSCALE] the same with
respect to the scalable conductances (SCALE_ORDER: GNa, GCaL, GKr, GKs, GK1,
Gto), whose values K(C_x) are the already scaled constants.

V is the same at every stage of a PDE step in tissue mode (hoist.py), so the
mixed form takes the body apart at what depends on V and constants alone:

    adj_hoist<R>(y_V, K, tissue, H)
    adj_rhs<R>(t, y, K, tissue, H, dydt)                    returns Iion_cm
    adj_rhs_vjp<R>(t, y, K, tissue, H, dbar, ibar, ybar, pbar, hbar)
    adj_hoist_vjp<R>(y_V, K, tissue, hbar)                  returns dV

adj_rhs_vjp adds the adjoint of the values H to hbar; the derivative being
linear in it, one adj_hoist_vjp of the sum over all stages replaces the part of
every stage's rhs_vjp that runs through them.  These four run in FP32, where the
roundings show: products that are added or subtracted are written as multiply-adds
(cfg_fma), which rounds once, and alike in every kernel, where a compiler's
contraction depends on what surrounds an expression.
"""
from __future__ import annotations

from typing import Dict, List, Tuple

from .cexpr import Bin, Call, Cond, Node, Num, Ref, Unary, Var, walk
from .emit import SCALABLE, SCALE_ORDER, _int_exponent, _is_half, ident
from .hoist import analyse
from .model import Assign, Fatal, If, Model, use_before_def

_CMP = ("==", "!=", "<", ">", "<=", ">=", "&&", "||")


def _expm1_arg(e: Node):
    """x of exp(x) - 1 (the GHK flux denominators), else None: evaluated as
    cfg_expm1(x), which in FP32 does not cancel to 0 as x -> 0."""
    if isinstance(e, Bin) and e.op == "-" and isinstance(e.r, Num) and \
            float(e.r.text.rstrip("fF")) == 1.0 and isinstance(e.l, Call) and e.l.fn == "exp":
        return e.l.args[0]
    return None


def tissue_mode_body(stmts) -> List[Assign]:
    """The statements with solveVmWithinODESolver = false resolved."""
    out: List[Assign] = []
    for st in stmts:
        if isinstance(st, Assign):
            out.append(st)
        elif isinstance(st, If):
            c = st.cond
            if isinstance(c, Var) and c.name == "solveVmWithinODESolver":
                out.extend(tissue_mode_body(st.orelse))
            elif isinstance(c, Unary) and c.op == "!" and isinstance(c.e, Var) and \
                    c.e.name == "solveVmWithinODESolver":
                out.extend(tissue_mode_body(st.then))
            else:
                raise ValueError(f"unsupported run-time if ({c}) in the adjoint")
        elif isinstance(st, Fatal):
            continue
    return out


class _Gen:
    """Three-address forward code and the matching reverse sweep."""

    def __init__(self, m: Model, early, fused: bool = False):
        self.m = m
        self.fused = fused
        self.product: Dict[str, Tuple[str, str]] = {}   # value -> its factors
        self.early = set(early)
        self.params = {v: k for k, v in SCALABLE[m.name].items()}   # constant -> scale key
        self.n = 0
        self.decl: List[str] = []           # hoisted temporaries
        self.defined: Dict[str, str] = {}   # algebraic -> current value name
        self.value: Dict[int, str] = {}     # id(node) -> value name
        self.alg_bar: Dict[str, str] = {}   # algebraic value name -> its adjoint accumulator
        self.states_read = set()
        self.varying: Dict[str, bool] = {}  # H slots that depend on V
        self.alg_ref: Dict[int, str] = {}

    def tmp(self, prefix="t") -> str:
        self.n += 1
        name = f"{prefix}{self.n}"
        self.decl.append(f"    R {name} = R(0);")
        return name

    # ---------------------------------------------------------------- forward
    def leaf(self, e: Node):
        if isinstance(e, Num):
            return e.text if e.is_int_literal else f"R({e.text})"
        if isinstance(e, Ref):
            if e.array == "STATES":
                self.states_read.add(e.name)
                return f"y_{e.name}"
            if e.array == "CONSTANTS":
                return f"p_{e.name}" if e.name in self.params else f"K(C_{e.name})"
            if e.array == "ALGEBRAIC":
                return self.defined.get(e.name, "R(0)")
            if e.array == "H":
                return f"H[{e.name}]"
            raise ValueError(f"read of {e.array} in the right-hand side")
        if isinstance(e, Var):
            if e.name == "tissueFlag":
                return "tissue"
            if e.name == "dimension":
                return "(tissue - 10)"
            if e.name == "solveVmWithinODESolver":
                return "false"
            if e.name == "VOI":
                return "t"
            raise ValueError(f"unknown variable {e.name}")
        return None

    def cond(self, e: Node, out: List[str], ind: str) -> str:
        """A boolean expression (never differentiated)."""
        if isinstance(e, Bin) and e.op in _CMP:
            return f"({self.cond_or_val(e.l, out, ind)} {e.op} {self.cond_or_val(e.r, out, ind)})"
        if isinstance(e, Unary) and e.op == "!":
            return f"(!{self.cond(e.e, out, ind)})"
        return f"({self.fwd(e, out, ind)} != R(0))"

    def cond_or_val(self, e: Node, out, ind) -> str:
        if isinstance(e, Bin) and e.op in _CMP or isinstance(e, Unary) and e.op == "!":
            return self.cond(e, out, ind)
        return self.fwd(e, out, ind)

    def binary(self, op: str, a: str, b: str, v: str) -> str:
        if self.fused and op in "+-":
            minus = "-" if op == "-" else ""
            # of two products the left one, the larger where currents are added up
            if a in self.product:
                p, q = self.product[a]
                return f"cfg_fma({p}, {q}, {minus}{b})"
            if b in self.product:
                p, q = self.product[b]
                return f"cfg_fma({minus}{p}, {q}, {a})"
        if op == "*":
            self.product[v] = (a, b)
        return f"({a} {op} {b})"

    def fwd(self, e: Node, out: List[str], ind: str) -> str:
        lf = self.leaf(e)
        if lf is not None:
            return lf
        x = _expm1_arg(e)
        if x is not None:
            a = self.fwd(x, out, ind)
            v = self.tmp()
            out.append(f"{ind}{v} = cfg_expm1({a});")
            self.value[id(e)] = v
            return v
        if isinstance(e, Unary):
            if e.op == "!":
                raise ValueError("logical not in an arithmetic position")
            a = self.fwd(e.e, out, ind)
            if e.op == "+":
                self.value[id(e)] = a
                return a
            v = self.tmp()
            out.append(f"{ind}{v} = (-{a});")
            self.value[id(e)] = v
            return v
        if isinstance(e, Bin):
            if e.op in _CMP:
                v = self.tmp()
                out.append(f"{ind}{v} = {self.cond(e, out, ind)} ? R(1) : R(0);")
                self.value[id(e)] = v
                return v
            a = self.fwd(e.l, out, ind)
            b = self.fwd(e.r, out, ind)
            v = self.tmp()
            out.append(f"{ind}{v} = {self.binary(e.op, a, b, v)};")
            self.value[id(e)] = v
            return v
        if isinstance(e, Cond):
            c = self.tmp("c")
            out.append(f"{ind}{c} = {self.cond(e.c, out, ind)} ? R(1) : R(0);")
            v = self.tmp()
            out.append(f"{ind}if ({c} != R(0)) {{")
            a = self.fwd(e.a, out, ind + "    ")
            out.append(f"{ind}    {v} = {a};")
            out.append(f"{ind}}} else {{")
            b = self.fwd(e.b, out, ind + "    ")
            out.append(f"{ind}    {v} = {b};")
            out.append(f"{ind}}}")
            self.value[id(e)] = v
            self.value[("cond", id(e))] = c
            return v
        if isinstance(e, Call):
            if e.fn == "computeIstim":
                return "R(0)"
            if e.fn == "tissueSelect":
                # tissueSelect(flag, endo, m, epi) as nested conditionals on tissue
                sel = Cond(Bin("==", Var("tissueFlag"), Num("3")), e.args[1],
                           Cond(Bin("==", Var("tissueFlag"), Num("2")), e.args[2], e.args[3]))
                v = self.fwd(sel, out, ind)
                self.value[id(e)] = v
                self.value[("alias", id(e))] = sel
                return v
            if e.fn == "heaviside":
                a = self.fwd(e.args[0], out, ind)
                v = self.tmp()
                out.append(f"{ind}{v} = ({a} > R(0)) ? R(1) : R(0);")
                self.value[id(e)] = v
                return v
            args = [self.fwd(x, out, ind) for x in e.args]
            v = self.tmp()
            if e.fn == "pow":
                n = _int_exponent(e.args[1])
                if n is not None:
                    out.append(f"{ind}{v} = cfg_ipow<{n}>({args[0]});")
                elif _is_half(e.args[1]):
                    out.append(f"{ind}{v} = cfg_sqrt({args[0]});")
                else:
                    out.append(f"{ind}{v} = cfg_pow({args[0]}, {args[1]});")
            elif e.fn in ("exp", "log", "sqrt", "tanh", "fabs", "floor"):
                out.append(f"{ind}{v} = cfg_{e.fn}({args[0]});")
            else:
                raise ValueError(f"{self.m.name}: no derivative rule for {e.fn}")
            self.value[id(e)] = v
            return v
        raise TypeError(e)

    # ---------------------------------------------------------------- reverse
    def acc(self, e: Node, g: str, out: List[str], ind: str):
        """Add the adjoint g of node e to its inputs."""
        if isinstance(e, Num) or isinstance(e, Var):
            return
        if isinstance(e, Ref):
            if e.array == "STATES":
                out.append(f"{ind}ybar[S_{e.name}] += {g};")
            elif e.array == "CONSTANTS" and e.name in self.params:
                out.append(f"{ind}pbar[SCALE_{self.params[e.name]}] += {g};")
            elif e.array == "H":
                if e.name in self.varying:
                    out.append(f"{ind}hbar[{e.name}] += {g};")
            elif e.array == "ALGEBRAIC" and id(e) in self.alg_ref:
                out.append(f"{ind}{self.alg_ref[id(e)]} += {g};")
            return
        val = lambda x: self.value.get(id(x)) or self.leaf(x)
        x = _expm1_arg(e)
        if x is not None:
            self.push(x, f"({g} * ({self.value[id(e)]} + R(1)))", out, ind)
            return
        if isinstance(e, Unary):
            if e.op == "+":
                self.acc(e.e, g, out, ind)
            else:
                self.push(e.e, f"(-{g})", out, ind)
            return
        if isinstance(e, Bin):
            if e.op in _CMP:
                return
            a, b, v = val(e.l), val(e.r), self.value[id(e)]
            if e.op == "+":
                self.push(e.l, g, out, ind)
                self.push(e.r, g, out, ind)
            elif e.op == "-":
                self.push(e.l, g, out, ind)
                self.push(e.r, f"(-{g})", out, ind)
            elif e.op == "*":
                self.push(e.l, f"({g} * {b})", out, ind)
                self.push(e.r, f"({g} * {a})", out, ind)
            elif e.op == "/":
                self.push(e.l, f"({g} / {b})", out, ind)
                self.push(e.r, f"(-{g} * {v} / {b})", out, ind)
            return
        if isinstance(e, Cond):
            c = self.value[("cond", id(e))]
            out.append(f"{ind}if ({c} != R(0)) {{")
            self.push(e.a, g, out, ind + "    ")
            out.append(f"{ind}}} else {{")
            self.push(e.b, g, out, ind + "    ")
            out.append(f"{ind}}}")
            return
        if isinstance(e, Call):
            if e.fn in ("computeIstim", "heaviside", "floor"):
                return
            if e.fn == "tissueSelect":
                self.acc(self.value[("alias", id(e))], g, out, ind)
                return
            v = self.value[id(e)]
            a = val(e.args[0])
            if e.fn == "exp":
                self.push(e.args[0], f"({g} * {v})", out, ind)
            elif e.fn == "log":
                self.push(e.args[0], f"({g} / {a})", out, ind)
            elif e.fn == "sqrt":
                self.push(e.args[0], f"({g} / (R(2) * {v}))", out, ind)
            elif e.fn == "tanh":
                self.push(e.args[0], f"({g} * (R(1) - {v} * {v}))", out, ind)
            elif e.fn == "fabs":
                self.push(e.args[0], f"({g} * ({a} >= R(0) ? R(1) : R(-1)))", out, ind)
            elif e.fn == "pow":
                n = _int_exponent(e.args[1])
                if n is not None:
                    d = "R(1)" if n == 1 else (f"R({n}) * {a}" if n == 2 else
                                               f"R({n}) * cfg_ipow<{n - 1}>({a})")
                    self.push(e.args[0], f"({g} * {d})", out, ind)
                elif _is_half(e.args[1]):
                    self.push(e.args[0], f"({g} / (R(2) * {v}))", out, ind)
                else:
                    b = val(e.args[1])
                    self.push(e.args[0], f"({g} * {b} * cfg_pow({a}, {b} - R(1)))", out, ind)
                    if not isinstance(e.args[1], Num):
                        self.push(e.args[1], f"({g} * {v} * cfg_log({a}))", out, ind)
            return
        raise TypeError(e)

    def push(self, e: Node, g: str, out, ind):
        """Adjoint g flows into node e: leaves accumulate, inner nodes get a
        temporary and propagate further."""
        if isinstance(e, (Num, Var)):
            return
        if isinstance(e, Ref):
            self.acc(e, g, out, ind)
            return
        t = self.tmp("g")
        out.append(f"{ind}{t} = {g};")
        self.acc(e, t, out, ind)


def _walk_body(gen: _Gen, body, fwd: List[str]):
    """Forward code of the statements; their (statement, adjoint name) pairs.
    Assignments to H (a value kept per cell) have H as target array."""
    targets: List[Tuple[Assign, str]] = []
    for st in body:
        t = st.target
        # record, for the reverse sweep, which value each algebraic read refers to
        for r in _alg_reads(st.expr):
            if r.name in gen.defined:
                gen.alg_ref[id(r)] = "b" + gen.defined[r.name]
        v = gen.fwd(st.expr, fwd, "    ")
        if t.array == "ALGEBRAIC":
            name = gen.tmp("a")
            fwd.append(f"    {name} = {v};")
            gen.defined[t.name] = name
            if v in gen.product:
                gen.product[name] = gen.product[v]
            gen.decl.append(f"    R b{name} = R(0);")
            targets.append((st, f"b{name}"))
        elif t.array == "RATES":
            targets.append((st, f"dbar[S_{t.name}]"))
        elif t.array == "H":
            targets.append((st, f"hbar[{t.name}]"))
        else:
            raise ValueError(f"assignment to {t.array} in the right-hand side")
    return targets


def _reverse(gen: _Gen, targets) -> List[str]:
    rev: List[str] = []
    for st, name in reversed(targets):
        if name.startswith("dbar"):
            rev.append(f"    {{ const R g0 = {name};")
            gen.push(st.expr, "g0", rev, "      ")
            rev.append("    }")
        else:
            gen.push(st.expr, name, rev, "    ")
    return rev


def _states_and_params(gen: _Gen) -> List[str]:
    return [f"    const R y_{s} = y[S_{s}];" for s in gen.m.states if s in gen.states_read] + \
           [f"    const R p_{c} = K(C_{c});" for c in gen.params]


def _without_v_rate(m: Model) -> List[Assign]:
    """The body without RATES of V: the PDE owns Vm."""
    return [st for st in tissue_mode_body(m.rates)
            if not (st.target.array == "RATES" and st.target.name == m.states[0])]


def emit_rhs_vjp(m: Model) -> str:
    gen = _Gen(m, use_before_def(m.rates))
    fwd: List[str] = []
    targets = _walk_body(gen, _without_v_rate(m), fwd)
    iion = gen.defined.get(m.iion_name)
    if iion is None:
        raise ValueError(f"{m.name}: the right-hand side does not compute {m.iion_name}")
    rev: List[str] = [f"    b{iion} += ibar;"] + _reverse(gen, targets)
    L: List[str] = []
    L.append("// Reverse-mode derivative of rhs<R, false> (tissue mode): adds to ybar the")
    L.append("// transposed Jacobian of (dydt without V, Iion_cm) with respect to the states")
    L.append("// applied to (dbar, ibar), and to pbar the same for the scalable conductances.")
    L.append("template <class R, class KS>")
    L.append("__device__ __noinline__ void rhs_vjp(double t, const R* y, const KS& K, int tissue, "
             "const R* dbar, R ibar, R* ybar, R* pbar)")
    L.append("{")
    L.append("    (void)t; (void)tissue;")
    L.extend(_states_and_params(gen))
    L.extend(gen.decl)
    L.extend(fwd)
    L.extend(rev)
    L.append("}")
    return "\n".join(L) + "\n"


def take_apart(m: Model):
    """The body without RATES of V as (statements of H, the other statements with
    H in them, H slot -> whether it depends on V).  H holds the algebraics of V
    and constants that the others read, and the largest subexpressions of the
    others that read V and constants (no scalable one) alone and hold a special
    function."""
    body = _without_v_rate(m)
    h = analyse(m, m.rates)
    inv = set(h.invariant)
    slots: Dict[Node, str] = {}
    varying: Dict[str, bool] = {}
    defined: set = set()

    def reads_v(e: Node) -> bool:
        return any(isinstance(n, Ref) and n.array in ("STATES", "ALGEBRAIC") for n in walk(e))

    def whole(e: Node) -> bool:
        special = False
        for n in walk(e):
            if isinstance(n, Var) and n.name not in ("tissueFlag", "dimension"):
                return False
            if isinstance(n, Call):
                if n.fn == "computeIstim":
                    return False
                special |= n.fn in ("exp", "log", "sqrt", "tanh", "tissueSelect") or (
                    n.fn == "pow" and _int_exponent(n.args[1]) is None)
            if isinstance(n, Ref) and (
                    (n.array == "STATES" and n.name != m.states[0]) or n.array == "RATES" or
                    (n.array == "CONSTANTS" and n.name in SCALABLE[m.name].values()) or
                    (n.array == "ALGEBRAIC" and n.name not in inv & defined)):
                return False
        return special

    def slot(e: Node) -> Ref:
        if e not in slots:
            slots[e] = str(len(slots))
            varying[slots[e]] = reads_v(e)
        return Ref("H", slots[e])

    def rewrite(e: Node) -> Node:
        if isinstance(e, (Num, Var)):
            return e
        if isinstance(e, Ref):
            if e.array == "ALGEBRAIC" and e.name in inv and e.name in defined:
                return slot(e)
            return Ref(e.array, e.name)
        if whole(e):
            return slot(e)
        if isinstance(e, Unary):
            return Unary(e.op, rewrite(e.e))
        if isinstance(e, Bin):
            return Bin(e.op, rewrite(e.l), rewrite(e.r))
        if isinstance(e, Cond):
            return Cond(rewrite(e.c), rewrite(e.a), rewrite(e.b))
        return Call(e.fn, tuple(rewrite(x) for x in e.args))

    first, rest = [], []
    for st in body:
        if st.target.array == "ALGEBRAIC" and st.target.name in inv:
            first.append(st)
            defined.add(st.target.name)
        else:
            rest.append(Assign(st.target, rewrite(st.expr), st.line))
    first += [Assign(Ref("H", k), e, 0) for e, k in slots.items()]
    return first, rest, varying


def emit_split(m: Model) -> str:
    first, rest, varying = take_apart(m)
    vm = m.states[0]
    L = [f"constexpr int ADJ_NH = {len(varying)};",
         "// What the right-hand side has of V and constants alone (the same at every",
         "// stage of a PDE step).",
         "template <class R, class KS>",
         f"__device__ __forceinline__ void adj_hoist(R y_{vm}, const KS& K, int tissue, R* H)",
         "{",
         "    (void)tissue;"]
    gen = _Gen(m, [], fused=True)
    fwd: List[str] = []
    targets = _walk_body(gen, first, fwd)
    L += gen.decl + fwd
    L += [f"    H[{st.target.name}] = {gen.value.get(id(st.expr)) or gen.leaf(st.expr)};"
          for st, _ in targets if st.target.array == "H"]
    L += ["}", "",
          "// Their derivative: the adjoint of V for the adjoint hbar of H.",
          "template <class R, class KS>",
          f"__device__ __forceinline__ R adj_hoist_vjp(R y_{vm}, const KS& K, int tissue, "
          "const R* hbar)",
          "{",
          "    (void)tissue;",
          f"    R ybar[1] = {{R(0)}};"]
    gen = _Gen(m, [], fused=True)
    fwd = []
    targets = _walk_body(gen, first, fwd)
    targets = [(st, n) for st, n in targets
               if not (st.target.array == "H" and not varying[st.target.name])]
    rev = [x.replace(f"ybar[S_{vm}]", "ybar[0]") for x in _reverse(gen, targets)]
    L += gen.decl + fwd + rev + ["    return ybar[0];", "}", ""]

    gen = _Gen(m, use_before_def(m.rates), fused=True)
    gen.varying = {k for k, v in varying.items() if v}
    fwd = []
    targets = _walk_body(gen, rest, fwd)
    iion = gen.defined[m.iion_name]
    L += ["// The right-hand side with them; returns Iion_cm.",
          "template <class R, class KS>",
          "__device__ __forceinline__ R adj_rhs(double t, const R* y, const KS& K, int tissue, "
          "const R* H, R* dydt)",
          "{",
          "    (void)t; (void)tissue;"]
    decl = [d for d in gen.decl if not d.startswith("    R ba")]
    L += _states_and_params(gen) + decl + fwd
    L += [f"    dydt[S_{st.target.name}] = {gen.value.get(id(st.expr)) or gen.leaf(st.expr)};"
          for st, _ in targets if st.target.array == "RATES"]
    L += [f"    return {iion};", "}", "",
          "// Its derivative: as rhs_vjp, and to hbar the adjoint of H.",
          "template <class R, class KS>",
          "__device__ __forceinline__ void adj_rhs_vjp(double t, const R* y, const KS& K, "
          "int tissue, const R* H, const R* dbar, R ibar, R* ybar, R* pbar, R* hbar)",
          "{",
          "    (void)t; (void)tissue;"]
    rev = [f"    b{iion} += ibar;"] + _reverse(gen, targets)
    L += _states_and_params(gen) + gen.decl + fwd + rev + ["}"]
    return "\n".join(L) + "\n"


def _alg_reads(e: Node):
    for n in walk(e):
        if isinstance(n, Ref) and n.array == "ALGEBRAIC":
            yield n


def emit_adjoint_header(m: Model, src_rel: str) -> str:
    ns = ident(m.name)
    L = [f"// Generated by cardiacfoam_gb300.cellml2cuda from {src_rel}: the reverse-mode",
         "// derivative of the model's tissue-mode right-hand side.  Regenerate with",
         "// `python -m cardiacfoam_gb300.cellml2cuda` instead of editing.",
         "#pragma once",
         "",
         f'#include "{ns}.cuh"',
         "",
         f"namespace cfg {{ namespace {ns} {{",
         ""]
    L.append(emit_rhs_vjp(m))
    L.append(emit_split(m))
    L.append(f"}} }}  // namespace cfg::{ns}")
    return "\n".join(L) + "\n"
