"""Emitter of the plain form's right-hand sides, ``csrc/models/<model>_plain.cuh``.

GB300 issues one FP64 instruction per SM partition every 64 clocks, so the
plain form's time is its FP64 instruction count.  The body that
:mod:`emit` writes for both forms is written here for double alone, with the
same operations in the same order but for

* products that are added or subtracted: one multiply-add, written out (the
  kernels are compiled without contraction, so that a value rounds alike in
  every kernel that evaluates it);
* divisions by a constant of the tissue, by a value of the membrane potential
  that the step keeps, or by a divisor several quotients share: the product
  with its reciprocal and one exact correction (``cfg_quotient``), three
  instructions for nine.

The file adds what the tissue step needs to take the linear gates out of the
stage loop (:mod:`gates`) and to share a cell between warps (:mod:`split`).
"""
from __future__ import annotations

from typing import Dict, List

from .cexpr import Bin, Call, Node, Num, Ref, Unary, refs, walk
from .emit import (_CudaPrinter, _Printer, _TissuePrinter, _cuda_body, _cuda_body_tissue,
                   _int_exponent, _is_int_expr, _predeclare_conditional_algebraics, _state_loads,
                   ident, scale_dependent_constants)
from .gates import linear_gates
from .hoist import analyse, invariant_statements
from .model import Assign, Model, iter_assigns, use_before_def
from .split import partition


def shared_divisors(m: Model, invariant=frozenset()) -> Dict[Node, int]:
    """Divisors that at least three top-level quotients of the right-hand side
    divide by (the normalisations of the exchanger's and the pump's states),
    whose operands are not all constants or invariants, numbered."""
    count: Dict[Node, int] = {}
    for st in m.rates:
        if isinstance(st, Assign) and isinstance(st.expr, Bin) and st.expr.op == "/":
            d = st.expr.r
            if isinstance(d, Bin) and any(r.array == "ALGEBRAIC" and r.name not in invariant
                                          for r in refs(d)):
                count[d] = count.get(d, 0) + 1
    return {d: k for k, d in enumerate(d for d, n in count.items() if n >= 3)}


class _Plain:
    """The double spelling of an expression, mixed into a printer."""

    def setup(self, m: Model, shared: Dict[Node, int]):
        self.scaled = set(scale_dependent_constants(m))
        self.shared = shared
        self.shared_done = set()
        return self

    def _tissue_constant(self, e: Node) -> bool:
        """Numbers and constants that do not change with a cell's conductance
        scales: known to the compiler in the kernels of one tissue."""
        return all(isinstance(n, (Num, Unary, Bin)) or
                   (isinstance(n, Ref) and n.array == "CONSTANTS" and n.name not in self.scaled) or
                   (isinstance(n, Call) and n.fn == "pow" and
                    _int_exponent(n.args[1]) is not None)
                   for n in walk(e))

    def _product(self, e: Node) -> bool:
        return (isinstance(e, Bin) and e.op == "*" and not self._tissue_constant(e) and
                not _is_int_expr(e.l) and not _is_int_expr(e.r) and not self._kept(e))

    def _kept(self, e: Node) -> bool:
        """A subexpression the step keeps in H."""
        return False

    def spell(self, e: Node):
        """The double form of e, or None where it is the common one."""
        if not isinstance(e, Bin) or self._tissue_constant(e):
            return None
        if e.op == "/" and self._tissue_constant(e.r):
            return f"cfg_cdiv<KS>({self(e.l)}, {self(e.r)})"
        if e.op == "/" and e.r in self.shared:
            return f"cfg_quotient({self(e.l)}, {_Printer.__call__(self, e.r)}, " \
                   f"r_{self.shared[e.r]})"
        if e.op in "+-" and self._product(e.l):
            c = self(e.r)
            return f"cfg_fma({self(e.l.l)}, {self(e.l.r)}, {c if e.op == '+' else '-' + c})"
        if e.op in "+-" and self._product(e.r):
            a = self(e.r.l)
            return f"cfg_fma({a if e.op == '+' else '-' + a}, {self(e.r.r)}, {self(e.l)})"
        return None

    def reciprocals(self, st, indent, out):
        """The reciprocal of a shared divisor, before its first quotient."""
        for d, k in self.shared.items():
            if k not in self.shared_done and isinstance(st, Assign) and any(
                    isinstance(n, Bin) and n.op == "/" and n.r == d for n in walk(st.expr)):
                out.append(f"{indent}const R r_{k} = R(1.0) / {_Printer.__call__(self, d)};")
                self.shared_done.add(k)


class _Body(_Plain, _CudaPrinter):
    def __call__(self, e: Node) -> str:
        if isinstance(e, Bin) and e.op == "-" and isinstance(e.l, Call) and e.l.fn == "exp":
            return _CudaPrinter.__call__(self, e)
        return self.spell(e) or _CudaPrinter.__call__(self, e)


class _TissueBody(_Plain, _TissuePrinter):
    def _kept(self, e: Node) -> bool:
        return self._extractable(e)

    def __call__(self, e: Node) -> str:
        if isinstance(e, Bin) and (self._slot_of(e.r) if e.op == "/" else None) is None and \
                not self._extractable(e) and \
                not (e.op == "-" and isinstance(e.l, Call) and e.l.fn == "exp"):
            s = self.spell(e)
            if s is not None:
                return s
        return _TissuePrinter.__call__(self, e)

    def _slot_of(self, e: Node):
        if isinstance(e, Ref):
            return self._slot(e)
        return "kept" if self._extractable(e) else None


def _statements(m: Model, stmts, pr, body, out):
    """body() of each top-level statement after the reciprocals it needs."""
    for st in stmts:
        pr.reciprocals(st, "    ", out)
        body(m, [st], pr, "    ", out)


def _function(name, args, lines, ret="double"):
    head = (f"template <class YS, class KS{', class HS' if 'HS&' in args else ''}>" if "YS&" in args
            else f"template <class KS{', class HS' if 'HS&' in args else ''}>")
    return [head, f"__device__ __forceinline__ {ret} {name}({args})", "{", "    using R = double;",
            *lines, "}"]


def emit_plain(m: Model, src_rel: str) -> str:
    ns = ident(m.name)
    h = analyse(m, m.rates)
    vm = m.states[0]
    void = "    (void)tissue; (void)K;"
    L: List[str] = [
        f"// Generated by cardiacfoam_gb300.cellml2cuda from {src_rel}: the right-hand",
        "// sides of the plain FP64 form (see cellml2cuda/emit_plain.py).  Regenerate with",
        "// `python -m cardiacfoam_gb300.cellml2cuda` instead of editing.",
        "#pragma once",
        f'#include "{ns}.cuh"',
        "",
        f"namespace cfg {{ namespace {ns} {{ namespace plain {{",
        "",
        "// rhs() of the common header"]
    early = use_before_def(m.rates)
    pr = _Body(m, early, "rhs").setup(m, shared_divisors(m))
    body: List[str] = []
    for name in _predeclare_conditional_algebraics(m, m.rates, body, "    "):
        body.append(f"    R a_{name} = R(0);")
        pr.defined.add(name)
    _statements(m, m.rates, pr, _cuda_body, body)
    L += ["template <bool SOLVE_VM, class YS, class KS>",
          "__device__ __forceinline__ double rhs(double t, const YS& Y, const KS& K, double* dydt, "
          "int tissue, const CfgStimulus& stim)", "{", "    using R = double;",
          void + " (void)stim; (void)t;", *_state_loads(m, pr), *body,
          f"    return a_{m.iion_name};", "}", ""]
    # the tissue form: pass 1 finds the slots read only as divisors
    recip: set = set()
    subtrees: Dict[Node, int] = {}
    rest: List[str] = []
    if h.needed:
        first = _TissuePrinter(m, early, h.invariant, h.needed)
        scratch: List[str] = []
        for name in _predeclare_conditional_algebraics(m, m.rates, scratch, "    "):
            if name not in h.invariant:
                first.defined.add(name)
        _cuda_body_tissue(m, m.rates, first, "    ", scratch)
        recip = {k for k in first.div_uses if k not in first.other_uses}
        recip.discard(f"H_{m.iion_name}")
        pr = _TissueBody(m, early, h.invariant, h.needed, frozenset(recip))
        pr.setup(m, shared_divisors(m, h.invariant))
        pr.subtrees = dict(first.subtrees)
        for name in _predeclare_conditional_algebraics(m, m.rates, rest, "    "):
            if name not in h.invariant:
                rest.append(f"    R a_{name} = R(0);")
                pr.defined.add(name)
        _statements(m, m.rates, pr, _cuda_body_tissue, rest)
        rest = _state_loads(m, pr) + rest
        rest.append(f"    return {'H(H_' if m.iion_name in h.invariant else 'a_'}{m.iion_name}"
                    f"{')' if m.iion_name in h.invariant else ''};")
        subtrees = dict(first.subtrees)
        if len(pr.subtrees) != len(subtrees):
            raise ValueError(f"{m.name}: the plain form keeps other values than the common one")
    L += ["// hoist() and rhs_tissue() of the common header; a slot read only as a divisor",
          "// holds its reciprocal too"]
    hoisted: List[str] = []
    if h.needed:
        stmts = invariant_statements(m.rates, h.invariant)
        pr = _Body(m, [], "rhs").setup(m, {})
        for name in _predeclare_conditional_algebraics(m, stmts, hoisted, "    "):
            hoisted.append(f"    R a_{name} = R(0);")
            pr.defined.add(name)
        _cuda_body(m, stmts, pr, "    ", hoisted)
        for a in h.needed:
            hoisted.append(f"    H[H_{a}] = " +
                           (f"CfgSlot::divisor(a_{a});" if f"H_{a}" in recip else f"a_{a};"))
        for e, k in sorted(subtrees.items(), key=lambda kv: kv[1]):
            slot = str(len(h.needed) + k)
            hoisted.append(f"    H[{slot}] = " +
                           (f"CfgSlot::divisor({pr(e)});" if slot in recip else f"{pr(e)};"))
    L += _function("hoist", f"double y_{vm}, const KS& K, int tissue, CfgSlot* H",
                   [void + f" (void)H; (void)y_{vm};", *hoisted], "void")
    args = "const YS& Y, const KS& K, const HS& H, double* dydt, int tissue"
    if h.needed:
        L += _function("rhs_tissue", args,
                       ["    constexpr bool SOLVE_VM = false;", "    constexpr double t = 0.0;",
                        "    const CfgStimulus stim{};",
                        void + " (void)H; (void)t; (void)stim;", *rest])
    else:
        L += _function("rhs_tissue", args,
                       ["    (void)H;", "    return rhs<false>(0.0, Y, K, dydt, tissue, "
                        "CfgStimulus{});"])
    # linear gates
    gates = linear_gates(m, h.invariant)
    pr = _TissueBody(m, [], h.invariant, h.needed, frozenset(recip)).setup(m, {})
    pr.hoisted_defined = set(h.invariant)
    pr.subtrees = dict(subtrees)
    decay = [f"    b[S_{s}] = {pr(e)};" for s, e in gates.items()]
    pr.states_read = set()
    slopes = [f"    d[S_{st.target.name}] = {pr(st.expr)};" for st in iter_assigns(m.rates)
              if st.target.array == "RATES" and st.target.name in gates]
    if len(pr.subtrees) != len(subtrees):
        raise ValueError(f"{m.name}: a gate needs a value H does not keep")
    mask = sum(1 << m.states.index(s) for s in gates)
    L += ["// States whose tissue-mode rate is a - b y with a and b functions of state 0 and",
          "// constants alone (bit i = state i): b of each, and their rates alone.",
          f"constexpr unsigned long long LIN_MASK = 0x{mask:x}ull;"]
    L += _function("gate_decay", f"double y_{vm}, const KS& K, const HS& H, int tissue, double* b",
                   [void + f" (void)H; (void)b; (void)y_{vm};", *decay], "void")
    L += _function("gate_rates", "const YS& Y, const KS& K, const HS& H, int tissue, double* d",
                   [void + " (void)H; (void)d; (void)Y;", *_state_loads(m, pr), *slopes], "void")
    for name, solve_vm in (("tissue", False), ("sv", True)):
        L += [f"// Warp of state i where four warps share a cell's step "
              f"({'Vm a state' if solve_vm else 'tissue mode'}; split.py).",
              f"CFG_HD constexpr int part_{name}(int i)", "{",
              "    constexpr signed char part[NS] = {" +
              ", ".join(map(str, partition(m, solve_vm))) + "};",
              "    return part[i];", "}"]
    L += ["", "// the model's traits with these right-hand sides",
          f"struct Model : {ns}::Model {{",
          "    static constexpr unsigned long long LIN_MASK = plain::LIN_MASK;",
          "    template <bool SV, class YS, class KS>",
          "    __device__ static __forceinline__ double rates(double t, const YS& Y, const KS& K, "
          "double* dydt, int tissue, const CfgStimulus& st) "
          "{ return plain::rhs<SV>(t, Y, K, dydt, tissue, st); }",
          "    template <class KS>",
          "    __device__ static __forceinline__ void hoist_vm(double v, const KS& K, int tissue, "
          "CfgSlot* H) { plain::hoist(v, K, tissue, H); }",
          "    template <class YS, class KS, class HS>",
          "    __device__ static __forceinline__ double rates_tissue(const YS& Y, const KS& K, "
          "const HS& H, double* dydt, int tissue) "
          "{ return plain::rhs_tissue(Y, K, H, dydt, tissue); }",
          "    template <class KS, class HS>",
          "    __device__ static __forceinline__ void decay(double v, const KS& K, const HS& H, "
          "int tissue, double* b) { plain::gate_decay(v, K, H, tissue, b); }",
          "    template <class YS, class KS, class HS>",
          "    __device__ static __forceinline__ void slopes(const YS& Y, const KS& K, "
          "const HS& H, int tissue, double* d) { plain::gate_rates(Y, K, H, tissue, d); }",
          "    CFG_HD static constexpr int part_tissue(int i) { return plain::part_tissue(i); }",
          "    CFG_HD static constexpr int part_sv(int i) { return plain::part_sv(i); }",
          "};", "", f"}} }} }}  // namespace cfg::{ns}::plain"]
    return "\n".join(L) + "\n"
