"""The FP32 right-hand side of the mixed adjoint rounds products that it adds or
subtracts once: they are written as multiply-adds, not left to a compiler."""
import re
from pathlib import Path

HEADER = (Path(__file__).resolve().parents[1] / "cardiacfoam_gb300" / "csrc" / "models" /
          "tnnp_adjoint.cuh")


def _function(text, name):
    body = text[text.index(f" {name}("):]
    return body[:body.index("\n}\n")]


def test_products_are_added_by_multiply_adds():
    text = HEADER.read_text()
    n = 0
    for name in ("adj_hoist", "adj_hoist_vjp", "adj_rhs", "adj_rhs_vjp"):
        products = set()
        for line in _function(text, name).splitlines():
            m = re.match(r"\s*(\w+) = (.*);$", line)
            if not m or m.group(1).startswith(("g", "ba")):      # the reverse sweep
                continue
            target, expr = m.groups()
            if re.match(r"a\d+$", target) and expr in products:
                products.add(target)
            op = re.match(r"\((\S+) ([-+*]) (\S+)\)$", expr)
            if op and op.group(2) == "*":
                products.add(target)
            elif op:
                assert not {op.group(1), op.group(3)} & products, (name, line)
            n += "cfg_fma(" in expr
    assert n > 50
