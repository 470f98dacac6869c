"""bench.py as source: each function once, every name a function uses defined,
and the kernels of a split solve counted as the library launches them."""
import ast
import builtins
import os
import symtable

from conftest import ROOT

SRC = open(os.path.join(ROOT, "bench.py")).read()


def test_every_top_level_name_is_defined_once():
    names = [d.name for d in ast.parse(SRC).body if isinstance(d, (ast.FunctionDef, ast.ClassDef))]
    assert sorted(names) == sorted(set(names))


def test_every_global_a_function_uses_exists():
    top = symtable.symtable(SRC, "bench.py", "exec")
    known = set(top.get_identifiers()) | set(dir(builtins))

    def missing(table):
        for s in table.get_symbols():
            if s.is_global() and s.is_referenced() and s.get_name() not in known | {"__file__", "__name__"}:
                yield table.get_name(), s.get_name()
        for child in table.get_children():
            yield from missing(child)

    assert not list(missing(top))


def test_kernels_of_a_split_solve():
    import bench

    # one iteration and one replacement that ends the solve: two mailbox
    # fills, the first residual, residual + solves + r'w, an iteration of
    # five, the replacement's residual, the final one
    assert bench.split_launches(1, 1) == 2 + 1 + 4 + 5 + 1 + 1
    # a further iteration, and a further replacement with its resume of four
    assert bench.split_launches(2, 1) - bench.split_launches(1, 1) == 5
    assert bench.split_launches(1, 2) - bench.split_launches(1, 1) == 1 + 4
