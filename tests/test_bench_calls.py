"""bench.py's calls of its own functions fit their signatures (its studies run on a GPU only)."""
import ast
import os

PATH = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bench.py")


def test_calls_fit_the_functions_they_name():
    tree = ast.parse(open(PATH).read())
    defs = {n.name: n.args for n in tree.body if isinstance(n, ast.FunctionDef)}
    checked = 0
    for call in ast.walk(tree):
        if not (isinstance(call, ast.Call) and isinstance(call.func, ast.Name) and call.func.id in defs):
            continue
        if any(isinstance(a, ast.Starred) for a in call.args) or any(k.arg is None for k in call.keywords):
            continue
        a = defs[call.func.id]
        names = [x.arg for x in a.posonlyargs + a.args]
        needed = set(names[:len(names) - len(a.defaults)])
        given = set(names[:len(call.args)]) | {k.arg for k in call.keywords}
        where = f"{call.func.id} at line {call.lineno}"
        assert a.vararg or len(call.args) <= len(names), where
        assert needed <= given, (where, needed - given)
        assert a.kwarg or given <= set(names) | {x.arg for x in a.kwonlyargs}, where
        checked += 1
    assert checked > 20
