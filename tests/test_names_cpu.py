"""Constants of the operator module have one meaning each."""
import ast
import collections

from vllm_b200.ops import cuda


def test_no_constant_is_set_twice():
    with open(cuda.__file__) as f:
        names = [n.id for s in ast.parse(f.read()).body if isinstance(s, (ast.Assign, ast.AnnAssign))
                 for t in (s.targets if isinstance(s, ast.Assign) else [s.target]) for n in ast.walk(t) if isinstance(n, ast.Name) and isinstance(n.ctx, ast.Store)]
    assert [n for n, k in collections.Counter(names).items() if k > 1] == []
