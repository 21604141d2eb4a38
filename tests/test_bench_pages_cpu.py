"""Page lists of the serving benchmarks lie within the caches that they make: a list that does not is read, and written, past the cache's end."""
import ast
import os

import krasis_b200

SOURCE = os.path.join(os.path.dirname(krasis_b200.__file__), "bench_seq.py")


def test_decoding_requests_have_their_pages():
    """Four requests of 40 pages of 64 tokens, whatever the prompt's length."""
    tree, seen = ast.parse(open(SOURCE).read()), 0
    for f in ast.walk(tree):
        if not isinstance(f, ast.FunctionDef) or "range(r * 40, r * 40 + 33)" not in ast.unparse(f):
            continue
        seen += 1
        calls = [c for c in ast.walk(f) if isinstance(c, ast.Call) and getattr(c.func, "attr", "") == "make_caches"]
        assert calls, f.name
        for c in calls:
            for tokens in (1, 512, 2048, 4096, 20000):
                assert eval(ast.unparse(c.args[0]), {"tokens": tokens, "max": max}) >= max(tokens, 4 * 40 * 64), (f.name, ast.unparse(c))
    assert seen >= 5
