"""CPU: a kernel's source is cut out of its file as inspect.getsource cuts it, without
the tokenizing that took a quarter of a kernel's first call (lang.py, _block)."""
import ast
import importlib.util
import inspect
import textwrap

import pytest

from vernondsl_b200 import lang

SOURCES = {
    "plain": """
def f(x):
    y = x + 1
    return y
z = 1
""",
    "nested, comments at the margin, blank lines": """
def outer():
    def f(x):
        # a comment

        y = x + 1
# at the margin
        for i in y:
            y = i

        return y
    # behind it
    return f
f = outer()
""",
    "last in the file, no newline": "def f(x):\n    return x",
    "decorators over several lines": """
def deco(*a):
    return lambda g: g

class K:
    @deco(1,
  2)
    @deco(
        3
    )
    def f(self, x: float):
        return x
f = K.f
""",
    "a header over several lines": """
def f(
    x: float,
    y: float = 2,
):
    return x
def g(): pass
""",
    "text at the margin inside strings and brackets": '''
def f(x):
    """One line,
another at the margin
    and back."""
    y = [x,
1,
  2]
    s = 1 + \\
2
    return """
def g(): pass
"""
def h(): pass
''',
    "tabs": "def f(x):\n\tif x:\n\t\ty = 1\n\treturn x\nz = 2\n",
    "a form feed in front of a line's indentation": "def f(x):\n    y = x\n\f    y = y + 1\n    return y\nz = 2\n",
    "a form feed between functions": "def f(x):\n    return x\n\f\ndef g(): pass\n",
    "one line": "def f(x): return x\nz = 3\n",
    "else at the margin of if": """
if True:
    def f(x):
        return 1
else:
    def f(x):
        return 2
""",
    "async": """
async def f(x):
    return x
def g(): pass
""",
}


@pytest.mark.parametrize("name", SOURCES)
def test_the_block_is_the_one_inspect_finds(tmp_path, name):
    path = tmp_path / "source.py"
    path.write_text(SOURCES[name])
    spec = importlib.util.spec_from_file_location("lang_source_under_test", path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)

    def parsed(get):
        try:
            return ast.dump(get(), include_attributes=False)
        except (SyntaxError, StopIteration) as e:
            return type(e)

    def by_inspect():
        tree = ast.parse(textwrap.dedent(inspect.getsource(mod.f)))
        return next(n for n in tree.body if isinstance(n, ast.FunctionDef))

    assert parsed(lambda: lang._parse(mod.f)) == parsed(by_inspect)


def test_an_ordinary_kernel_is_not_tokenized(monkeypatch):
    def tokenizes(lines):
        raise AssertionError("the block was looked for by tokenizing")

    monkeypatch.setattr(inspect, "getblock", tokenizes)
    with lang.plan_only():
        o = lang.field(float, (4, 8))

        @lang.kernel
        def double(s: float):
            for i, j in o:
                # twice
                o[i, j] = s * 2.0

        double(1.5)
    assert double.last_tape is not None


def test_a_function_without_source_is_refused_as_before():
    scope = {}
    exec("def f(x):\n    return x\n", scope)
    with pytest.raises(OSError):
        lang._parse(scope["f"])
