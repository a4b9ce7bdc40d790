"""Kernels that are launched while the one before them still runs, and what they read through helpers: a function that takes its argument for
memory that stays the same (__ldg) is found by what it does, not by its name.  Read from the sources."""
import re

from tests.test_overlapped_launches import _closing, _functions

# Rows and codebooks of an encode: written two launches ago or earlier.
ALLOWED = {
    "rvq_stages_kernel": {"P.x", "book"},
}


def _split(args):
    out, depth, last = [], 0, 0
    for i, c in enumerate(args):
        depth += (c in "([{") - (c in ")]}")
        if c == "," and depth == 0:
            out.append(args[last:i])
            last = i + 1
    return out + [args[last:]]


def _root(expression):
    expression = re.sub(r"reinterpret_cast<[^>]*>\(|static_cast<[^>]*>\(", "", expression)
    name = re.match(r"[\s(&*]*([A-Za-z_][\w.]*)", expression)
    return name.group(1) if name else None


def _calls(body, name):
    for m in re.finditer(r"\b%s\s*(?:<[\w\s,:]*>)?\(" % name, body):
        yield _split(body[m.end():_closing(body, m.end() - 1, "()")])


def _readers(functions):
    """name -> positions of the arguments that it, or a function that it hands them to, reads with __ldg"""
    found = {"__ldg": {0}}
    while True:
        before = sum(map(len, found.values()))
        for name, params, body in functions:
            own = [re.sub(r"\W*$", "", p.split("=")[0]).split("[")[0].split()[-1].lstrip("*&(") if p.strip() else "" for p in _split(params)]
            for reader, at in list(found.items()):
                for args in _calls(body, reader):
                    for i in at:
                        root = _root(args[i]) if i < len(args) else None
                        if root in own:
                            found.setdefault(name, set()).add(own.index(root))
        if sum(map(len, found.values())) == before:
            return found


def test_what_helpers_take_for_invariant():
    functions = list(_functions())
    readers = _readers(functions)
    assert readers["load4"] == {1}
    for name, _, body in functions:
        if "after_previous_kernel();" not in body or name not in ALLOWED:
            continue
        taken = {_root(args[i]) for reader, at in readers.items() for args in _calls(body, reader) for i in at if i < len(args)}
        assert taken == ALLOWED[name], f"{name} reads {sorted(taken)} as invariant"


def test_a_planted_read_is_found():
    functions = [(n, p, b.replace("load4(v[i], P.x + row", "load4(v[i], P.frames + row") if n == "rvq_stages_kernel" else b) for n, p, b in _functions()]
    readers = _readers(functions)
    body = next(b for n, _, b in functions if n == "rvq_stages_kernel")
    taken = {_root(args[i]) for reader, at in readers.items() for args in _calls(body, reader) for i in at if i < len(args)}
    assert "P.frames" in taken
