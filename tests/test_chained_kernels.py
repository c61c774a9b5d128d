"""Kernels launched before their predecessor has finished (pdl.cuh) wait in
their first statement, and read nothing through a __restrict__ pointer to
const: the compiler may take such a load for one of constant memory and move
it above the wait.  Checked in the sources, for the kernels, the functions
that they call and the functors that they take."""
import re

import pytest

from .conftest import ROOT

CSRC = ROOT / "anelastic_solve_b200" / "csrc"
RESTRICT_CONST = re.compile(r"const\s+[\w:<>]+\s*\*\s*__restrict__")


def definitions(path):
    """(name, text) of the functions, kernels and structs of a file, split
    where a line starts one at the margin or in a namespace."""
    text = re.sub(r"//.*", "", path.read_text())
    heads = [m.start() for m in re.finditer(r"^(?=template\s*<|__global__|__device__|static |inline |struct |[\w:<>]+[ *&]+\w+\()",
                                            text, re.M)]
    for a, b in zip(heads, heads[1:] + [len(text)]):
        t = text[a:b]
        m = re.match(r"struct (\w+)", t) or re.search(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\([^)]*\)", "", t))
        if m:
            yield m.group(1), t


DEFS = [(p.name, n, t) for p in sorted(CSRC.glob("*.cu*")) for n, t in definitions(p)]
CHAINED = [(f, n, t) for f, n, t in DEFS if "__global__" in t and "chain_enter();" in t]


def reached(file, text):
    """The definitions that a kernel's text names, and those that these
    name; the functors of its file where it takes some."""
    todo, seen = [text], {}
    if re.search(r"\bIn in\b", text):
        todo += [t for f, n, t in DEFS if f == file and "operator()" in t]
    while todo:
        t = todo.pop()
        seen[t] = True
        words = set(re.findall(r"\w+", t))
        todo += [u for f, n, u in DEFS if n in words and u not in seen and u not in todo
                 and "__global__" not in u and (f == file or f.endswith(".cuh"))]
    return seen


def test_every_chained_launch_is_of_a_kernel_that_waits():
    names = {n for _, n, _ in CHAINED}
    assert len(names) > 15
    for p in CSRC.glob("*.cu"):
        for k in re.findall(r"launch_chained\(\s*(k_\w+)", p.read_text()):
            assert k in names, (p.name, k)


@pytest.mark.parametrize("file,name,text", CHAINED, ids=[n for _, n, _ in CHAINED])
def test_no_restrict_pointers_to_const(file, name, text):
    body = text[text.index("{"):]
    assert re.match(r"\{\s*chain_enter\(\);", body), f"{name} does not wait first"
    for t in reached(file, text):
        assert not RESTRICT_CONST.search(t), f"{name} reaches {t[:120]}"
