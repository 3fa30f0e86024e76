"""A kernel that waits for the grid before it (griddep_wait) overlaps that
grid, which writes its inputs: it must not read them through non-coherent
loads, which are for memory that no one writes while the kernel runs."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "glsl-tree-construction_gb300", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def closing(text, i, pair):
    """One past the bracket that closes the one at text[i]."""
    depth = 0
    for j in range(i, len(text)):
        depth += {pair[0]: 1, pair[1]: -1}.get(text[j], 0)
        if depth == 0:
            return j + 1


def functions(text):
    """(name, parameter list, body) of every device function and kernel."""
    for m in re.finditer(r"__(?:global__|device__)\b[^;{=]*?\b(\w+)(?=\()", text):
        name, p = m.group(1), m.end()
        while name in ("__launch_bounds__", "max", "min"):  # an attribute: the name follows it
            p = closing(text, p, "()")
            n = re.compile(r"\s*(\w+)(?=\()").match(text, p)
            if n is None:
                break
            name, p = n.group(1), n.end()
        e = closing(text, p, "()")
        b = re.compile(r"\s*\{").match(text, e)
        if b:
            yield name, text[p:e], text[b.end() - 1:closing(text, b.end() - 1, "{}")]


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_no_non_coherent_loads_behind_the_wait(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    assert "__ldg(" not in text and ".nc." not in text
    for name, params, body in functions(text):
        if "griddep_wait();" in body or (path.endswith("_dev.cuh") or path.endswith("karras.cuh")):
            for p in params.split(","):
                assert not (re.search(r"\bconst\b", p) and "__restrict__" in p), (name, p.strip())


def test_the_scan_finds_the_kernels():
    found = [n for f in FILES for n, _, body in functions(re.sub(r"//[^\n]*", "", open(f).read()))
             if "griddep_wait();" in body]
    calls = sum(len(re.findall(r"griddep_wait\(\);", re.sub(r"//[^\n]*", "", open(f).read()))) for f in FILES)
    assert len(found) == calls > 0
