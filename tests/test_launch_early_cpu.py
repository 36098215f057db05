"""Kernels that may be resident while the kernel ahead of them still writes (launch_early) read global memory in ways that stay
behind grid_wait() and see those writes: no read-only loads, no no-alias parameters, no hinted loads the compiler may move. Checked in
the source, over the kernels and every device function that they call."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "aitemplate_b200" / "csrc"
FORBIDDEN = re.compile(r"__ldg\s*\(|__ldc[agsv]\s*\(|__ldlu\s*\(|__restrict__|ld\.global\.nc")


def _code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def _functions(code):
    """name -> text from the qualifier to the closing brace, of every __global__ and __device__ function."""
    found = {}
    for m in re.finditer(r"__(global|device)__\b", code):
        brace, semi = code.find("{", m.start()), code.find(";", m.start())
        if brace < 0 or (0 <= semi < brace):
            continue  # a variable
        name = re.findall(r"([A-Za-z_]\w*)\s*\(", re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", code[m.start():brace]))
        depth, end = 0, brace
        for end in range(brace, len(code)):
            depth += {"{": 1, "}": -1}.get(code[end], 0)
            if depth == 0:
                break
        if name:
            found.setdefault(name[0], []).append((m.group(1), code[m.start():end + 1]))
    return found


@pytest.fixture(scope="module")
def functions():
    every = {}
    for path in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
        for name, texts in _functions(_code(path)).items():
            every.setdefault(name, []).extend(texts)
    return every


def _reached(functions, name):
    seen, todo = set(), [name]
    while todo:
        at = todo.pop()
        if at in seen:
            continue
        seen.add(at)
        for _, text in functions[at]:
            todo += [f for f in set(re.findall(r"\b([A-Za-z_]\w*)\s*(?:<[^;{}()]*>)?\s*\(", text)) if f in functions and f != at]
    return seen


def test_kernels_launched_early_wait(functions):
    waiting = {n for n, texts in functions.items() if any(kind == "global" and "grid_wait()" in text for kind, text in texts)}
    assert len(waiting) >= 10
    for path in CSRC.glob("*.cu*"):
        code = _code(path)
        for at in re.finditer(r"launch_early\(\s*(?:vec \? )?&(\w+)", code):
            assert at.group(1) in waiting, at.group(1)


def test_no_read_only_loads_behind_grid_wait(functions):
    kernels = [n for n, texts in functions.items() if any(kind == "global" and "grid_wait()" in text for kind, text in texts)]
    bad = {(k, f, hit) for k in kernels for f in _reached(functions, k) for _, text in functions[f] for hit in FORBIDDEN.findall(text)}
    assert not bad, sorted(bad)
