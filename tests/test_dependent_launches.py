"""Kernels launched while the launch before them drains (csrc/launch.cuh) must
not let the compiler read through the read-only path, or move a load above the
wait: a __restrict__ pointer declares that nobody else writes what it points to
for the kernel's whole life, and before the wait the previous launch still does.
Checked on the sources, for each such kernel and every device function it calls."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "1dsweptcuda_gb300" / "csrc"
WAIT = "wait_for_previous_launch"
# written by an ordinary launch that has completed before the first of the dependent ones starts
STAGED = {("k_forward", "weights")}


def _balanced(text, start, opening, closing):
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == opening) - (text[i] == closing)
        if depth == 0:
            return i
    raise ValueError("unbalanced")


def _functions():
    """name -> [(is a kernel, parameters, body)] of the device functions."""
    out = {}
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)
        for m in re.finditer(r"\b(__global__|__device__)\b", text):
            end = re.compile(r"[{;]").search(text, m.end())
            header = text[m.start():end.start()].rstrip()
            if end.group() == ";" or not header.endswith(")"):
                continue
            depth, i = 0, len(header) - 1
            while True:
                depth += (header[i] == ")") - (header[i] == "(")
                if depth == 0:
                    break
                i -= 1
            name = re.search(r"(\w+)\s*$", header[:i]).group(1)
            body = text[end.start():_balanced(text, end.start(), "{", "}") + 1]
            out.setdefault(name, []).append((m.group(1) == "__global__", header[i + 1:-1], body))
    return out


FUNCTIONS = _functions()
DEPENDENT = sorted(n for n, fs in FUNCTIONS.items() for k, _, body in fs if k and WAIT in body)


def _reached(kernel):
    seen, todo = set(), [kernel]
    while todo:
        name = todo.pop()
        if name in seen:
            continue
        seen.add(name)
        for _, _, body in FUNCTIONS[name]:
            todo += [w for w in set(re.findall(r"\b\w+\b", body)) if w in FUNCTIONS]
    return seen


def test_every_dependent_launch_has_a_kernel_that_waits():
    launched = set()
    for path in CSRC.glob("*.cu*"):
        launched |= set(re.findall(r"launch_dependent\(\s*(?:\w+::)*(k_\w+)", path.read_text()))
    assert len(launched) >= 12 and launched <= set(DEPENDENT)


@pytest.mark.parametrize("kernel", DEPENDENT)
def test_no_pointer_is_declared_unaliased(kernel):
    for name in sorted(_reached(kernel)):
        for _, params, body in FUNCTIONS[name]:
            for p in params.split(","):
                if "__restrict__" in p:
                    assert (name, re.search(r"(\w+)\s*$", p).group(1)) in STAGED, "%s: %s" % (name, p.strip())
            assert "__ldg(" not in body and "ld.global.nc" not in body, name
