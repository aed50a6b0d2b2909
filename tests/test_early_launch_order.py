"""Kernels that may start before the kernel in front of them has ended: none of their CTAs may end before it has."""
import re
from pathlib import Path

import pytest

SOURCES = Path(__file__).resolve().parents[1] / "actlizela_b200" / "csrc" / "backends" / "sm100"
WAIT = "wait_for_previous_kernel();"


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def _body(code, kernel):
    """Text of a kernel from its parameter list to the brace that closes it."""
    at = re.search(r"__launch_bounds__\([^)]*(?:<[^)]*)?\)\s+" + kernel + r"\s*\(", code)
    assert at, kernel
    start = code.index("{", code.index(")", at.end()))
    depth = 0
    for i in range(start, len(code)):
        depth += {"{": 1, "}": -1}.get(code[i], 0)
        if depth == 0:
            return code[start:i]
    raise AssertionError(kernel)


def _early_kernels():
    for path in sorted(SOURCES.glob("*.cu")):
        code = _code(path)
        names = {name for m in re.finditer(r"return launch_early\(", code) for name in re.findall(r"\b\w+_kernel\b", code[m.end():m.end() + 100])}
        if "attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization" in code:
            names.add("out_proj_skinny_kernel")
        for name in sorted(names):
            yield pytest.param(code, name, id=name)


@pytest.mark.parametrize("code,kernel", list(_early_kernels()))
def test_no_cta_ends_before_the_kernel_in_front(code, kernel):
    """A CTA that returns without the wait lets the launch end while the kernel in front of it still runs: the next
    launch then writes to memory (the call's scratch, given back by then) that kernel still reads."""
    body = _body(code, kernel)
    assert WAIT in body
    leaves = [m.start() for m in re.finditer(r"\breturn\b", body)]
    assert all(body.index(WAIT) < at for at in leaves)
