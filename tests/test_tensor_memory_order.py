"""Tensor memory behind a wait: tcgen05 instructions of a thread are ordered behind what an mbarrier announced only by a
``tcgen05.fence::after_thread_sync`` between the wait and the instruction.  Read off the sources, without a GPU."""
import re
from pathlib import Path

import pytest

SOURCES = Path(__file__).resolve().parents[1] / "actlizela_b200" / "csrc" / "backends" / "sm100"
FENCE = "tc_fence_after()"
EVENT = re.compile(r"(?P<fence>tc_fence_after\(\))|(?P<access>\b(?:tmem_(?:ld|st)\d+|mma_[st]s)\()"
                   r"|\b(?:mbar_wait|warp_wait)\((?P<wait>[^,]+),|(?P<lock>\bacc_lock\()")
KERNELS = {"gdn_fused.cu": ("prepare_chunk", "forward_umma_kernel"), "gdn_umma.cu": ("prepare_umma_kernel", "walk_umma_kernel"),
           "out_proj.cu": ("out_proj_umma_kernel", "out_proj_skinny_kernel")}
# Waits behind which the thread itself touches no tensor memory that the barrier guards.
ELSEWHERE = {
    ("prepare_chunk", "&bar->u[group]"): "the product has read its operand in shared memory",
    ("walk_umma_kernel", "bar_ofree + (c & 1)"): "passed on with the operand; the issuer's own fence follows",
}


def _body(file, name):
    """Text between the braces of a function, comments and its blank lines aside."""
    code = re.sub(r"//[^\n]*", "", (SOURCES / file).read_text())
    at = re.search(r"(?:\)\s+|__device__ __forceinline__ bool )" + name + r"\(", code).end()
    start = code.index("{", at)
    depth = 0
    for i in range(start, len(code)):
        depth += {"{": 1, "}": -1}.get(code[i], 0)
        if depth == 0:
            return code[start + 1:i]
    raise AssertionError(name)


def _header(text):
    """What opens a block: its keyword with the ``else`` in front of it, if any."""
    text = text.rstrip()
    if text.endswith(")"):
        depth, at = 0, len(text)
        while at:
            at -= 1
            depth += {")": 1, "(": -1}.get(text[at], 0)
            if depth == 0:
                break
        text = text[:at]
    return " ".join(re.search(r"(?:\belse\s+)?\w*\s*$", text).group().split())


def _tree(text):
    """Statements in order: text, or (keyword, statements) for a block."""
    root, stack, at = [], [], 0
    level = root
    for m in re.finditer(r"[{}]", text):
        level.append(text[at:m.start()])
        at = m.end()
        if m.group() == "{":
            block = (_header(text[:m.start()]), [])
            level.append(block)
            stack.append(level)
            level = block[1]
        else:
            level = stack.pop()
    level.append(text[at:])
    return root


def _walk(level, pending, name, found, seen):
    """Waits that no fence has followed yet on some way through `level`; accesses that they reach go to `found`."""
    entry = pending                   # in front of the first branch of an if / else chain
    for part in level:
        if isinstance(part, str):
            for m in EVENT.finditer(part):
                if m["fence"]:
                    pending = frozenset()
                elif m["access"]:
                    seen["accesses"] += 1
                    if pending:
                        found.append((m["access"], sorted(pending)))
                else:
                    seen["waits"] += 1
                    bar = " ".join(m["wait"].split()) if m["wait"] else "lock"
                    if (name, bar) not in ELSEWHERE:
                        pending |= {bar}
            continue
        header, inner = part
        if not header.startswith("else"):
            entry = pending
        end = _walk(inner, entry, name, found, seen)
        if header in ("for", "while"):
            end = _walk(inner, end, name, found, seen)                # round again, with what the first turn left
        pending = pending | end if header in ("if", "else if", "else", "for", "while") else end      # taken or not
    return pending


def _violations(name, body):
    found, seen = [], {"waits": 0, "accesses": 0}
    _walk(_tree(body), frozenset(), name, found, seen)
    return found, seen


@pytest.mark.parametrize("file,name", [(f, n) for f, names in KERNELS.items() for n in names])
def test_fence_between_every_wait_and_tensor_memory(file, name):
    body = _body(file, name)
    found, seen = _violations(name, body)
    assert seen["waits"] and seen["accesses"]
    assert not found, found
    assert _violations(name, body.replace(FENCE, ""))[0]            # without its fences the same kernel is caught
