"""What the kernels' sources promise about programmatic dependent launch (csrc/common.cuh), read from the sources: no GPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pygpukit_b200" / "csrc"


def strip(text):
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def kernels(path):
    """(name, parameters, body) of every kernel that is defined in a source file"""
    text = strip(path.read_text(encoding="utf-8"))
    for m in re.finditer(r"__global__\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(?:static\s+)?void\s*(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        at, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        params, rest = text[m.end():at - 1], text[at:]
        if not rest.lstrip().startswith("{"):
            continue                                     # a declaration
        at, depth = at + rest.index("{") + 1, 1
        begin = at
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(1), params, text[begin:at - 1]


def all_kernels():
    return [(f.name, *k) for f in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]) for k in kernels(f)]


@pytest.mark.parametrize("where,name,body", [(f, n, b) for f, n, _, b in all_kernels() if "tmem_alloc(" in b], ids=lambda x: x if len(x) < 50 else "")
def test_tensor_memory_is_held_before_dependents_may_start(where, name, body):
    """A dependent block that took the columns first would wait for a grid that waits for them: the allocation, and the barrier behind
    which every thread knows of it, come before griddep_launch."""
    assert "griddep_launch()" in body
    head = body[:body.index("griddep_launch()")]
    assert "tmem_alloc(" in head, f"{where}: {name} lets its dependents start before it holds its tensor memory"
    assert "__syncthreads()" in head[head.rindex("tmem_alloc("):]
