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


def dependents():
    """Files whose kernels are always launched as dependents, and the headers they share.  (fp8_scan_codes_kernel is launched plainly.)"""
    sources = [f for f in sorted(CSRC.glob("*.cu")) if re.search(r"launch_waiting\(|ProgrammaticStreamSerialization", strip(f.read_text(encoding="utf-8")))]
    return sources + [CSRC / "common.cuh", CSRC / "gemv_common.cuh", CSRC / "tc_common.cuh", CSRC / "tma.cuh"]


def test_dependent_kernels_do_not_load_through_the_read_only_path():
    """Their lifetime overlaps that of the kernel which writes what they read."""
    assert len(dependents()) > 15
    for f in dependents():
        text = strip(f.read_text(encoding="utf-8"))
        for name, _, body in kernels(f):
            if name == "fp8_scan_codes_kernel":
                text = text.replace(body, "")
        assert "__ldg(" not in text and "global.nc" not in text, f.name


def test_other_kernels_read_only_weights_through_the_read_only_path():
    """Kernels that are dependents under set_pdl alone: weights are older than the launch before, rows are not."""
    weights = {"gemm_tc_f8.cu": ["p.S"], "gemm_w8a16.cu": ["reinterpret_cast<const uint32_t*>(B"], "gemv_fp8.cu": ["reinterpret_cast<const uint4*>(B)"],
               "seq_gla.cu": ["wp", "a.w2"], "step.cu": ["gv", "(t ? sj.S1", "gamma", "cs", "sn"]}
    for f in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        for arg in re.findall(r"__ldg\(([^;]*)", strip(f.read_text(encoding="utf-8"))):
            assert any(arg.startswith(w) for w in weights.get(f.name, [])), (f.name, arg)


@pytest.mark.parametrize("where,name,params", [(f.name, n, p) for f in dependents() for n, p, b in kernels(f) if "griddep_wait" in b and "__restrict__" in p],
                         ids=lambda x: x if len(x) < 40 else "")
def test_dependent_kernels_load_through_plain_pointers(where, name, params):
    """__restrict__ lets the compiler move a load ahead of the wait: only pointers that a kernel stores through may have it."""
    body = next(b for n, p, b in kernels(CSRC / where) if n == name and p == params)
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", params)
    for p in re.findall(r"\*\s*__restrict__\s+(\w+)", params):
        uses = re.findall(r"[^;{}]*\b%s\b[^;{}]*" % p, body)
        assert uses
        for use in uses:                                     # `p[...] = x`, `*p = x`, a store helper, or a pointer that is stored through
            assert re.search(r"\b(st|mst<DT>)\(%s\b|\b%s\[.*\]\s*=[^=]|\*%s\s*=[^=]|(?:uint4|uint16_t)\* ?dst\w*\s*=" % (p, p, p), use) or re.fullmatch(r"\s*if \(%s\).*" % p, use), (name, use)


def test_register_shares_of_a_block_fit_its_launch():
    """setmaxnreg.inc waits until the block has the registers that others of its warps gave up: a kernel that asks for shares adds them up,
    fits an SM with them, and refuses to launch where the compiler gave the block fewer."""
    for f in sorted(CSRC.glob("*.cu")):
        text = strip(f.read_text(encoding="utf-8"))
        if "setmaxnreg" not in text:
            continue
        names = {n: int(eval(v, {}, {})) for n, v in re.findall(r"\b(P_\w+) = ([0-9]+)(?=[,;])", text)}
        total = 32 * (names["P_SUMS"] * names["P_SUMS_REGS"] + names["P_CONV"] * names["P_CONV_REGS"] + 4 * names["P_REST_REGS"])
        assert total <= 65536 and total % (32 * (names["P_SUMS"] + names["P_CONV"] + 4)) == 0
        assert re.search(r"numRegs \* P_THREADS < P_REGS\) return cudaErrorInvalidConfiguration", text), f.name
        assert not re.search(r"registers_(?:up|down)<\d", text)
