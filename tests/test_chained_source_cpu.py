"""Rules of memory order, checked on the sources. Chained launches: a kernel that may be resident while the kernels before
it still write its item tables, row maxima and planes calls chain_wait() and promises nothing constant about that data
(no __restrict__; __ldg only on the caller's operands, which are constant from a call's first launch on). The GEMM's job ring: a
warp whose lane 0 waited on an mbarrier touches the ring after __syncwarp(), as a shuffle orders no memory. Inline assembly: what
reads or writes memory, or waits for it, is volatile and clobbers memory (a load without them is a function of its address
to the compiler, which may keep its value over a refill)."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "os2-xe_b200", "csrc")
FILES = {f: open(os.path.join(SRC, f)).read() for f in os.listdir(SRC) if f.endswith((".cu", ".cuh"))}
CHAINED = sorted({(f, k) for f, text in FILES.items() for k in re.findall(r"launch_chained\((\w+)\s*<", text)})
# functions of the chained kernels that read their items
HELPERS = [("oz2_split.cu", h) for h in ("find_item", "split_consts", "SplitFetch", "edge", "split_tiles")] + [("oz2_gemm.cu", "decode")]
OPERANDS = {"scale_kernel": {"X", "row"}}  # pointers into op(A), op(B) read through __ldg


def body(text, name):
    """the definition of `name`, from its parameter list to its closing brace"""
    for m in re.finditer(r"\b%s\(" % name, text):
        depth, i = 0, m.end() - 1
        while True:  # past the parameter list
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        if not re.match(r"\s*\{", text[i:]):
            continue  # a call or a declaration
        while True:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
            if depth == 0 and text[i - 1] == "}":
                return text[m.start():i]
    raise AssertionError(name)


def test_the_chained_kernels_are_found():
    assert {k for _, k in CHAINED} == {"scale_kernel", "split_kernel", "gemm_i8_modm_kernel", "crt_kernel"}


@pytest.mark.parametrize("where,name", CHAINED + HELPERS)
def test_no_constant_promise(where, name):
    text = body(FILES[where], name)
    if (where, name) in CHAINED:
        assert "dev::chain_wait();" in text
    assert "__restrict__" not in text
    for arg in re.findall(r"__ldg\((\w+)", text):
        assert arg in OPERANDS.get(name, ()), arg


def test_job_ring_is_ordered():
    text = body(FILES["oz2_gemm.cu"], "gemm_i8_modm_kernel")
    waits = [m.end() for m in re.finditer(r"mbar_wait\(jobs_(?:full|empty)\(", text)]
    assert len(waits) == 2
    for at in waits:
        use = text.index("job_ring[", at)
        assert "__syncwarp();" in text[at:use]


def asm_statements(text):
    for m in re.finditer(r"\basm\s*(volatile)?\s*\(", text):
        depth, i, quoted = 1, m.end(), False
        while depth:
            c = text[i]
            if c == '"':
                quoted = not quoted
            elif not quoted:
                depth += {"(": 1, ")": -1}.get(c, 0)
            i += 1
        yield m.group(1), text[m.end():i]


@pytest.mark.parametrize("where", sorted(FILES))
def test_assembly_that_touches_memory(where):
    for volatile, stmt in asm_statements(FILES[where]):
        code = " ".join(re.findall(r'"((?:[^"\\]|\\.)*)"', stmt.split('"=')[0]))
        if re.search(r"\b(ld|st|atom|red|cp)\.|mbarrier|tcgen05|fence|griddepcontrol", code):
            assert volatile and '"memory"' in stmt, code
