"""Kernels that may start before their predecessor has finished (wd_pdl_wait)
read data that was not there when they started.  const __restrict__ on an
operand lets the compiler use loads for data that never changes during the
kernel, so neither their parameters nor the structures that carry their
operands may have it."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "ipcc2021-final_gb300" / "csrc"


def body(text, start):
    """The braces' content that opens at or after start."""
    i = text.index("{", start)
    depth, j = 1, i + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
    return text[i:j]


def early_kernels():
    for f in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"__global__\s+void\b", text):
            head = text[m.start():text.index("{", m.start())]
            if ";" in head or "wd_pdl_wait" not in body(text, m.start()):
                continue
            yield f.name, head


def structs():
    out = {}
    for f in CSRC.glob("*.cu*"):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"\bstruct\s+(\w+)[^;{()]*\{", text):
            out[m.group(1)] = body(text, m.start())
    return out


def test_operands_are_not_promised_constant():
    kernels, defs = list(early_kernels()), structs()
    assert len(kernels) >= 12
    for name, head in kernels:
        assert "__restrict__" not in head, (name, head)
        for t in re.findall(r"\bconst\s+(\w+)\s+\w+", head):
            assert "__restrict__" not in defs.get(t, ""), (name, t)


def test_no_loads_for_constant_data():
    """Nor are they read with __ldg, which is the same promise; the one file
    that does holds kernels that are launched in the ordinary way only."""
    for f in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        if "__ldg(" in text or "ld.global.nc" in text:
            assert f.name == "wd_h16_tma.cuh" and "wd_pdl_wait" not in text and "wd_launch" not in text, f.name
