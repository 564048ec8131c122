"""Rules that the chained kernels (started while the launch before them drains)
keep, read off their sources: a missing wait or a load through the read-only path
changes no result that a test on one GPU would be sure to see."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fdtd_accelerate_gb300", "csrc")


def source(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def block(text, at):
    """The brace block that opens at or after position at."""
    a = text.index("{", at)
    depth = 0
    for i in range(a, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[a:i + 1]
    raise ValueError("unbalanced braces")


def kernels():
    """name -> body of every kernel definition."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = source(path)
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            out[m.group(1)] = block(text, m.end())
    return out


KERNELS = kernels()
CHAINED = sorted(k for k, body in KERNELS.items() if "grid_wait" in body or "grid_release" in body)


def test_chained_kernels_are_found():
    assert CHAINED == ["k_edge_e", "k_edge_h", "k_symp_pair", "k_yee_fused"]


@pytest.mark.parametrize("name", CHAINED)
def test_every_thread_waits(name):
    """grid_wait() under no condition but the kernel's template arguments."""
    body = KERNELS[name]
    waits = [m.start() for m in re.finditer(r"\bgrid_wait\(\)", body)]
    assert waits
    for at in waits:
        start = max(body.rfind(c, 0, at) for c in ";{}")
        assert not body[start + 1:at].strip(), "conditional: " + body[start + 1:at]
        depth, heads = 0, []
        for i in range(at - 1, 0, -1):
            if body[i] == "}":
                depth += 1
            elif body[i] == "{":
                if depth == 0:
                    heads.append(body[max(body.rfind(c, 0, i) for c in ";{}") + 1:i].strip())
                else:
                    depth -= 1
        assert set(heads) <= {"if (!BATCH)", "else"}, heads
    assert not re.search(r"\breturn;", body[:waits[0]])


@pytest.mark.parametrize("name", ["symp_pair.cu", "symp_group.cuh", "yee_fused.cuh", "yee_fused.cu"])
def test_read_only_loads_of_tables_alone(name):
    """The launch before a chained kernel may write its fields and psi while the kernel
    is resident: only the CPML tables (and a wave's 1-D arrays) go through __ldg."""
    text = source(os.path.join(CSRC, name))
    assert not re.search(r"#define[^\n]*__ldg|ld\.global\.nc", text)
    text = text.replace("return RO ? __ldg(p) : *p;", "")  # the edge kernels' loads, below
    for arg in re.findall(r"__ldg\(([^;]*)", text):
        assert re.match(r"T\.(b|a|km1) \+ s", arg) or (name == "yee_fused.cuh" and arg.startswith("f1d + at")), arg


def test_edge_kernels_of_chained_launches():
    """The edge kernels' read-only forms are launched the plain way."""
    text = source(os.path.join(CSRC, "symp_pair.cu"))
    forms = re.findall(r"launch\((\w+), ([^;]*k_edge_[he][^;]*);", text)
    assert len(forms) == 5
    for chained, kernel in forms:
        names = set(re.findall(r"k_edge_h<\w+, (\w+)>", kernel) + re.findall(r"k_edge_e<(\w+)>", kernel))
        assert names and names <= {"true": {"PLAIN", "SPLIT_COMP"}, "false": {"READ_ONLY"}}[chained], kernel
    assert re.search(r"RO = FORM == READ_ONLY,", text)


def test_one_dimensional_arrays_of_a_wave():
    """The fused kernel reads them through __ldg: the kernels that write them start
    nothing before their own end, and the offset is known after the wait only."""
    writers = [k for k, body in KERNELS.items() if "1d" in k or "1D" in body or "e1d[" in body or "h1d[" in body]
    assert writers and not set(writers) & set(CHAINED)
    text = source(os.path.join(CSRC, "yee_fused.cuh"))
    assert re.search(r"const int at = \(ix >= 0 \? ix : ax \+ p\.tvo\) \+ zero,", text)
    assert re.search(r"grid_wait\(\);\s*if \(TFSF\) asm volatile\(\"\" : \"\+r\"\(zero\) : : \"memory\"\);", text)


@pytest.mark.parametrize("name", ["k_adj_e4", "k_adj_h4"])
def test_written_arrays_are_not_read_as_read_only(name):
    """No array that the adjoint cell kernels store to is loaded through ld4 / ldp /
    __ldg in the same kernel."""
    body = KERNELS[name]
    stored = set(re.findall(r"\bst4\(([\w.\[\]]+)", body))
    assert len(stored) >= 3
    assert not stored & set(re.findall(r"\b(?:ld4|ldp|__ldg)\(([\w.\[\]]+)", body))
