"""Rules of the programmatic dependent launches, checked on the kernel sources.

A kernel launched with launch_after() is live while the kernel before it still
writes; only after_previous() orders the two.  So it has to call
after_previous(), and it may read nothing that another kernel writes through
__ldg or a __restrict__ pointer: both promise that the data is constant for
the kernel's lifetime, and a load so marked may be moved above the wait.  The
GELU tables are constant: written once per process, with a host wait.
"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "heterogeneous_mhd_gb300" / "csrc"
CONSTANT = {"gelu_tab", "grad_tab"}
SHARED = {"su", "sb"}  # tiles in shared memory


def strip_comments(text):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def block(text, start):
    """The balanced {...} that begins at or after `start`."""
    i = text.index("{", start)
    depth = 0
    for k in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[i:k + 1]
    raise AssertionError("unbalanced braces")


def functions(text):
    """(kernel name or None, signature, body) of every __global__ and __device__ function."""
    for m in re.finditer(r"__(global|device)__", text):
        brace = text.find("{", m.end())
        semi = text.find(";", m.end())
        if brace < 0 or (0 <= semi < brace):
            continue
        sig = text[m.end():brace]
        name = re.search(r"\b(k_\w+)\s*\(", sig)
        yield (name.group(1) if m.group(1) == "global" and name else None), sig, block(text, brace)


def sources():
    return {p.name: strip_comments(p.read_text()) for p in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))}


def test_dependent_kernels_wait_for_the_kernel_before():
    src = sources()
    waits = {name: "after_previous()" in body
             for text in src.values() for name, _, body in functions(text) if name}
    launched = set()
    for text in src.values():
        for m in re.finditer(r"launch_after\(([^,]+),", text):
            launched |= set(re.findall(r"\bk_\w+", m.group(1)))
    assert len(launched) >= 30
    assert sorted(k for k in launched if not waits[k]) == []


def test_dependent_kernels_read_through_plain_loads():
    bad = []
    for fname, text in sources().items():
        for m in re.finditer(r"__ldg\(\s*(\w+)", text):
            if m.group(1) not in CONSTANT:
                bad.append((fname, m.group(0)))
        for name, sig, body in functions(text):
            if name and "after_previous()" not in body:
                continue  # launched when the work before it has ended
            for p in re.findall(r"__restrict__\s+(\w+)", sig):
                if p not in CONSTANT | SHARED:
                    bad.append((fname, name or sig.split("(")[0].split()[-1], p))
    assert bad == []
