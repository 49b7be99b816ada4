"""Kernels launched under programmatic dependent launch, by their sources:
before grid_dependency_wait() a kernel may read only its constant tables and
write only shared memory, because what its predecessor writes (and where its
own stores land among the predecessor's) is ordered by that wait alone."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gtom_b200" / "csrc"


def _body(text, at):
    """The text between the braces that open at or after `at`."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i]
    raise AssertionError("unbalanced braces")


def _waiting_kernels():
    out = []
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", text):
            head = re.search(r"(\w+)\(\s*(?:const |float|double|int|uint|BrickGrid|ArrayFetch|GridFinalArgs|SegBin|TcArgs)", text[m.start():])
            body = _body(text, m.start() + head.start())
            if "grid_dependency_wait()" in body:
                out.append((path.name, head.group(1), body))
    return out


def test_the_waiting_kernels_are_found():
    names = {k for _, k, _ in _waiting_kernels()}
    assert {"gridgen_final_z_kernel", "gridsym_final_z_kernel", "gridgen_z_kernel", "backproject_segment_kernel",
            "diff2_tc_kernel", "segment_fill_kernel"} <= names


@pytest.mark.parametrize("file,kernel,body", _waiting_kernels(), ids=lambda v: v if len(str(v)) < 60 else "")
def test_nothing_but_tables_before_the_wait(file, kernel, body):
    before = body[:body.index("grid_dependency_wait()")]
    # stores through anything but the kernel's shared arrays
    for m in re.finditer(r"([\w.]+)\[[^;=]*\]\s*[-+*]?=[^=]", before):
        assert m.group(1) in ("tw", "sv", "sw"), f"{file}: {kernel} stores to {m.group(1)} before its wait"
    # reads of the caller's data through the final map's columns or by __ldg
    assert ".value(" not in before and ".zero(" not in before and "GridColumn" not in before, f"{file}: {kernel}"
    assert "__ldg" not in before, f"{file}: {kernel}"
