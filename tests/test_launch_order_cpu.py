"""Kernels whose grid may be set up while the kernel before them still writes
(they begin with after_previous()) read by ordinary loads: no __ldg, no
parameter that lets the compiler take the read-only path, in them or in the
helpers that read earlier kernels' arrays for them."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "nexusbvh_gb300" / "csrc"
HELPERS = ["load_box", "load_child_pair", "delta", "mesh_of", "load_tile", "climb_tile", "climb_between",
           "merge_between", "load_entry", "local_sort"]


def block(text, at):
    """The brace-matched block that starts at or after `at`."""
    i = text.index("{", at)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError("unbalanced braces")


def kernels():
    """(name, signature, body) of the kernels that begin with after_previous()."""
    out = []
    for f in sorted(CSRC.glob("*.cu")):
        text = f.read_text()
        for m in re.finditer(r"__global__[^;{]*?\bvoid\s+(\w+)\s*\(", text):
            start = text.index("{", m.end())
            body = block(text, m.end())
            if "after_previous();" in body:
                out.append((m.group(1), text[m.start():start], body))
    return out


def test_they_are_found():
    names = {k[0] for k in kernels()}
    assert {"scene_bounds_kernel", "morton_kernel", "sort_cluster_kernel", "hploc_kernel", "bvh8_lists_kernel",
            "bvh8_group_kernel", "finalize_kernel"} <= names


def test_the_wait_comes_first():
    for name, _, body in kernels():
        assert body[1:].lstrip().startswith("after_previous();"), name


@pytest.mark.parametrize("name,signature,body", kernels(), ids=lambda v: v if re.fullmatch(r"\w+", v) else "")
def test_kernels(name, signature, body):
    assert "__restrict__" not in signature
    reads = re.findall(r"(?:__ldg|__ldcs)\(([^)]*)", body)
    assert [r for r in reads if not r.startswith("seg.")] == []  # a batch's offsets: no kernel of the build writes them


@pytest.mark.parametrize("name", HELPERS)
def test_helpers(name):
    found = 0
    for f in sorted(CSRC.glob("*.cu*")):
        text = f.read_text()
        for m in re.finditer(r"__device__[^;{}]*?\b%s\([^;{]*\{" % name, text):
            found += 1
            assert "__restrict__" not in m.group(0), f.name
            assert "__ldg" not in block(text, m.end() - 1), f.name
    assert found


def test_launches_with_attributes_leave_no_error_behind():
    """cudaLaunchKernelEx returns its error and also keeps it for the next
    cudaGetLastError, which would fail the launch after it."""
    for f in sorted(CSRC.iterdir()):
        text = f.read_text()
        for m in re.finditer(r"cudaLaunchKernelEx\(", text):
            assert f.name == "pipeline.h" and "cudaGetLastError();" in text[m.start():m.start() + 120], f.name
