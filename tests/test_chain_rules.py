"""Kernels that wait for their predecessor inside (programmatic launches) must not read what it
writes as read-only data: such loads may be moved over the wait. Checked on the sources:
only arrays complete before a chain starts are __restrict__ inputs or arguments of __ldg."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "project1_b200" / "csrc"
COMPLETE = {"M", "prm.kOff", "col"}     # the products (col: one of their columns), plane-wave offsets
OUTPUTS = {"F"}


def _kernels():
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__\s+void\s+(?:__\w+__\([^)]*\)\s*)*(\w+)\s*\(([^{};]*)\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            if "await_previous()" in text[m.end():i]:
                yield m.group(1), m.group(2), text[m.end():i]


def test_chained_kernels_are_found():
    names = {k[0] for k in _kernels()}
    assert {"split_quantize_kernel", "split_quantize_real_kernel", "split_gram_kernel", "split_gram_finish_kernel",
            "zgemm_gather_kernel", "sweep_panels_kernel"} <= names


@pytest.mark.parametrize("kernel", list(_kernels()), ids=lambda k: k[0])
def test_predecessors_data_is_read_with_ordinary_loads(kernel):
    _, params, body = kernel
    for p in re.findall(r"__restrict__\s+(\w+)", params):
        assert p in COMPLETE | OUTPUTS, f"{p} is __restrict__"
    for a in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?([\w.]+)", body):
        assert a in COMPLETE, f"{a} is read through __ldg"
