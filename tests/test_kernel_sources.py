"""Orderings that a wrong result would show too rarely to be tested by results,
checked in the kernels' sources, on the CPU."""
from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "fdtd_gb300" / "csrc"


def _kernels():
    """(file, name, parameters, body) of every __global__ function."""
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__\s+void\s+", text):
            at = m.end()
            bounds = re.match(r"__launch_bounds__\s*\(", text[at:])
            if bounds:
                at = _close(text, at + bounds.end() - 1, "()")
            name = re.match(r"\s*(\w+)\s*\(", text[at:])
            p0 = at + name.end() - 1
            p1 = _close(text, p0, "()")
            b0 = text.index("{", p1)
            yield path.name, name.group(1), text[p0 + 1:p1 - 1], text[b0:_close(text, b0, "{}")]


def _close(text, at, pair):
    depth = 0
    for k in range(at, len(text)):
        depth += (text[k] == pair[0]) - (text[k] == pair[1])
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced source")


def test_tensor_maps_in_global_memory_are_acquired_before_use():
    """A batch's tensor maps are rewritten in place by host copies whenever a
    solve joins or leaves; a block that uses them must acquire them through the
    tensor-map proxy first, with a barrier between."""
    seen = 0
    for file, name, params, body in _kernels():
        if "BatchDesc" not in params or not re.search(r"\bd\.s?maps\[", body):
            continue
        seen += 1
        acquire = body.find("acquire_tensor_maps<")
        use = re.search(r"(strip|fused)_unit<", body).start()
        assert 0 <= acquire < use, (file, name)
        assert "__syncthreads();" in body[acquire:use], (file, name)
    assert seen == 2


def test_kernels_launched_early_take_no_read_only_pointers():
    """A programmatic dependent begins while the grid before it still writes:
    const __restrict__ promises the compiler data constant from the kernel's first
    instruction on, ahead of griddepcontrol.wait."""
    seen = 0
    for file, name, params, body in _kernels():
        if "pdl_begin();" not in body and "griddepcontrol.wait" not in body:
            continue
        seen += 1
        assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", params + body), (file, name)
    assert seen >= 8


def test_records_of_the_batched_kernels_have_no_fields_shorter_than_a_word():
    """16-bit fields of a work unit's record were read wrong by compiled code."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "native.cuh").read_text())
    for name in ("BatchUnit", "BatchMurBlock"):
        body = re.search(rf"struct[^;{{]*\b{name}\s*{{([^}}]*)}}", text).group(1)
        fields = [f.strip() for f in body.split(";") if f.strip()]
        assert fields, name
        for f in fields:
            assert not re.search(r"\b(short|char|u?int8_t|u?int16_t|bool)\b", f), (name, f)
