"""Shared-memory arrays that a kernel reads or writes as 8- or 16-byte vectors.

A vector access faults unless its address is a multiple of the vector's size,
and an array of scalars is placed only at a multiple of its element's size:
every such array has to be declared with the vector's alignment."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fiber3d_b200" / "csrc"
VECTOR = {"double2": 16, "longlong2": 16, "float4": 16, "uint4": 16, "int4": 16, "float2": 8, "uint2": 8, "int2": 8}
SCALAR = {"double": 8, "int64_t": 8, "uint64_t": 8, "float": 4, "unsigned": 4, "int": 4, "int32_t": 4, "uint32_t": 4}
CAST = re.compile(r"reinterpret_cast<\s*(?:const\s+)?(%s)\s*\*\s*>\(\s*&?\s*(?:\w+\.)*(\w+)" % "|".join(VECTOR))
ARRAY = r"(__shared__\s+)?(?:__align__\((\d+)\)\s+)?\b(%s)\s+(?:[\w\[\], ]*,\s*)?%%s\s*\[" % "|".join(SCALAR)


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


@pytest.mark.parametrize("path", sorted(p for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh")),
                         ids=lambda p: p.name)
def test_arrays_read_as_vectors_are_aligned(path):
    code = _code(path)
    structs = [s.group(0) for s in re.finditer(r"struct \w+Shared \{.*?\n\};", code, flags=re.S)]
    bad = []
    for vector, name in set(CAST.findall(code)):
        for m in re.finditer(ARRAY % re.escape(name), code):
            shared, align, scalar = m.groups()
            if not shared and not any(m.group(0) in s for s in structs):
                continue  # a thread's own array
            if max(int(align or 0), SCALAR[scalar]) < VECTOR[vector]:
                bad.append(f"{name}: {scalar} read as {vector}")
    assert not bad


def test_the_scan_finds_what_it_is_for():
    found = {name for p in CSRC.glob("*.cu") for _, name in CAST.findall(_code(p))}
    assert {"s_key", "hi", "cand"} <= found
