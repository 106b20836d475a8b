"""Shared arrays that a kernel reads in wider words than it declares them in say
their alignment: a declared uint32_t array is aligned to 4 bytes only, and an
8- or 16-byte access to it is legal by the luck of the layout."""
from __future__ import annotations

import os
import re

from conftest import PKG

CSRC = os.path.join(PKG, "csrc")
BYTES = {"uint8_t": 1, "uint16_t": 2, "uint32_t": 4, "unsigned": 4, "int": 4, "float": 4}
WIDE = {"uint2", "int2", "float2", "uint64_t", "double", "ulonglong2", "uint4", "int4", "float4", "longlong"}


def unaligned_views(text: str) -> list[str]:
    """Wider views of shared arrays that are declared in narrow words without an alignment."""
    shared = set()
    for m in re.finditer(r"__shared__\s+((?:__align__\(\d+\)|alignas\(\d+\))\s+)?(\w+)\s+([^;]*);", text):
        if not m.group(1) and m.group(2) in BYTES:
            shared |= set(re.findall(r"(\w+)\s*\[", m.group(3)))
    # Pointers set from such an array point into it too.
    while True:
        more = {m.group(1) for m in re.finditer(r"\*\s*(\w+)\s*=\s*([^;]*);", text)
                if "reinterpret_cast" not in m.group(2) and shared & set(re.findall(r"\w+", m.group(2)))}
        if more <= shared:
            break
        shared |= more
    return [m.group(0) for m in re.finditer(r"reinterpret_cast<(?:const )?(\w+)\*>\(\s*&?(\w+)", text)
            if m.group(1) in WIDE and m.group(2) in shared]


def test_the_check_finds_a_view_through_a_pointer():
    text = "__shared__ uint32_t a[4]; uint32_t* b = x ? a : nullptr; auto c = reinterpret_cast<uint2*>(b);"
    assert unaligned_views(text) == ["reinterpret_cast<uint2*>(b"]
    assert unaligned_views(text.replace("__shared__", "__shared__ __align__(16)")) == []


def test_wider_views_of_shared_arrays_are_aligned():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                for kernel in f.read().split("__global__"):
                    assert unaligned_views(kernel) == [], name
