"""Kernels launched before their predecessor ends: a const __restrict__ parameter tells the compiler
that nothing writes its memory, so loads through it may move above the wait.  Every such parameter that
other kernels write is therefore made known only by the wait (pdl_wait_for, pdl_entry_for); the
topology's (lists, items, chunks, codes), written when a grid is created, need not be.  (What a kernel
stores depends on what it has loaded, so its outputs cannot move; they are not read through.)"""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cirrus_b200" / "csrc"
MUTABLE = re.compile(r"^const (?:float|double|T|float2|Scalars|InstParams|uint8_t) ?\* ?__restrict__ (\w+)$")
# (the attribute's own parentheses, then the name)
KERNEL = re.compile(r"(?:__global__ void(?: __launch_bounds__\([^()]*(?:\([^()]*\)[^()]*)*\))?|__device__ __forceinline__ void) (k_\w+)\(")


def kernels(text):
    """(name, parameters, body) of the k_ functions."""
    for m in KERNEL.finditer(text):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        j = text.index("{", i)
        yield m.group(1), [" ".join(p.split()) for p in text[m.end():i - 1].split(",")], text[j:text.index("\n}\n", j)]


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_written_pointers_are_known_after_the_wait(path):
    for name, params, body in kernels(path.read_text()):
        if "pdl_" not in body:
            continue  # launched in plain stream order, or passes its parameters on
        mutable = {MUTABLE.match(p).group(1) for p in params if MUTABLE.match(p)}
        assert not mutable or "pdl_entry();" not in body, name
        assert not mutable or not re.search(r"pdl_wait\(\);(?!\s*return;)", body), name
        for names in re.findall(r"pdl_(?:wait|entry)_for\(([^)]*)\);", body):
            assert mutable <= {n.strip() for n in names.split(",")}, (name, names)


def test_kernels_are_found():
    """The scan above sees the library's kernels."""
    names = {n for p in CSRC.glob("*.cu") for n, _, body in kernels(p.read_text()) if "pdl_" in body}
    assert {"k_laplacian_fused_body", "k_bottom", "k_inst_reduce", "k_amg_sweep", "k_divergence", "k_presmooth_wide"} <= names
