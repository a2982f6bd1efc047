"""Kernels that start while their predecessor drains (launch_pdl): what the sources must keep to, checked on the text.

Such a kernel's lifetime begins while its predecessor may still be writing.  So every one of them waits first, and
reads what the stream produced through ordinary loads: the read-only path (__ldg, ld.global.nc) presumes data that
does not change during the kernel, and accesses through __restrict__ pointers may be moved across the wait."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fsd_b200" / "csrc"
SOURCES = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu*"))}
# parameters that are written once, or by launches that do not overlap: tables, and the matrix A and its list
TABLES = {"tw_global", "table", "gridk", "pn", "plist", "A"}
# outputs that the kernel only writes, each value computed from data read after the wait
OUTPUTS = {"k_inner_g": {"z"}}


def functions(text):
    """(kernel?, name, signature, body) of the functions of a file."""
    head = r"(__global__|__device__ __forceinline__|__host__ __device__)((?:[^;{}()]|\((?:[^()]|\([^()]*\))*\))*)\{"
    for m in re.finditer(head, text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        sig = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", m.group(2))
        name = re.search(r"(\w+(?:\(\))?)\s*\(", sig)
        yield m.group(1) == "__global__", name.group(1) if name else "", sig, text[m.end():i - 1]


ALL = {(f, n): (k, s, b) for f, t in SOURCES.items() for k, n, s, b in functions(t)}
OVERLAPPED = {k: v for k, v in ALL.items() if v[0] and "pdl_wait()" in v[2]}
LAUNCHED = {k for t in SOURCES.values() for m in re.findall(r"launch_pdl\(([^,]*)", t) for k in re.findall(r"\bk_\w+", m)}


def test_every_overlapped_launch_is_of_a_kernel_that_waits_first():
    assert len(LAUNCHED) > 40
    assert LAUNCHED == {n for _, n in OVERLAPPED}
    for (f, n), (_, _, body) in OVERLAPPED.items():
        assert re.match(r"\s*pdl_wait\(\);", body), f"{f}: {n}"


@pytest.mark.parametrize("key", sorted(OVERLAPPED), ids=lambda k: k[1])
def test_overlapped_kernels_read_the_stream_by_ordinary_loads(key):
    _, sig, body = OVERLAPPED[key]
    assert set(re.findall(r"__restrict__\s+(\w+)", sig)) <= TABLES | OUTPUTS.get(key[1], set())
    # its own text and that of the helpers it calls, to any depth
    seen, todo = {}, {key[1]: body}
    while todo:
        name, text = todo.popitem()
        seen[name] = text
        for (f, n), (kernel, s, b) in ALL.items():
            if not kernel and n not in seen and re.search(rf"\b{n}\b\s*[<(]", text):
                if n not in ("load8_const", "lub_interp"):  # tables
                    assert "__restrict__" not in re.sub(r"__restrict__ (" + "|".join(TABLES) + r")\b", "", s), n
                    todo[n] = b
    for name, text in seen.items():
        assert "__ldg" not in text and "ld.global.nc" not in text, name


def test_read_only_loads_are_of_tables_or_in_ordinary_kernels():
    found = set()
    for f, t in SOURCES.items():
        for kernel, n, _, body in functions(t):
            if "__ldg" in body or "ld.global.nc" in body:
                assert n in ("res_interp", "lub_interp", "load8_const") or (kernel and (f, n) not in OVERLAPPED), (f, n)
                found.add(n)
    assert {"lub_interp", "load8_const"} <= found
