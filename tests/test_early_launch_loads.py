"""Kernels that are put in place before the kernel ahead has ended read global
memory by coherent loads that stay behind their wait (ld_ca, ld_cg, ld_cs).

A non-coherent load (__ldg, or a plain read through a `const __restrict__`
pointer) takes its data as unchanging while the kernel is resident, and neither
it nor the plain cache-operator intrinsics are ordered behind the wait; such a
read could return what was there before the kernel ahead stored its results,
and these are indices and counts.  No run shows this reliably, so the sources
are read instead."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "kascade_b200" / "csrc"
FORBIDDEN = re.compile(r"__ldg\b|__ldc[agsv]\b|__ldlu\b|\bld_out_nc_keep\b|ld\.global\.nc")


def _source(path: Path) -> str:
    s = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", s)


def _body(s: str, at: int) -> int:
    """The end of the brace block that opens at or after `at`."""
    i = s.index("{", at)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(s[i], 0)
        i += 1
        if depth == 0:
            return i


def _kernels():
    """(file, name, parameters, body) of every kernel, and each file's rest."""
    out, rest = [], {}
    for path in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
        s, keep, pos = _source(path), [], 0
        for m in re.finditer(r"__global__\b.*?\b(k_\w+)\s*\(", s, flags=re.S):
            if m.start() < pos:
                continue
            end, depth, i = _body(s, m.end()), 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(s[i], 0)
                i += 1
            out.append((path.name, m.group(1), s[m.end():i - 1], s[i:end]))
            keep.append(s[pos:m.start()])
            pos = end
        rest[path.name] = "".join(keep) + s[pos:]
    return out, rest


KERNELS, REST = _kernels()
EARLY = [k for k in KERNELS if "kernel_begin()" in k[3]]


def test_early_kernels_are_found():
    assert len(EARLY) >= 14 and len(KERNELS) > len(EARLY)


def test_every_kernel_started_early_waits_first():
    early = {k[1] for k in EARLY}
    for name, text in REST.items():
        for m in re.finditer(r"\blaunch\(\s*ctx,\s*(k_\w+)", text):
            assert m.group(1) in early, f"{name}: {m.group(1)} is started early but does not wait"
    for file, name, _, body in EARLY:
        assert body.lstrip("{ \n").startswith("kernel_begin();"), f"{file}: {name} does not wait first"


@pytest.mark.parametrize("kernel", EARLY, ids=lambda k: f"{k[0]}:{k[1]}")
def test_early_kernel_loads(kernel):
    file, name, params, body = kernel
    assert not FORBIDDEN.search(body), f"{file}: {name}: {FORBIDDEN.search(body).group(0)}"
    assert not re.search(r"\bconst\b[^,]*\*\s*__restrict__", params), f"{file}: {name}: const __restrict__ input"


@pytest.mark.parametrize("file", ["common.cuh", "ranker.cuh", "ranker.cu", "tree.cu", "batch.cu", "tma.cuh"])
def test_device_functions_they_share(file):
    text = REST[file]
    if file == "common.cuh":  # the one non-coherent load, for kernels started plainly
        m = re.search(r"\bOut ld_out_nc_keep\(", text)
        text = text[:m.start()] + text[_body(text, m.end()):]
    assert not FORBIDDEN.search(text), f"{file}: {FORBIDDEN.search(text).group(0)}"
    assert not re.search(r"\bconst\b[^,;{]*\*\s*__restrict__", text), f"{file}: const __restrict__"
