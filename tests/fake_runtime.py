"""The library's host code on a CUDA runtime without a device
(tests/cpp/fake_cudart.cpp): its own objects, linked with that instead."""
from __future__ import annotations

import ctypes
import importlib.util
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
DEVICE = 1 << 41  # an address for what the caller holds on the device


class Segment(ctypes.Structure):
    _fields_ = [("offset", ctypes.c_uint64), ("size", ctypes.c_uint64), ("kind", ctypes.c_uint32),
                ("reserved", ctypes.c_uint32)]


class Opts(ctypes.Structure):
    _fields_ = [(n, ctypes.c_uint32) for n in (
        "struct_size", "algorithm", "ruler_spacing", "ruler_spacing_deep", "max_levels", "base_case_size",
        "chains_per_thread", "block_size", "validate", "async_", "profile", "seed", "level0_mode", "max_chain")]


def load(tmp: Path) -> ctypes.CDLL:
    spec = importlib.util.spec_from_file_location("kascade_b200_build", ROOT / "kascade_b200" / "build.py")
    kbuild = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(kbuild)
    kbuild.build()
    objects = [kbuild.BUILD / (s.stem + ".o") for s in sorted(kbuild.CSRC.glob("*.cu"))]
    out = tmp / "libkascade_fake.so"
    cuda = Path(kbuild.nvcc()).resolve().parents[1]
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-Wl,--no-undefined",
                    f"-I{cuda}/include", str(ROOT / "tests" / "cpp" / "fake_cudart.cpp"), *map(str, objects), "-o",
                    str(out), "-lpthread"], check=True)
    lib = ctypes.CDLL(str(out))
    lib.fake_launches.restype = ctypes.c_char_p
    lib.fake_stream.restype = ctypes.c_void_p
    for f in ("fake_used", "fake_peak"):
        getattr(lib, f).restype = ctypes.c_size_t
    lib.fake_reset.argtypes = [ctypes.c_size_t]
    lib.fake_priority.argtypes = [ctypes.c_size_t]
    return lib


def opts(lib, **kw) -> Opts:
    o = Opts()
    lib.kascade_opts_init(ctypes.byref(o))
    assert o.struct_size == ctypes.sizeof(o)
    for k, v in kw.items():
        setattr(o, k, v)
    return o


def segments(sizes, kinds):
    segs, at = (Segment * len(sizes))(), 0
    for i, (n, k) in enumerate(zip(sizes, kinds)):
        segs[i] = Segment(at, n, k, 0)
        at += n
    return segs, at


def launches(lib):
    """(kernel's mangled name, stream) of what was launched since fake_reset."""
    rows = lib.fake_launches().decode().splitlines()
    return [(r.rsplit(" ", 1)[0], int(r.rsplit(" ", 1)[1])) for r in rows]
