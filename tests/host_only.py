"""The library's host code on a CUDA runtime without a GPU (tests/cpp/host_only.cu
and host_runtime.cpp): kernels do not run, launches are written down."""
import ctypes as C
import os
import shutil
import subprocess

from opensayal_gb300 import native
from opensayal_gb300.fluid import default_config
from tests.conftest import ROOT

CPP = ROOT / "tests" / "cpp"
LIB = ROOT / "oracle" / "build" / "libhost_only.so"
SOURCES = [CPP / "host_only.cu", CPP / "host_runtime.cpp"]

OTHER, PROJECT, DIFFUSE, BATCH_PROJECT, BATCH_DIFFUSE = range(5)


class HostLaunch(C.Structure):
    _fields_ = [(k, C.c_int32) for k in ("kind", "tiles", "cluster", "cooperative", "pdl",
                                         "n", "K", "D", "R", "warps", "halo", "tiles_y")]
    _fields_ += [("smem", C.c_uint64), ("limit", C.c_uint64)]
    _fields_ += [(k, C.c_void_p) for k in ("fn", "ui", "vi", "uo", "vo", "err")]


class HostState(C.Structure):
    _fields_ = [("fail_malloc_from", C.c_int64), ("fail_attribute", C.c_int32),
                ("limits_lowered", C.c_int32)]


def build():
    csrc = ROOT / "opensayal_gb300" / "csrc"
    deps = [*SOURCES, CPP / "host_only.h", *csrc.glob("*.cu*"), *(ROOT / "include").rglob("*.h*")]
    if LIB.exists() and all(d.stat().st_mtime <= LIB.stat().st_mtime for d in deps):
        return LIB
    LIB.parent.mkdir(parents=True, exist_ok=True)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    objects = [LIB.with_suffix(f".{k}.o") for k in range(2)]
    # The device code is not used: PTX, without the assembler's time.
    cmds = [[f"{cuda}/bin/nvcc", "-std=c++17", "-O1", "--use_fast_math", "-gencode",
             "arch=compute_103a,code=compute_103a", "-Xcompiler", "-fPIC,-fno-gnu-unique",
             "-diag-suppress", "177", "-c", "-o", str(objects[0]), str(SOURCES[0])],
            ["g++", "-std=c++17", "-O1", "-fPIC", f"-I{cuda}/include", "-c", "-o",
             str(objects[1]), str(SOURCES[1])],
            # The runtime calls bind to the ones here, whatever the process has loaded
            # (and what inline functions keep is this library's own: no unique symbols).
            ["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", str(LIB),
             *map(str, objects), "-lpthread"]]
    for cmd in cmds:
        subprocess.run(cmd, check=True, capture_output=True, text=True)
    return LIB


def load(copy_to=None):
    """The library; a copy in a folder has a state of its own."""
    path = build()
    if copy_to is not None:
        path = shutil.copy(path, copy_to)
    lib = C.CDLL(str(path))
    for name, res, args in native.SIGNATURES:
        fn = getattr(lib, name)
        fn.argtypes, fn.restype = args, res
    lib.host_launches.argtypes = [C.POINTER(HostLaunch), C.c_int32]
    lib.state = HostState.in_dll(lib, "host_state")
    return lib


def launches(lib, *kinds):
    """The launches since the last call, of the given kinds only."""
    buf = (HostLaunch * 4096)()
    n = lib.host_launches(buf, len(buf))
    return [x for x in buf[:n] if not kinds or x.kind in kinds]


def segments(lib, x, storage):
    """The segments of sweeps of tile launch x: (sweeps, messages, round, exchange)."""
    out = []
    while True:
        more = [C.c_int32() for _ in range(3)]
        sweeps = lib.host_segment(x.kind == PROJECT, x.n, x.K, x.D, storage, len(out),
                                  *map(C.byref, more))
        if not sweeps:
            return out
        out.append((sweeps, *(m.value for m in more)))


class Handle:
    """A tunnel of the host-only library."""

    def __init__(self, lib, cfg):
        self.lib, self.h = lib, C.c_void_p()
        self.rc = lib.os_create(C.byref(cfg), C.byref(self.h))
        self.error = lib.os_last_error().decode() if self.rc else ""
        launches(lib)

    def fields(self):
        view = native.OsFieldsView()
        assert self.lib.os_fields(self.h, C.byref(view)) == native.OS_OK
        return view

    def update(self):
        return self.lib.os_update(self.h, None, 0.05)

    def close(self):
        self.lib.os_destroy(self.h)

    def __enter__(self):
        assert self.rc == native.OS_OK, self.error
        return self

    def __exit__(self, *exc):
        self.close()


def tunnel(w, h, **over):
    c = default_config(w, h)
    c.tunnel_speed, c.viscosity = 2.0, 0.02
    for k, v in over.items():
        setattr(c, k, v)
    return c
