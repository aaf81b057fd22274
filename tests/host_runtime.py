"""The library's objects linked with a CUDA runtime that needs no GPU
(host_runtime.cpp): what the launchers and the C interface do on the host."""
import ctypes
import functools
import glob
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
PKG = os.path.join(ROOT, "weighted_bte_b200")


@functools.lru_cache(maxsize=None)
def library():
    from weighted_bte_b200 import build

    build.build(verbose=False)
    objects = glob.glob(os.path.join(PKG, "_build", "-".join(build.DEFAULT_DEFINES), "*.o"))
    assert len(objects) == len(build.SOURCES)
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    lib = os.path.join(tempfile.mkdtemp(), "libhost.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", include, "-I", build.CSRC,
                    "-o", lib, os.path.join(HERE, "host_runtime.cpp")] + objects, check=True)
    h = ctypes.CDLL(lib)
    for name in ("fake_live", "fake_peak", "fake_allocations"):
        getattr(h, name).restype = ctypes.c_uint64
    h.fake_log.restype = ctypes.c_char_p
    h.fake_buffer.restype = ctypes.c_void_p
    return h


def log(h):
    """[(kernel, blocks, threads)] launched and [(address, bytes)] copied on the device."""
    launches, copies = [], []
    for line in h.fake_log().decode().splitlines():
        what, a, *rest = line.split()
        if what == "launch":
            launches.append((a, int(rest[0]), int(rest[1])))
        else:
            copies.append((int(a), int(rest[0])))
    return launches, copies


def i64(*values):
    return [ctypes.c_int64(v) for v in values]
