"""The engine's library on a stand-in CUDA runtime (fake_cudart.cpp): its host code -- what it
allocates, captures and launches -- runs without a GPU.  Kernels and copies do nothing."""
import ctypes
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def load(tmp):
    """The library linked with the stand-in, with the engine's prototypes."""
    from das_gb300 import _lib, build
    build.build()
    objs = [os.path.join(build.BUILD, os.path.basename(s) + ".o") for s in build._sources()]
    if not all(os.path.exists(o) for o in objs):
        build.build(force=True)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))),
                        "include")
    out = os.path.join(str(tmp), "libwave2d_fake.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + cuda,
                    os.path.join(HERE, "fake_cudart.cpp"), *objs, "-Wl,-Bsymbolic", "-o", out],
                   check=True)
    lib = ctypes.CDLL(out)
    for name, (res, args) in _lib._SIGS.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    lib.fake_used.restype = ctypes.c_ulonglong
    lib.fake_set_total.argtypes = [ctypes.c_ulonglong]
    return lib


def counts(lib, clear=True):
    """Launches since the last clear, by kind."""
    c = (ctypes.c_longlong * 5)()
    lib.fake_counts(c, 1 if clear else 0)
    return dict(zip(("plain", "cooperative", "captured_cooperative", "graph", "captures"), c))
