"""The library's host code on a CUDA runtime without a device (fake_cuda.cpp): es_native and es_mitm
bound to it for the length of a `with` block.  Test infrastructure only."""
import contextlib
import ctypes as C
import importlib.util
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def build(out_dir) -> str:
    spec = importlib.util.spec_from_file_location("es_build", os.path.join(ROOT, "erdos-selfridge_gb300", "build.py"))
    es_build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(es_build)
    es_build.build()   # the objects below are those of the library
    obj = os.path.join(ROOT, "erdos-selfridge_gb300", "_build")
    so = os.path.join(str(out_dir), "libfake.so")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", cuda, "-o", so,
                    os.path.join(ROOT, "tests", "fake_cuda.cpp")] +
                   [os.path.join(obj, f"{s}.cu.o") for s in ("es_abi", "es_cascade", "es_mitm")] + ["-lpthread"],
                   check=True, capture_output=True)
    return so


@contextlib.contextmanager
def bound(so: str):
    import es_native as N
    kept = N._lib, N.LIB_PATH
    N._lib, N.LIB_PATH = None, so
    try:
        L = N.lib()
        L.fake_fail_alloc.argtypes, L.fake_fail_alloc.restype = [C.c_long], C.c_long
        yield L
    finally:
        N._lib, N.LIB_PATH = kept
