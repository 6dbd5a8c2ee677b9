"""The library linked with a runtime that has no device (tests/fake_cuda.cpp): host code alone, on the
CPU.  Not a test module."""
import ctypes as C
import os
import subprocess

from grainrecon_b200 import _lib
from grainrecon_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))
HOOK = C.CFUNCTYPE(C.c_int, C.c_char_p, C.POINTER(C.c_void_p))


class Fake:
    def __init__(self, folder):
        B.build()
        objs = [os.path.join(B.BUILD_DIR, s.replace(".cu", ".o")) for s in B.SOURCES]
        if any(not os.path.exists(o) for o in objs):
            B.build(force=True)
        self.path = os.path.join(str(folder), "libfake.so")
        subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-Wl,-Bsymbolic",
                        os.path.join(HERE, "fake_cuda.cpp"), *objs, "-lpthread", "-o", self.path], check=True)
        old, path, _lib._lib, _lib.LIB_PATH = _lib._lib, _lib.LIB_PATH, None, self.path
        try:
            self.lib = _lib.load()
        finally:
            _lib._lib, _lib.LIB_PATH = old, path
        for name, res, args in (("alloc", C.c_void_p, [C.c_size_t]), ("limit", None, [C.c_size_t]), ("reset", None, []),
                                ("hook", None, [HOOK]), ("fail", None, [C.c_char_p, C.c_int, C.c_int]),
                                ("used", C.c_size_t, []), ("largest", C.c_size_t, []), ("stray", C.c_int, []),
                                ("launched", C.c_char_p, [])):
            f = getattr(self.lib, "fake_" + name)
            f.restype, f.argtypes = res, args
            if name not in ("hook", "fail", "launched"):
                setattr(self, name, f)

    def fail(self, name, after=0, code=2):
        self.lib.fake_fail(name.encode(), after, code)

    def launched(self):
        return self.lib.fake_launched().decode().split()

    def on_launch(self, f):
        """f(name, args): args[i] is the address of the kernel's argument i."""
        self._keep = HOOK(lambda n, a: f(n.decode(), a) or 0)
        self.lib.fake_hook(self._keep)

    def context(self):
        old, _lib._lib = _lib._lib, self.lib
        try:
            return _lib.Context(0)
        finally:
            _lib._lib = old


def pointer(args, i):
    """Argument i, a pointer, as an integer."""
    return C.cast(args[i], C.POINTER(C.c_uint64))[0]


def code_map(fake, distinct):
    """Has the map coding see one upper half of keys in use and `distinct` values."""
    def launch(name, args):
        if "number_halves_k" in name:
            C.c_int.from_address(pointer(args, 3)).value = 1
        elif "popc_k" in name:
            words = C.cast(args[1], C.POINTER(C.c_int64))[0]
            C.c_uint32.from_address(pointer(args, 2) + 4 * (words - 1)).value = distinct
    fake.on_launch(launch)
