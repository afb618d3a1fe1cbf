"""The library on a stand-in for the CUDA runtime (runtime.cpp): its own
objects, linked with that instead of with CUDA, so that its host side runs
and is checked without a GPU.  Kernels do nothing there."""
import collections
import ctypes as C
import glob
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
Op = collections.namedtuple("Op", "kind stream name early captured grid block dst bytes")


def build(build_module):
    """Path of the library linked with the stand-in (made when stale)."""
    b = build_module
    b.build_library()
    out = os.path.join(b.OBJ_DIR, "fake", "libfesomc_fake.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    src = os.path.join(HERE, "runtime.cpp")
    objs = sorted(glob.glob(os.path.join(b.OBJ_DIR, "*.o")))
    if b._stale(out, [src] + objs):
        inc = os.path.join(os.path.dirname(os.path.dirname(b._nvcc())), "include")
        tmp = out + ".%d" % os.getpid()
        subprocess.run([b._cxx(), "-O1", "-fPIC", "-shared", "-std=c++17", "-I", inc, src] + objs + ["-Wl,-Bsymbolic", "-lpthread", "-o", tmp],
                       check=True, capture_output=True, text=True)
        os.replace(tmp, out)
    return out


class Log:
    """The stand-in's log and switches."""

    def __init__(self, lib):
        self.lib = lib
        lib.fake_pinned_bytes.restype = C.c_longlong
        for f in (lib.fake_fail_copy, lib.fake_fail_malloc):
            f.argtypes = [C.c_longlong]

    def clear(self):
        self.lib.fake_clear()

    def ops(self):
        out = []
        for i in range(self.lib.fake_ops()):
            k, s, n, e, c, g, b, d, z = (C.c_char(), C.c_void_p(), C.c_char_p(), C.c_int(), C.c_int(), C.c_uint(),
                                         C.c_uint(), C.c_void_p(), C.c_size_t())
            self.lib.fake_op(i, *[C.byref(x) for x in (k, s, n, e, c, g, b, d, z)])
            out.append(Op(k.value.decode(), s.value, n.value.decode(), bool(e.value), bool(c.value), g.value, b.value,
                          d.value, z.value))
        return out
