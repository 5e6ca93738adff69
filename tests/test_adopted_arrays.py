"""Arrays over callee-allocated blocks: the block is freed once, when the last array over it goes, and
not at the interpreter's exit, where other code (handlers registered earlier, other threads' objects)
may still read the array."""
import ctypes as C
import gc
import os
import subprocess
import sys

import numpy as np

from geye_gb300 import dpm

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _malloc(n):
    libc = C.CDLL(None)
    libc.malloc.restype, libc.malloc.argtypes = C.c_void_p, [C.c_size_t]
    p = libc.malloc(4 * n)
    return C.cast(p, C.POINTER(C.c_float))


def test_the_block_is_freed_with_the_last_array(monkeypatch):
    freed = []

    class Lib:
        @staticmethod
        def geye_free(p):
            freed.append(p)

    monkeypatch.setattr(dpm, "lib", lambda: Lib)
    for n in (0, 1, 1000):
        p = _malloc(max(n, 1))
        at = C.cast(p, C.c_void_p).value
        a = dpm._adopted(p, n)
        assert a.dtype == np.float32 and a.shape == (n,)
        part = a[: n // 2].reshape(1, -1)
        del a
        gc.collect()
        assert not freed
        del part
        gc.collect()
        assert freed == [at]
        freed.clear()


def test_arrays_are_whole_at_exit():
    code = """
import atexit, ctypes as C, numpy as np
held = {}
atexit.register(lambda: print("sum", int(held["a"].sum()), flush=True))   # (runs after what is registered later)
from geye_gb300 import dpm
libc = C.CDLL(None)
libc.malloc.restype, libc.malloc.argtypes = C.c_void_p, [C.c_size_t]
n = 4 << 20
held["a"] = dpm._adopted(C.cast(libc.malloc(4 * n), C.POINTER(C.c_float)), n)
held["a"][:] = 1.0
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert (r.returncode, r.stdout.split()) == (0, ["sum", str(4 << 20)]), (r.returncode, r.stdout, r.stderr[-2000:])
