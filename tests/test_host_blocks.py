"""Blocks handed to C callers (calc_f_pyramid's levels, get_boxes, nms, flip_feat) are malloc's: code
written for the reference's functions frees them with free().  geye_free takes them too, and any other
malloc'ed pointer, and keeps large ones for the next call, a bounded number of bytes of them.  In a
process of its own, since the C library aborts on a pointer that is not its own."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import os
import ctypes as C
import geye_gb300 as g
L, libc = g.lib(), C.CDLL(None)
alloc, ref = L._ZN4geye10host_allocEm, L._ZN4geye13host_pool_refEi   # geye::host_alloc, geye::host_pool_ref
alloc.restype, alloc.argtypes = C.c_void_p, [C.c_size_t]
ref.restype, ref.argtypes = None, [C.c_int]
L.geye_free.restype, L.geye_free.argtypes = None, [C.c_void_p]
libc.malloc.restype, libc.malloc.argtypes = C.c_void_p, [C.c_size_t]
libc.free.restype, libc.free.argtypes = None, [C.c_void_p]
libc.malloc_usable_size.restype, libc.malloc_usable_size.argtypes = C.c_size_t, [C.c_void_p]
def new(n):
    p = alloc(n)
    assert p and libc.malloc_usable_size(p) >= max(n, 1)
    C.memset(p, 7, n)
    return p
"""

CASES = {
    "freed_by_the_c_library": """
for kept in (0, 1):       # without a context, and with the blocks of one kept
    ref(kept)
    for n in (0, 1, 1000, (1 << 20) - 1, 1 << 20, 15 << 20):
        libc.free(new(n))
        L.geye_free(new(n))
        libc.free(new(n))  # (a kept block)
ref(-1)
""",
    "geye_free_of_a_malloc_block": """
for kept in (0, 1):
    ref(kept)
    for n in (1, 100, 1 << 20, 9 << 20):
        L.geye_free(libc.malloc(n))
L.geye_free(None)
ref(-1)
""",
    "kept_blocks_are_reused_and_bounded": """
ref(1)
p = new(2 << 20)
L.geye_free(p)
assert new(2 << 20) == p       # kept
L.geye_free(p)
assert new(3 << 19) == p       # and for a smaller block, of half its size at least
big = [new(40 << 20) for _ in range(8)]
L.geye_free(p)
for q in big:
    L.geye_free(q)
def rss():
    return int(open('/proc/self/statm').read().split()[1]) * os.sysconf('SC_PAGE_SIZE')
with_kept = rss()
ref(-1)
assert 128 << 20 < with_kept - rss() <= (256 << 20) + (1 << 20)
""",
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_host_blocks(case):
    r = subprocess.run([sys.executable, "-c", PRELUDE + CASES[case]], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
