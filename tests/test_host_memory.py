"""A C entry that cannot allocate host memory returns an error; nothing is thrown through the C boundary (CPU: the
allocation comes before any device call)."""
import os
import subprocess
import sys

from mestrado_gb300 import build as engine_build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes as C, resource, sys
lib = C.CDLL(sys.argv[1])
lib.gbivf_last_error.restype = C.c_char_p
resource.setrlimit(resource.RLIMIT_AS, (64 << 30, 64 << 30))
one = (C.c_void_p * 1)(None)
size = (C.c_int * 1)(0)
out = C.c_void_p()
# a codebook of 256 x 2^30 floats
rc = lib.gbivf_index_create_from_lists(C.byref(out), 0, 1 << 30, 1, None, 1, 256, one, size, one, one)
print(rc, out.value, lib.gbivf_last_error().decode())
"""


def test_create_without_host_memory():
    engine_build.build()
    r = subprocess.run([sys.executable, "-c", CHILD, engine_build.LIB], capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split()[:2] == ["3", "None"], r.stdout  # GBIVF_ERR_NOMEM
