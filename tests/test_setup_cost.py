"""The split stage kernel's set-up: a block of at most 48 KB of shared memory needs no opt-in, so its variants are
neither looked up nor loaded -- shown by preparing them where the runtime could not answer (no CUDA device)."""
import os
import subprocess
import sys

import pytest

from hom3_b200 import _ffi

PREPARE, BYTES = "_ZN3h3c13split_prepareEibjbm", "_ZN3h3c16split_smem_bytesEib"

CODE = """
import ctypes as C, sys
L = C.CDLL(sys.argv[1])
prepare, bytes_ = L[sys.argv[2]], L[sys.argv[3]]
prepare.restype, prepare.argtypes = C.c_bool, [C.c_int, C.c_bool, C.c_uint, C.c_bool, C.c_size_t]
bytes_.restype, bytes_.argtypes = C.c_size_t, [C.c_int, C.c_bool]
nd, mixed = int(sys.argv[4]), bool(int(sys.argv[5]))
print(bytes_(nd, mixed), prepare(nd, mixed, 1, False, bytes_(nd, mixed)))
"""


@pytest.mark.parametrize("nd,mixed,free", [(2, 0, True), (2, 1, True), (3, 1, True), (3, 0, False)])
def test_only_3d_fp64_needs_the_runtime(nd, mixed, free):
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    out = subprocess.run([sys.executable, "-c", CODE, _ffi.LIB_PATH, PREPARE, BYTES, str(nd), str(mixed)], env=env,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    nbytes, ok = out.stdout.split()
    assert (int(nbytes) + 1024 <= 48 * 1024) == free
    assert ok == str(free)
