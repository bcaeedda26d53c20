"""Determinant-list builds whose allocations fail (on the host, tests/cpp/alloc_fail.cpp):
the connection masks are an aid, so a build without memory for them, or for the matrix
beside them, scans the list again and gives the same matrix."""
import os
import subprocess
import sys

import pytest

from ciflow_gb300 import build as B

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes, sys
sys.path.insert(0, {root!r})
sys.path.insert(0, {root!r} + "/oracle")
import numpy as np
import oracle as O
from ciflow_gb300 import _abi as A
from ciflow_gb300.ciflow import FCI_File, Hamiltonian
from ciflow_gb300.synthetic import make_integrals
from tests.helpers import crs_sha256
from tests.test_gpu_dets import random_list, upper_sha

fail = ctypes.CDLL({lib!r}).alloc_fail_set
fail.argtypes = [ctypes.c_size_t, ctypes.c_int]
n = 1000
ints = make_integrals(14, 3, 3, nchol=5, seed=2)
up, down = random_list(14, 3, 3, n, seed=2)
ham = Hamiltonian.from_integrals(ints)
m = O.build_dets(ints, up, down)
want = crs_sha256(m.row, m.col, m.val)
words = (n + 31) // 32
masks = words * words * 32 * 4
fail(masks, -1)
assert upper_sha(FCI_File(ham, up=up, down=down)) == want
mixed = FCI_File(ham, up=up, down=down, precision=A.MIXED).get_mat()
assert np.array_equal(mixed.upper()[2], m.val.astype(np.float32).astype(np.float64))
columns = 4 * mixed.nnz_full
assert columns != masks
fail(columns, 1)  # with the masks held
assert upper_sha(FCI_File(ham, up=up, down=down)) == want
fail(columns, -1)
try:
    FCI_File(ham, up=up, down=down)
except A.CigpuError:
    print("refused")
fail(0, 0)
assert upper_sha(FCI_File(ham, up=up, down=down)) == want
print("done")
"""


def test_list_build_without_memory_for_the_masks(tmp_path):
    lib = str(tmp_path / "alloc_fail.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", os.path.join(ROOT, "tests", "cpp", "alloc_fail.cpp"),
                    "-o", lib, "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=lib + " " + B.LIB)
    out = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, lib=lib)], env=env, capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.split() == ["refused", "done"]
