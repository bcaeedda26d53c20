"""FP32 sums of the mixed solver's basis kernels (ciflow_gb300/csrc/lanczos.cu): a
thread's chain of several terms must not lose what a single term's sum kept. The harness
(tests/cpp/test_vec_sums.cu) sums terms of 1 and 2^-24, which plain FP32 chains drop."""
import os
import subprocess

import pytest

from ciflow_gb300 import _abi as A
from ciflow_gb300 import build as B

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_chains_keep_their_small_terms(tmp_path):
    A.lib()
    exe = str(tmp_path / "test_vec_sums")
    lib = os.path.dirname(B.LIB)
    subprocess.run([B.nvcc(), *B.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                    os.path.join(ROOT, "tests", "cpp", "test_vec_sums.cu"), "-o", exe, "-L" + lib, "-lcigpu",
                    "-Xlinker", "-rpath=" + lib], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    errors = [(name, float(e)) for name, e in (line.split() for line in out.stdout.splitlines())]
    assert {name for name, _ in errors} == {"dots", "couple", "step"}
    # the sums are exact below the warp and round in FP64 above: at most 2^11 additions of
    # 2^-53 each in a chain (608 blocks, their warps, the lanes' running sums)
    for name, err in errors:
        assert err <= 2.0 ** -42, (name, err)
