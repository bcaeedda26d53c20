"""The CRS matvec's lanes per row (ciflow_gb300/csrc/row_shape.h): few lanes only where
every row has the mean's length. A list's long rows are chains of rounds."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIST, DOCI, FCI = 0, 1, 2


def test_row_shape(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "test_row_shape")
    subprocess.run([gxx, "-O1", "-std=c++17", os.path.join(ROOT, "tests", "cpp", "test_row_shape.cpp"), "-o", exe], check=True)
    # (rows, elements per row, FP64, kind): lanes, chunks per lane
    cases = {(125970, 97, 1, DOCI): (4, 2), (12000, 65, 1, DOCI): (4, 2), (11999, 65, 1, DOCI): (8, 5),
             (125970, 97, 0, DOCI): (8, 5), (39711, 181, 1, DOCI): (4, 2), (487635, 225, 1, DOCI): (32, 4),
             (10584, 504, 1, FCI): (32, 2), (10584, 504, 0, FCI): (32, 4),
             # lists: the mean says nothing of the longest row
             (12000, 190, 1, LIST): (8, 5), (40000, 60, 1, LIST): (8, 5), (200000, 20, 1, LIST): (8, 5),
             (52705, 1717, 1, LIST): (32, 4), (1, 1, 1, LIST): (8, 5)}
    text = "".join(f"{n} {n * row} {fp64} {kind}\n" for n, row, fp64, kind in cases)
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
    for line, (case, shape) in zip(out, cases.items()):
        assert tuple(int(v) for v in line.split()) == shape, case
