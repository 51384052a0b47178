"""The error of the Gram kernel's entries (csrc/dense.cu) is one of their own terms, also
where columns are nearly orthogonal or very different in norm: the kernel itself, against
long double, at row counts around its 32-row slabs and 128-row chunks.

A chunk has n <= 128 rows. Its second float gathers what n additions round away, about
sqrt(n) 2^-25 of the terms' sum as a random walk, and each of its own additions rounds
that by 2^-25: n 2^-50 = 2^-43. Eight times that, for the largest of some 10^4 entries:
2^-40."""
import glob
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_entries_against_long_double(tmp_path):
    import build as B
    exe = str(tmp_path / "gram_check")
    subprocess.run([B.NVCC] + B.ARCH + ["-O1", "-std=c++17", "-I" + B.INCLUDE, "-I" + B.CSRC,
                    os.path.join(HERE, "native", "gram_check.cu"), "-o", exe]
                   + glob.glob(os.path.join(B.BUILD, "*.o")) + ["-Xcompiler", "-pthread"],
                   check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    lines = [line.split() for line in out.splitlines()]
    assert len(lines) == 60
    for kind, rows, cols, bits in lines:
        assert float(bits) <= -40, (kind, rows, cols, bits)
