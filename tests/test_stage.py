"""Which tables a 2-D trace CTA stages in shared memory (csrc/tabstage.cuh), on the CPU:
those that the launch's step reads. A batch of several profile types takes the general
step, for environments with packed segments as well."""
import os
import subprocess

import pytest

from bellhopcuda_b200 import build as BUILD

HERE = os.path.dirname(os.path.abspath(__file__))
N2, C, S, P = 0, 1, 2, 3   # SspType


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("stage") / "check")
    subprocess.run([BUILD.nvcc(), *BUILD.ARCH, "-std=c++17", "-I" + BUILD.CSRC, os.path.join(HERE, "stage_check.cu"), "-o",
                    exe], check=True)
    return exe


# SEG Z C CZ COEF N2 N2Z RHO QR QC QCZ BTOP BBOT RR
@pytest.mark.parametrize("ssp,packed,tables", [(C, 1, "10000000000111"), (S, 1, "10000000000111"), (P, 1, "10000000000111"),
                                               (C, 0, "01110001000111"), (S, 0, "01001001000111"),
                                               (P, 0, "01001001000111"), (N2, 0, "01000111000111")])
def test_tables(program, ssp, packed, tables):
    got, used = subprocess.check_output([program, str(ssp), str(packed)], text=True).split()
    assert got == tables and 0 < int(used) <= 32 * 1024
