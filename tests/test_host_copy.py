"""HostCopy (csrc/hostcopy.h) on the CPU, over a fake of the runtime calls it makes:
which copies go through the ring (512 KB pieces), that the bytes arrive, and that an
error which was pending before the copy is still there after it, unless a probe of the
copy's own failed."""
import os
import shutil
import subprocess

import pytest

from bellhopcuda_b200 import build as BUILD

HERE = os.path.dirname(os.path.abspath(__file__))
MB = 1 << 20


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("hostcopy") / "check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-pthread", "-I" + os.path.join(HERE, "fake_cuda"),
                    "-I" + BUILD.CSRC, os.path.join(HERE, "host_copy_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("nbytes,how,pieces", [(1, 0, 1), (32 * MB - 1, 0, 1), (32 * MB, 0, 64), (33 * MB + 5, 0, 67),
                                               (33 * MB, 1, 1), (33 * MB, 2, 1), (33 * MB, 3, 1)])
@pytest.mark.parametrize("before", [0, 1])
def test_copy(program, nbytes, how, pieces, before):
    equal, copies, after = map(int, subprocess.check_output([program, str(nbytes), str(how), str(before)]).split())
    assert equal == 1 and copies == pieces
    assert after == (0 if how in (2, 3) else before)
