"""The bounds-checked build (`feram_b200/build.py --checked`) of the runtime
x-y and k-space kernels, emulated on the host: `tests/host_emu/bounds_emu.cpp`
runs them with FG_BOUNDS_CHECK on shapes as the library makes them, which must
record nothing, and on shapes whose strides, lengths or tiles do not fit their
arrays, which must be recorded."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "host_emu", "bounds_emu.cpp")
CUDA_INC = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.isdir(CUDA_INC):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("bounds") / "bounds_emu")
    subprocess.run([gxx, "-std=c++20", "-O1", "-I", CUDA_INC, "-I", os.path.join(ROOT, "feram_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.dirname(SRC), SRC, "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=600).stdout
    return {n: (int(a), int(b)) for n, a, b in (line.split() for line in out.splitlines())}


def test_every_case_ran(lines):
    assert len(lines) == 2 * (7 * 6 * 2 + 6 * 3 + 2)


@pytest.mark.parametrize("kernel", ["fwd", "inv", "z", "zct"])
def test_indices_out_of_range_are_recorded_and_only_those(lines, kernel):
    mine = {n: v for n, v in lines.items() if n.startswith(kernel + "_")}
    assert mine
    assert not {n: v for n, v in mine.items() if v[0] != v[1]}
