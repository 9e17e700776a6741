"""The runtime two-stage FFT kernels (planes and lengths without a
compile-time instance) emulated on the host.

`tests/host_emu/gen_emu.cpp` runs `k_xy_fwd_gen`, `k_xy_inv_gen` and the
runtime form of `k_z_lane` block by block behind `kernel_emu.h`, against
direct DFTs, on shapes that reach every radix, odd Lx/2, row groups cut by Ly
and tiles cut by Lx/2 and Ly, in FP64 and FP32.

Tolerances as for the other emulated kernels: a few roundings of the largest
term; the z pass runs a forward and an inverse transform, its energy sums the
squares of FP32 spectra."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "host_emu", "gen_emu.cpp")
CUDA_INC = "/usr/local/cuda/include"
TOL = {"f64": 4e-15, "f32": 2e-6}


@pytest.fixture(scope="module")
def emu_lines(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.isdir(CUDA_INC):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("genemu") / "gen_emu")
    subprocess.run([gxx, "-std=c++20", "-O1", "-I", CUDA_INC, "-I", os.path.join(ROOT, "feram_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.dirname(SRC), SRC, "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=600).stdout
    return {n: (float(a), float(b)) for n, a, b in (line.split() for line in out.splitlines())}


def test_every_case_ran(emu_lines):
    assert len(emu_lines) == 2 * (29 + 1 + 39) and not [n for n in emu_lines if "nosplit" in n]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("kind", ["xy", "z"])
def test_kernels_give_the_transforms(emu_lines, kind, prec):
    bad = {n: v for n, v in emu_lines.items() if n.startswith(f"{kind}_{prec}") and not max(v) <= TOL[prec]}
    assert not bad, bad
