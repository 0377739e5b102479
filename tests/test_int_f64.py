"""The FP64 products, reciprocals, quotients and roots on the integer pipes
(csrc/int_f64.cuh) by themselves: every seed argument of the reciprocal and the
root, against FP64 arithmetic, bit for bit.  On the host with seeds moved by up to 2 units in the last place:
a relative error of 2^-23 (reciprocal) or 2^-22.9 (root), the hardware
approximations' bounds, is at most 2 units of a value in [1/2, 1).  On the GPU
with the hardware's own seeds."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "fd-weno-eulerequation_gb300", "csrc")
SOURCE = os.path.join(ROOT, "tests", "int_f64_check.cu")


def _mismatches(program):
    r = subprocess.run([program], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return dict(zip(("product", "reciprocal", "quotient", "root"), map(int, r.stdout.split())))


@pytest.mark.parametrize("units", [-2, -1, 0, 1, 2])
def test_every_seed_moved_by_units_in_the_last_place(units, tmp_path):
    header = open(os.path.join(CSRC, "int_f64.cuh")).read()
    for seed in ("1.0f / x", "1.0f / __builtin_sqrtf(x)"):
        assert header.count(f"return {seed};") == 1
        header = header.replace(f"return {seed};", f"return moved({seed});")
    (tmp_path / "int_f64.cuh").write_text(
        "#include <cstring>\n"
        "inline float moved(float x) {\n"
        "  unsigned u;\n"
        "  std::memcpy(&u, &x, 4);\n"
        f"  u += unsigned({units});\n"
        "  std::memcpy(&x, &u, 4);\n"
        "  return x;\n"
        "}\n" + header.replace("#pragma once", ""))
    program = str(tmp_path / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(tmp_path), "-x", "c++", SOURCE, "-o", program],
                   check=True)
    assert not any(_mismatches(program).values()), _mismatches(program)


@pytest.mark.gpu
def test_every_seed_of_the_hardware(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    program = str(tmp_path / "check")
    subprocess.run([os.path.join(cuda, "bin", "nvcc"), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-fmad=false", "-I", CSRC, SOURCE, "-o", program], check=True)
    assert not any(_mismatches(program).values()), _mismatches(program)
